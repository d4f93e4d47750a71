"""The LBVH's bottom-up tree kernel at the sizes where its tiles (256 leaves),
their windows (32 keys either side) and their groups (32 tiles, then 32
groups) begin and end, and on tie runs inside a tile, over a tile's end and
longer than a tile, and either side of the sort's two forms; bit for bit against the restatement, as the other LBVH
tests are."""
import numpy as np
import pytest

from operatorgraph_gb300 import grammar as G
from operatorgraph_gb300 import scenes

pytestmark = pytest.mark.gpu

BOUNDS = (-10.0, -10.0, -10.0, 10.0, 10.0, 10.0)


def _records(n, ties, seed=3):
    rng = np.random.default_rng(seed + n)
    rec = np.zeros(n, G.TERMINAL_DT)
    m = rng.uniform(-0.5, 0.5, (n, 12)).astype(np.float32)
    m[:, [3, 7, 11]] = rng.uniform(-9.0, 9.0, (n, 3)).astype(np.float32)
    path = rng.integers(0, 1 << 64, n, dtype=np.uint64)
    if ties != "none":
        cells = {"short": max(1, n // 3000), "long": max(1, n // 40000), "equal": max(1, n // 700)}[ties]
        at = rng.uniform(-9.0, 9.0, (cells, 3)).astype(np.float32)
        m[:, [3, 7, 11]] = at[rng.integers(0, cells, n)]
    if ties == "long":  # runs of about 40,000 / 4 leaves: the top bits of the hash take four values
        path = (path & np.uint64((1 << 50) - 1)) | (rng.integers(0, 4, n, dtype=np.uint64) << np.uint64(60))
    if ties == "equal":  # no path at all: the terminal index decides
        path[:] = 0
    rec["m"] = m
    rec["path"] = path
    rec["rule"] = np.where(rng.random(n) < 0.3, np.uint32(0x80000001), np.uint32(1))
    return rec


SIZES = [2, 3, 31, 33, 255, 256, 257, 288, 289, 512, 513, 8191, 8192, 8193, 30011]


@pytest.mark.parametrize("n,ties", [(n, t) for n in SIZES for t in ("none", "short", "equal")]
                         + [(262144, "none"), (262145, "short"), (290017, "equal"), (90001, "long")]
                         # the sort's small and large forms, and a large one with more tiles than counting groups
                         + [(622592, "short"), (622593, "none"), (2500001, "short")])
def test_tree_bit_exact(n, ties):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import oracle
    from operatorgraph_gb300.engine import Engine

    rec = _records(n, ties)
    nodes, lp, aabb, lt, keys = oracle.lbvh(rec, BOUNDS)
    eng = Engine(scenes.menger_table(0.5), node_capacity=1 << 12, max_terminals=n + 300)
    d = torch.from_numpy(rec.view(np.uint8).reshape(n, 64).copy()).cuda()
    count = torch.tensor([n], dtype=torch.int64, device="cuda")
    pad = torch.zeros((n + 300, 64), dtype=torch.uint8, device="cuda")
    pad[:n] = d
    for counted in (False, True):
        bv = eng.lbvh(pad, n + 300, BOUNDS, count=count) if counted else eng.lbvh(d, n, BOUNDS)
        torch.cuda.synchronize()
        assert np.array_equal(bv["keys"].cpu().numpy().view(np.uint64)[:n], keys)
        assert np.array_equal(bv["leafTerminal"].cpu().numpy().view(np.uint32)[:n], lt)
        assert np.array_equal(bv["nodes"].cpu().numpy()[: n - 1], nodes)
        assert np.array_equal(bv["leafParents"].cpu().numpy().view(np.uint32)[:n], lp)
        assert np.array_equal(bv["aabbs"].cpu().numpy()[: n - 1], aabb)
        if counted:
            assert (bv["keys"][n:] == -1).all()
    eng.release()


def test_boxes_of_infinite_and_nan_records_follow_the_corners():
    """A record with an infinite or NaN entry: the box is the fminf / fmaxf over its corners, NaN corners left out."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import oracle
    from operatorgraph_gb300.engine import Engine

    n = 600
    rec = _records(n, "none")
    rng = np.random.default_rng(5)
    for v in (np.inf, -np.inf, np.nan, 3e38, -3e38):
        rows = rng.integers(0, n, 12)
        rec["m"][rows, rng.choice([0, 1, 2, 4, 5, 6, 8, 9, 10], 12)] = v
    nodes, lp, aabb, lt, keys = oracle.lbvh(rec, BOUNDS)
    eng = Engine(scenes.menger_table(0.5), node_capacity=1 << 12, max_terminals=n)
    bv = eng.lbvh(torch.from_numpy(rec.view(np.uint8).reshape(n, 64).copy()).cuda(), n, BOUNDS)
    torch.cuda.synchronize()
    assert np.array_equal(bv["nodes"].cpu().numpy(), nodes)
    assert np.array_equal(bv["aabbs"].cpu().numpy(), aabb)
    eng.release()
