"""The small sort's ranking, whose lanes find the others of their digit through a
mask per digit: few digits, so that a warp's turns use the same masks one after
another, against the restatement's order."""
import numpy as np
import pytest

from operatorgraph_gb300 import grammar as G
from operatorgraph_gb300 import scenes

pytestmark = pytest.mark.gpu

BOUNDS = (-10.0, -10.0, -10.0, 10.0, 10.0, 10.0)


@pytest.mark.parametrize("n,cells", [(129, 1), (2047, 2), (2049, 3), (20011, 2), (20011, 40)])
def test_recurring_digits(n, cells):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import oracle
    from operatorgraph_gb300.engine import Engine

    rng = np.random.default_rng(n + cells)
    rec = np.zeros(n, G.TERMINAL_DT)
    rec["m"] = rng.uniform(-0.5, 0.5, (n, 12)).astype(np.float32)
    at = rng.uniform(-9.0, 9.0, (cells, 3)).astype(np.float32)
    rec["m"][:, [3, 7, 11]] = at[rng.integers(0, cells, n)]
    rec["path"] = rng.integers(0, 1 << 50, n, dtype=np.uint64) | (rng.integers(0, 3, n, dtype=np.uint64) << np.uint64(60))
    rec["rule"] = 1
    nodes, _, _, leaf, keys = oracle.lbvh(rec, BOUNDS)
    eng = Engine(scenes.menger_table(0.5), node_capacity=1 << 12, max_terminals=n)
    t = torch.from_numpy(rec.view(np.uint8).reshape(n, 64).copy()).cuda()
    for _ in range(3):
        bv = eng.lbvh(t, n, BOUNDS)
        torch.cuda.synchronize()
        assert np.array_equal(bv["keys"].cpu().numpy().view(np.uint64), keys)
        assert np.array_equal(bv["leafTerminal"].cpu().numpy().view(np.uint32), leaf)
        assert np.array_equal(bv["nodes"].cpu().numpy(), nodes)
    eng.release()
