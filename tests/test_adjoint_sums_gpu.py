"""The adjoint's closed-form sums (rules whose children pass their gradients on
unchanged) against its general replay: the same grammar with a Scale by one
between a split and its children, which the sums do not cover, must give the
same terminals and, to FP32 summation order, the same gradients.  Every split
and form that the sums accept (and Subdivides of nine block factors, which
they do not), with frame codes and with general frames, on levels narrow
enough for eight lanes an item and on wide ones; children that are terminals,
and children that are work items of several pages."""
import numpy as np
import pytest

from operatorgraph_gb300 import grammar as G
from operatorgraph_gb300.grammar import DispatchTable, Entry, block, scalar

pytestmark = pytest.mark.gpu

SPLITS = (["static", "faces", "replicate"] + [f"dynamic{n}" for n in (1, 2, 4, 5, 8, 9)]
          + [f"repeat{mode}{how}" for mode in (0, 1, 2) for how in ("absolute", "relative")])


def _table(split, blocks, plain, rotate):
    """Root -> [Rotate] -> split -> [Scale] -> a terminal, or a Repeat of 11 pieces, each a terminal."""
    par = (lambda k, v: block(k)) if blocks else (lambda k, v: scalar(v))
    rot, cut, one, rows, one2, leaf = range(6)
    quad = split == "faces"
    scale, rep, gen = ((G.QUAD_SCALE, G.QUAD_REPEAT, G.QUAD_GENERATE) if quad else
                       (G.BOX_SCALE, G.BOX_REPEAT, G.BOX_GENERATE))
    term, many = (one2, one) if not plain else (leaf, rows)
    values = [-0.7, 0.11, -1.3, 0.07, -0.4, 0.05, 0.13, -0.9, 0.06]
    if split == "static":
        op, params, succ = G.BOX_SUBDIVIDE3, [scalar(1), par(0, values[0]), scalar(0.0), par(2, values[2])], [term, term, many]
    elif split == "faces":
        op, params, succ = G.BOX_COMPONENT_SPLIT, [], [term, many, term]
    elif split == "replicate":
        op, params, succ = G.BOX_REPLICATE, [], [term, many, term]
    elif split.startswith("dynamic"):
        n = int(split[7:])
        op, params = G.BOX_SUBDIVIDE, [scalar(2)] + [par(k, values[k]) for k in range(n)]
        succ = [many if k % 3 == 1 else term for k in range(n)]
    else:
        mode, relative = int(split[6]), split.endswith("relative")
        op, params, succ = G.BOX_REPEAT, [scalar(0), par(0, -0.19 if relative else 0.23), scalar(mode)], [many]
    entries = [
        Entry(G.BOX_ROTATE, [scalar(20), scalar(-35), scalar(10)], [(cut, 0)]),
        Entry(op, params, [(s, 0) for s in succ]),
        Entry(scale, [scalar(-1), scalar(-1), scalar(-1)], [(rows, 0)]),
        Entry(rep, [scalar(0 if quad else 1), scalar(-0.0915), scalar(0)], [(term, 0)]),
        Entry(scale, [scalar(-1), scalar(-1), scalar(-1)], [(leaf, 0)]),
        Entry(gen, [scalar(1)], []),
    ]
    first = np.array([-0.19 if split.endswith("relative") else 0.23], np.float32) if split.startswith("repeat") else None
    blk = np.array(values, np.float32)
    if first is not None:
        blk[0] = first[0]
    if not rotate:  # without a Rotate rule in the table the frame-code kernels run
        entries[rot] = Entry(G.BOX_DISCARD, [], [])
    return DispatchTable(entries).to_array(), (rot if rotate else cut), blk


def _gradients(torch, split, blocks, plain, rotate, n):
    from operatorgraph_gb300.autograd import axioms_tensor
    from operatorgraph_gb300.engine import Engine

    entries, root, values = _table(split, blocks, plain, rotate)
    rng = np.random.default_rng(7)
    ax = G.make_axioms(n)
    ax["entry"] = root
    ax["shape"] = G.SHAPE_BOX
    ax["size"] = rng.uniform(0.9, 1.6, (n, 3)).astype(np.float32)
    ax["position"] = rng.uniform(-1.0, 1.0, (n, 3)).astype(np.float32)
    blk = torch.from_numpy(np.tile(values, (n, 1)) * rng.uniform(0.9, 1.1, (n, 9)).astype(np.float32)).cuda().contiguous()
    cap = 150 * n + 4096
    eng = Engine(entries, node_capacity=40 * n + (1 << 19), max_terminals=cap, block_stride=9, record_tape=True)
    axioms = axioms_tensor(ax)
    out, count, _ = eng.execute(axioms, blocks=blk, capacity=cap)
    g_sizes, g_blk = torch.zeros((n, 3), device="cuda"), torch.zeros((n, 9), device="cuda")
    eng.adjoint_raw(out.data_ptr(), g_blk.data_ptr(), n, g_sizes.data_ptr(), grad_stride=16)  # L = |M|^2 / 2
    torch.cuda.synchronize()
    assert eng.report()["status"] == 0
    m = out[:count].view(torch.float32).view(count, 16)[:, :12].double()
    total = float((m * m).sum())
    eng.release()
    return count, total, g_sizes.cpu().numpy().astype(np.float64), g_blk.cpu().numpy().astype(np.float64)


@pytest.mark.parametrize("n", [3, 40000])
@pytest.mark.parametrize("rotate", [False, True])
@pytest.mark.parametrize("blocks", [False, True])
@pytest.mark.parametrize("split", SPLITS)
def test_sums_match_the_general_replay(split, blocks, rotate, n):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    a = _gradients(torch, split, blocks, True, rotate, n)
    b = _gradients(torch, split, blocks, False, rotate, n)
    assert a[0] == b[0] and abs(a[1] - b[1]) <= 1e-12 * b[1]
    assert np.abs(b[2]).max() > 0
    pairs = [(a[2], b[2])]
    # no parameter, or one without effect: a single relative share is the whole, and pieces adjusted to fill depend
    # on their extent through their (frozen) number alone
    if blocks and split not in ("faces", "replicate", "dynamic1", "repeat2absolute", "repeat2relative"):
        assert np.abs(b[3]).max() > 0
        pairs.append((a[3], b[3]))
    # sums of up to 130 terms in two orders: 130 eps of the largest magnitudes, with the factor gradients'
    # cancellation of a few between W and Q / R
    for x, y in pairs:
        assert np.abs(x - y).max() <= 5e-5 * np.abs(y).max(), (np.abs(x - y).max(), np.abs(y).max())


@pytest.mark.parametrize("blocks", [False, True])
def test_the_two_launch_shapes_agree(blocks):
    """Either side of the capacity (2^21 terminals) from which an engine launches k_adjoint_wide."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from operatorgraph_gb300 import scenes
    from operatorgraph_gb300.autograd import axioms_tensor
    from operatorgraph_gb300.engine import Engine

    b = scenes.mixed(500, blocks=blocks)
    axioms = axioms_tensor(b["axioms"])
    blk = torch.from_numpy(b["blocks"]).cuda() if blocks else None
    grads = []
    for cap in ((1 << 21) - 1, 1 << 21):
        eng = Engine(b["entries"], node_capacity=1 << 22, max_terminals=cap, block_stride=b["block_stride"],
                     record_tape=True)
        out, _, _ = eng.execute(axioms, blocks=blk, capacity=cap)
        g = torch.zeros((500, 3), device="cuda")
        gb = torch.zeros_like(blk) if blocks else None
        eng.adjoint_raw(out.data_ptr(), gb.data_ptr() if blocks else None, 500 if blocks else 0, g.data_ptr(),
                        grad_stride=16)
        torch.cuda.synchronize()
        assert eng.report()["status"] == 0
        grads.append([g.cpu().numpy().astype(np.float64)] + ([gb.cpu().numpy().astype(np.float64)] if blocks else []))
        eng.release()
    for x, y in zip(*grads):  # up to 10^4 terminals an axiom
        assert np.abs(y).max() > 0 and np.abs(x - y).max() <= 1e-4 * np.abs(y).max()


def test_one_tape_serves_many_reverse_passes():
    """The reverse launches of one derivation share their barrier words: more launches than there are words."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from operatorgraph_gb300 import scenes
    from operatorgraph_gb300.autograd import axioms_tensor
    from operatorgraph_gb300.engine import Engine

    b = scenes.city(50)
    axioms = axioms_tensor(b["axioms"])
    eng = Engine(b["entries"], node_capacity=1 << 20, max_terminals=1 << 18, record_tape=True)
    out, _, _ = eng.execute(axioms, capacity=1 << 18)
    grads = []
    for _ in range(7):
        g = torch.full((50, 3), float("nan"), device="cuda")
        eng.adjoint_raw(out.data_ptr(), None, 0, g.data_ptr(), grad_stride=16)
        torch.cuda.synchronize()
        assert eng.report()["status"] == 0
        grads.append(g.cpu().numpy().astype(np.float64))
    eng.release()
    for g in grads[1:]:  # one building's terminals in another order of summation
        assert np.abs(g - grads[0]).max() <= 1e-5 * np.abs(grads[0]).max()
