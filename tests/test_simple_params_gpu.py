"""Tables of scalars, block values and the custom attribute only derive with
kernels that evaluate nothing else.  The same table with an unreachable rule
that draws a random number derives with the others: the terminals and the
gradients of the tape have to be the same, whatever form of the kernel an
engine runs."""
import numpy as np
import pytest

from operatorgraph_gb300 import grammar as G
from operatorgraph_gb300 import scenes
from operatorgraph_gb300.grammar import DispatchTable, Entry, block, scalar, shape_attr

pytestmark = pytest.mark.gpu


def _torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _chains(n, blocks, affine):
    """Every operator that reads parameters: Repeats of the three modes (absolute, relative), Subdivides, Extrude by
    the custom attribute, a static random choice between equal successors, and (affine) Translate and Scale."""
    par = (lambda k, v: block(k)) if blocks else (lambda k, v: scalar(v))
    e = [
        Entry(G.QUAD_EXTRUDE, [scalar(2), shape_attr(16)], [(1, 0)]),
        Entry(G.BOX_REPEAT, [scalar(0), par(0, -0.3), scalar(0)], [(2, 0)]),
        Entry(G.BOX_REPEAT, [scalar(1), par(1, 0.31), scalar(1)], [(3, 0)]),
        Entry(G.BOX_REPEAT, [scalar(2), par(2, 0.27), scalar(2)], [(4, 0)]),
        Entry(G.BOX_SUBDIVIDE, [scalar(0), par(3, -0.4), scalar(-0.6), scalar(-0.05)], [(7, 0), (5, 0), (9, 0)]),
        Entry(G.BOX_TRANSLATE, [par(4, 0.1), scalar(0.2), scalar(-0.1)], [(6, 0)]),
        Entry(G.BOX_SCALE, [scalar(-1), par(5, 0.8), scalar(-0.5)], [(7, 0)]),
        Entry(G.BOX_IF_SIZE_LESS, [scalar(0), par(6, 0.1)], [(9, 0), (8, 0)]),
        Entry(G.BOX_COMPONENT_SPLIT, [], [(10, 0), (10, 0), (10, 0)]),
        Entry(G.BOX_GENERATE, [shape_attr(16)], []),
        Entry(G.QUAD_GENERATE, [scalar(2)], []),
    ]
    if not affine:
        e[4] = Entry(G.BOX_SUBDIVIDE, [scalar(0), par(3, -0.4), scalar(-0.6), scalar(-0.05)], [(7, 0), (7, 0), (9, 0)])
        e[5] = e[6] = Entry(G.BOX_DISCARD, [], [])
    rng = np.random.default_rng(11)
    ax = G.make_axioms(n)
    ax["entry"], ax["shape"] = 0, G.SHAPE_QUAD
    ax["size"] = rng.uniform(0.8, 1.5, (n, 3)).astype(np.float32)
    ax["position"] = rng.uniform(-2.0, 2.0, (n, 3)).astype(np.float32)
    ax["custom"] = rng.uniform(0.4, 1.2, n).astype(np.float32)
    ax["block"] = np.arange(n)
    values = np.array([-0.3, 0.31, 0.27, -0.4, 0.1, 0.8, 0.1], np.float32)
    return {"entries": DispatchTable(e).to_array(), "axioms": ax,
            "blocks": np.tile(values, (n, 1)) * rng.uniform(0.9, 1.1, (n, 7)).astype(np.float32) if blocks else None}


BATCHES = {
    "building": lambda: scenes.building(),
    "city": lambda: scenes.city(150),
    "menger": lambda: scenes.menger(0.15, 9),
    "mixed": lambda: scenes.mixed(90),
    "mixed blocks": lambda: scenes.mixed(90, blocks=True),
    "chains": lambda: _chains(70, False, True),
    "chains blocks": lambda: _chains(70, True, True),
    "splits blocks": lambda: _chains(70, True, False),
}


@pytest.mark.parametrize("form", ["leaves", "no_inline", "dynamic_chunks", "host_levels"])
@pytest.mark.parametrize("name", list(BATCHES))
def test_simple_tables_derive_as_the_general_kernels(name, form):
    torch = _torch()
    from operatorgraph_gb300.autograd import axioms_tensor
    from operatorgraph_gb300.engine import Engine, terminals_to_numpy

    b = BATCHES[name]()
    b["axioms"]["position"] = 0.0  # coordinates of one size, so that the gradients' terms are comparable
    entries, n = np.ascontiguousarray(b["entries"], dtype=G.ENTRY_DT), len(b["axioms"])
    drawing = DispatchTable([Entry(G.BOX_IF_SIZE_LESS, [scalar(0), G.rand(0.1, 0.2)], [(0, 0), (0, 0)])]).to_array()
    blk = None
    if b.get("blocks") is not None:
        blk = torch.from_numpy(np.ascontiguousarray(b["blocks"], np.float32).reshape(n, -1)).cuda()
    cap = 1 << 19
    found = []
    for table in (entries, np.concatenate([entries, drawing])):
        eng = Engine(table, node_capacity=1 << 20, max_terminals=cap, record_tape=form == "leaves",
                     block_stride=0 if blk is None else blk.shape[1], no_inline=form != "leaves",
                     dynamic_chunks=form == "dynamic_chunks")
        axioms = axioms_tensor(b["axioms"])
        out, count, _ = eng.execute(axioms, blocks=blk, capacity=cap, plain=form == "host_levels")
        assert eng.report()["status"] == 0 and 0 < count <= cap
        grads = None
        if form == "leaves":
            g_sizes = torch.zeros((n, 3), device="cuda")
            g_blk = torch.zeros((n, 1 if blk is None else blk.shape[1]), device="cuda")
            eng.adjoint_raw(out.data_ptr(), 0 if blk is None else g_blk.data_ptr(), 0 if blk is None else n,
                            g_sizes.data_ptr(), grad_stride=16)
            torch.cuda.synchronize()
            assert eng.report()["status"] == 0
            grads = (g_sizes.cpu().numpy().astype(np.float64), g_blk.cpu().numpy().astype(np.float64))
        t = G.sort_terminals(terminals_to_numpy(out, count), by_path=True)
        found.append((t, grads))
        eng.release()
    (t0, g0), (t1, g1) = found
    assert len(t0) == len(t1)
    for field in ("path", "rule", "custom", "m"):
        assert np.array_equal(t0[field], t1[field])
    if g0 is not None:
        # One adjoint, one tape: only the order of the FP32 sums may differ.  An axiom
        # has at most 8,000 terminals: 8000 * 2^-24 = 5e-4 of the largest sum.
        for a, c in zip(g0, g1):
            assert np.isfinite(a).all() and np.abs(a - c).max() <= 5e-4 * np.abs(c).max()
