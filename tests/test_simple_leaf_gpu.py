"""Leaf children expanded in place by the kernels of simple tables (scalars, block
values and the custom attribute), against the general kernels' (the same table
with an unreachable rule that draws a random number): leaf Subdivides with
scalar and with block factors."""
import numpy as np
import pytest

from operatorgraph_gb300 import grammar as G
from operatorgraph_gb300 import scenes
from operatorgraph_gb300.grammar import DispatchTable, Entry

pytestmark = pytest.mark.gpu

BATCHES = {
    "building": lambda: scenes.building(),
    "city": lambda: scenes.city(150),
    "menger": lambda: scenes.menger(0.15, 9),
    "facades": lambda: scenes.facades(40),
    "mixed": lambda: scenes.mixed(90),
    "mixed blocks": lambda: scenes.mixed(90, blocks=True),  # the windows' wall widths are block factors
}


@pytest.mark.parametrize("group", [False, True])
@pytest.mark.parametrize("name", list(BATCHES))
def test_leaf_children_in_place(name, group):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from operatorgraph_gb300.engine import Engine, terminals_to_numpy

    b = BATCHES[name]()
    entries, n = np.ascontiguousarray(b["entries"], dtype=G.ENTRY_DT), len(b["axioms"])
    drawing = DispatchTable([Entry(G.BOX_IF_SIZE_LESS, [G.scalar(0), G.rand(0.1, 0.2)], [(0, 0), (0, 0)])]).to_array()
    blk = None
    if b["blocks"] is not None:  # values of each axiom's own
        own = b["blocks"].reshape(n, -1) * np.random.default_rng(4).uniform(0.9, 1.1, (n, 1)).astype(np.float32)
        blk = torch.from_numpy(np.ascontiguousarray(own)).cuda()
    found = []
    for table in (entries, np.concatenate([entries, drawing])):
        eng = Engine(table, node_capacity=1 << 20, max_terminals=1 << 19, block_stride=b["block_stride"],
                     group_axioms=group)
        out, count, rep = eng.execute(b["axioms"], blocks=blk, capacity=1 << 19)
        assert rep["status"] == 0 and count > 0
        found.append((G.sort_terminals(terminals_to_numpy(out, count), by_path=True), rep["levels"]))
        eng.release()
    (t0, l0), (t1, l1) = found
    assert len(t0) == len(t1) and l0 == l1
    for field in ("path", "rule", "custom", "m"):
        assert np.array_equal(t0[field], t1[field])


def test_grouped_engines_of_either_size():
    """Engines that group axioms take the general kernels from 2^27 terminals of capacity on."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from operatorgraph_gb300.engine import Engine, terminals_to_numpy

    b = scenes.mixed(90)
    found = []
    for cap in (1 << 19, (1 << 27) - 1, 1 << 27):
        eng = Engine(b["entries"], node_capacity=1 << 20, max_terminals=cap, group_axioms=True)
        out, count, rep = eng.execute(b["axioms"], capacity=1 << 19)
        assert rep["status"] == 0
        found.append(G.sort_terminals(terminals_to_numpy(out, count), by_path=True))
        eng.release()
    assert len(found[0]) > 0 and all(np.array_equal(found[0], t) for t in found[1:])
