"""A derivation stops at the end of the level in which a status is raised, in
every build of the kernels: the levels that the report and pga_engine_levels
give for a table whose first axiom fails in the seeding or in a known level
while the second has many levels to go."""
import numpy as np
import pytest

from operatorgraph_gb300 import grammar as G
from operatorgraph_gb300.grammar import DispatchTable, Entry, block, scalar

pytestmark = pytest.mark.gpu

BAD_PARAM = 5
SPLITS = 6


def _table(build):
    """Entries 0 .. 5: splits one into the next (the last makes terminals), 10 .. 15: the same, but the last makes
    a Repeat of extent 0; 20: a chain that fails at once."""
    one = block(0) if build == "blocks" else scalar(-1)
    e = []
    for base in (0, 10):
        for k in range(SPLITS):
            nxt = base + k + 1
            e.append(Entry(G.BOX_SUBDIVIDE, [scalar(k % 3), one, scalar(-1)], [(nxt, 0), (nxt, 0)]))
        e.append(Entry(G.BOX_GENERATE, [scalar(0)], []) if base == 0 else
                 Entry(G.BOX_REPEAT, [scalar(0), scalar(0), scalar(0)], [(6, 0)]))
        e += [Entry(G.BOX_DISCARD, [], [])] * (10 - SPLITS - 1)
    e.append(Entry(G.BOX_IF_SIZE_LESS, [scalar(5), scalar(1)], [(6, 0), (6, 0)]))
    if build == "draws":  # not reached: the table no longer is one of scalars
        e.append(Entry(G.BOX_IF_SIZE_LESS, [scalar(0), G.rand(0.1, 0.2)], [(6, 0), (6, 0)]))
    if build == "turns":
        e.append(Entry(G.BOX_ROTATE, [scalar(10), scalar(20), scalar(30)], [(6, 0)]))
    return DispatchTable(e).to_array()


@pytest.mark.parametrize("build", ["scalars", "blocks", "draws", "turns"])
@pytest.mark.parametrize("entry,levels", [(20, 0), (16, 1), (15, 2), (12, 5), (0, SPLITS)])
def test_levels_of_a_failed_derivation(build, entry, levels):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from operatorgraph_gb300.engine import Engine

    ax = G.make_axioms(3000)  # many blocks' worth, the failing one in the first
    ax["entry"], ax["shape"], ax["size"], ax["block"] = 0, G.SHAPE_BOX, 1.0, 0
    ax["entry"][0] = entry
    blk = torch.full((1,), -1.0, device="cuda")
    eng = Engine(_table(build), node_capacity=1 << 20, max_terminals=1 << 18, block_stride=1, no_inline=True)
    _, _, rep = eng.execute(ax, blocks=blk, capacity=1 << 18, check=False)
    assert rep["status"] == (BAD_PARAM if entry else 0)
    starts, _ = eng.levels()
    assert rep["levels"] == levels and len(starts) == levels + 1
    eng.release()
