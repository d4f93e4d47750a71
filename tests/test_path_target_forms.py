"""PathTarget made and used in other ways: made where nothing may be read back,
restored from what an object of an earlier version holds, on strided paths, and
with a path that occurs twice."""
import warnings

import pytest

torch = pytest.importorskip("torch")

from operatorgraph_gb300.autograd import PathTarget, centres_extents  # noqa: E402


def test_made_without_reading_the_paths_back():
    """On tensors without values, as under the capture of a graph, where a read-back is an error."""
    t = PathTarget(torch.empty(5, 12, device="meta"), torch.empty(5, dtype=torch.int64, device="meta"))
    assert t.paths.shape == (5,) and t.c.shape == (5, 3) and t.e.shape == (5, 3)


@pytest.mark.parametrize("check", [True, False])
def test_restored_from_paths_centres_and_extents(check):
    g = torch.Generator().manual_seed(2)
    M, paths = torch.randn(20, 12, generator=g, dtype=torch.float64), torch.randperm(90, generator=g)[:20]
    old = PathTarget.__new__(PathTarget)
    order = torch.argsort(paths)
    old.__dict__.update(paths=paths[order], c=centres_extents(M[order])[0], e=centres_extents(M[order])[1])
    assert float(old.sse(M, paths, check=check)) == 0.0
    if check:
        with pytest.raises(ValueError):
            old.sse(M, paths + 1)


def test_paths_inside_a_larger_record():
    g = torch.Generator().manual_seed(3)
    M, rows = torch.randn(20, 12, generator=g, dtype=torch.float64), torch.zeros(20, 8, dtype=torch.int64)
    rows[:, 7] = torch.randperm(90, generator=g)[:20]
    target = PathTarget(M, rows[:, 7])
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert float(target.sse(M, rows[:, 7])) == 0.0


@pytest.mark.parametrize("check", [True, False])
def test_a_doubled_path_pairs_one_way_or_the_other(check):
    g = torch.Generator().manual_seed(5)
    M, T = (torch.randn(57, 12, generator=g, dtype=torch.float64) for _ in range(2))
    paths = torch.randperm(300, generator=g)[:57] * 7 - 2 * 57
    paths[1] = paths[0]
    shuffle = torch.randperm(57, generator=g)
    mine = M[shuffle].clone().requires_grad_()
    loss = PathTarget(T, paths).sse(mine, paths[shuffle], check=check)
    loss.backward()
    found = []
    for swap in (False, True):
        other = T.clone()
        if swap:
            other[[0, 1]] = T[[1, 0]]
        a = M.clone().requires_grad_()
        (c, e), (ct, et) = centres_extents(a), centres_extents(other)
        want = ((c - ct) ** 2).sum() + ((e - et) ** 2).sum()
        want.backward()
        # two orders of a 342-term sum in FP64
        found.append(torch.allclose(loss, want, rtol=1e-13, atol=0)
                     and torch.allclose(mine.grad, a.grad[shuffle], rtol=1e-13, atol=0))
    assert sum(found) == 1
    with pytest.raises(ValueError):  # the path once only
        once = paths[shuffle].clone()
        once[(shuffle == 1).nonzero()[0, 0]] = 10**6
        PathTarget(T, paths).sse(M[shuffle], once)
