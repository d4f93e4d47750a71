"""PathTarget on the CPU: the loss matched by path against the loss over both
sides sorted by path, whichever side is put in order; gradients and the check."""
import pytest

torch = pytest.importorskip("torch")

from operatorgraph_gb300.autograd import PathTarget, centres_extents  # noqa: E402


def _case(n, seed, double_path=False):
    g = torch.Generator().manual_seed(seed)
    M, T = (torch.randn(n, 12, generator=g, dtype=torch.float64) for _ in range(2))
    paths = torch.randperm(4 * n + 4, generator=g)[:n] * 7 - 2 * n
    if double_path and n > 1:
        paths[1] = paths[0]
    return M, T, paths, torch.randperm(n, generator=g)


@pytest.mark.parametrize("n,double_path,check", [(0, False, True), (1, False, True), (2, False, True), (57, False, True),
                                                 (57, False, False), (57, True, True)])
def test_sse_is_the_loss_over_both_sides_sorted_by_path(n, double_path, check):
    M, T, paths, shuffle = _case(n, 3 + n, double_path)
    target = PathTarget(T, paths)
    mine = M[shuffle].clone().requires_grad_()
    loss = target.sse(mine, paths[shuffle], check=check)
    loss.backward()
    a = M[shuffle].clone().requires_grad_()
    order = torch.argsort(paths[shuffle])
    (c, e), (ct, et) = centres_extents(a[order]), centres_extents(T[torch.argsort(paths)])
    want = ((c - ct) ** 2).sum() + ((e - et) ** 2).sum()
    want.backward()
    if double_path:  # equal paths may pair either way round
        return
    # two orders of a 57-term sum in FP64
    assert torch.allclose(loss, want, rtol=1e-13, atol=0)
    assert torch.allclose(mine.grad, a.grad, rtol=1e-13, atol=0)


def test_other_paths_are_refused():
    M, T, paths, shuffle = _case(9, 1)
    target = PathTarget(T, paths)
    for k, v in ((0, 10**6), (4, -(10**6)), (5, None)):
        other = paths[shuffle].clone()
        other[k] = other[(k + 1) % 9] if v is None else v
        with pytest.raises(ValueError):
            target.sse(M, other)
    with pytest.raises(ValueError):
        target.sse(M[:8], paths[:8])
    with pytest.raises(RuntimeError):
        target.sse(M[:8], paths[:8], check=False)


def test_centres_do_not_alias_the_transforms():
    M = torch.randn(4, 12)
    c, _ = centres_extents(M)
    c += 1.0
    assert torch.equal(c - 1.0, M[:, [3, 7, 11]]) or torch.allclose(c - 1.0, M[:, [3, 7, 11]])
