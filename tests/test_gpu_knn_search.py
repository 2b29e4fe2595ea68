"""k-NN beyond one thread per query: a warp or several per query, and the search among sorted leaves.
Indices and distances have to equal the oracle's bit for bit, as everywhere."""
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


def _points(kind, B, D, n, g):
    p = torch.randn(B, D, n, generator=g)
    if kind == "sphere":
        return p / p.norm(dim=1, keepdim=True)
    if kind == "lattice":  # few distinct positions: most distances tie
        return torch.randint(0, 12, (B, D, n), generator=g).float()
    if kind == "spot":     # nearly all points in one cell of the curve: the all-pairs kernels take over
        p *= 1e-4
        p[:, :, ::100] *= 1e4
    if kind == "gaps":     # coordinates that are no numbers or infinite
        p[:, :, ::7] = float("nan")
        p[:, 0, ::11] = float("inf")
    return p


# (kind, B, D, M, N, k): above 5e7 pairs the leaves are searched; M = 32 * 32 leaves' minimum, one leaf
# more than a node / a group, odd counts; below, 1 to 32 warps share a query
CASES = [("sphere", 1, 3, 1025, 50001, 9), ("sphere", 1, 3, 32 * 1024 + 33, 2000, 9), ("cloud", 2, 3, 5000, 6000, 32),
         ("lattice", 1, 3, 8000, 8001, 16), ("spot", 1, 3, 9000, 6000, 5), ("gaps", 1, 3, 7001, 8000, 9),
         ("cloud", 1, 2, 7500, 7500, 1), ("sphere", 3, 1, 4999, 3500, 7),
         ("cloud", 1, 3, 40000, 7, 9), ("lattice", 2, 3, 5000, 40, 32), ("gaps", 1, 4, 3000, 300, 8),
         ("cloud", 1, 9, 1100, 65, 3), ("lattice", 1, 3, 33, 20001, 4)]


@pytest.mark.parametrize("kind,B,D,M,N,k", CASES)
def test_knn_search_against_oracle(kind, B, D, M, N, k):
    from mappedconvolutions_b200 import host
    g = torch.Generator().manual_seed(M + N)
    ref = _points(kind, B, D, M, g)
    query = _points(kind, B, D, N, g)
    idx, dist = host.impl.knn_forward(ref.cuda(), query.cuda(), k)
    if kind == "gaps":
        # such references are nobody's neighbours, such queries have none (index 0, infinite distance)
        keep = torch.isfinite(ref[0]).all(0).nonzero().flatten()
        lost = ~torch.isfinite(query[0]).all(0)
        want_idx, want_dist = oracle.knn_forward(ref[:, :, keep].contiguous(), query, k)
        want_idx = keep[want_idx - 1] + 1
        want_idx[:, :, lost], want_dist[:, :, lost] = 0, float("inf")
    else:
        want_idx, want_dist = oracle.knn_forward(ref, query, k)
    assert torch.equal(idx.cpu(), want_idx)
    assert torch.equal(dist.cpu(), want_dist)


def test_knn_of_a_set_with_itself():
    from mappedconvolutions_b200 import host
    p = _points("sphere", 1, 3, 9001, torch.Generator().manual_seed(1))
    d = p.cuda()
    idx, dist = host.impl.knn_forward(d, d, 9)
    want_idx, want_dist = oracle.knn_forward(p, p, 9)
    assert torch.equal(idx.cpu(), want_idx) and torch.equal(dist.cpu(), want_dist)


# Queries that no box rules anything out for: at the centre of a sphere of references, or far away from all; all of
# them, some of them (listed for the all-pairs kernels one by one), in one batch element of two
@pytest.mark.parametrize("B,D,M,N,k,share", [(1, 3, 70001, 900, 9, 1.0), (1, 3, 9001, 7001, 9, 1.0), (1, 3, 40000, 30000, 5, 0.8),
                                             (1, 3, 40000, 2000, 20, 0.02), (2, 2, 20000, 3000, 9, 0.5),
                                             (1, 1, 40000, 1300, 3, 0.5)])
def test_queries_at_the_same_distance_from_everything(B, D, M, N, k, share):
    from mappedconvolutions_b200 import host
    g = torch.Generator().manual_seed(M)
    ref, query = _points("sphere", B, D, M, g), _points("sphere", B, D, N, g)
    if D == 1:
        ref = torch.randn(B, D, M, generator=g)
    n = int(share * N)
    where = torch.randperm(N, generator=g)[:n]
    query[0, :, where[::2]] *= 1e-3
    query[0, :, where[1::2]] *= 1e4
    idx, dist = host.impl.knn_forward(ref.cuda(), query.cuda(), k)
    want_idx, want_dist = oracle.knn_forward(ref, query, k)
    assert torch.equal(idx.cpu(), want_idx)
    assert torch.equal(dist.cpu(), want_dist)
