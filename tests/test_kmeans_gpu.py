"""Clustering kernels against the CPU oracle: assignments, counts, member lists bit-exact; centroids and value
sums bit-exact as well (exact sums, one rounding)."""
import os

import numpy as np
import pytest
import torch

from oracle import kmeans_oracle as ko

pytestmark = pytest.mark.gpu


def _data(g, t, d, seed, dtype):
    gen = torch.Generator().manual_seed(seed)
    x = torch.randn(g, t, d, generator=gen)
    x[..., 5] *= 8
    return x.to(dtype)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("g,t,k,d", [(2, 500, 64, 64), (3, 4096, 96, 128), (1, 1000, 32, 128)])
def test_train_step(dtype, g, t, k, d):
    from longcontext_sqattn_paddle_b200.cache_hub import kmeans as km
    data = _data(g, t, d, 1, dtype)
    cent = data[:, ko.init_centroid_indices(t, k)].contiguous()
    cent[:, 3] = cent[:, 1]  # duplicate centroid: exact ties must go to the lower index
    for norm in (True, False):
        rc, ridx, rcnt = ko.k_means_train(data, cent, norm)
        dc = cent.clone().cuda()
        _, idx, cnt = km.k_means_train(data.cuda(), dc, norm)
        assert torch.equal(idx.cpu(), ridx)
        assert torch.equal(cnt.cpu(), rcnt)
        assert torch.equal(dc.cpu().view(torch.int16), rc.view(torch.int16))
        cent = rc


def test_segment_k_means_full():
    from longcontext_sqattn_paddle_b200.cache_hub import segment_k_means
    g, t, k, d = 4, 8192, 128, 128
    key, val = _data(g, t, d, 2, torch.bfloat16), _data(g, t, d, 3, torch.bfloat16)
    for segs in (1, 4):
        rc, rvs, rcl, rcs, ridx = ko.segment_k_means(key, val, k, 10, segs)
        c, vs, cl, cs, idx = segment_k_means(key.cuda(), val.cuda(), k, 10, segs, return_indices=True)
        assert torch.equal(idx.cpu(), ridx)
        assert torch.equal(cs.cpu(), rcs)
        assert torch.equal(cl.cpu(), rcl)
        assert torch.equal(c.cpu().view(torch.int16), rc.view(torch.int16))
        assert torch.equal(vs.cpu().view(torch.int16), rvs.view(torch.int16))


def test_kmeans_reference_golden(golden_dir):
    from longcontext_sqattn_paddle_b200.cache_hub import kmeans as km
    z = np.load(os.path.join(golden_dir, "kmeans.npz"))
    g = {n: torch.from_numpy(z[n]) for n in z.files}
    cent = g["cent0"].clone().cuda()
    for it, norm in enumerate((True, False)):
        _, idx, cnt = km.k_means_train(g["data"].cuda(), cent, norm)
        assert torch.equal(idx.cpu(), g[f"idx{it}"])
        assert torch.equal(cnt.cpu(), g[f"cnt{it}"])
        cent = g[f"cent{it + 1}"].clone().cuda()


def test_clustered_retrieval_ragged_decode():
    """Ragged batch, Llama-3-8B head geometry: selected token indices bit-exact against the oracle's retrieval
    rule; attention over the gathered tokens within the decode tolerance (2e-2) with 16-bit P.  With FP8 P the
    rounding of p*448 is taken relative to the running maximum, which a split-KV kernel restarts per key range
    and per warp, so individual e4m3 decisions (6 % steps) differ from the sequential oracle: 6e-2 there."""
    from longcontext_sqattn_paddle_b200.cache_hub import ClusteredKV, RaggedClusteredDecoder
    from oracle import sqattn_oracle as so
    hq, hkv, d, budget = 32, 8, 128, 1024
    lens = [3000, 9000, 5000]
    keys = [_data(hkv, n, d, 10 + i, torch.bfloat16) for i, n in enumerate(lens)]
    vals = [_data(hkv, n, d, 20 + i, torch.bfloat16) for i, n in enumerate(lens)]
    caches = [ClusteredKV(k.cuda(), v.cuda()) for k, v in zip(keys, vals)]
    dec = RaggedClusteredDecoder(caches, budget=budget)
    g = torch.Generator().manual_seed(30)
    q = torch.randn(len(lens), hq, 1, d, generator=g).to(torch.bfloat16)
    out = dec.step(q.cuda()).cpu()
    out16 = RaggedClusteredDecoder(caches, budget=budget, p_fp8=False).step(q.cuda()).cpu()
    # the per-sequence entry points select the same tokens; the attention then only differs in where the planner,
    # which sees the counts on the host there, cuts the key ranges
    idx_b, cnt_b = dec.idx.clone(), dec.count.clone()
    out_u = dec.step_unbatched(q.cuda()).cpu()
    assert torch.equal(cnt_b, dec.count)
    for i in range(len(lens)):
        for h in range(hkv):
            assert torch.equal(idx_b[i, h, :cnt_b[i, h]], dec.idx[i, h, :cnt_b[i, h]])
    assert (out_u.float() - out.float()).abs().max().item() < 3e-2
    groups = hq // hkv
    for i, n in enumerate(lens):
        k = ko.init_centroid_indices(n, caches[i].k).numel()
        rc, _, rcl, rcs, _ = ko.segment_k_means(keys[i], vals[i], k, 10, 1)
        assert torch.equal(caches[i].cluster_size.cpu(), rcs) and torch.equal(caches[i].clusters.cpu(), rcl)
        qm = torch.zeros(hkv, d)
        for h in range(groups):   # fp32, heads added in order, one division
            qm = qm + q[i, :, 0].view(hkv, groups, d)[:, h].float()
        qm = qm / float(groups)
        sel = ko.select_clusters(qm, rc, rcs, rcl, budget)
        cnt = dec.count[i].cpu()
        for h in range(hkv):
            assert int(cnt[h]) == sel[h].numel() and sel[h].numel() >= budget
            assert torch.equal(dec.idx[i, h, :cnt[h]].cpu(), sel[h])
            kq = keys[i][h, sel[h].long()][None, None]     # [1,1,n,d]
            vq = vals[i][h, sel[h].long()][None, None]
            qh = q[i, h * groups:(h + 1) * groups][None]   # [1,groups,1,d]
            ro = so.decode(qh, kq, vq, output_dtype=torch.bfloat16, is_P_fp8_quant=True, center_k=False, mask_tail=True)
            assert (out[i, h * groups:(h + 1) * groups].float() - ro[0].float()).abs().max().item() < 6e-2
            ro = so.decode(qh, kq, vq, output_dtype=torch.bfloat16, center_k=False, mask_tail=True)
            assert (out16[i, h * groups:(h + 1) * groups].float() - ro[0].float()).abs().max().item() < 2e-2


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("t,d", [(1, 128), (63, 128), (64, 64), (65, 128), (257, 128), (5000, 64), (20000, 128)])
def test_member_sums_and_lists_with_uneven_clusters(dtype, t, d):
    """Sums and sorted lists where they are cut into ranges: one cluster holds half of the tokens, others one or none.
    The fp64 sum of 16-bit values is exact, so the sums are compared exactly."""
    from longcontext_sqattn_paddle_b200.cache_hub import kmeans as km
    g, k = 2, 96
    gen = torch.Generator().manual_seed(t + d)
    idx = torch.randint(0, k - 5, (g, t), generator=gen, dtype=torch.int32)      # the last clusters stay empty
    idx[torch.rand(g, t, generator=gen) < 0.5] = 7
    val = torch.randn(g, t, d, generator=gen).to(dtype)
    val[0, 0, 0], val[1, t - 1, 1] = 0.0, 6e-8                                    # zero and a subnormal of the half type
    sums = torch.zeros(g, k, d, dtype=torch.float64)
    sums.scatter_add_(1, idx.long()[..., None].expand(-1, -1, d), val.double())
    got = km.index_add(val.cuda(), idx.cuda(), k)
    assert torch.equal(got.cpu(), sums.float().to(dtype))
    n = torch.stack([torch.bincount(r.long(), minlength=k) for r in idx])
    width = int(n.max())
    lists, size = km.reverse_index(idx.cuda(), k, width)
    assert torch.equal(size.cpu().long(), n)
    for b in range(g):
        for c in range(k):
            assert torch.equal(lists[b, c, :n[b, c]].cpu().long(), (idx[b] == c).nonzero()[:, 0])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("g,t,k,d", [(1, 1, 32, 128), (2, 255, 96, 64), (3, 20001, 288, 128), (7, 6000, 544, 64)])
def test_assignment_over_many_items(dtype, g, t, k, d):
    """More 256-token items than CTAs, groups that end inside an item, centroid counts that end inside a tile.  Exact
    arg-max: keys that are zero (every score ties, below any exponent), centroids that are repeated (lowest index), and a
    NaN key, which has no arg-max but must get some centroid."""
    from longcontext_sqattn_paddle_b200.cache_hub import kmeans as km
    gen = torch.Generator(device="cuda").manual_seed(t)
    data = torch.randn(g, t, d, generator=gen, device="cuda").to(dtype)
    cent = torch.randn(g, k, d, generator=gen, device="cuda").to(dtype)
    cent[:, k // 2:k // 2 + 8] = cent[:, :8]
    data[:, ::7] = 0.0
    data[:, 1::11] *= 1e-6 if dtype == torch.float16 else 1e-30
    want = (data.double() @ cent.double().transpose(1, 2)).argmax(-1)
    want[(data == 0).all(-1)] = 0
    want = torch.where((want >= k // 2) & (want < k // 2 + 8), want - k // 2, want)
    nan = t // 2
    if t > 1:
        data[0, nan, 3] = float("nan")
    _, idx, counts = km.k_means_train(data, cent.clone(), True)
    if t > 1:
        assert 0 <= idx[0, nan].item() < k
        want[0, nan] = idx[0, nan]
    assert torch.equal(idx.long(), want)
    assert torch.equal(counts.long(), torch.stack([torch.bincount(r.long(), minlength=k) for r in idx]))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("g,t,k,d", [(1, 300, 32, 128), (2, 700, 160, 64), (1, 513, 416, 128)])
def test_assignment_among_negative_and_close_scores(dtype, g, t, k, d):
    """Every score is negative and most lie within a few parts in a thousand of each other, so that the largest one is
    a small negative number of the scan's units; exact arg-max, lowest index on ties."""
    from longcontext_sqattn_paddle_b200.cache_hub import kmeans as km
    gen = torch.Generator().manual_seed(31 * k + d)
    data = (torch.rand(g, t, d, generator=gen) + 0.5).to(dtype)
    cent = (-1.0 - 2.0 ** -6 * torch.rand(g, k, d, generator=gen)).to(dtype)
    cent[:, k // 2:] = cent[:, : k - k // 2].roll(1, 2)
    _, idx, _ = km.k_means_train(data.cuda(), cent.cuda().clone(), False)
    assert torch.equal(idx.cpu(), ko.assign(data, cent).to(idx.dtype))


@pytest.mark.parametrize("key_exp,cent_exp", [(0, 0), (-90, 0), (0, -90), (-80, -70), (100, 30)])
@pytest.mark.parametrize("d", [64, 128])
def test_assignment_where_fp32_has_no_squares_of_the_norms(d, key_exp, cent_exp):
    """Exact arg-max of bf16 keys and centroids whose squared norms underflow or overflow in fp32.  The centroids of a group
    differ from each other by last places of every other channel, which the keys hardly weigh (2^-12 of the others): fp32
    sums put up to two thirds of the keys on another one.  Eight-bit integers times powers of two, so that the sums are
    exact in fp64 in any order."""
    from longcontext_sqattn_paddle_b200.cache_hub import kmeans as km
    g, t, k = 2, 700, 96
    gen = torch.Generator().manual_seed(d)

    def pick(lo, hi, *shape):
        return torch.randint(lo, hi, shape, generator=gen).double() * (2.0 * torch.randint(0, 2, shape, generator=gen) - 1.0)

    data, base = pick(128, 256, g, t, d), pick(130, 254, g, 1, d)
    data[..., 1::2] *= 2.0 ** -12
    bump = torch.zeros(g, k, d, dtype=torch.float64)
    bump[..., 1::2] = torch.randint(-1, 2, (g, k, d // 2), generator=gen).double()
    data, cent = (data * 2.0 ** key_exp).bfloat16(), ((base + bump) * 2.0 ** cent_exp).bfloat16()
    score = data.double() @ cent.double().transpose(1, 2)
    want = torch.where(score == score.amax(-1, keepdim=True), torch.arange(k), k).amin(-1)
    _, idx, _ = km.k_means_train(data.cuda(), cent.cuda(), True)
    assert torch.equal(idx.cpu().long(), want)


@pytest.mark.parametrize("g,t,k", [(2, 700, 1024), (1, 5000, 9600), (3, 20000, 4992)])
def test_member_lists_with_fewer_ranges_than_usual(g, t, k):
    """Clusters of few tokens: the counters of the sort's token ranges fit only a few times into the scratch."""
    from longcontext_sqattn_paddle_b200.cache_hub import kmeans as km
    idx = torch.randint(0, k, (g, t), generator=torch.Generator().manual_seed(k), dtype=torch.int32)
    n = torch.stack([torch.bincount(r.long(), minlength=k) for r in idx])
    lists, size = (r.cpu().long() for r in km.reverse_index(idx.cuda(), k, int(n.max())))
    assert torch.equal(size, n)
    for b in range(g):
        order = torch.sort(idx[b].long(), stable=True).indices          # members one cluster after another, in token order
        assert torch.equal(lists[b][torch.arange(lists.shape[2]) < n[b][:, None]], order)


def _exact_assignment(data, cent):
    """Largest fp64 score, lowest index on ties; a score that is not a number is never taken, 0 where none is left."""
    score = data.double() @ cent.double().transpose(1, 2)
    score = score.nan_to_num(nan=-float("inf"), posinf=float("inf"), neginf=-float("inf"))
    best = score.amax(-1, keepdim=True)
    k = cent.shape[1]
    return torch.where(score == best, torch.arange(k, device=data.device), k).amin(-1)


@pytest.mark.parametrize("g,t,k,d,twice,zeros", [
    (2, 10000, 6144, 128, 64, 0), (1, 20000, 6176, 128, 64, 0), (2, 7000, 9600, 64, 4800, 0), (1, 10000, 12320, 128, 64, 0),
    (1, 5000, 24608, 128, 12304, 0), (1, 2500, 49152, 64, 64, 0), (1, 900, 12320, 128, 6160, 0), (2, 9000, 64, 128, 32, 4500),
    (8, 30000, 64, 64, 8, 0), (8, 100000, 64, 64, 8, 0), (8, 250, 1024, 128, 8, 0)])
def test_many_centroids_and_long_lists(g, t, k, d, twice, zeros):
    """Every number of tokens that a sweep of the re-scoring takes (8, 4, 2 and 1 as their scores' memory allows, 1 in small
    calls), up to the most centroids a group may have; ranks counted by CTAs and, above 8192 clusters, by warps; and more listed
    tokens than the list holds.  ``twice`` centroids are there twice: their tokens are re-scored, and the lower index wins.
    Exact indices, counts and sums."""
    from longcontext_sqattn_paddle_b200.cache_hub import kmeans as km
    gen = torch.Generator(device="cuda").manual_seed(k + t)
    data = torch.randn(g, t, d, generator=gen, device="cuda").bfloat16()
    data[:, t - zeros:] = 0.0
    cent = torch.randn(g, k, d, generator=gen, device="cuda").bfloat16()
    cent[:, k - twice:] = cent[:, :twice]
    want = _exact_assignment(data, cent)
    want = torch.where(want >= k - twice, want - (k - twice), want)
    new, idx, counts = km.k_means_train(data, cent.clone(), False)
    assert torch.equal(idx.long(), want)
    n = torch.stack([torch.bincount(r, minlength=k) for r in want])
    assert torch.equal(counts.long(), n)
    sums = torch.zeros(g, k, d, dtype=torch.float64, device="cuda").scatter_add_(1, want[..., None].expand(-1, -1, d), data.double())
    mean = torch.where(n[..., None] > 0, (sums.float() / n[..., None].float()).bfloat16(), cent)
    assert torch.equal(new, mean)
    assert torch.equal(km.index_add(data, idx, k), sums.float().bfloat16())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("t,k,d", [(300, 32, 128), (700, 64, 64), (2000, 416, 128)])
def test_assignment_with_infinities_and_nans(dtype, t, k, d):
    """Infinite and NaN elements in keys, then in centroids: the largest score that is a number, whatever stands beside it."""
    from longcontext_sqattn_paddle_b200.cache_hub import kmeans as km
    gen = torch.Generator(device="cuda").manual_seed(t)
    data = torch.randn(2, t, d, generator=gen, device="cuda").to(dtype)
    cent = torch.randn(2, k, d, generator=gen, device="cuda").to(dtype)
    odd = data.clone()
    odd[:, 3::7, 1], odd[:, 5::11, 2], odd[:, 4::13, 0] = float("inf"), -float("inf"), float("nan")
    wild = cent.clone()
    wild[0, 3, :] = float("nan")
    wild[0, 7, 3], wild[0, 9, 4], wild[1, k - 1, 5] = float("inf"), -float("inf"), float("nan")
    for x, c in ((odd, cent), (data, wild), (odd, wild)):
        _, idx, _ = km.k_means_train(x, c.clone(), False)
        assert torch.equal(idx.long(), _exact_assignment(x, c))
