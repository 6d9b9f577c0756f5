"""Window calibration: threshold search on CPU (host logic) and the fused histogram kernel against the dense-map
restatement of the reference."""
import numpy as np
import pytest
import torch

from oracle import window_search_oracle as wo


def test_threshold_search_matches_reference_rules(tmp_path):
    from longcontext_sqattn_paddle_b200.sqattn import window_search as ws
    rng = np.random.default_rng(0)
    for _ in range(20):
        h = rng.random(200) * (rng.random(200) > 0.3)
        for thr in (0.5, 0.9, 0.99, 1.0):
            assert ws.find_optimal_relative_window(h, thr, 200) == wo.find_optimal_relative_window(h, thr, 200)
        h2 = rng.random(1000)
        for thr in (0.5, 0.95):
            assert ws.find_optimal_window(h2, thr) == wo.find_optimal_window(h2, thr)
    assert ws.find_optimal_relative_window(np.zeros(200), 0.9, 200) == 0.1   # the fallback the shipped reference always hits
    assert ws.find_optimal_window(np.zeros(10), 0.9) == 1
    alloc = {1: ws.bits_alloc_entry([{"bit8_relative": 0.1, "bit4_relative": 0.3}] * 4, True)}
    ws.save_bits_alloc(tmp_path / "b.json", alloc)
    assert ws.load_bits_alloc(tmp_path / "b.json") == alloc and alloc[1]["sink"] == 256


@pytest.mark.gpu
@pytest.mark.parametrize("relative,sink", [(True, 64), (True, 256), (False, 0), (False, 32)])
def test_histogram_kernel_matches_dense_map(relative, sink):
    from longcontext_sqattn_paddle_b200.sqattn import window_search as ws
    hq, hkv, n, d, bins = 4, 2, 700, 128, 200
    g = torch.Generator().manual_seed(1)
    q = torch.randn(hq, n, d, generator=g).to(torch.bfloat16)
    k = torch.randn(hkv, n, d, generator=g).to(torch.bfloat16)
    nb = bins if relative else n
    hist = ws.attention_histograms(q.cuda(), k.cuda(), relative=relative, num_bins=nb, sink_len=sink).cpu().numpy()
    a = wo.attention_map(q, k)
    for h in range(hq):
        ref = wo.relative_histogram_with_sink(a[h], bins, sink) if relative else wo.absolute_histogram_with_sink(a[h], n, sink)
        assert np.allclose(hist[h], ref, rtol=2e-3, atol=2e-3 * ref.max())
        for thr in (0.8, 0.95):
            if relative:
                assert abs(ws.find_optimal_relative_window(hist[h], thr, bins) - wo.find_optimal_relative_window(ref, thr, bins)) <= 1.0 / bins
            else:
                assert ws.find_optimal_window(hist[h], thr) == wo.find_optimal_window(ref, thr)

    class Args:
        use_relative_distance, bit8_thres, bit4_thres, relative_bins, sink_window_size = relative, 0.8, 0.95, bins, sink

    b8, b4, windows = ws.calibrate_windows([(q.cuda(), k.cuda())], Args(), max_len=n)
    assert len(windows) == hq and b8 <= b4


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,bins,sink", [(1, 128, 200, 0), (5, 64, 7, 256), (127, 128, 1, 0), (128, 128, 100, 5), (129, 128, 200, 0),
                                           (257, 64, 256, 256), (1000, 128, 3, 130), (2311, 128, 200, 256), (2500, 64, 100, 77)])
def test_relative_histogram_at_tile_and_bin_edges(n, d, bins, sink):
    """Rows that end inside a tile, sinks that do, bins narrower and wider than the kernel's key groups.  All weights are
    positive, so a bin's relative error is at most that of a pair: 2^-22 of the exponential plus the rounding of an fp32
    score of magnitude <= 40 summed over 128 products (3e-6 each way)."""
    from longcontext_sqattn_paddle_b200.sqattn import window_search as ws
    for dtype in (torch.bfloat16, torch.float16):
        g = torch.Generator().manual_seed(n)
        q, k = torch.randn(4, n, d, generator=g).to(dtype), torch.randn(2, n, d, generator=g).to(dtype)
        k[..., 5::32] *= 8.0
        hist = ws.attention_histograms(q.cuda(), k.cuda(), relative=True, num_bins=bins, sink_len=sink).cpu().numpy()
        a = wo.attention_map(q, k)
        for h in range(4):
            np.testing.assert_allclose(hist[h], wo.relative_histogram_with_sink(a[h], bins, sink), rtol=5e-5, atol=1e-30)


@pytest.mark.gpu
@pytest.mark.parametrize("n,bins", [(8, 200), (40, 248), (200, 200), (1000, 200), (3000, 100)])
def test_relative_histogram_keeps_fp32_precision_in_bins_narrower_than_a_key(n, bins):
    """Without a sink, rows of a few keys have all their weight in bins much narrower than a key.  All terms of a bin are
    positive, so its relative error is a pair's: 2^-22 of the exponential, 2^-23 * 10 * 4 / 8 = 6e-7 of an fp32 score of
    magnitude <= 10 summed over 64 products, and 1e-6 for some sixteen roundings of sums, weight and normalisation."""
    from longcontext_sqattn_paddle_b200.sqattn import window_search as ws
    g = torch.Generator().manual_seed(n)
    q, k = ((torch.randn(h, n, 64, generator=g) * 0.5).to(torch.bfloat16) for h in (4, 2))
    hist = ws.attention_histograms(q.cuda(), k.cuda(), relative=True, num_bins=bins, sink_len=0).cpu().numpy()
    a = wo.attention_map(q, k)
    for h in range(4):
        np.testing.assert_allclose(hist[h], wo.relative_histogram_with_sink(a[h], bins, 0), rtol=2e-6, atol=1e-30)


def test_unaligned_inputs_are_refused_before_a_kernel_reads_them():
    from longcontext_sqattn_paddle_b200 import _lib as L
    for q, k in ((0x1008, 0x2000), (0x1000, 0x2002)):
        for d in (32, 64, 128):
            assert L.lib.sqattn_window_histogram(q, k, L.BF16, 4, 2, 100, d, 1, 50, 0, 0x3000, None) == L.ERR_INVALID_ARG


@pytest.mark.gpu
@pytest.mark.parametrize("relative", [True, False])
def test_histograms_of_views(relative):
    """Token-major views of both inputs (each has to be copied, and the copies have to live together), and unaligned ones."""
    from longcontext_sqattn_paddle_b200.sqattn import window_search as ws
    n, d, bins = 900, 64, 100
    g = torch.Generator(device="cuda").manual_seed(7)
    q, k = (torch.randn(h, n, d, generator=g, device="cuda").to(torch.bfloat16) for h in (4, 2))

    def hist(a, b):
        return ws.attention_histograms(a, b, relative=relative, num_bins=bins if relative else n, sink_len=64).cpu().numpy()

    want = hist(q, k)
    token_major = [t.transpose(0, 1).contiguous().transpose(0, 1) for t in (q, k)]
    shifted = [torch.cat([t.new_zeros(3), t.flatten()])[3:].view(t.shape) for t in (q, k)]
    for a, b in (token_major, shifted):
        np.testing.assert_allclose(hist(a, b), want, rtol=1e-5)        # the same values, a block's fp32 sums in another order


@pytest.mark.gpu
@pytest.mark.parametrize("n,bins,sink", [(33001, 200, 0), (40000, 96, 256), (65001, 100, 0)])
def test_relative_histogram_of_rows_beyond_31250_keys(n, bins, sink):
    """There the reference's fp32 expression can put the key beside a bin's edge on either side, and the kernel asks the
    expression itself.  The definition in fp64 on the GPU, bins in fp32 as the reference has them; the bar is that of
    test_relative_histogram_at_tile_and_bin_edges (one key on the wrong side of an edge moves a bin by 1 / keys per bin)."""
    from longcontext_sqattn_paddle_b200.sqattn import window_search as ws
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k = (torch.randn(1, n, 64, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    hist = ws.attention_histograms(q, k, relative=True, num_bins=bins, sink_len=sink)
    ref = torch.zeros(bins, dtype=torch.float64, device="cuda")
    cols, kt = torch.arange(n, device="cuda")[None], k[0].double().T
    for r in range(0, n, 512):
        rows = torch.arange(r, min(r + 512, n), device="cuda")[:, None]
        a = torch.softmax((q[0, r:r + 512].double() @ kt / 8.0).masked_fill(cols > rows, float("-inf")), -1)
        rel = (rows - cols).float() / torch.clamp(rows.float() - sink, min=1)
        rel[rows.squeeze(1) <= sink] = 0
        b = torch.clamp((rel * bins).floor().long(), 0, bins - 1)
        w = (a * (rel * bins + 1)).masked_fill((cols > rows) | (cols < sink), 0.0)
        ref += torch.zeros(len(rows), bins, dtype=torch.float64, device="cuda").scatter_add_(1, b, w).sum(0)
    np.testing.assert_allclose(hist[0].cpu().numpy(), ref.cpu().numpy(), rtol=5e-5)
