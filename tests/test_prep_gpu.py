"""The fused input preparation (K centring + fake quantisers + q scaling) against the oracle's restatement of
the adapter.  Integer grids make this almost always bit-exact; a value may land on the neighbouring grid point
when the fp32 K mean differs in its last bit (different summation order), so a tiny fraction of mismatches by
one quantisation step is allowed for K and none for Q and V."""
import pytest
import torch

from oracle import sqattn_oracle as so

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,hq,hkv,d", [(300, 4, 2, 128), (1024, 28, 4, 128), (77, 6, 3, 64)])
@pytest.mark.parametrize("qk_qtype,v_qtype", [("int", "int"), ("e4m3", "e5m2"), ("e5m2", "e4m3")])
def test_prep_matches_adapter(dtype, n, hq, hkv, d, qk_qtype, v_qtype):
    from longcontext_sqattn_paddle_b200 import ops
    q, k, v = so.make_inputs(3, 2, n, hq, hkv, d, dtype)
    q8, q4, k8, k4, v8 = (t.cpu() for t in ops.prep_qkv(q.cuda(), k.cuda(), v.cuda(), qk_qtype=qk_qtype, v_qtype=v_qtype))
    groups = hq // hkv
    r8, r4, rk8, rk4, rv8 = so.prep_qkv(q, k, v, groups, qk_qtype, v_qtype)
    r8, r4 = so.scale_q(r8, d), so.scale_q(r4, d)
    rk8, rk4, rv8 = rk8[:, ::groups], rk4[:, ::groups], rv8[:, ::groups]
    exact = qk_qtype == "int"

    def frac_bad(a, b):
        return (a.float() != b.float()).float().mean().item()

    assert frac_bad(q4, r4) == 0 and frac_bad(k4, rk4) < 2e-3
    if exact:
        assert frac_bad(q8, r8) == 0
        assert frac_bad(k8, rk8) < 2e-3
    else:  # emulated float formats go through log2/exp2: compare by value
        assert (q8.float() - r8.float()).abs().max().item() < 2e-2 * r8.float().abs().max().item()
        assert frac_bad(q8, r8) < 1e-3 and frac_bad(k8, rk8) < 3e-3
    if v_qtype == "int":
        assert frac_bad(v8, rv8.to(torch.float16)) == 0
    else:
        assert frac_bad(v8, rv8.to(torch.float16)) < 1e-3
    assert v8.dtype == torch.float16


def test_operator_boundary():
    """attention_fn installed with types.MethodType like the reference's process_model does."""
    from longcontext_sqattn_paddle_b200.sqattn import process_model
    hq, hkv, n, d = 8, 2, 700, 128

    class Layer:
        num_key_value_groups = hq // hkv

        def prefill_attention(self, q, k, v, mask):
            raise AssertionError("not replaced")

    class Model:
        layers = [Layer(), Layer(), Layer()]

    class Args:
        qk_qtype, v_qtype, use_relative_distance = "int", "int", True

    model = process_model(Model(), "SQAttn", {1: {"bit8": [0.2] * hq, "bit4": [0.4] * hq, "sink": 256}}, Args())
    q, k, v = so.make_inputs(5, 1, n, hq, hkv, d, torch.bfloat16)
    out = model.layers[1].prefill_attention(q.cuda(), k.cuda(), v.cuda(), None)
    assert out.shape == (1, n, hq * d) and out.dtype == torch.bfloat16
    ref = so.attention_fn(q, k, v, hq // hkv, [0.2] * hq, [0.4] * hq, 256)
    assert (out.float().cpu() - ref.float()).abs().max().item() < 2e-2
    with pytest.raises(AssertionError):
        model.layers[0].prefill_attention(q, k, v, None)
    with pytest.raises(ValueError):
        process_model(Model(), "Nope", {}, Args())

    class AbsArgs:
        qk_qtype, v_qtype, use_relative_distance = "int", "int", False

    model = process_model(Model(), "SQAttn", {2: {"bit8": [128] * hq, "bit4": [256] * hq, "sink": 256}}, AbsArgs())
    out = model.layers[2].prefill_attention(q.cuda(), k.cuda(), v.cuda(), None)
    ref = so.attention_fn(q, k, v, hq // hkv, [128] * hq, [256] * hq, 256, use_relative_distance=False)
    assert (out.float().cpu() - ref.float()).abs().max().item() < 2e-2


@pytest.mark.parametrize("n", [1280 + 384, 1700])
def test_host_pipeline_matches_operator(n):
    """Pinned host tensors in, pinned host tensor out, chunked over query rows: bit-identical to the one-shot
    operator (the last chunk is ragged; 1700 tokens: the sequence does not end on a 128-row tile either)."""
    from longcontext_sqattn_paddle_b200.sqattn import HostPrefillPipeline, mp_triton_wrapper
    hq, hkv, d = 8, 2, 128
    q, k, v = so.make_inputs(13, 1, n, hq, hkv, d, torch.bfloat16)

    class Layer:
        num_key_value_groups = hq // hkv

    class Args:
        qk_qtype, v_qtype, use_relative_distance = "int", "int", True

    ref = mp_triton_wrapper(0, [0.2] * hq, [0.4] * hq, 256, Args())(Layer(), q.cuda(), k.cuda(), v.cuda(), None)
    for edge in (512, 128):   # short first and last chunks
        pipe = HostPrefillPipeline([0.2] * hq, [0.4] * hq, 256, Args(), chunk_rows=512, edge_rows=edge)
        assert pipe._bounds(n)[0] == (0, edge) and pipe._bounds(n)[-1][1] == n
        for _ in range(2):   # buffers are reused across calls
            out = pipe(q.pin_memory(), k.pin_memory(), v.pin_memory())
            torch.cuda.synchronize()
            assert out.is_pinned() and torch.equal(out, ref.cpu())
    with pytest.raises(ValueError):
        pipe(q, k, v)   # pageable host memory


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("qtype", ["int", "e4m3", "e5m2"])
def test_q_fake_quant_inside_the_attention_kernel_is_bit_identical(dtype, qtype):
    """The operator hands the raw query to the attention kernel, which fake-quantises and scales every 128-row tile
    in shared memory; the result must be the one obtained from the stand-alone preparation of Q (same device
    functions), for a strided query view of a fused projection, a ragged last tile and a sharded launch."""
    from longcontext_sqattn_paddle_b200 import _lib as L, ops
    hq, hkv, n, d = 8, 2, 1000, 128
    q, k, v = so.make_inputs(17, 1, n, hq, hkv, d, dtype)
    fused = torch.zeros(1, n, (hq + 2 * hkv) * d, dtype=dtype, device="cuda")
    fused[..., :hq * d] = q.cuda().reshape(1, n, hq * d)
    query = fused[..., :hq * d].view(1, n, hq, d)                   # row stride (Hq + 2 Hkv) * D
    q8, _, k8, _, v8 = ops.prep_qkv(query, k.cuda(), v.cuda(), qk_qtype=qtype, skip_bit4=True)
    r8, r4 = [0.2] * hq, [0.4] * hq
    kw = dict(mode=L.MODE_RELATIVE_WINDOW, win8=r8, win4=r4, sink=128, out_dtype=dtype, return_lse=True, p_fp8_mode=L.P_FP8_STAGE2)
    o_ref, lse_ref = ops.prefill(q8, k8, q8, k8, v8, layout="HND", q_is_scaled=True, **kw)
    o, lse = ops.prefill(query, k8, query, k8, v8, layout="NHD", kv_layout="HND", q_fake_quant=qtype, **kw)
    assert torch.equal(o.permute(0, 2, 1, 3), o_ref) and torch.equal(lse, lse_ref)
    # a shard: rows [256, 768) of the sequence
    o, lse = ops.prefill(query[:, 256:768], k8, query[:, 256:768], k8, v8, layout="NHD", kv_layout="HND",
                         q_fake_quant=qtype, q_row_offset=256, **kw)
    assert torch.equal(o.permute(0, 2, 1, 3), o_ref[:, :, 256:768]) and torch.equal(lse, lse_ref[:, :, 256:768])
    with pytest.raises(ValueError):   # two operand sets (absolute windows) keep the stand-alone preparation
        ops.prefill(query, k8, q8.permute(0, 2, 1, 3), k8, v8, layout="NHD", kv_layout="HND", q_fake_quant=qtype, **kw)
    torch.cuda.synchronize()
    ops.check_device_status()


@pytest.mark.parametrize("n,hq,hkv,d", [(1, 4, 2, 128), (63, 4, 1, 64), (8257, 28, 4, 128), (20011, 32, 8, 128), (16500, 32, 8, 64)])
def test_prep_of_slices_equals_the_whole(n, hq, hkv, d):
    """Rows are independent given K's mean: a whole call, whose K blocks add the mean up themselves, equals calls on slices
    that are given the mean, bit for bit (row blocks that end anywhere); so do calls that prepare one tensor at a time."""
    from longcontext_sqattn_paddle_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(n)
    qkv = torch.randn(1, n, (hq + 2 * hkv) * d, generator=g, device="cuda", dtype=torch.bfloat16)
    q, k, v = (t.view(1, n, -1, d) for t in qkv.split([hq * d, hkv * d, hkv * d], dim=-1))
    whole = ops.prep_qkv(q, k, v)
    mean = ops.k_column_sums(k) / torch.tensor(float(n), device="cuda")
    step = 1000
    for r in range(0, n, step):
        part = ops.prep_qkv(q[:, r:r + step], k[:, r:r + step], v[:, r:r + step], k_mean=mean)
        for w, p in zip(whole, part):
            assert torch.equal(w[:, :, r:r + step], p)
    one = ops.prep_qkv(q, None, None)[:2] + ops.prep_qkv(None, k, None)[2:4] + ops.prep_qkv(None, None, v)[4:]
    assert all(torch.equal(w, o) for w, o in zip(whole, one))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,d", [(1, 128), (3, 64), (65, 128), (130, 64)])
def test_query_rows_bit_for_bit(dtype, n, d):
    """Rows of very different ranges beside each other (a row's scale comes from one of its lanes), rows of zeros, values that
    round to a zero of either sign, and quotients on half-integers: the bits of the oracle, on the int8 and the int4 grid."""
    from longcontext_sqattn_paddle_b200 import ops
    q, k, v = so.make_inputs(5, 1, n, 4, 2, d, dtype)
    gen = torch.Generator().manual_seed(n)
    q *= torch.exp2(torch.randint(-8, 9, (1, n, 4, 1), generator=gen).float()).to(dtype)
    q[:, :, 1, ::3] *= 2.0 ** -9
    q[:, ::2, 2] = 0.0
    q[:, :, 3] = (torch.randint(-254, 255, (1, n, d), generator=gen) / 2).to(dtype)   # a range of 127: halves are ties
    q[:, :, 3, 0] = 127.0
    q8, q4, *_ = ops.prep_qkv(q.cuda(), k.cuda(), v.cuda())
    r8, r4, *_ = so.prep_qkv(q, k, v, 2, "int", "int")
    for got, want in ((q8, so.scale_q(r8, d)), (q4, so.scale_q(r4, d))):
        assert torch.equal(got.cpu().view(torch.int16), want.contiguous().view(torch.int16))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("qtype", ["e4m3", "e5m2"])
@pytest.mark.parametrize("n,d", [(1, 128), (3, 64), (65, 128), (130, 64)])
def test_emulated_float_rows_do_not_depend_on_their_place(dtype, qtype, n, d):
    """A thread takes its four rows one after another: a row's bits are those of the same row in another place, beside rows of
    other ranges and rows of zeros, on both outputs."""
    from longcontext_sqattn_paddle_b200 import ops
    q, *_ = so.make_inputs(6, 1, n, 4, 2, d, dtype)
    q *= torch.exp2(torch.randint(-8, 9, (1, n, 4, 1), generator=torch.Generator().manual_seed(n)).float()).to(dtype)
    q[:, ::2, 2] = 0.0
    q = q.cuda()
    whole = ops.prep_qkv(q, None, None, qk_qtype=qtype)[:2]
    bits = lambda t: t.contiguous().view(torch.int16)
    for shift in (1, 8, 16, n // 2):
        moved = ops.prep_qkv(q.roll(shift, 1), None, None, qk_qtype=qtype)[:2]
        assert all(torch.equal(bits(a.roll(shift, 2)), bits(b)) for a, b in zip(whole, moved))
    alone = ops.prep_qkv(q[:, n - 1:], None, None, qk_qtype=qtype)[:2]
    assert all(torch.equal(bits(a[:, :, n - 1:]), bits(b)) for a, b in zip(whole, alone))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_a_nan_in_v_ends_on_the_lowest_step_whatever_lies_beside_it(dtype):
    """The clamp of the integer grid turns a NaN into -128 steps of its channel (the range is taken over the other heads),
    also where none of the channels that one thread holds sits near a half.  The other values are what they are without it."""
    from longcontext_sqattn_paddle_b200 import ops
    g = torch.Generator().manual_seed(5)
    v = torch.randn(1, 200, 6, 64, generator=g).to(dtype)
    heads, chans = torch.arange(200) % 6, torch.arange(200) * 7 % 64
    at = (0, torch.arange(200), heads, chans)
    zero = v.clone()
    zero[at] = 0.0                                        # a zero leaves the range to the other heads as a NaN does
    bad = v.clone()
    bad[at] = float("nan")
    want, got = (ops.prep_qkv(None, None, t.cuda())[4].cpu().transpose(1, 2) for t in (zero, bad))
    step = (zero.float().abs().amax((0, 2)).clamp_min(1e-5) / 127.0)[torch.arange(200), chans]
    assert torch.equal(got[at], (step * -128.0).to(dtype).to(torch.float16))
    want, got = want.clone(), got.clone()
    want[at] = got[at] = 0.0
    assert torch.equal(want, got)


@pytest.mark.parametrize("key_shape,value_shape", [((1, 200, 2, 64), (1, 200, 2, 64)), ((1, 300, 2, 64), (1, 300, 1, 64)),
                                                   ((1, 300, 2, 128), (1, 300, 2, 128)), ((2, 300, 2, 64), (2, 300, 2, 64))])
def test_shapes_that_do_not_fit_the_queries_are_refused(key_shape, value_shape):
    """One length and one head_dim go down for all three tensors: others are refused before anything is launched."""
    from longcontext_sqattn_paddle_b200 import ops
    make = lambda shape: torch.zeros(shape, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(ValueError, match="one batch, length and head_dim"):
        ops.prep_qkv(make((1, 300, 4, 64)), make(key_shape), make(value_shape))


@pytest.mark.parametrize("keys,values,value_heads", [(300, 300, 2), (301, 300, 2), (300, 452, 2), (1000, 600, 3)])
def test_of_longer_keys_and_values_the_first_rows_are_prepared(keys, values, value_heads):
    """Keys and values that reach beyond the queries (a cache with room, a chunk's queries) are prepared up to the queries' length."""
    from longcontext_sqattn_paddle_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(keys + values)
    make = lambda n, h: torch.randn(1, n, h, 128, generator=gen, device="cuda").bfloat16()
    q, k, v = make(300, 4), make(keys, 2), make(values, value_heads)
    got, want = ops.prep_qkv(q, k, v), ops.prep_qkv(q, k[:, :300], v[:, :300, :2])
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    assert torch.equal(ops.prep_qkv(None, k[:, :300], v)[4], want[4])
