"""INT8 path parity: bit-exact K codes/scales, INT8-QK^T forward, fp16 backward."""
import numpy as np
import pytest
import torch

import cases
import util
from oracle import attention_oracle as orc
from util import DEV, maxdiff

pytestmark = pytest.mark.gpu
INT8_GRAD_TOL = 5e-2  # the reference's own bar for this path (tests/test_compare_implementations.py:27)


def test_golden_k_quantiser_bit_exact(golden):
    from flash_attn_triton_b200 import _ops
    g = golden("int8_kquant")
    k = cases.k_with_outliers(21, 4, 192, 128)
    assert cases.checksum(k) == str(g["checksum"])
    k8, s_k = _ops.quantize_k_int8(k.to(DEV))
    assert np.array_equal(k8.cpu().numpy(), g["k8"])
    assert np.array_equal(s_k.cpu().numpy().view(np.uint32), g["s_k"].view(np.uint32))


@pytest.mark.parametrize("D", [32, 64, 128, 256])
def test_k_quantiser_bit_exact_vs_oracle(D):
    from flash_attn_triton_b200 import _ops
    k = cases.k_with_outliers(500 + D, 3, 5, 333, D)
    # rounding ties and the amax<1 clamp
    k[0, 0, 0] = 0.0
    k[0, 0, 1, :] = 0.25
    k[0, 0, 2, 0] = 127.0
    k[0, 0, 2, 1:] = torch.linspace(-60, 60, D - 1).half() + 0.5
    k8, s_k = _ops.quantize_k_int8(k.to(DEV))
    r8, rs = orc.quantize_k_rows_ref(k)
    assert np.array_equal(k8.cpu().numpy(), r8)
    assert np.array_equal(s_k.cpu().numpy().view(np.uint32), rs.view(np.uint32))


@pytest.mark.parametrize("causal", [0, 1])
def test_golden_int8_forward(golden, causal):
    from flash_attn_triton_b200 import _ops
    g = golden(f"int8_fwd_causal{causal}")
    q, k, v = cases.int8_case(30, 1, 2, 256, 128)
    assert cases.checksum(q, k, v) == str(g["checksum"])
    o, lse, _, _ = _ops.int8_forward(q.to(DEV), k.to(DEV), v.to(DEV), bool(causal), 1.0 / 128 ** 0.5)
    assert maxdiff(o, g["out"]) <= util.FWD_TOL
    assert maxdiff(lse, g["lse2"]) <= util.FWD_TOL


@pytest.mark.parametrize("shape", [(2, 2, 128, 64), (1, 3, 320, 128), (1, 1, 64, 32), (1, 2, 192, 256)])
@pytest.mark.parametrize("causal", [False, True])
def test_int8_forward_backward_vs_oracle(shape, causal):
    import flash_attn_triton_b200 as fa
    B, H, S, D = shape
    q, k, v = cases.int8_case(600 + S, B, H, S, D)
    do = torch.from_numpy(np.random.default_rng(S).standard_normal((B, H, S, D), dtype=np.float32)).half()
    qd, kd, vd = (t.to(DEV).requires_grad_() for t in (q, k, v))
    out = fa.attention_int8(qd, kd, vd, causal=causal, sm_scale=0.125)
    ro, _, _, _ = orc.attention_int8_ref(q, k, v, causal=causal, sm_scale=0.125)
    assert maxdiff(out, ro) <= util.FWD_TOL
    dq, dk, dv = torch.autograd.grad((out.float() * do.to(DEV).float()).sum(), (qd, kd, vd))
    # backward = fp16 dense backward with the INT8 forward's LSE and output
    # (attention_kernel_int8.py:256-267), restated by attention_int8_grads_ref
    rdq, rdk, rdv = orc.attention_int8_grads_ref(q, k, v, do, causal=causal, sm_scale=0.125)
    # K carries x8 outliers, so dq reaches magnitudes of 20-30 where one fp16 rounding step
    # of the stored gradient is already 1.6e-2: allow that step on top of the 1e-2 bar
    for t, r in ((dq, rdq), (dk, rdk), (dv, rdv)):
        assert util.excess(t, r) <= util.GRAD_TOL


@pytest.mark.parametrize("causal", [0, 1])
def test_golden_int8_backward(golden, causal):
    """Shape of the reference's own INT8 test: gradients of the reference, and (without K
    outliers) its 5e-2 bar against the fp32 attention gradients."""
    import flash_attn_triton_b200 as fa
    g = golden(f"int8_bwd_causal{causal}")
    q, k, v = cases.int8_case(31, 2, 2, 128, 64)
    do = cases.randn16(np.random.default_rng(32), 2, 2, 128, 64)
    qd, kd, vd = (t.to(DEV).requires_grad_() for t in (q, k, v))
    out = fa.attention_int8(qd, kd, vd, causal=bool(causal), sm_scale=0.125)
    dq, dk, dv = torch.autograd.grad((out.float() * do.to(DEV).float()).sum(), (qd, kd, vd))
    assert maxdiff(out, g["out"]) <= util.FWD_TOL
    for n, t in (("dq", dq), ("dk", dk), ("dv", dv)):
        assert maxdiff(t, g[n]) <= util.GRAD_TOL, n
    rng = np.random.default_rng(9)
    q, k, v, do = (cases.randn16(rng, 2, 2, 128, 64) for _ in range(4))
    qd, kd, vd = (t.to(DEV).requires_grad_() for t in (q, k, v))
    out = fa.attention_int8(qd, kd, vd, causal=bool(causal), sm_scale=0.125)
    grads = torch.autograd.grad((out.float() * do.to(DEV).float()).sum(), (qd, kd, vd))
    tr = lambda t: t.transpose(1, 2)
    ro, _, rdq, rdk, rdv = orc.attention_grads_ref(tr(q), tr(k), tr(v), tr(do), softmax_scale=0.125,
                                                   causal=bool(causal))
    assert maxdiff(tr(out), ro) <= INT8_GRAD_TOL
    for t, r in zip(grads, (rdq, rdk, rdv)):
        assert util.excess(tr(t), r, rel=2e-2) <= INT8_GRAD_TOL  # atol and rtol of the reference's test


@pytest.mark.parametrize("causal", [0, 1])
def test_golden_int8_padded(golden, causal):
    """A padded call: 150 valid tokens in 192 rows, seq_len_k = seq_len_q = 150
    (attention_kernel_int8.py:108-118, :245), against the reference's outputs and gradients."""
    import flash_attn_triton_b200 as fa
    g = golden(f"int8_padded_causal{causal}")
    q, k, v = cases.int8_case(33, 1, 2, 192, 64)
    do = cases.randn16(np.random.default_rng(34), 1, 2, 192, 64)
    qd, kd, vd = (t.to(DEV).requires_grad_() for t in (q, k, v))
    out = fa.attention_int8(qd, kd, vd, causal=bool(causal), sm_scale=0.125, seq_len_k=150, seq_len_q=150)
    dq, dk, dv = torch.autograd.grad((out.float() * do.to(DEV).float()).sum(), (qd, kd, vd))
    assert maxdiff(out, g["out"]) <= util.FWD_TOL
    # the reference's dq of the padded query rows is not meaningful under a causal mask (it skips
    # the key-length mask there); everything a caller keeps is compared
    assert maxdiff(dq[:, :, :150], g["dq"][:, :, :150]) <= util.GRAD_TOL
    assert maxdiff(dk, g["dk"]) <= util.GRAD_TOL and maxdiff(dv, g["dv"]) <= util.GRAD_TOL
    assert not dk[:, :, 150:].any() and not dv[:, :, 150:].any()
    # D = 128 takes the tcgen05 kernel: same call against the oracle, with a causal offset too
    q, k, v = cases.int8_case(35, 1, 2, 320, 128)
    for lk, lq in ((300, 300), (257, 200)):
        o = fa.attention_int8(q.to(DEV), k.to(DEV), v.to(DEV), causal=bool(causal), seq_len_k=lk, seq_len_q=lq)
        ro, _, _, _ = orc.attention_int8_ref(q, k, v, causal=bool(causal), seq_len_k=lk, seq_len_q=lq)
        assert maxdiff(o, ro) <= util.FWD_TOL, (lk, lq)
    with pytest.raises(ValueError):
        fa.attention_int8(q.to(DEV), k.to(DEV), v.to(DEV), seq_len_k=321)


def test_int8_value_errors():
    import flash_attn_triton_b200 as fa
    q = torch.zeros(1, 1, 64, 64, device=DEV, dtype=torch.float16)
    with pytest.raises(ValueError):
        fa.attention_int8(q[..., :16], q[..., :16], q[..., :16])
    with pytest.raises(ValueError):
        fa.attention_int8(q[:, :, :50], q[:, :, :50], q[:, :, :50])
    with pytest.raises(ValueError):
        fa.attention_int8(q.transpose(1, 2), q.transpose(1, 2), q.transpose(1, 2).contiguous())
    with pytest.raises(ValueError):
        fa.attention_int8(q.cpu(), q.cpu(), q.cpu())


def test_config5_shape():
    """B8 H32 S8192 D128 with 1 % x8 K outliers: codes/scales bit-exact on four (batch, head)
    slices (numpy oracle), forward finite and checked on the same four against the int8-math oracle."""
    from flash_attn_triton_b200 import _ops
    import flash_attn_triton_b200 as fa
    B, H, S, D = 8, 32, 8192, 128
    g = torch.Generator(device=DEV).manual_seed(5)
    q = torch.randn(B, H, S, D, device=DEV, dtype=torch.float16, generator=g)
    v = torch.randn(B, H, S, D, device=DEV, dtype=torch.float16, generator=g)
    k = torch.randn(B, H, S, D, device=DEV, dtype=torch.float16, generator=g)
    k = torch.where(torch.rand(B, H, S, D, device=DEV, generator=g) < 0.01, k * 8, k)
    k8, s_k = _ops.quantize_k_int8(k)
    slices = [(0, 0), (1, 2), (4, 17), (7, 31)]            # first, last and two in between
    for b, h in slices:
        r8, rs = orc.quantize_k_rows_ref(k[b, h].cpu())
        assert np.array_equal(k8[b, h].cpu().numpy(), r8) and np.array_equal(s_k[b, h].cpu().numpy(), rs), (b, h)
    # dequantised codes reproduce k to half a step everywhere (size-independent property)
    err = (k8.float() * s_k[..., None] - k.float()).abs()
    assert (err <= 0.5001 * s_k[..., None]).all()
    for causal in (False, True):
        out = fa.attention_int8(q, k, v, causal=causal)
        assert torch.isfinite(out).all()
        for b, h in slices:
            sl = (slice(b, b + 1), slice(h, h + 1))
            ro, _, _, _ = orc.attention_int8_ref(q[sl].cpu(), k[sl].cpu(), v[sl].cpu(), causal=causal)
            assert maxdiff(out[sl], ro) <= util.FWD_TOL, (b, h, causal)


@pytest.mark.parametrize("B,H,S,lk,causal", [(2, 60, 512, 512, True), (1, 26, 1088, 1088, False), (1, 8, 2048, 2048, True),
                                             (1, 26, 1088, 900, True)])
def test_head_dim_64_on_tcgen05(B, H, S, lk, causal):
    """Problems large enough for the codes held as 16-bit floats, key columns of very different scales among them."""
    import flash_attn_triton_b200 as fa
    q, k, v = cases.int8_case(700 + S, B, H, S, 64)
    k[0, 0, :, 5] *= 8
    kw = {} if lk == S else dict(seq_len_k=lk, seq_len_q=lk)
    out = fa.attention_int8(q.to(DEV), k.to(DEV), v.to(DEV), causal=causal, **kw)
    ro, _, _, _ = orc.attention_int8_ref(q, k, v, causal=causal, **kw)
    assert maxdiff(out[:, :, :lk], ro[:, :, :lk]) <= util.FWD_TOL


@pytest.mark.parametrize("S", [960, 1024, 2048])
@pytest.mark.parametrize("D", [64, 128])
def test_an_entry_has_the_same_result_in_any_batch(S, D):
    import flash_attn_triton_b200 as fa
    g = torch.Generator(DEV).manual_seed(S)
    q, k, v = (torch.randn(6, 16, S, D, device=DEV, dtype=torch.half, generator=g) for _ in range(3))
    whole = fa.attention_int8(q, k, v, causal=True)
    assert torch.equal(fa.attention_int8(q[:1], k[:1], v[:1], causal=True), whole[:1])
    assert torch.equal(fa.attention_int8(*(t[:1, :2].contiguous() for t in (q, k, v)), causal=True), whole[:1, :2])


@pytest.mark.parametrize("S,D", [(256, 128), (1088, 128), (1088, 64)])
def test_query_rows_with_infinities_and_zeros(S, D):
    """A row with an infinity has an infinite scale and a path of its own; rows of zeros, of both signs, and of the largest and
    the smallest values beside it stay what they are without it."""
    import flash_attn_triton_b200 as fa
    g = torch.Generator(DEV).manual_seed(S + D)
    q, k, v = (torch.randn(2, 32, S, D, device=DEV, dtype=torch.half, generator=g) for _ in range(3))
    q[0, 0, 0] = 0.0
    q[0, 0, 1] = -0.0
    q[0, 0, 2, ::2], q[0, 0, 3] = 65504.0, 6e-8
    want = fa.attention_int8(q, k, v)
    q[0, 0, 5, 7] = float("inf")
    out = fa.attention_int8(q, k, v)
    out[0, 0, 5] = want[0, 0, 5]
    assert torch.equal(out, want)
    mean = v[0, 0].float().mean(0)                   # scores of zero: every key alike
    assert (out[0, 0, :2].float() - mean).abs().max() <= 2e-3


def query_rows(D):
    """Rows of finite fp16 values whose quotients by the row's scale lie next to a rounding boundary (below and above every half from 0.5 to
    126.5), one row or more for every largest value >= 1 that there is; and random rows."""
    amax = np.arange(0x3c00, 0x7c00, dtype=np.uint16).view(np.float16)
    s = amax.astype(np.float32) / np.float32(127.0)
    halves = (np.arange(127, dtype=np.float64) + 0.5)[None, :] * s[:, None].astype(np.float64)
    near = np.minimum(halves, amax[:, None].astype(np.float64)).astype(np.float16)
    near = np.minimum(near, amax[:, None])
    below = np.minimum(np.maximum(near.view(np.uint16).astype(np.int32) - 1, 0).astype(np.uint16).view(np.float16), amax[:, None])
    above = np.minimum((near.view(np.uint16) + 1).view(np.float16), amax[:, None])
    x = np.concatenate([near, below, above], 1)                       # 381 values a row
    sign = np.where(np.arange(x.shape[1]) % 3 == 0, -1, 1).astype(np.float16)
    x = x * sign
    per = D - 1
    x = np.pad(x, ((0, 0), (0, -x.shape[1] % per))).reshape(len(amax), -1, per)
    x = np.concatenate([np.repeat(amax[:, None, None], x.shape[1], 1), x], 2).reshape(-1, D)
    g = np.random.default_rng(D)
    more = (g.standard_normal((4096, D)) * np.exp(g.uniform(-8, 9, (4096, 1)))).astype(np.float16)
    more[::7, ::5] = -0.0
    x = np.concatenate([x, more])
    assert np.isfinite(x).all()
    return x[:len(x) // 1024 * 1024]


@pytest.mark.parametrize("D", [128, 64])
def test_query_codes_are_those_of_a_division(D):
    """The quantiser's quotient (a reciprocal and a correction step) against an fp32 division, where a last-bit error changes the code, as
    int8 and as 16-bit floats with the sign of a zero."""
    import ctypes as C
    from flash_attn_triton_b200 import _native as N
    x = query_rows(D)
    r8, rs = orc.quantize_q_rows_ref(torch.from_numpy(x))
    amax = np.maximum(np.abs(x.astype(np.float32)).max(1, keepdims=True), np.float32(1.0))
    inverse = np.float32(1.0) / (amax / np.float32(127.0))
    wrong = np.trunc(np.abs(x.astype(np.float32) * inverse) + np.float32(0.5)) * np.sign(x)
    assert (wrong.astype(np.int8) != r8.reshape(x.shape)).any()       # a quotient without the correction would be seen
    heads, S = len(x) // 1024, 1024
    q = torch.from_numpy(x).to(DEV).view(1, heads, S, D)
    k, v, o = torch.randn_like(q), torch.randn_like(q), torch.empty_like(q)
    s_k, s_q = (torch.empty(heads * S, dtype=torch.float32, device=DEV) for _ in range(2))
    a = N.Int8Args()
    a.device, a.impl, a.batch, a.heads, a.seqlen, a.head_dim = 0, N.IMPL_AUTO, 1, heads, S, D
    a.q, a.s_k, a.v, a.o, a.softmax_scale, a.sq_scratch = q.data_ptr(), s_k.data_ptr(), v.data_ptr(), o.data_ptr(), 0.1, s_q.data_ptr()
    lib, stream = N.lib(), N.stream_ptr(q.device)
    if D == 64:
        codes = torch.zeros(lib.fa_int8_codes16_bytes(C.byref(a)), dtype=torch.uint8, device=DEV)
        assert codes.numel() >= 2 * q.numel()
        N.check(lib.fa_fwd_int8_codes16(C.byref(a), k.data_ptr(), s_k.data_ptr(), codes.data_ptr(), stream), "fa_fwd_int8_codes16")
        got = codes.view(torch.float16)[:q.numel()].cpu().numpy().reshape(x.shape)
        want = np.copysign(r8.reshape(x.shape).astype(np.float16), x)
        assert np.array_equal(got.view(np.uint16), want.view(np.uint16))
    else:
        k8, q8 = torch.zeros_like(q, dtype=torch.int8), torch.zeros_like(q, dtype=torch.int8)
        N.check(lib.fa_quantize_k_int8(k.data_ptr(), k8.data_ptr(), s_k.data_ptr(), heads * S, D, 0, stream), "fa_quantize_k_int8")
        a.k8, a.q8_scratch = k8.data_ptr(), q8.data_ptr()
        N.check(lib.fa_fwd_int8(C.byref(a), stream), "fa_fwd_int8")
        assert np.array_equal(q8.cpu().numpy().reshape(x.shape), r8.reshape(x.shape))
    assert np.array_equal(s_q.cpu().numpy().view(np.uint32), rs.reshape(-1).view(np.uint32))


@pytest.mark.parametrize("S", [1024, 1088, 2112])
@pytest.mark.parametrize("causal", [True, False])
def test_head_dim_64_entries_do_not_depend_on_the_batch(S, causal):
    """From 1024 tokens on a batch takes the kernel with two CTAs per SM, one entry of it the two-tile kernel: bit for bit equal."""
    import flash_attn_triton_b200 as fa
    B, H = 6, 16
    assert 2 * B * H * (S // 128) > 5 * torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator("cuda").manual_seed(S)
    q, k, v = (torch.randn(B, H, S, 64, device="cuda", dtype=torch.half, generator=g) for _ in range(3))
    k[:, :, ::37] *= 8                                # outlier keys
    got = fa.attention_int8(q, k, v, causal=causal)
    for b in (0, B - 1):
        assert torch.equal(got[b:b + 1], fa.attention_int8(q[b:b + 1].contiguous(), k[b:b + 1].contiguous(), v[b:b + 1].contiguous(), causal=causal))
