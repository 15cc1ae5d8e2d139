"""Decode attention on the GPU against the oracle composition (through the C ABI).

Parity definition for the int8-KV form: out = Cast(DecodeAttentionValid_f32(Cast(q),
Dequantize(K), Dequantize(V), ...)). Tolerance: max|err| / max|ref| <= 1e-2 for bf16 output
(the reference's own bf16 attention bound is 3e-2, crates/hologram-compute/tests/conformance.rs:1390);
<= 2e-4 when q/out are f32 (isolates the kernel's own arithmetic from the final bf16 truncation).
"""
import numpy as np
import pytest

import hologram_b200 as hb
from hologram_b200 import kernel_call as kc
from oracle import oracle as orc
from helpers import norm_max_err, synth_bf16

pytestmark = pytest.mark.gpu
BF, F32 = kc.DTYPE_BF16, kc.DTYPE_F32


def make_q8_case(b, h, kv, past, d, seed, dtype=BF, m=1, sigma=1.0):
    rng = np.random.default_rng(seed)
    if dtype == BF:
        q = synth_bf16(b * h * m * d, 1.0, seed + 1)
    else:
        q = rng.standard_normal(b * h * m * d).astype(np.float32)
    src = {}
    for off, (name, rows) in enumerate((("kp", b * kv * past), ("vp", b * kv * past), ("kn", b * kv * m), ("vn", b * kv * m))):
        x = synth_bf16(rows * d, sigma, seed + 101 * (off + 2))
        src[name] = x
    quant = {k: orc.quantize_rows_i8(v, BF, v.size // d, d) for k, v in src.items()}
    return q, src, quant


def run_q8(backend, q, quant, valid_len, b, h, kv, m, past, d, dtype, scale_bits=0):
    ws = hb.DeviceWorkspace(backend, 12)
    ws.put(0, q)
    slot = 1
    for name in ("kp", "vp", "kn", "vn"):
        codes, scales = quant[name]
        ws.put(slot, codes if codes.size else np.zeros(16, np.int8))
        ws.put(slot + 1, scales if scales.size else np.zeros(4, np.float32))
        slot += 2
    ws.put(9, np.array([valid_len], dtype=np.uint32))
    es = 2 if dtype != F32 else 4
    ws.alloc(10, b * h * m * d * es)
    call = kc.DecodeAttentionValidQ8Call(kc.rb(0), kc.rb(1), kc.rb(2), kc.rb(3), kc.rb(4), kc.rb(5), kc.rb(6), kc.rb(7),
                                         kc.rb(8), kc.rb(9), kc.rb(10), b, h, kv, m, past, m, d, scale_bits, dtype)
    backend.dispatch(kc.KernelCall.DecodeAttentionValidQ8(call), ws)
    out = ws.read(10, b * h * m * d * es, np.uint16 if dtype != F32 else np.float32)
    ws.close()
    return out


def oracle_q8(q, quant, valid_len, b, h, kv, m, past, d, dtype, scale_bits=0):
    rc, out = orc.decode_attention_valid_q8(q, dtype, quant["kp"][0], quant["kp"][1], quant["vp"][0], quant["vp"][1],
                                            quant["kn"][0], quant["kn"][1], quant["vn"][0], quant["vn"][1], valid_len,
                                            b, h, kv, m, past, m, d, scale_bits)
    assert rc == 0
    return out


def as_f32(x, dtype):
    return x if dtype == F32 else orc.bf16_to_f32(x)


@pytest.mark.parametrize("b,h,kv,past,valid,dtype,tol", [
    (2, 32, 8, 1024, 1024, BF, 1e-2),
    (2, 32, 8, 1024, 1024, F32, 2e-4),
    (3, 8, 2, 1156, 700, BF, 1e-2),       # ragged valid_len inside a tile, past not a tile multiple
    (3, 8, 2, 1156, 700, F32, 2e-4),
    (1, 4, 4, 512, 512, F32, 2e-4),       # multi-head (group 1)
    (2, 8, 4, 384, 100, F32, 2e-4),       # group 2
    (1, 4, 1, 12, 12, F32, 2e-4),         # bucket smaller than a tile
    (1, 4, 1, 4096, 5, F32, 2e-4),        # realized prefix far below the bucket
    (2, 16, 2, 256, 256, F32, 2e-4),      # group 8: served by the general-shape kernel
    (1, 4, 2, 130, 130, F32, 2e-4),       # bucket not a multiple of 4: general-shape kernel
])
def test_q8_attention_matches_oracle(backend, b, h, kv, past, valid, dtype, tol):
    d = 128
    q, _, quant = make_q8_case(b, h, kv, past, d, seed=past + h, dtype=dtype)
    got = run_q8(backend, q, quant, valid, b, h, kv, 1, past, d, dtype)
    want = oracle_q8(q, quant, valid, b, h, kv, 1, past, d, dtype)
    assert norm_max_err(as_f32(got, dtype), as_f32(want, dtype)) <= tol


def test_q8_unrealized_rows_are_never_read(backend):
    # padded == tight (tests/decode_attention_valid.rs:226-282): bytes beyond valid_len do not matter
    b, h, kv, past, d, valid = 2, 8, 2, 512, 128, 300
    q, _, quant = make_q8_case(b, h, kv, past, d, seed=77, dtype=F32)
    a = run_q8(backend, q, quant, valid, b, h, kv, 1, past, d, F32)
    rng = np.random.default_rng(1)
    dirty = dict(quant)
    for name in ("kp", "vp"):
        codes, scales = (v.copy() for v in quant[name])
        c3 = codes.reshape(b * kv, past, d)
        c3[:, valid:, :] = rng.integers(-128, 128, size=c3[:, valid:, :].shape)
        s2 = scales.reshape(b * kv, past)
        s2[:, valid:] = np.float32(np.nan)
        dirty[name] = (codes, scales)
    bdirty = run_q8(backend, q, dirty, valid, b, h, kv, 1, past, d, F32)
    assert np.array_equal(a.view(np.uint32), bdirty.view(np.uint32))
    # valid_len beyond the bucket means the whole bucket
    full = run_q8(backend, q, quant, past, b, h, kv, 1, past, d, F32)
    over = run_q8(backend, q, quant, 10 ** 9, b, h, kv, 1, past, d, F32)
    assert np.array_equal(full.view(np.uint32), over.view(np.uint32))


def test_q8_extreme_rows(backend):
    # a zero query head, zero-scale (all-zero) K/V rows, one huge V row, a dominant key
    b, h, kv, past, d = 1, 4, 1, 640, 128
    q, src, _ = make_q8_case(b, h, kv, past, d, seed=5, dtype=F32)
    q = q.reshape(h, d)
    q[1] = 0.0
    q[2] *= 40.0          # very peaked softmax
    q[3] *= 1e-3
    q = q.reshape(-1)
    kp = orc.bf16_to_f32(src["kp"]).reshape(past, d)
    vp = orc.bf16_to_f32(src["vp"]).reshape(past, d)
    kp[10] = 0.0
    vp[11] = 0.0
    vp[500] *= 3e4
    kp[600] *= 30.0
    src["kp"], src["vp"] = orc.f32_to_bf16_rne(kp.reshape(-1)), orc.f32_to_bf16_rne(vp.reshape(-1))
    quant = {k: orc.quantize_rows_i8(v, BF, v.size // d, d) for k, v in src.items()}
    got = run_q8(backend, q, quant, past, b, h, kv, 1, past, d, F32)
    want = oracle_q8(q, quant, past, b, h, kv, 1, past, d, F32)
    got, want = got.reshape(h, d), want.reshape(h, d)
    for head in range(h):
        assert norm_max_err(got[head], want[head]) <= 5e-4, head


def test_q8_explicit_scale_and_general_kernel_shapes(backend):
    import struct
    sb = struct.unpack("<I", struct.pack("<f", 0.05))[0]
    for (b, h, kv, m, past, d) in [(2, 8, 2, 1, 256, 128), (1, 6, 3, 4, 40, 64), (1, 2, 2, 3, 0, 32)]:
        q, _, quant = make_q8_case(b, h, kv, past, d, seed=d + m, dtype=F32, m=m)
        got = run_q8(backend, q, quant, past, b, h, kv, m, past, d, F32, scale_bits=sb)
        want = oracle_q8(q, quant, past, b, h, kv, m, past, d, F32, scale_bits=sb)
        assert norm_max_err(got, want) <= 2e-4


def test_unquantized_decode_attention_valid(backend):
    # the reference variant itself (KernelCall::DecodeAttentionValid, wire 121) in bf16 and f32
    b, h, kv, m, past, d = 1, 4, 2, 4, 12, 16
    for dtype, tol in ((F32, 1e-5), (BF, 3e-2)):
        rng = np.random.default_rng(3)
        arrs = [rng.standard_normal(n).astype(np.float32) for n in
                (b * h * m * d, b * kv * past * d, b * kv * past * d, b * kv * m * d, b * kv * m * d)]
        if dtype == BF:
            arrs = [orc.f32_to_bf16_rne(a) for a in arrs]
        for valid in (0, 5, 12, 99):
            ws = hb.DeviceWorkspace(backend, 7)
            for i, a in enumerate(arrs):
                ws.put(i, a)
            ws.put(5, np.array([valid], dtype=np.uint32))
            ws.alloc(6, arrs[0].nbytes)
            call = kc.DecodeAttentionValidCall(kc.rb(0), kc.rb(1), kc.rb(2), kc.rb(3), kc.rb(4), kc.rb(5), kc.rb(6),
                                               b, h, kv, m, past, m, d, 0, dtype)
            backend.dispatch(kc.KernelCall.DecodeAttentionValid(call), ws)
            got = ws.read(6, arrs[0].nbytes, np.float32 if dtype == F32 else np.uint16)
            rc, want = orc.decode_attention_valid(*arrs, valid, b, h, kv, m, past, m, d, 0, dtype)
            assert rc == 0
            assert norm_max_err(as_f32(got, dtype), as_f32(want, dtype)) <= tol
    # geometry refusals (float_kernels.rs:4205-4220)
    ws = hb.DeviceWorkspace(backend, 7)
    for i in range(7):
        ws.alloc(i, 4096)
    for bad in (kc.DecodeAttentionValidCall(kc.rb(0), kc.rb(1), kc.rb(2), kc.rb(3), kc.rb(4), kc.rb(5), kc.rb(6), 1, 4, 2, 2, 4, 1, 16, 0, F32),
                kc.DecodeAttentionValidCall(kc.rb(0), kc.rb(1), kc.rb(2), kc.rb(3), kc.rb(4), kc.rb(5), kc.rb(6), 1, 4, 3, 1, 4, 1, 16, 0, F32)):
        with pytest.raises(hb.BackendError) as e:
            backend.dispatch(kc.KernelCall.DecodeAttentionValid(bad), ws)
        assert e.value.variant == "UnsupportedOp"


def test_mask_form_decode_attention(backend):
    # KernelCall::DecodeAttention (wire 119): additive f32 mask [q_rows, past + new], every key takes
    # part, -inf erases exactly, an all-erased row is the zero vector, q_rows independent of new_len
    b, h, kv, m, past, new, d = 2, 4, 2, 3, 37, 2, 32
    l = past + new
    for dtype, tol in ((F32, 1e-5), (BF, 3e-2)):
        rng = np.random.default_rng(8)
        arrs = [rng.standard_normal(n).astype(np.float32) for n in
                (b * h * m * d, b * kv * past * d, b * kv * past * d, b * kv * new * d, b * kv * new * d)]
        if dtype == BF:
            arrs = [orc.f32_to_bf16_rne(a) for a in arrs]
        mask = np.where(rng.random((m, l)) < 0.3, -np.inf, 0.0).astype(np.float32)
        mask[0, 5] = 0.75            # a finite bias
        mask[1, :] = -np.inf         # every key erased: zero vector
        for scale_bits in (0, int(np.float32(0.2).view(np.uint32))):
            ws = hb.DeviceWorkspace(backend, 7)
            for i, a in enumerate(arrs):
                ws.put(i, a)
            ws.put(5, mask)
            ws.alloc(6, arrs[0].nbytes)
            call = kc.DecodeAttentionCall(kc.rb(0), kc.rb(1), kc.rb(2), kc.rb(3), kc.rb(4), kc.rb(5), kc.rb(6),
                                          b, h, kv, m, past, new, d, scale_bits, dtype)
            backend.dispatch(kc.KernelCall.DecodeAttention(call), ws)
            got = as_f32(ws.read(6, arrs[0].nbytes, np.float32 if dtype == F32 else np.uint16), dtype)
            want = as_f32(orc.decode_attention_mask(*arrs, mask, b, h, kv, m, past, new, d, scale_bits, dtype), dtype)
            assert norm_max_err(got, want) <= tol
            assert not np.any(got.reshape(b * h, m, d)[:, 1, :])
    # the realized-length mask reproduces the scalar form (decode step: m = new = 1)
    b, h, kv, past, d, valid = 1, 4, 2, 24, 16, 9
    rng = np.random.default_rng(4)
    arrs = [rng.standard_normal(n).astype(np.float32) for n in (b * h * d, b * kv * past * d, b * kv * past * d, b * kv * d, b * kv * d)]
    mask = np.zeros((1, past + 1), np.float32)
    mask[0, valid:past] = -np.inf
    ws = hb.DeviceWorkspace(backend, 9)
    for i, a in enumerate(arrs):
        ws.put(i, a)
    ws.put(5, mask)
    ws.put(6, np.array([valid], dtype=np.uint32))
    ws.alloc(7, arrs[0].nbytes)
    ws.alloc(8, arrs[0].nbytes)
    backend.dispatch(kc.KernelCall.DecodeAttention(kc.DecodeAttentionCall(
        kc.rb(0), kc.rb(1), kc.rb(2), kc.rb(3), kc.rb(4), kc.rb(5), kc.rb(7), b, h, kv, 1, past, 1, d, 0, F32)), ws)
    backend.dispatch(kc.KernelCall.DecodeAttentionValid(kc.DecodeAttentionValidCall(
        kc.rb(0), kc.rb(1), kc.rb(2), kc.rb(3), kc.rb(4), kc.rb(6), kc.rb(8), b, h, kv, 1, past, 1, d, 0, F32)), ws)
    assert norm_max_err(ws.read(7, arrs[0].nbytes, np.float32), ws.read(8, arrs[0].nbytes, np.float32)) <= 1e-6
    # refusals: no key at all; heads not a multiple of kv_heads
    for bad in (kc.DecodeAttentionCall(kc.rb(0), kc.rb(1), kc.rb(2), kc.rb(3), kc.rb(4), kc.rb(5), kc.rb(7), 1, 4, 2, 1, 0, 0, 16, 0, F32),
                kc.DecodeAttentionCall(kc.rb(0), kc.rb(1), kc.rb(2), kc.rb(3), kc.rb(4), kc.rb(5), kc.rb(7), 1, 4, 3, 1, 4, 1, 16, 0, F32)):
        with pytest.raises(hb.BackendError) as e:
            backend.dispatch(kc.KernelCall.DecodeAttention(bad), ws)
        assert e.value.variant == "UnsupportedOp"


def test_config4_full_size_codes_and_attention(backend):
    # batch 32, 32 query / 8 kv heads, head_dim 128, 8192 cached positions: quantizer codes
    # bit-exact on the full cache, attention within tolerance of the oracle on every row.
    b, h, kv, past, d = 32, 32, 8, 8192, 128
    rows = b * kv * past
    q = synth_bf16(b * h * d, 1.0, 0xC4)
    ws = hb.DeviceWorkspace(backend, 12)
    ws.put(0, q)
    quant = {}
    slot = 1
    for name, nrows, seed in (("kp", rows, 1), ("vp", rows, 2), ("kn", b * kv, 3), ("vn", b * kv, 4)):
        src = synth_bf16(nrows * d, 1.0, 0xC4 + seed)
        quant[name] = orc.quantize_rows_i8(src, BF, nrows, d)
        tmp = hb.DeviceWorkspace(backend, 1)
        tmp.put(0, src)
        ptr, nbytes = tmp.slot(0)
        ws.alloc(slot, nrows * d)
        ws.alloc(slot + 1, nrows * 4)
        stage = hb.DeviceWorkspace(backend, 3)
        stage.bind(0, ptr, nbytes)
        for j in (0, 1):
            p, nb = ws.slot(slot + j)
            stage.bind(1 + j, p, nb)
        backend.dispatch(kc.KernelCall.QuantizeRowsI8(kc.QuantizeRowsI8Call(kc.rb(0), kc.rb(1), kc.rb(2), nrows, d, BF)), stage)
        backend.synchronize()
        assert np.array_equal(ws.read(slot, nrows * d, np.int8), quant[name][0]), name
        assert np.array_equal(ws.read(slot + 1, nrows * 4, np.uint32), quant[name][1].view(np.uint32)), name
        tmp.close()
        slot += 2
    ws.put(9, np.array([past], dtype=np.uint32))
    ws.alloc(10, b * h * d * 2)
    call = kc.DecodeAttentionValidQ8Call(kc.rb(0), kc.rb(1), kc.rb(2), kc.rb(3), kc.rb(4), kc.rb(5), kc.rb(6), kc.rb(7),
                                         kc.rb(8), kc.rb(9), kc.rb(10), b, h, kv, 1, past, 1, d, 0, BF)
    backend.dispatch(kc.KernelCall.DecodeAttentionValidQ8(call), ws)
    got = orc.bf16_to_f32(ws.read(10, b * h * d * 2, np.uint16))
    want = orc.bf16_to_f32(oracle_q8(q, quant, past, b, h, kv, 1, past, d, BF))
    err = norm_max_err(got, want)
    print(f"config-4 attention: max|err|/max|ref| = {err:.3e}")
    assert err <= 1e-2


def test_legacy_attention_prefill_form(backend):
    # KernelCall::Attention (wire 69; attention_float, cpu/float_kernels.rs:2244-2395): the reference's own
    # conformance cases plus a longer bf16 prefill; online softmax on the GPU against the CPU's two-pass row
    from helpers import ATTENTION_CASES
    cases = [(c, kc.DTYPE_F32) for c in ATTENTION_CASES] + [((2, 8, 2, 160, 128, True, None), BF), ((1, 4, 4, 96, 64, False, None), BF)]
    for idx, ((b, h, hkv, s, d, causal, mult), dt) in enumerate(cases):
        rng = np.random.default_rng(0x8c0 + idx)
        q, k, v = (rng.standard_normal(n).astype(np.float32) for n in (b * h * s * d, b * hkv * s * d, b * hkv * s * d))
        if dt == BF:
            q, k, v = (orc.f32_to_bf16_rne(x) for x in (q, k, v))
        bits = int(np.float32(mult).view(np.uint32)) if mult else 0
        kvh = hkv if hkv != h else 0
        ws = hb.DeviceWorkspace(backend, 4)
        for i, x in enumerate((q, k, v)):
            ws.put(i, x)
        ws.alloc(3, q.nbytes)
        call = kc.AttentionCall(kc.rb(0), kc.rb(1), kc.rb(2), kc.rb(3), b, h, s, d, kvh, int(causal), bits, dt)
        backend.dispatch(kc.KernelCall.Attention(call), ws)
        want = orc.attention(q, k, v, b, h, kvh, s, d, causal, bits, dt)
        got = ws.read(3, q.nbytes, q.dtype)
        if dt == BF:
            got, want = orc.bf16_to_f32(got), orc.bf16_to_f32(want)
        assert norm_max_err(got, want) <= (1e-2 if dt == BF else 2e-4), (idx, norm_max_err(got, want))
        ws.close()


def run_attention(backend, q, k, v, b, h, kv, s, d, causal, dtype, scale_bits=0):
    ws = hb.DeviceWorkspace(backend, 4)
    for i, x in enumerate((q, k, v)):
        ws.put(i, x)
    ws.alloc(3, q.nbytes)
    backend.dispatch(kc.KernelCall.Attention(kc.AttentionCall(kc.rb(0), kc.rb(1), kc.rb(2), kc.rb(3), b, h, s, d, kv if kv != h else 0, int(causal), scale_bits, dtype)), ws)
    out = ws.read(3, q.nbytes, q.dtype)
    ws.close()
    return out


def attention_inputs(b, h, kv, s, d, dtype, seed, sigma=1.0):
    rng = np.random.default_rng(seed)
    x = [rng.standard_normal(n).astype(np.float32) for n in (b * h * s * d, b * kv * s * d, b * kv * s * d)]
    x[0] *= sigma
    return x if dtype == F32 else [orc.f32_to_bf16_rne(t) if dtype == BF else t.astype(np.float16).view(np.uint16) for t in x]


def wide(x, dtype):
    return x if dtype == F32 else orc.bf16_to_f32(x) if dtype == BF else x.view(np.float16).astype(np.float32)


# one unit in the last place of the output: bf16 is truncated, f16 rounded; f32 sums stay two orders below what they are held to
ATTENTION_TOL = {BF: 2.0 ** -7, kc.DTYPE_F16: 2.0 ** -10, F32: 2e-5}


@pytest.mark.parametrize("dtype", [BF, kc.DTYPE_F16])
@pytest.mark.parametrize("b,h,kv,s,d,causal,sigma", [
    (1, 2, 1, 16, 16, True, 1.0), (1, 3, 3, 127, 64, False, 1.0), (2, 4, 2, 128, 128, True, 1.0), (1, 2, 2, 129, 80, False, 1.0),
    (1, 2, 1, 257, 80, True, 6.0),         # peaked rows: the running maximum grows and O is rescaled
    (1, 160, 8, 300, 64, True, 1.0),       # two query tiles a CTA, the second past the end or short
    (2, 80, 16, 513, 128, False, 6.0), (1, 150, 150, 385, 48, True, 1.0)])
def test_attention_of_16_bit_sequences(backend, b, h, kv, s, d, causal, sigma, dtype):
    from helpers import attention_f64
    q, k, v = attention_inputs(b, h, kv, s, d, dtype, s + d, sigma)
    got = wide(run_attention(backend, q, k, v, b, h, kv, s, d, causal, dtype), dtype)
    assert norm_max_err(got, attention_f64(wide(q, dtype), wide(k, dtype), wide(v, dtype), b, h, kv, s, d, causal, None)) <= ATTENTION_TOL[dtype]


@pytest.mark.parametrize("dtype", [BF, kc.DTYPE_F16, F32])
def test_attention_of_sequences_with_values_that_are_not_finite(backend, dtype, monkeypatch):
    # an infinite value row, a NaN key and scores of plus infinity reach exactly the rows that see them
    b, h, kv, s, d = 1, 4, 2, 200, 64
    q, k, v = attention_inputs(b, h, kv, s, d, dtype, 9)
    inf, nan = (0x7f80, 0x7fc0) if dtype == BF else (0x7c00, 0x7e00) if dtype != F32 else (np.inf, np.nan)
    v.reshape(kv, s, d)[0, 150, 3] = inf
    k.reshape(kv, s, d)[1, 60, 5] = nan
    v.reshape(kv, s, d)[1, 190, 7] = nan
    got = wide(run_attention(backend, q, k, v, b, h, kv, s, d, True, dtype), dtype).reshape(h, s, d)
    monkeypatch.setenv("HOLO_ATTN_FORCE_GENERIC", "1")
    want = wide(run_attention(backend, q, k, v, b, h, kv, s, d, True, dtype), dtype).reshape(h, s, d)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isposinf(got), np.isposinf(want))
    assert np.isfinite(got[:2, :150]).all() and np.isinf(got[:2, 150:, 3]).all() and np.isfinite(got[2:, :60]).all() and np.isnan(got[2:, 60:]).all()
    fine = np.isfinite(want)
    assert np.max(np.abs(got[fine] - want[fine])) <= ATTENTION_TOL[dtype] * np.max(np.abs(want[fine]))


@pytest.mark.parametrize("dtype", [F32, BF, kc.DTYPE_F16])
@pytest.mark.parametrize("b,h,kv,past,valid,d,sigma", [
    (1, 1, 1, 0, 0, 64, 1.0), (1, 12, 2, 100, 0, 128, 1.0), (1, 12, 2, 1531, 1531, 128, 1.0), (1, 32, 8, 3000, 2999, 128, 4.0),
    (2, 4, 4, 77, 5, 80, 1.0), (1, 8, 1, 4097, 4000, 64, 4.0), (1, 3, 1, 700, 10 ** 9, 256, 1.0), (1, 10, 1, 2100, 2100, 200, 1.0),
    (3, 5, 5, 999, 640, 200, 1.0), (8, 64, 16, 301, 300, 64, 1.0), (1, 7, 7, 513, 513, 16, 4.0)])
def test_single_token_attention_over_a_float_cache(backend, b, h, kv, past, valid, d, sigma, dtype):
    # clusters of every size and several of them per kv head, caches shorter than what they were cut for, padded row blocks
    rng = np.random.default_rng(past + d)
    arrs = [rng.standard_normal(n).astype(np.float32) for n in (b * h * d, b * kv * past * d, b * kv * past * d, b * kv * d, b * kv * d)]
    arrs[0] *= sigma
    if dtype != F32:
        arrs = [orc.f32_to_bf16_rne(x) if dtype == BF else x.astype(np.float16).view(np.uint16) for x in arrs]
    rc, want = orc.decode_attention_valid(*arrs, valid, b, h, kv, 1, past, 1, d, 0, dtype)
    assert rc == 0
    hidden = min(valid, past)          # bytes past the valid rows, NaN among them, are never read
    for x in arrs[1:3]:
        x.reshape(b * kv, past, d)[:, hidden:] = np.nan if dtype == F32 else 0x7fc0 if dtype == BF else 0x7e00
    ws = hb.DeviceWorkspace(backend, 7)
    for i, x in enumerate(arrs):
        ws.put(i, x if x.size else np.zeros(16, x.dtype))
    ws.put(5, np.array([valid], dtype=np.uint32))
    ws.alloc(6, arrs[0].nbytes)
    call = kc.KernelCall.DecodeAttentionValid(kc.DecodeAttentionValidCall(*[kc.rb(i) for i in range(7)], b, h, kv, 1, past, 1, d, 0, dtype))
    for _ in range(2):                 # the second launch finds the counters as the first one did
        backend.dispatch(call, ws)
        got = ws.read(6, arrs[0].nbytes, arrs[0].dtype)
        assert norm_max_err(wide(got, dtype), wide(want, dtype)) <= ATTENTION_TOL[dtype]
    ws.close()


def run_decode(backend, arrs, valid, b, h, kv, m, past, d, dtype):
    ws = hb.DeviceWorkspace(backend, 7)
    for i, x in enumerate(arrs):
        ws.put(i, x)
    ws.put(5, np.array([valid], dtype=np.uint32))
    ws.alloc(6, arrs[0].nbytes)
    backend.dispatch(kc.KernelCall.DecodeAttentionValid(kc.DecodeAttentionValidCall(*[kc.rb(i) for i in range(7)], b, h, kv, m, past, m, d, 0, dtype)), ws)
    out = ws.read(6, arrs[0].nbytes, arrs[0].dtype)
    ws.close()
    return out


@pytest.mark.parametrize("dtype", [F32, BF])
def test_recorded_calls_of_one_context_share_nothing(dtype):
    # two graphs recorded from one context, replayed side by side on two streams: each gives its own call's result every time
    import torch
    b, h, kv, past, d = 1, 12, 2, 4000, 128
    be, kind = hb.B200Backend(0), torch.float32 if dtype == F32 else torch.bfloat16
    stream = torch.cuda.Stream()
    be.set_stream(stream.cuda_stream)
    g = torch.Generator(device="cuda").manual_seed(7)
    graphs, outs, wants, kept = [], [], [], []
    for _ in range(2):
        x = [torch.randn(n, generator=g, device="cuda").to(kind) for n in (b * h * d, b * kv * past * d, b * kv * past * d, b * kv * d, b * kv * d)]
        x += [torch.tensor([past], dtype=torch.int32, device="cuda"), torch.empty(b * h * d, device="cuda", dtype=kind)]
        torch.cuda.synchronize()
        ws = hb.DeviceWorkspace(be, 7)
        for i, t in enumerate(x):
            ws.bind(i, t.data_ptr(), t.numel() * t.element_size())
        call = kc.KernelCall.DecodeAttentionValid(kc.DecodeAttentionValidCall(*[kc.rb(i) for i in range(7)], b, h, kv, 1, past, 1, d, 0, dtype))
        be.dispatch(call, ws)
        be.synchronize()
        wants.append(x[6].double().clone())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            be.dispatch(call, ws)
        graphs.append(graph)
        outs.append(x[6])
        kept.append((x, ws))
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream() for _ in graphs], [[], []]
    for _ in range(50):
        for i, graph in enumerate(graphs):
            with torch.cuda.stream(streams[i]):
                outs[i].fill_(float("nan"))
                graph.replay()
                got[i].append(outs[i].clone())
    torch.cuda.synchronize()
    tol = 2.0 ** -7 if dtype == BF else 2e-5      # ATTENTION_TOL: the recorded call adds up in another order
    for want, results in zip(wants, got):
        for r in results:
            assert (r.double() - want).abs().max() <= tol * want.abs().max()
    for x, ws in kept:
        ws.close()
    del graphs
    be.close()


@pytest.mark.parametrize("b,h,kv,s,d,causal,sigma", [
    (1, 1, 1, 2, 4, True, 1.0), (1, 4, 2, 63, 64, True, 1.0), (2, 3, 3, 65, 64, False, 6.0), (1, 12, 12, 381, 64, False, 1.0), (1, 60, 20, 200, 64, True, 1.0),
    (1, 4, 1, 129, 80, True, 6.0), (1, 2, 2, 100, 96, False, 1.0), (1, 40, 8, 257, 128, True, 1.0), (1, 3, 3, 320, 112, False, 6.0), (1, 2, 1, 70, 20, True, 1.0)])
def test_attention_of_f32_sequences(backend, b, h, kv, s, d, causal, sigma):
    from helpers import attention_f64
    q, k, v = attention_inputs(b, h, kv, s, d, F32, s + d, sigma)
    got = run_attention(backend, q, k, v, b, h, kv, s, d, causal, F32)
    assert norm_max_err(got, attention_f64(q, k, v, b, h, kv, s, d, causal, None)) <= ATTENTION_TOL[F32]


@pytest.mark.parametrize("past,valid,m,d", [(100, 100, 5, 64), (70, 0, 33, 128), (64, 64, 64, 64), (300, 211, 130, 96)])
def test_chunk_of_f32_rows_after_a_cache(backend, past, valid, m, d):
    b, h, kv = 2, 6, 2
    rng = np.random.default_rng(past + m)
    arrs = [rng.standard_normal(n).astype(np.float32) for n in (b * h * m * d, b * kv * past * d, b * kv * past * d, b * kv * m * d, b * kv * m * d)]
    rc, want = orc.decode_attention_valid(*arrs, valid, b, h, kv, m, past, m, d, 0, F32)
    assert rc == 0
    for x in arrs[1:3]:
        x.reshape(b * kv, past, d)[:, valid:] = np.nan        # never read
    ws = hb.DeviceWorkspace(backend, 7)
    for i, x in enumerate(arrs):
        ws.put(i, x)
    ws.put(5, np.array([valid], dtype=np.uint32))
    ws.alloc(6, arrs[0].nbytes)
    backend.dispatch(kc.KernelCall.DecodeAttentionValid(kc.DecodeAttentionValidCall(*[kc.rb(i) for i in range(7)], b, h, kv, m, past, m, d, 0, F32)), ws)
    assert norm_max_err(ws.read(6, arrs[0].nbytes, np.float32), want) <= ATTENTION_TOL[F32]
    ws.close()


SPECIAL = {BF: (0x7f80, 0xff80, 0x7fc0), kc.DTYPE_F16: (0x7c00, 0xfc00, 0x7e00), F32: (np.inf, -np.inf, np.nan)}


def same_as_general(backend, monkeypatch, run, dtype):
    """A route's output and the general routine's: NaN and infinities in the same places, other values within the tolerance."""
    got = wide(run(), dtype)
    monkeypatch.setenv("HOLO_ATTN_FORCE_GENERIC", "1")
    want = wide(run(), dtype)
    monkeypatch.delenv("HOLO_ATTN_FORCE_GENERIC")
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    fine = np.isfinite(want)
    assert fine.any() and not fine.all() and np.isinf(want).any() and np.isnan(want).any()
    assert np.max(np.abs(got[fine] - want[fine])) <= ATTENTION_TOL[dtype] * np.max(np.abs(want[fine]))


@pytest.mark.parametrize("dtype", [F32, BF, kc.DTYPE_F16])
@pytest.mark.parametrize("b,h,kv,s,d,causal,sigma", [(1, 4, 2, 200, 64, True, 1.0), (1, 4, 2, 131, 64, False, 6.0), (2, 3, 3, 70, 128, True, 6.0), (1, 2, 2, 300, 128, False, 1.0),
                                                     (1, 80, 4, 300, 48, True, 1.0), (1, 4, 4, 260, 80, True, 1.0)])
def test_infinities_and_nan_reach_the_rows_that_see_them(backend, monkeypatch, dtype, b, h, kv, s, d, causal, sigma):
    # infinite values of both signs in one column, in a column each, a value row of NaN, a NaN key, a query and a key whose product is infinite
    q, k, v = attention_inputs(b, h, kv, s, d, dtype, 3 * s + d, sigma)
    inf, ninf, nan = SPECIAL[dtype]
    q4, k4, v4 = q.reshape(b, h, s, d), k.reshape(b, kv, s, d), v.reshape(b, kv, s, d)
    v4[0, 0, 5, 2], v4[0, 0, s // 2, 2], v4[0, 0, s // 3, 7], v4[0, 0, s - 2, 9] = inf, ninf, ninf, inf
    if causal:
        v4[0, kv - 1, s - 20] = nan
        k4[0, kv - 1, s - 9, 1] = nan
    big = {F32: 3e38, BF: 0x7f61, kc.DTYPE_F16: inf}[dtype]     # 3e38; its square, and an infinity times anything but zero, is infinite
    q4[b - 1, h - 1, s - 30, 0] = big
    k4[b - 1, kv - 1, 17, 0] = big
    same_as_general(backend, monkeypatch, lambda: run_attention(backend, q, k, v, b, h, kv, s, d, causal, dtype), dtype)


@pytest.mark.parametrize("dtype", [F32, BF, kc.DTYPE_F16])
def test_one_row_sees_infinities_and_nan_of_its_cache(backend, monkeypatch, dtype):
    # keys split over warps, a cluster and clusters: one column's infinities meet, one stays, an infinite score in the other kv head
    b, h, kv, past, d = 1, 4, 2, 700, 64
    rng = np.random.default_rng(13)
    arrs = [rng.standard_normal(n).astype(np.float32) for n in (b * h * d, b * kv * past * d, b * kv * past * d, b * kv * d, b * kv * d)]
    if dtype != F32:
        arrs = [orc.f32_to_bf16_rne(x) if dtype == BF else x.astype(np.float16).view(np.uint16) for x in arrs]
    inf, ninf, nan = SPECIAL[dtype]
    arrs[0].reshape(h, d)[2:, 0] = (0x3f80, 0xbf80) if dtype == BF else (0x3c00, 0xbc00) if dtype != F32 else (1.0, -1.0)   # one row's score is +inf, the other's -inf
    v, k = arrs[2].reshape(kv, past, d), arrs[1].reshape(kv, past, d)
    v[0, 5, 2], v[0, 600, 2], v[0, 300, 7], arrs[4].reshape(kv, d)[0, 9] = inf, ninf, ninf, inf
    k[1, 417, 0] = inf
    same_as_general(backend, monkeypatch, lambda: run_decode(backend, arrs, past, b, h, kv, 1, past, d, dtype), dtype)


# up to 64 query rows of a kv head that all see the same keys: blocks of one, four and eight rows, the last one padded
@pytest.mark.parametrize("b,h,kv,s,d,dtype", [(1, 3, 3, 2, 64, BF), (1, 8, 2, 7, 64, kc.DTYPE_F16), (2, 12, 4, 15, 64, BF), (1, 4, 1, 15, 128, kc.DTYPE_F16), (1, 4, 2, 9, 200, BF),
                                              (1, 5, 5, 3, 16, kc.DTYPE_F16), (1, 4, 2, 5, 160, F32), (1, 2, 1, 30, 256, F32), (3, 2, 2, 2, 132, F32)])
def test_short_sequences_without_the_causal_law(backend, b, h, kv, s, d, dtype):
    from helpers import attention_f64
    q, k, v = attention_inputs(b, h, kv, s, d, dtype, s + d, 2.0)
    got = wide(run_attention(backend, q, k, v, b, h, kv, s, d, False, dtype), dtype)
    assert norm_max_err(got, attention_f64(wide(q, dtype), wide(k, dtype), wide(v, dtype), b, h, kv, s, d, False, None)) <= ATTENTION_TOL[dtype]


@pytest.mark.parametrize("dtype", [BF, kc.DTYPE_F16])
def test_weights_are_held_in_more_than_16_bits(backend, dtype):
    # Values of +A and -A: a cell whose sum nearly cancels shows the weights' own error, which elsewhere is below the output's last bit.
    # Unit: A times the 2-norm of the row's weights, which is at least A / 8 for 64 keys. Two bf16 terms err by at most 2^-17 of a weight,
    # so by 2^-14 units; the output's rounding by 2^-7 of the at most 2^-6 units that are looked at: together under 2^-12. One term would
    # err by 2^-9 of each weight, 2^-9.8 units on average. f16: 2^-14 where one term errs by 2^-12.8 on average.
    b, h, s, d, a = 1, 8, 64, 64, 1024.0
    q, k, v = attention_inputs(b, h, h, s, d, dtype, 21)
    v = np.where(wide(v, dtype) > 0, a, -a).astype(np.float32)
    stored = orc.f32_to_bf16_rne(v) if dtype == BF else v.astype(np.float16).view(np.uint16)
    got = wide(run_attention(backend, q, k, stored, b, h, h, s, d, False, dtype), dtype).reshape(h, s, d).astype(np.float64)
    q4, k4, v4 = (x.astype(np.float64).reshape(h, s, d) for x in (wide(q, dtype), wide(k, dtype), v))
    e = np.einsum("hqd,hkd->hqk", q4, k4) / np.sqrt(d)
    w = np.exp(e - e.max(-1, keepdims=True))
    w /= w.sum(-1, keepdims=True)
    want, unit = np.einsum("hqk,hkd->hqd", w, v4), a * np.sqrt((w * w).sum(-1, keepdims=True))
    near = np.abs(want) <= 2.0 ** -6 * unit
    assert near.sum() > 200
    assert (np.abs(got - want) / unit)[near].max() <= (2.0 ** -12 if dtype == BF else 2.0 ** -14)


# ---- routes ----
def times(call, tensors, monkeypatch):
    """us of a call's launch on the device: the route that is taken, the general routine"""
    import torch
    be, stream, best = hb.B200Backend(0), torch.cuda.Stream(), []
    be.set_stream(stream.cuda_stream)
    ws = hb.DeviceWorkspace(be, len(tensors))
    for i, t in enumerate(tensors):
        ws.bind(i, t.data_ptr(), t.numel() * t.element_size())
    torch.cuda.synchronize()
    for general in (False, True):
        if general:
            monkeypatch.setenv("HOLO_ATTN_FORCE_GENERIC", "1")
        low = 1e9
        with torch.cuda.stream(stream):
            for _ in range(5):
                ends = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                be.dispatch(call, ws)
                torch.cuda._sleep(2000000)            # 1 ms: the launches are all queued before the first one starts
                ends[0].record()
                for _ in range(20):
                    be.dispatch(call, ws)
                ends[1].record()
                stream.synchronize()
                low = min(low, ends[0].elapsed_time(ends[1]) * 50)
        best.append(low)
    monkeypatch.delenv("HOLO_ATTN_FORCE_GENERIC")
    ws.close()
    be.close()
    return best


def device_tensors(shapes, dtype, seed=5):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(s, generator=g, device="cuda").to({F32: torch.float32, BF: torch.bfloat16, kc.DTYPE_F16: torch.float16}[dtype]) for s in shapes]


@pytest.mark.parametrize("dtype", [BF, kc.DTYPE_F16])
@pytest.mark.parametrize("d", [64, 80, 128])
@pytest.mark.parametrize("causal", [True, False])
def test_long_sequences_repeat_their_bits(d, dtype, causal):
    # a tile's next scores are issued behind the product that still reads the weights they overwrite: a product that was overtaken, once in
    # forty calls of 16 heads x 12 tiles x 12 tiles, would give other bits
    import torch
    b, h, kv, s = 1, 16, 4, 1500
    be, stream = hb.B200Backend(0), torch.cuda.Stream()
    be.set_stream(stream.cuda_stream)
    x = device_tensors([(b, h, s, d), (b, kv, s, d), (b, kv, s, d)], dtype)
    out = torch.zeros((40,) + tuple(x[0].shape), dtype=x[0].dtype, device="cuda")
    torch.cuda.synchronize()
    for o in out:
        ws = hb.DeviceWorkspace(be, 4)
        for i, t in enumerate(x + [o]):
            ws.bind(i, t.data_ptr(), t.numel() * t.element_size())
        be.dispatch(kc.KernelCall.Attention(kc.AttentionCall(*[kc.rb(i) for i in range(4)], b, h, s, d, kv, int(causal), 0, dtype)), ws)
        ws.close()
    stream.synchronize()
    be.close()
    bits = out.view(torch.int16)
    assert bits[0].any() and (bits == bits[0]).all()


@pytest.mark.parametrize("b,h,kv,past,d,dtype", [(64, 32, 32, 3, 64, F32), (64, 32, 32, 7, 64, BF), (256, 12, 12, 3, 128, BF), (32, 12, 12, 3, 64, kc.DTYPE_F16),
                                                 (64, 32, 32, 23, 64, F32), (16, 32, 8, 3, 64, F32), (1, 12, 2, 3, 128, F32)])
def test_one_row_of_many_short_caches_takes_the_quicker_route(monkeypatch, b, h, kv, past, d, dtype):
    # the split kernel took 40 us on the first call, the general routine 25: it must not lose more than the 15 % that boxes and estimates differ by
    import torch
    x = device_tensors([(b, h, 1, d), (b, kv, past, d), (b, kv, past, d), (b, kv, 1, d), (b, kv, 1, d)], dtype)
    x += [torch.tensor([past], dtype=torch.int32, device="cuda"), torch.empty_like(x[0])]
    now, general = times(kc.KernelCall.DecodeAttentionValid(kc.DecodeAttentionValidCall(*[kc.rb(i) for i in range(7)], b, h, kv, 1, past, 1, d, 0, dtype)), x, monkeypatch)
    assert now <= 1.15 * general, (now, general)


@pytest.mark.parametrize("b,h,kv,s,d,causal", [(64, 32, 32, 2, 128, True), (32, 32, 32, 2, 64, False), (1, 12, 12, 8, 128, True), (1, 12, 12, 4, 64, False),
                                               (1, 12, 12, 8, 96, True), (32, 32, 32, 4, 128, False), (1, 12, 12, 64, 64, True), (32, 32, 32, 16, 96, True)])
def test_a_few_f32_rows_take_the_quicker_route(monkeypatch, b, h, kv, s, d, causal):
    # tiles of 64 keys and of 32 or 64 rows took 167 us on the first call, the general routine 52
    import torch
    x = device_tensors([(b, h, s, d), (b, kv, s, d), (b, kv, s, d)], F32)
    x.append(torch.empty_like(x[0]))
    now, general = times(kc.KernelCall.Attention(kc.AttentionCall(*[kc.rb(i) for i in range(4)], b, h, s, d, 0, int(causal), 0, F32)), x, monkeypatch)
    assert now <= 1.15 * general, (now, general)


@pytest.mark.parametrize("dtype", [F32, BF, kc.DTYPE_F16])
@pytest.mark.parametrize("b,h,kv,s,d,causal", [(1, 12, 12, 128, 64, True), (1, 1, 1, 128, 128, False), (1, 8, 8, 381, 64, True), (1, 32, 8, 512, 128, False)])
def test_a_value_that_is_not_finite_costs_no_more_than_the_general_routine(monkeypatch, b, h, kv, s, d, causal, dtype):
    # every row sees it, in one column: f32, 12 heads of 128 rows took 718 us where the general routine takes 87
    import torch
    x = device_tensors([(b, h, s, d), (b, kv, s, d), (b, kv, s, d)], dtype)
    x[2][:, :, 0, 3] = float("inf")
    x.append(torch.empty_like(x[0]))
    now, general = times(kc.KernelCall.Attention(kc.AttentionCall(*[kc.rb(i) for i in range(4)], b, h, s, d, kv if kv != h else 0, int(causal), 0, dtype)), x, monkeypatch)
    assert now <= 1.15 * general, (now, general)


@pytest.mark.parametrize("d", [64, 128])
def test_large_finite_values_stay_finite(backend, d):
    # the tiles' weights refer to a maximum that lags by up to 2^8: a value near the type's largest overflows there and is computed again
    b, h, s = 1, 2, 300
    q, k, v = attention_inputs(b, h, h, s, d, BF, 11, 6.0)
    v.reshape(h, s, d)[:, ::7, 3] = orc.f32_to_bf16_rne(np.full(1, 2e37, np.float32))[0]
    got = wide(run_attention(backend, q, k, v, b, h, h, s, d, False, BF), BF).reshape(h, s, d).astype(np.float64)
    from helpers import attention_f64
    want = attention_f64(wide(q, BF), wide(k, BF), wide(v, BF), b, h, h, s, d, False, None).reshape(h, s, d)
    assert np.isfinite(got).all()
    assert np.abs(got - want)[..., 3].max() <= 2.0 ** -7 * np.abs(want[..., 3]).max()
