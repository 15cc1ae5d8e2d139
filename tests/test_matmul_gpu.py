"""bf16 matmul (+ fused epilogues) on the GPU against the oracle (through the C ABI).

Tolerance: max|err| / max|ref| <= 1e-2 against the oracle's ascending-k fused-multiply-add
chain truncated to bf16 (the reference's own bf16 bound vs f64 is 8e-3,
crates/hologram-compute/tests/conformance.rs:256). Shapes that take the per-cell kernel run
the reference's exact recurrence and must match bit for bit.
"""
import numpy as np
import pytest

import hologram_b200 as hb
from hologram_b200 import kernel_call as kc
from oracle import oracle as orc
from helpers import norm_max_err

pytestmark = pytest.mark.gpu
BF = kc.DTYPE_BF16


def synth(m, k, n, seed):
    rng = np.random.default_rng(seed)
    s = np.float32(1.0 / np.sqrt(k))
    a = orc.f32_to_bf16_rne(rng.standard_normal(m * k, dtype=np.float32) * s)
    b = orc.f32_to_bf16_rne(rng.standard_normal(k * n, dtype=np.float32) * s)
    return a, b


def run(backend, a, b, m, k, n, act=0, residual=None):
    ws = hb.DeviceWorkspace(backend, 4)
    ws.put(0, a)
    ws.put(1, b)
    ws.alloc(2, m * n * 2 + 64)
    mm = kc.MatMulCall(kc.rb(0), kc.rb(1), kc.rb(2), m, k, n, BF, 0)
    if residual is not None:
        ws.put(3, residual)
        call = kc.KernelCall.MatMulAdd(kc.MatMulAddCall(mm, kc.rb(3)))
    elif act:
        call = kc.KernelCall.MatMulActivation(kc.MatMulActivationCall(mm, act))
    else:
        call = kc.KernelCall.MatMul(mm)
    backend.dispatch(call, ws)
    out = ws.read(kc.rb(2, 0, m * n * 2), m * n * 2, np.uint16)
    assert not ws.read(kc.rb(2, m * n * 2), 64).any()
    ws.close()
    return out


@pytest.mark.parametrize("m,k,n", [(3, 37, 16), (5, 64, 20), (1, 8, 8), (7, 33, 9)])
def test_small_and_odd_shapes_are_bit_exact(backend, m, k, n):
    a, b = synth(m, k, n, m + k + n)
    assert np.array_equal(run(backend, a, b, m, k, n), orc.matmul(a, b, m, k, n, BF))


@pytest.mark.parametrize("m,k,n", [
    (128, 64, 128), (128, 256, 256), (200, 192, 512), (64, 512, 1024), (16, 4096, 1024), (64, 4096, 4096),
    (256, 1000 * 8, 136), (129, 72, 8 * 33), (1024, 1024, 1024), (40, 2048, 512), (100, 4096, 256), (64, 14336, 4096),
])
def test_tensor_core_path_within_tolerance(backend, m, k, n):
    a, b = synth(m, k, n, m * 7 + n)
    got = orc.bf16_to_f32(run(backend, a, b, m, k, n))
    want = orc.bf16_to_f32(orc.matmul(a, b, m, k, n, BF))
    assert norm_max_err(got, want) <= 1e-2


def test_fused_epilogues(backend):
    m, k, n = 64, 1024, 2048
    a, b = synth(m, k, n, 21)
    r = orc.f32_to_bf16_rne(np.random.default_rng(22).standard_normal(m * n, dtype=np.float32))
    plain = run(backend, a, b, m, k, n)
    silu = run(backend, a, b, m, k, n, act=kc.FUSED_SILU)
    add = run(backend, a, b, m, k, n, residual=r)
    # the epilogue acts on the truncated product exactly as the unfused pair would
    assert np.array_equal(silu, orc.unary_lut(kc.LUT_SILU, BF, plain))
    assert np.array_equal(add, orc.binary(0, plain, r, BF))
    want = orc.bf16_to_f32(orc.matmul(a, b, m, k, n, BF, act=kc.FUSED_SILU))
    assert norm_max_err(orc.bf16_to_f32(silu), want) <= 1e-2
    # split-K route (few tiles): same identities
    m, k, n = 16, 4096, 512
    a, b = synth(m, k, n, 23)
    r = orc.f32_to_bf16_rne(np.random.default_rng(24).standard_normal(m * n, dtype=np.float32))
    plain = run(backend, a, b, m, k, n)
    assert np.array_equal(run(backend, a, b, m, k, n, act=kc.FUSED_GELU), orc.unary_lut(kc.LUT_GELU, BF, plain))
    assert np.array_equal(run(backend, a, b, m, k, n, residual=r), orc.binary(0, plain, r, BF))


def test_refusals(backend):
    ws = hb.DeviceWorkspace(backend, 3)
    for i in range(3):
        ws.alloc(i, 1 << 16)
    with pytest.raises(hb.BackendError) as e:
        backend.dispatch(kc.KernelCall.MatMul(kc.MatMulCall(kc.rb(0), kc.rb(1), kc.rb(2), 64, 64, 64, kc.DTYPE_F64, 0)), ws)
    assert e.value.variant == "UnsupportedOp"
    with pytest.raises(hb.BackendError) as e:   # A shorter than m*k
        backend.dispatch(kc.KernelCall.MatMul(kc.MatMulCall(kc.rb(0), kc.rb(1), kc.rb(2), 1024, 64, 8, BF, 0)), ws)
    assert e.value.variant == "SlotOutOfRange" and e.value.slot == 0
    # m == 0 is a no-op (float_kernels.rs:302-304)
    backend.dispatch(kc.KernelCall.MatMul(kc.MatMulCall(kc.rb(0), kc.rb(1), kc.rb(2), 0, 64, 64, BF, 0)), ws)


def test_config3_prefill_4096_cubed(backend):
    m = k = n = 4096
    a, b = synth(m, k, n, 0xC3)
    got = orc.bf16_to_f32(run(backend, a, b, m, k, n))
    want = orc.bf16_to_f32(orc.matmul(a, b, m, k, n, BF))
    err = norm_max_err(got, want)
    print(f"4096^3 matmul: max|err|/max|ref| = {err:.3e}")
    assert err <= 1e-2


def test_config3_decode_16x4096x14336(backend):
    m, k, n = 16, 4096, 14336
    a, b = synth(m, k, n, 0xC3 + 1)
    got = orc.bf16_to_f32(run(backend, a, b, m, k, n))
    want = orc.bf16_to_f32(orc.matmul(a, b, m, k, n, BF))
    err = norm_max_err(got, want)
    print(f"16x4096x14336 matmul: max|err|/max|ref| = {err:.3e}")
    assert err <= 1e-2


def run_dt(backend, a, b, m, k, n, dt, act=0, residual=None):
    es = 4 if dt == kc.DTYPE_F32 else 2
    ws = hb.DeviceWorkspace(backend, 4)
    ws.put(0, a)
    ws.put(1, b)
    ws.alloc(2, m * n * es)
    mm = kc.MatMulCall(kc.rb(0), kc.rb(1), kc.rb(2), m, k, n, dt, 0)
    if residual is not None:
        ws.put(3, residual)
        call = kc.KernelCall.MatMulAdd(kc.MatMulAddCall(mm, kc.rb(3)))
    elif act:
        call = kc.KernelCall.MatMulActivation(kc.MatMulActivationCall(mm, act))
    else:
        call = kc.KernelCall.MatMul(mm)
    backend.dispatch(call, ws)
    out = ws.read(2, m * n * es, np.float32 if dt == kc.DTYPE_F32 else np.uint16)
    ws.close()
    return out


def f16_to_f32(h):
    return h.view(np.float16).astype(np.float32)


@pytest.mark.parametrize("m,k,n", [(64, 1024, 2048), (16, 4096, 512), (200, 192, 512), (5, 64, 20)])
def test_f16_matmul(backend, m, k, n):
    # f16 takes the same tensor-core kernel (operand format f16, the reference's add-half narrow);
    # the last shape takes the per-cell kernel and is bit-exact
    rng = np.random.default_rng(m + n)
    s = np.float32(1.0 / np.sqrt(k))
    a = (rng.standard_normal(m * k, dtype=np.float32) * s).astype(np.float16).view(np.uint16)
    b = (rng.standard_normal(k * n, dtype=np.float32) * s).astype(np.float16).view(np.uint16)
    r = rng.standard_normal(m * n, dtype=np.float32).astype(np.float16).view(np.uint16)
    F16 = kc.DTYPE_F16
    plain = run_dt(backend, a, b, m, k, n, F16)
    want = orc.matmul(a, b, m, k, n, F16)
    if (m, k, n) == (5, 64, 20):
        assert np.array_equal(plain, want)
    else:
        assert norm_max_err(f16_to_f32(plain), f16_to_f32(want)) <= 2e-3
    # fused epilogues act on the narrowed product exactly as the unfused pair
    assert np.array_equal(run_dt(backend, a, b, m, k, n, F16, act=kc.FUSED_SILU), orc.unary_lut(kc.LUT_SILU, F16, plain))
    assert np.array_equal(run_dt(backend, a, b, m, k, n, F16, residual=r), orc.binary(0, plain, r, F16))


@pytest.mark.parametrize("m,k,n", [(8, 256, 64), (33, 100, 20), (64, 512, 128)])
def test_f32_matmul_is_the_reference_recurrence(backend, m, k, n):
    # every f32 product runs the per-cell ascending-k fused-multiply-add chain: bit-exact;
    # the fused activation is the scalar function on the f32 product (no table for 32-bit patterns)
    rng = np.random.default_rng(m * n)
    a = rng.standard_normal(m * k, dtype=np.float32)
    b = rng.standard_normal(k * n, dtype=np.float32) * np.float32(1.0 / np.sqrt(k))
    r = rng.standard_normal(m * n, dtype=np.float32)
    F32 = kc.DTYPE_F32
    assert np.array_equal(run_dt(backend, a, b, m, k, n, F32).view(np.uint32), orc.matmul(a, b, m, k, n, F32).view(np.uint32))
    assert np.array_equal(run_dt(backend, a, b, m, k, n, F32, residual=r).view(np.uint32),
                          orc.matmul(a, b, m, k, n, F32, residual=r).view(np.uint32))
    got = run_dt(backend, a, b, m, k, n, F32, act=kc.FUSED_GELU)
    want = orc.matmul(a, b, m, k, n, F32, act=kc.FUSED_GELU)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("dtype", [kc.DTYPE_F32, BF, kc.DTYPE_F16])
@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (1, 33, 41), (3, 31, 1003), (5, 100, 64), (16, 37, 531), (33, 65, 130), (129, 7, 8 * 37), (200, 70, 2055),
                                   (500, 50, 771), (1025, 36, 1801), (4, 96, 7),
                                   # every ring goes round: four full steps of k and a part of one, 16-byte copies and single ones
                                   (5, 645, 1003), (8, 772, 516), (33, 389, 130), (40, 324, 268), (300, 323, 771), (300, 388, 772), (1025, 197, 1801), (1100, 196, 1804),
                                   # one thread per cell and its neighbours: short chains, few rows of a wide B
                                   (1, 9, 100001), (1, 150, 100001), (3, 60, 100001), (8, 81, 60000), (2, 100, 60000), (9, 12, 2001), (9, 20, 33), (64, 24, 517), (64, 25, 517),
                                   (300, 4, 7), (300, 12, 1001), (1200, 20, 65), (2001, 12, 33)])
def test_every_tile_of_the_per_cell_kernel_is_bit_exact(backend, dtype, m, k, n):
    # edges of the tiles and of the k steps, pitches that are multiples of four elements and that are not, columns of the
    # multiply-then-add tail alone and beside full tiles, chains whose sums are -0 and subnormal
    rng = np.random.default_rng(m + 3 * k + 5 * n)
    a, b, r = rng.standard_normal(m * k, dtype=np.float32), rng.standard_normal(k * n, dtype=np.float32), rng.standard_normal(m * n, dtype=np.float32)
    if dtype == kc.DTYPE_F32:
        a[:k] = np.float32(-1e-30)
        b[::n] = np.float32(1e-30)
    else:
        narrow = orc.f32_to_bf16_rne if dtype == BF else (lambda x: x.astype(np.float16).view(np.uint16))
        a, b, r = narrow(a), narrow(b), narrow(r)
    bits = np.uint32 if dtype == kc.DTYPE_F32 else np.uint16
    assert np.array_equal(run_dt(backend, a, b, m, k, n, dtype).view(bits), orc.matmul(a, b, m, k, n, dtype).view(bits))
    assert np.array_equal(run_dt(backend, a, b, m, k, n, dtype, residual=r).view(bits), orc.matmul(a, b, m, k, n, dtype, residual=r).view(bits))


@pytest.mark.parametrize("dtype,m,k,n,act", [(kc.DTYPE_F32, 5, 64, 24, kc.FUSED_GELU), (kc.DTYPE_F32, 3, 33, 17, kc.FUSED_SILU),
                                             (BF, 4, 128, 40, kc.FUSED_TANH), (kc.DTYPE_F16, 6, 72, 16, kc.FUSED_SIGMOID)])
def test_matmul_add_activation_is_the_three_calls(backend, dtype, m, k, n, act):
    # MatMulAddActivation (cpu/float_kernels.rs:899-938): act(A . B + residual) with nothing narrowed between the add and
    # the activation; served on the exact per-cell kernel, so every bit must match. For f32, where the reference forms
    # the triple at load, it is also bit-identical to MatMul -> Add -> activation run separately.
    rng = np.random.default_rng(m * 100 + n)
    if dtype == kc.DTYPE_F32:
        a = rng.standard_normal(m * k, dtype=np.float32) * np.float32(0.2)
        b = rng.standard_normal(k * n, dtype=np.float32) * np.float32(0.2)
        r = rng.standard_normal(m * n, dtype=np.float32)
        store = np.float32
    else:
        narrow = orc.f32_to_bf16_rne if dtype == BF else (lambda x: np.asarray(x, dtype=np.float32).astype(np.float16).view(np.uint16))
        a, b = narrow(rng.standard_normal(m * k, dtype=np.float32) * np.float32(0.2)), narrow(rng.standard_normal(k * n, dtype=np.float32) * np.float32(0.2))
        r = narrow(rng.standard_normal(m * n, dtype=np.float32))
        store = np.uint16
    es = np.dtype(store).itemsize
    ws = hb.DeviceWorkspace(backend, 4)
    ws.put(0, a)
    ws.put(1, b)
    ws.put(3, r)
    ws.alloc(2, m * n * es)
    mm = kc.MatMulCall(kc.rb(0), kc.rb(1), kc.rb(2), m, k, n, dtype, 0)
    backend.dispatch(kc.KernelCall.MatMulAddActivation(kc.MatMulAddActivationCall(mm, kc.rb(3), act)), ws)
    got = ws.read(2, m * n * es, store)
    want = orc.matmul_add_activation(a, b, r, m, k, n, dtype, act)
    assert np.array_equal(got.view(np.uint32 if es == 4 else np.uint16), want.view(np.uint32 if es == 4 else np.uint16))
    with pytest.raises(hb.BackendError) as e:       # an activation with no table-backed scalar form is refused, loudly
        backend.dispatch(kc.KernelCall.MatMulAddActivation(kc.MatMulAddActivationCall(mm, kc.rb(3), kc.FUSED_RELU)), ws)
    assert e.value.variant == "UnsupportedOp"
    ws.close()


def test_session_forms_the_f32_triple_at_load(backend):
    # fuse_matmul_epilogue (session.rs:2220-2226, 2279-2318): matmul -> add -> activation collapses to one call for f32
    # only; for bf16 the Add is absorbed (MatMulAdd) and the activation stays a call of its own
    from hologram_b200 import holo
    m, k, n = 4, 32, 16
    rng = np.random.default_rng(3)
    outs = {}
    for dtype, store in ((kc.DTYPE_F32, np.float32), (BF, np.uint16)):
        es = np.dtype(store).itemsize
        w = holo.HoloWriter()
        if dtype == BF:
            wt, bias = orc.f32_to_bf16_rne(rng.standard_normal(k * n, dtype=np.float32) * np.float32(0.2)), orc.f32_to_bf16_rne(rng.standard_normal(m * n, dtype=np.float32))
            x = orc.f32_to_bf16_rne(rng.standard_normal(m * k, dtype=np.float32))
        else:
            wt, bias = rng.standard_normal(k * n, dtype=np.float32) * np.float32(0.2), rng.standard_normal(m * n, dtype=np.float32)
            x = rng.standard_normal(m * k, dtype=np.float32)
        w.add_constant(1, dtype, wt.tobytes(), by_reference=False)
        w.add_constant(2, dtype, bias.tobytes(), by_reference=False)
        w.inputs = [holo.Port("x", 0, m * k, dtype, [m, k])]
        w.outputs = [holo.Port("y", 5, m * n, dtype, [m, n])]
        rb = lambda s, cnt: kc.rb(s, 0, cnt * es)
        w.calls = [kc.KernelCall.MatMul(kc.MatMulCall(rb(0, m * k), rb(1, k * n), rb(3, m * n), m, k, n, dtype, 0)),
                   kc.KernelCall.Add(kc.BinaryCall(rb(3, m * n), rb(2, m * n), rb(4, m * n), m * n, 16 if es == 2 else 32, dtype)),
                   kc.KernelCall.Gelu(kc.UnaryCall(rb(4, m * n), rb(5, m * n), m * n, 16 if es == 2 else 32, dtype))]
        w.exec_plan = [[0], [1], [2]]
        if dtype == kc.DTYPE_F32:
            sess = hb.InferenceSession(backend, w.finish())
            assert sess.n_calls == 1 and sess.call(0).kind == kc.K_MATMUL_ADD_ACTIVATION and sess.fused_count == 2
            sess.write("x", x)
            sess.execute()
            got = sess.read("y", np.float32)
            assert np.array_equal(got.view(np.uint32), orc.matmul_add_activation(x, wt, bias, m, k, n, dtype, kc.FUSED_GELU).view(np.uint32))
            sess.close()
        else:
            # a 16-bit Gelu over an Add is a LUT call the session keeps; only the Add is absorbed
            sess = hb.InferenceSession(backend, w.finish())
            assert [sess.call(i).kind for i in range(sess.n_calls)] == [kc.K_MATMUL_ADD, kc.K_GELU]
            sess.close()


@pytest.mark.parametrize("m,k,n,act,res", [(4096, 256, 2560, 0, False), (2500, 320, 2320, kc.FUSED_SILU, False), (2304, 192, 2304, 0, True),
                                           (1333, 128, 8200, 0, False)])
def test_persistent_tile_kernels_within_tolerance(backend, monkeypatch, m, k, n, act, res):
    # shapes of one 128 x 256 tile per SM and more: the CTA-pair kernel (tcgen05 cta_group::2) by its estimated time, the one-CTA
    # persistent kernel without it; ragged edges in both directions, fused epilogues.
    # Both must agree with the CPU chain within the tensor-core tolerance, and with each other and with the
    # one-tile-per-CTA kernel bit for bit (same k order per cell: the accumulation order inside one MMA chain is fixed).
    a, b = synth(m, k, n, m + n)
    r = orc.f32_to_bf16_rne(np.random.default_rng(1).standard_normal(m * n, dtype=np.float32)) if res else None
    want = orc.bf16_to_f32(orc.matmul(a, b, m, k, n, BF, act=act, residual=r))
    outs = {}
    for mode, env in (("pair", {}), ("persistent", {"HOLO_GEMM_PAIR": "0"}), ("classic", {"HOLO_GEMM_PERSISTENT": "0"})):
        for key in ("HOLO_GEMM_PAIR", "HOLO_GEMM_PERSISTENT"):
            monkeypatch.delenv(key, raising=False)
        for key, val in env.items():
            monkeypatch.setenv(key, val)
        outs[mode] = run(backend, a, b, m, k, n, act=act, residual=r)
        err = norm_max_err(orc.bf16_to_f32(outs[mode]), want)
        assert err <= 1e-2, (mode, err)
    backend.synchronize()
    assert np.array_equal(outs["pair"], outs["classic"]) and np.array_equal(outs["persistent"], outs["classic"])


@pytest.mark.parametrize("pairs", ["", "2"], ids=["all-pairs", "two-pairs"])
@pytest.mark.parametrize("kernel", ["halves", "pairs"])
@pytest.mark.parametrize("m,k,n,act,res", [(257, 4160, 392, 0, False), (1000, 2544, 1936, kc.FUSED_SILU, False), (1000, 2496, 1928, 0, False), (900, 2600, 1936, 0, True), (130, 8000, 264, 0, True), (300, 2000, 136, 0, False),
                                           (300, 2056, 136, 0, False), (300, 2120, 136, 0, False), (260, 1536, 2056, 0, False), (513, 1984, 640, 0, True), (129, 64, 8200, 0, False)])
def test_few_row_tiles_of_a_long_k_on_pairs(backend, monkeypatch, m, k, n, act, res, kernel, pairs):
    # 256 x 128 and 256 x 256 items, three or two k-blocks a stage (remainders of 0, 1 and 2 among these), ragged last tiles, some with no
    # column for the pair's second CTA. Two pairs walk up to 33 items each: ring phases and accumulator buffers carry over from item to item.
    # The kernel is named, so that no rule can take these shapes elsewhere.
    # The tolerance is the other tensor-core kernels'; the k order per cell is theirs, so the bits are too.
    a, b = synth(m, k, n, m + n)
    r = orc.f32_to_bf16_rne(np.random.default_rng(1).standard_normal(m * n, dtype=np.float32)) if res else None
    monkeypatch.setenv("HOLO_GEMM_KERNEL", kernel)
    if pairs:
        monkeypatch.setenv("HOLO_GEMM_PAIR_GRID", pairs)
    got = run(backend, a, b, m, k, n, act=act, residual=r)
    want = orc.bf16_to_f32(orc.matmul(a, b, m, k, n, BF, act=act, residual=r))
    assert norm_max_err(orc.bf16_to_f32(got), want) <= 1e-2
    monkeypatch.setenv("HOLO_GEMM_KERNEL", "tile")
    assert np.array_equal(got, run(backend, a, b, m, k, n, act=act, residual=r))


@pytest.mark.parametrize("m,k,n", [(2790, 2048, 1648), (898, 448, 4672)])
def test_several_rounds_of_half_width_items(backend, monkeypatch, m, k, n):
    # more 256 x 128 items than pairs of SMs, as the rule itself chooses them; one or two k-blocks are left over in the last stage
    a, b = synth(m, k, n, m + n)
    monkeypatch.setenv("HOLO_GEMM_KERNEL", "halves")
    got = run(backend, a, b, m, k, n)
    monkeypatch.setenv("HOLO_GEMM_KERNEL", "tile")
    assert np.array_equal(got, run(backend, a, b, m, k, n))


@pytest.mark.parametrize("pairs", ["", "2"], ids=["all-pairs", "two-pairs"])
@pytest.mark.parametrize("kernel", ["walk", "pairs", "halves"])
@pytest.mark.parametrize("m,k,n", [(300, 456, 200), (520, 1032, 648)])
def test_f16_products_on_every_kernel(backend, monkeypatch, m, k, n, kernel, pairs):
    monkeypatch.setenv("HOLO_GEMM_KERNEL", kernel)
    if pairs:
        monkeypatch.setenv("HOLO_GEMM_PAIR_GRID", pairs)
    test_f16_matmul(backend, m, k, n)


@pytest.mark.parametrize("bn", [64, 128])
@pytest.mark.parametrize("splits", [2, 3, 5, 7, 8])
@pytest.mark.parametrize("m,n,act,res", [(1, 200, 0, True), (7, 328, kc.FUSED_SILU, False), (16, 136, 0, True)])
def test_few_rows_add_up_any_split(backend, monkeypatch, m, n, act, res, splits, bn):
    # the parts of a K split are written to the CTA that adds them up: every splits-th row, ragged last tiles; the other kernels' tolerance
    k = 9 * 64 + 24
    a, b = synth(m, k, n, m + n)
    r = orc.f32_to_bf16_rne(np.random.default_rng(1).standard_normal(m * n, dtype=np.float32)) if res else None
    monkeypatch.setenv("HOLO_GEMM_SPLITS", str(splits))
    monkeypatch.setenv("HOLO_GEMM_BN", str(bn))
    got = run(backend, a, b, m, k, n, act=act, residual=r)
    want = orc.bf16_to_f32(orc.matmul(a, b, m, k, n, BF, act=act, residual=r))
    assert norm_max_err(orc.bf16_to_f32(got), want) <= 1e-2
