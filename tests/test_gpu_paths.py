"""GPU tests of the paths around the kernels: chained and grouped layer stacks, non-finite
activations on the device-pointer entry points, activations that are not 16-byte aligned, and a
bounded device wait that is made to run out (the kernel returns by itself, the call reports
TB_TIMEOUT, the next call works)."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as orc
from tritium_b200 import _lib, errors
from tritium_b200.format import SaltV2Codec, SaltV2Tensor
from tritium_b200.synth import bf16_bits_to_f32, f32_to_bf16_bits, make_activations

from gpu_common import exact_group_sums, rel_l2, uniform_pair

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backend():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device: there is no CPU path to fall back to")
    from tritium_b200 import B200Backend
    b = B200Backend(0)
    yield b
    b.close()


def to_dev_bf16(x):
    import torch
    return torch.from_numpy(f32_to_bf16_bits(x).view(np.int16).copy()).cuda().view(torch.bfloat16).reshape(x.shape)


def bf16_round(v):
    return bf16_bits_to_f32(f32_to_bf16_bits(np.ascontiguousarray(v, np.float32)))


# ------------------------------------------------------------------ layer stacks
@pytest.mark.parametrize("chain", [[0, 0, 1], [0, 1, 1]], ids=["group_then_chain", "chain_of_three"])
@pytest.mark.parametrize("m", [2, 6, 20])
def test_chained_stack_matches_layer_by_layer_oracle(backend, chain, m):
    """chain[i] = 1 feeds layer i with the bf16 output of layer i-1; the others read the stack input.
    Decode kernel (one and two passes) and tensor-core kernel."""
    import torch
    from tritium_b200 import LinearStack
    k = 512
    pairs = [uniform_pair(k, k, 2, seed=200 + i) for i in range(3)]
    weights = [backend.upload_salt_v2(prod, SaltV2Codec.B3) for prod, _ in pairs]
    stack = LinearStack(backend, weights, chain, max_m=m)
    x = make_activations(m, k, seed=23, bf16=True)
    y_last = torch.zeros(m, k, dtype=torch.float32, device="cuda")
    stream = torch.cuda.Stream()
    for flags in (0, _lib.TB_FWD_PDL):
        y_last.zero_()
        with torch.cuda.stream(stream):
            stack.forward_dev(to_dev_bf16(x), y_last=y_last, flags=flags, stream=stream)
        stream.synchronize()
        backend.check(stream)
        prev, want = None, None
        for i, (_, orac) in enumerate(pairs):
            want = orc.a8_linear(orac, bf16_round(prev) if chain[i] else x, dump=False)[0]
            prev = want
        assert rel_l2(y_last.cpu().numpy(), want) <= 2e-2, flags   # two bf16 hand-offs on the way
    stack.close()


@pytest.mark.parametrize("m,flags", [(6, 0), (6, _lib.TB_FWD_PDL), (20, 0)], ids=["m6", "m6_pdl", "m20_tensor_core"])
def test_grouped_stack_beyond_four_tokens(backend, m, flags):
    """A grouped run (layers that read the stack input) takes more than four tokens: the grouped
    launch is repeated per pass of four tokens; above sixteen the tensor-core kernel runs per layer.
    Every layer's output is read back from the group buffer."""
    import torch
    from tritium_b200 import LinearStack
    n, k, planes = 96, 1024, 2
    pairs = [uniform_pair(n, k, planes, seed=300 + i) for i in range(4)]
    weights = [backend.upload_salt_v2(prod, SaltV2Codec.B3) for prod, _ in pairs]
    stack = LinearStack(backend, weights, [0] * 4, max_m=max(m, 8))
    x = make_activations(m, k, seed=29, bf16=True)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        stack.forward_dev(to_dev_bf16(x), flags=flags, stream=stream)
    stream.synchronize()
    backend.check(stream)
    for i, (_, orac) in enumerate(pairs):
        want = orc.a8_linear(orac, x, dump=False)[0]
        assert rel_l2(bf16_bits_to_f32(stack.read_output(i, m)), want) <= 1e-2, i
    got = stack.forward_host(f32_to_bf16_bits(x), m, x_is_bf16=True)
    for i, (_, orac) in enumerate(pairs):
        assert rel_l2(bf16_bits_to_f32(got[i]), orc.a8_linear(orac, x, dump=False)[0]) <= 1e-2, i
    # the last layer belongs to a group: a y_last pointer is refused, not ignored
    with pytest.raises(errors.InvalidInput):
        stack.forward_dev(to_dev_bf16(x), y_last=torch.zeros(m, n, dtype=torch.float32, device="cuda"), stream=stream)
    stack.close()


# ------------------------------------------------------------------ input checks on device pointers
@pytest.mark.parametrize("bad", [float("nan"), float("inf")], ids=["nan", "inf"])
@pytest.mark.parametrize("m", [2, 24], ids=["decode", "tensor_core"])
def test_nonfinite_bf16_activation_is_reported(backend, bad, m):
    """quantize_act_int8 (crates/tritium-spec/src/lib.rs:351-378) would carry a NaN through to the
    output; the device paths report it instead of returning clamped codes."""
    import torch
    n, k = 64, 512
    prod, _ = uniform_pair(n, k, 1, seed=9)
    resident = backend.upload_salt_v2(prod, SaltV2Codec.B3)
    backend.reserve(resident, m)
    x = make_activations(m, k, seed=3, bf16=True)
    x[m - 1, 77] = bad
    x_dev = torch.from_numpy(x).cuda().to(torch.bfloat16)
    y_dev = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        backend.forward_dev(resident, x_dev, y_dev, a8=True, stream=stream)
    with pytest.raises(errors.InvalidInput, match="non-finite"):
        backend.check(stream)
    if m <= 4:
        L = _lib.load()
        errors.check(L.tb_linear_forward_a8_static(backend._h, resident._h, C.c_void_p(x_dev.data_ptr()), _lib.TB_BF16, None,
                                                   C.c_uint32(m), C.c_void_p(y_dev.data_ptr()), _lib.TB_F32, C.c_void_p(stream.cuda_stream)))
        with pytest.raises(errors.InvalidInput, match="non-finite"):
            backend.check(stream)
    # the status word is clear again and the next call is clean
    x[m - 1, 77] = 1.0
    with torch.cuda.stream(stream):
        backend.forward_dev(resident, torch.from_numpy(x).cuda().to(torch.bfloat16), y_dev, a8=True, stream=stream)
    backend.check(stream)


def test_unaligned_activation_pointer_takes_the_scratch_path(backend):
    """The one-launch path reads activations with 16-byte loads; a pointer that is only 2-byte
    aligned goes through the preparation kernel and gives the same bits."""
    import torch
    n, k, m = 80, 768, 3
    prod, orac = uniform_pair(n, k, 3, seed=13)
    resident = backend.upload_salt_v2(prod, SaltV2Codec.B3)
    x = make_activations(m, k, seed=4, bf16=True)
    flat = torch.zeros(m * k + 8, dtype=torch.bfloat16, device="cuda")
    aligned, shifted = flat[:m * k].view(m, k), flat[1:m * k + 1].view(m, k)
    want_dev = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    got_dev = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        aligned.copy_(torch.from_numpy(x))
        backend.forward_dev(resident, aligned, want_dev, a8=True, stream=stream)
        stream.synchronize()
        shifted.copy_(torch.from_numpy(x))
        assert shifted.data_ptr() % 16 != 0
        backend.forward_dev(resident, shifted, got_dev, a8=True, stream=stream)
    stream.synchronize()
    backend.check(stream)
    assert torch.equal(want_dev, got_dev)
    assert rel_l2(got_dev.cpu().numpy(), orc.a8_linear(orac, x, dump=False)[0]) <= 1e-5


# ------------------------------------------------------------------ a bounded wait that runs out
def test_bounded_wait_runs_out_and_the_context_stays_usable(backend):
    """The hook makes one kernel wait for bytes that nobody copies.  The wait has a limit: the kernel
    returns by itself (no trap, no fault), the status word says so, tb_backend_check turns it into
    TB_TIMEOUT, and the same backend computes correct results right after."""
    import torch
    L = _lib.load()
    n, k, m = 64, 512, 2
    prod, orac = uniform_pair(n, k, 2, seed=17)
    resident = backend.upload_salt_v2(prod, SaltV2Codec.B3)
    x = make_activations(m, k, seed=5, bf16=True)
    x_dev = to_dev_bf16(x)
    y_dev = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    stream = torch.cuda.Stream()

    def static_call():
        errors.check(L.tb_linear_forward_a8_static(backend._h, resident._h, C.c_void_p(x_dev.data_ptr()), _lib.TB_BF16, None,
                                                   C.c_uint32(m), C.c_void_p(y_dev.data_ptr()), _lib.TB_F32, C.c_void_p(stream.cuda_stream)))

    static_call()                       # resolves the scratch address; clean
    backend.check(stream)
    errors.check(L.tb_backend_inject_wait_timeout(backend._h, 1))
    static_call()
    with pytest.raises(errors.Timeout, match="bounded device wait"):
        backend.check(stream)
    y_dev.zero_()
    static_call()                       # the hook disarmed itself
    backend.check(stream)
    assert rel_l2(y_dev.cpu().numpy(), orc.a8_linear(orac, x, dump=False)[0]) <= 1e-5


# ------------------------------------------------------------------ package file -> device through seeks
def test_upload_from_seekable_package_file(backend, tmp_path):
    """upload_salt_v2_from_reader: a multi-tensor package on disk, one tensor uploaded through seeks,
    forward bit-identical to the upload from arenas."""
    from tritium_b200 import format as fmt
    a, oa = uniform_pair(48, 512, 2, seed=61)
    b2, ob = uniform_pair(32, 768, 3, seed=62)
    a.name, b2.name = "blk.0.attn_q", "blk.0.ffn_up"
    path = tmp_path / "two.tslt2"
    path.write_bytes(fmt.write_salt_v2_package_multi([a, b2], SaltV2Codec.B3))
    x = make_activations(2, 768, seed=6)
    with open(path, "rb") as f:
        streamed = backend.upload_salt_v2_from_reader(f, "blk.0.ffn_up")
    want = np.stack([orc.matvec(ob, x[i]) for i in range(2)])
    got = backend.salt_v2_forward_exact(streamed, x, 2).output
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    y, acc, _ = backend.linear_forward_a8(streamed, x, 2, dump=True)
    want_y, want_acc, _ = orc.a8_linear(ob, x)
    assert np.array_equal(acc, want_acc) and rel_l2(y, want_y) <= 1e-5
    with open(path, "rb") as f:
        with pytest.raises(errors.InvalidInput):
            backend.upload_salt_v2_from_reader(f, "blk.9.none")


# ------------------------------------------------------------------ SALT V1 multi-plane operator
@pytest.mark.parametrize("t_planes", [1, 2, 3])
@pytest.mark.parametrize("m", [1, 4, 24])
def test_salt_v1_planes_match_the_reference_row_dot(backend, t_planes, m):
    """Plane-major TQ2_0 planes with per-block f16 scales (tq2_0_add.cu:640-719): the int8 path against
    SaltLinear::forward (quantise, PackedSaltMatrix::row_dot, scale), the fp32 path against row_dot on
    the raw activations, both under the reference's own 1e-4 rule (crates/tritium-testkit/src/vector.rs:113-126)."""
    rng = np.random.default_rng(100 + t_planes)
    n, k = 72, 700                                       # k is not a multiple of 256: rows are padded with zero trits
    trits = rng.integers(-1, 2, (t_planes, n, k)).astype(np.int8)
    nb = (k + 255) // 256
    block_scales = (0.01 + 0.05 * rng.random((t_planes, n, nb))).astype(np.float16).view(np.uint16)
    planes = orc.salt_v1_pack(trits, block_scales)
    handle = backend.upload_salt_v1(planes, t_planes, n, k)
    assert handle.rows == n and handle.columns == nb * 256
    x = make_activations(m, k, seed=40 + m)
    xp = np.zeros((m, nb * 256), np.float32)
    xp[:, :k] = x
    want = orc.salt_v1_forward_a8(planes, t_planes, n, k, x)
    _, s = orc.quantize_act_int8(x, m, k)
    y, _, receipt = backend.linear_forward_a8(handle, xp, m)
    assert receipt.kernel == (1 if m <= 8 else 2)
    for r in range(m):
        assert np.all(np.abs(y[r] - want[r]) <= 1e-4 * np.maximum(max(float(s[r]), 1e-30), np.abs(want[r])))
    want_f32 = orc.salt_v1_matmul(planes, t_planes, n, k, x)
    got_f32 = backend.salt_v2_forward_fast(handle, xp, m).output
    assert np.all(np.abs(got_f32 - want_f32) <= 1e-4 * np.maximum(1.0, np.abs(want_f32)))
    with pytest.raises(errors.UnsupportedFormat):
        backend.upload_salt_v1(planes + planes[: len(planes) // t_planes], t_planes + 3, n, k)


# ------------------------------------------------------------------ RMSNorm prologue, residual epilogue
@pytest.mark.parametrize("codec", [SaltV2Codec.B3, SaltV2Codec.D2])
@pytest.mark.parametrize("n,k,planes,m,x_bf16,zero_centered,with_residual", [
    (192, 2560, 3, 1, False, False, True),     # one launch: the norm runs inside the decode kernel's table builder
    (192, 2560, 2, 2, True, True, False),
    (200, 768, 1, 3, False, True, True),
    (192, 1280, 3, 4, True, False, True),
    (96, 8192, 2, 4, False, False, True),      # large tables: norm kernel, preparation kernel, decode kernel
    (160, 2560, 3, 6, False, True, True),      # two passes
    (256, 1024, 2, 40, False, False, True),    # tensor-core kernel behind the norm kernel
])
def test_norm_linear_matches_the_reference_arithmetic(backend, codec, n, k, planes, m, x_bf16, zero_centered, with_residual):
    """RMSNorm in the canonical reduction order, the int8 quantiser, the packed linear and
    ``residual + y`` in one rounding.  Every float operation of the prologue is the reference's, so
    the result must equal, bit for bit, the plain int8 forward of rows the oracle normalised, with
    the residual added once in fp32; and it must agree with the oracle's whole chain."""
    import torch
    prod, orac = uniform_pair(n, k, planes, seed=91)
    resident = backend.upload_salt_v2(prod, codec)
    backend.reserve(resident, m)
    rng = np.random.default_rng(5 + m)
    x = make_activations(m, k, seed=17, bf16=x_bf16) * np.float32(3.7)
    if x_bf16:
        x = bf16_bits_to_f32(f32_to_bf16_bits(x))
    w_norm = (rng.standard_normal(k) * 0.3 + (0.0 if zero_centered else 1.0)).astype(np.float32)
    residual = rng.standard_normal((m, n)).astype(np.float32) if with_residual else None
    eps = 1e-6
    normed = orc.rmsnorm(x, w_norm, eps, zero_centered)
    stream = torch.cuda.Stream()
    x_dev = torch.from_numpy(x).cuda()
    if x_bf16:
        x_dev = x_dev.to(torch.bfloat16)
    plain = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    got = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    got_bf16 = torch.zeros(m, n, dtype=torch.bfloat16, device="cuda")
    w_dev = torch.from_numpy(w_norm).cuda()
    r_dev = torch.from_numpy(residual).cuda() if with_residual else None
    with torch.cuda.stream(stream):
        backend.forward_dev(resident, torch.from_numpy(normed).cuda(), plain, a8=True, stream=stream)
        backend.norm_linear_forward_dev(resident, x_dev, got, norm_weight=w_dev, eps=eps, zero_centered=zero_centered,
                                        residual=r_dev, stream=stream)
        backend.norm_linear_forward_dev(resident, x_dev, got_bf16, norm_weight=w_dev, eps=eps, zero_centered=zero_centered,
                                        residual=r_dev, stream=stream)
    stream.synchronize()
    backend.check(stream)
    want = plain.cpu().numpy()
    if with_residual:
        want = (residual + want).astype(np.float32)
    assert np.array_equal(got.cpu().numpy(), want)
    assert np.array_equal(got_bf16.view(torch.int16).cpu().numpy().view(np.uint16), f32_to_bf16_bits(want))
    chain = orc.norm_a8_linear(orac, x, w_norm, eps, zero_centered, residual)
    plain_chain = orc.norm_a8_linear(orac, x, w_norm, eps, zero_centered, None)
    # the tolerance belongs to the linear's output; the residual is added exactly once on both sides
    assert rel_l2(got.cpu().numpy() - (residual if with_residual else 0), plain_chain) <= 1e-5
    assert np.allclose(got.cpu().numpy(), chain, rtol=0, atol=1e-4 * float(np.abs(plain_chain).max()))


def test_residual_epilogue_alone_and_argument_checks(backend):
    import torch
    n, k, m = 128, 1024, 2
    prod, orac = uniform_pair(n, k, 3, seed=8)
    resident = backend.upload_salt_v2(prod, SaltV2Codec.B3)
    x = make_activations(m, k, seed=3, bf16=True)
    residual = np.random.default_rng(1).standard_normal((m, n)).astype(np.float32)
    x_dev = torch.from_numpy(x).cuda().to(torch.bfloat16)
    y = torch.from_numpy(residual).cuda()          # residual aliases the fp32 output: x = x + linear(h)
    plain = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    backend.forward_dev(resident, x_dev, plain, a8=True)
    backend.norm_linear_forward_dev(resident, x_dev, y, residual=y)
    torch.cuda.synchronize()
    backend.check()
    assert np.array_equal(y.cpu().numpy(), (residual + plain.cpu().numpy()).astype(np.float32))
    with pytest.raises(errors.InvalidInput, match="non-negative"):
        backend.norm_linear_forward_dev(resident, x_dev, y, norm_weight=torch.ones(k, device="cuda"), eps=float("nan"))
    with pytest.raises(KeyError):
        backend.norm_linear_forward_dev(resident, torch.zeros(m, k, dtype=torch.int8, device="cuda"), y)


def test_backend_freed_before_its_weights():
    """Handles may be dropped in any order: freeing the backend first leaves the weights' free call
    valid, refuses further work on the released context, and poisons nothing for the next context."""
    import torch
    from tritium_b200 import B200Backend
    first = B200Backend(0)
    prod, orac = uniform_pair(64, 512, 2, seed=3)
    resident = first.upload_salt_v2(prod, SaltV2Codec.B3)
    released = C.c_void_p(first._h.value)
    first.close()                                   # the context is only marked released
    x_dev = torch.zeros(1, 512, dtype=torch.bfloat16, device="cuda")
    y_dev = torch.zeros(1, 64, dtype=torch.float32, device="cuda")
    args = _lib.ForwardArgs()
    args.x, args.x_dtype, args.m, args.y, args.y_dtype, args.flags = x_dev.data_ptr(), _lib.TB_BF16, 1, y_dev.data_ptr(), _lib.TB_F32, _lib.TB_FWD_A8
    # the pointer stays valid while the weights live, and work on it is refused
    assert _lib.load().tb_linear_forward_dev(released, resident._h, C.byref(args), None) == _lib.TB_INVALID_INPUT
    assert "freed" in _lib.last_error()
    resident.free()                                 # the last dependant destroys the released context
    second = B200Backend(0)
    prod2, orac2 = uniform_pair(64, 512, 2, seed=4)
    again = second.upload_salt_v2(prod2, SaltV2Codec.B3)
    x = make_activations(40, 512, seed=1, bf16=True)   # the tensor-core route checks the runtime's last error first
    y, _, _ = second.linear_forward_a8(again, x, 40, x_is_bf16=False)
    assert rel_l2(y, orc.a8_linear(orac2, x, dump=False)[0]) <= 1e-5
    second.close()


# ------------------------------------------------------------------ few tokens on the tensor cores (9..64 tokens)
@pytest.mark.parametrize("codec", [SaltV2Codec.B3, SaltV2Codec.D2])
@pytest.mark.parametrize("m,n,k,planes", [
    (9, 200, 768, 3),       # smallest batch that takes the tensor-core route; K split three ways; ragged rows
    (20, 256, 1024, 2),
    (32, 6912, 2560, 3),    # the benchmark's layer: 54 row tiles, two K splits
    (33, 384, 2560, 3),     # 64-token tile
    (64, 1000, 1536, 1),
    (48, 19200, 512, 2),    # more row tiles than SMs: no split, several tiles per CTA
])
def test_few_token_tensor_core_kernel_is_exact(backend, codec, m, n, k, planes):
    """Batches of 9 to 64 tokens run one pass of the tensor-core kernel with a tile of 32 or 64 (accumulator ring,
    sums in registers, K split over CTAs with a fixed-order combine).  The int32 group sums must be
    the oracle's bit for bit, with and without the dump, and two runs must give the same bits."""
    import torch
    prod, orac = uniform_pair(n, k, planes, seed=m + planes)
    resident = backend.upload_salt_v2(prod, codec)
    backend.reserve(resident, m)
    x = make_activations(m, k, seed=3, bf16=True)
    x_dev = torch.from_numpy(x).cuda().to(torch.bfloat16)
    residual = np.random.default_rng(m).standard_normal((m, n)).astype(np.float32)
    r_dev = torch.from_numpy(residual).cuda()
    y = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    y2 = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    y3 = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    dump = torch.zeros(m, n, k // 128, planes, dtype=torch.int32, device="cuda")
    backend.forward_dev(resident, x_dev, y, a8=True, acc_dump=dump)
    backend.forward_dev(resident, x_dev, y2, a8=True)
    backend.norm_linear_forward_dev(resident, x_dev, y3, residual=r_dev)      # residual epilogue, also behind the split combine
    torch.cuda.synchronize()
    backend.check()
    # the oracle is a scalar program: the big layers are checked on their last 300 rows
    if n <= 2048:
        sample = slice(0, n)
        want, want_dump, _ = orc.a8_linear(orac, x, dump=True)
    else:
        from gpu_common import oracle_rows
        sample = slice(n - 300, n)
        want, want_dump, _ = orc.a8_linear(oracle_rows(prod, np.arange(n - 300, n)), x, dump=True)
    assert np.array_equal(dump.cpu().numpy()[:, sample], want_dump[..., :planes])
    assert torch.equal(y, y2)
    assert rel_l2(y.cpu().numpy()[:, sample], want) <= 1e-5
    assert np.array_equal(y3.cpu().numpy(), (residual + y.cpu().numpy()).astype(np.float32))


# ------------------------------------------------------------------ squared-ReLU gate in front of the down projection
@pytest.mark.parametrize("codec", [SaltV2Codec.B3, SaltV2Codec.D2])
@pytest.mark.parametrize("n,k,planes,m", [
    (192, 1024, 2, 1),      # tables built in the decode kernel
    (160, 6912, 1, 4),      # the 2B-class down projection's width: preparation kernel
    (256, 2560, 3, 6),      # two passes
    (256, 1536, 2, 40),     # tensor-core kernel, one tile of 64 tokens
    (128, 1024, 1, 200),    # two tiles of 128
])
def test_relu2_gate_prologue_is_bit_identical(backend, codec, n, k, planes, m):
    """(max(gate, 0)^2) * up is computed where the activations are quantised; elementwise and
    association-preserving, so the result equals the plain int8 forward of gated rows bit for bit."""
    import torch
    prod, orac = uniform_pair(n, k, planes, seed=21)
    resident = backend.upload_salt_v2(prod, codec)
    backend.reserve(resident, m)
    rng = np.random.default_rng(m)
    gate = rng.standard_normal((m, k)).astype(np.float32)
    up = rng.standard_normal((m, k)).astype(np.float32)
    gated = orc.relu2_gate(gate, up)
    plain = torch.zeros(m, n, dtype=torch.float32, device="cuda")
    got = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
    backend.forward_dev(resident, torch.from_numpy(gated).cuda(), plain, a8=True)
    backend.norm_linear_forward_dev(resident, torch.from_numpy(gate).cuda(), got, relu2_up=torch.from_numpy(up).cuda())
    torch.cuda.synchronize()
    backend.check()
    assert torch.equal(got, plain)
    assert rel_l2(got.cpu().numpy(), orc.a8_linear(orac, gated, dump=False)[0]) <= 1e-5
    with pytest.raises(errors.InvalidInput, match="not combined"):
        backend.norm_linear_forward_dev(resident, torch.from_numpy(gate).cuda(), got, relu2_up=torch.from_numpy(up).cuda(),
                                        norm_weight=torch.ones(k, device="cuda"))


@pytest.mark.gpu
@pytest.mark.parametrize("codec", [SaltV2Codec.B3, SaltV2Codec.D2])
@pytest.mark.parametrize("k,m", [(256, 1), (256, 4), (1024, 3), (1024, 4), (1280, 4), (2048, 2), (2304, 2), (4096, 1), (4096, 2), (4352, 1),
                                 (4352, 2), (8192, 1), (8448, 1)])
def test_activation_tables_where_their_passes_end(backend, codec, k, m):
    """Tables built in the decode kernel: one (tile column, token) pair, a full pass of 16 and one more, the
    largest number it takes and one more (then the preparation kernel).  fp32, bf16 and int8
    activations (whole int8 range): int32 group sums equal to the oracle's, outputs within 1e-5."""
    import torch
    n = 20
    prod, orac = uniform_pair(n, k, 1, seed=k + m)
    resident = backend.upload_salt_v2(prod, codec)
    x = make_activations(m, k, seed=m, bf16=True)
    want, want_acc, _ = orc.a8_linear(orac, x)
    acc = torch.full((m, n, k // 128, 1), 7, dtype=torch.int32, device="cuda")
    y = torch.zeros(m, n, device="cuda")
    for xt in (torch.from_numpy(x).cuda(), to_dev_bf16(x)):
        backend.forward_dev(resident, xt, y, acc_dump=acc)
        backend.check()
        assert np.array_equal(acc.cpu().numpy(), want_acc[..., :1])
        assert rel_l2(y.cpu().numpy(), want) <= 1e-5
    q = np.random.default_rng(k).integers(-128, 128, (m, k)).astype(np.int8)
    scale = torch.linspace(0.5, 1.5, m, device="cuda")
    backend.forward_dev(resident, torch.from_numpy(q).cuda(), y, act_scale=scale, acc_dump=acc)
    backend.check()
    sums = exact_group_sums(prod.raw[0], q)
    assert np.array_equal(acc.cpu().numpy(), sums)
    per_group = prod.raw[1][0].astype(np.float16).astype(np.float64)   # as the artifact stores them
    ref = (sums[..., 0] * per_group).sum(axis=2) * scale.double().cpu().numpy()[:, None]
    assert rel_l2(y.cpu().numpy(), ref) <= 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("codec", [SaltV2Codec.B3, SaltV2Codec.D2])
@pytest.mark.parametrize("k,planes", [(256, 1), (512, 1), (768, 1), (1280, 2), (768, 3), (2304, 3)])
def test_tensor_core_tiles_at_their_edges(backend, codec, k, planes):
    """Token tiles of 32, 64 and 128 (one and several) at their first and last token and one past it, with
    rows whose tile-planes start on every 4-byte residue of a 16-byte line, a ragged last row tile, and as
    few tile columns as there can be: int32 group sums and outputs against the oracle.  Group sums are
    exact; an output is at most 54 fp32 additions, each within 2^-24 of the partial sum, behind a
    product and in front of another one: 1e-5 relative leaves more than twice that.  The kernel without
    the dump is another instantiation: its outputs (fp32, bf16, with a residual) follow bit for bit."""
    import torch
    n = 133
    prod, orac = uniform_pair(n, k, planes, seed=k + planes)
    resident = backend.upload_salt_v2(prod, codec)
    backend.reserve(resident, 300)
    for m in (9, 32, 33, 64, 65, 128, 129, 256, 257):
        x = make_activations(m, k, seed=m, bf16=True)
        x_dev = torch.from_numpy(x).cuda().to(torch.bfloat16)
        y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
        dump = torch.zeros(m, n, k // 128, planes, dtype=torch.int32, device="cuda")
        backend.forward_dev(resident, x_dev, y, a8=True, acc_dump=dump)
        torch.cuda.synchronize()
        backend.check()
        want, want_dump, _ = orc.a8_linear(orac, x, dump=True)
        assert np.array_equal(dump.cpu().numpy(), want_dump[..., :planes]), m
        assert rel_l2(y.cpu().numpy(), want) <= 1e-5, m
        outputs_follow_without_the_dump(backend, resident, x_dev, y)


def outputs_follow_without_the_dump(backend, resident, x_dev, y):
    """The same call without the dump, in fp32, in bf16 and with a residual, against the dump form's fp32 outputs."""
    import torch
    y2, y16 = torch.full_like(y, float("nan")), torch.full_like(y, float("nan"), dtype=torch.bfloat16)
    y3, residual = torch.full_like(y, float("nan")), torch.randn(y.shape, device="cuda")
    backend.forward_dev(resident, x_dev, y2, a8=True)
    backend.forward_dev(resident, x_dev, y16, a8=True)
    backend.norm_linear_forward_dev(resident, x_dev, y3, residual=residual)
    torch.cuda.synchronize()
    backend.check()
    assert torch.equal(y, y2) and torch.equal(y.to(torch.bfloat16), y16) and torch.equal(residual + y, y3), y.shape


@pytest.mark.gpu
@pytest.mark.parametrize("codec", [SaltV2Codec.B3, SaltV2Codec.D2])
@pytest.mark.parametrize("k,planes", [(1280, 1), (1024, 2), (512, 3)])
def test_wide_token_tiles_at_their_edges(backend, codec, k, planes):
    """Token tiles of 256, which take more than four tile-planes per row and row tiles enough to fill the
    GPU: 76 of them (the last one ragged) at one token more than a tile of 128 holds, at a full tile, and at
    three tiles, where each CTA has several.  Sampled rows against the oracle, as in the test above."""
    import torch
    from gpu_common import oracle_rows, product_only, sample_rows
    n = 9605
    prod = product_only(n, k, planes, seed=k)
    rows = sample_rows(n)
    orac, resident = oracle_rows(prod, rows), backend.upload_salt_v2(prod, codec)
    backend.reserve(resident, 700)
    for m in (129, 256, 700):
        x = make_activations(m, k, seed=m, bf16=True)
        x_dev = torch.from_numpy(x).cuda().to(torch.bfloat16)
        y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
        dump = torch.zeros(m, n, k // 128, planes, dtype=torch.int32, device="cuda")
        backend.forward_dev(resident, x_dev, y, a8=True, acc_dump=dump)
        torch.cuda.synchronize()
        backend.check()
        want, want_dump, _ = orc.a8_linear(orac, x, dump=True)
        at = torch.from_numpy(rows).cuda()
        assert np.array_equal(dump[:, at].cpu().numpy(), want_dump[..., :planes]), m
        assert rel_l2(y[:, at].cpu().numpy(), want) <= 1e-5, m
        outputs_follow_without_the_dump(backend, resident, x_dev, y)


@pytest.mark.gpu
@pytest.mark.parametrize("codec", [SaltV2Codec.B3, SaltV2Codec.D2])
@pytest.mark.parametrize("k,planes", [(2560, 1), (3072, 1), (3328, 2), (2304, 3)])
def test_tiles_of_128_tokens_that_split_k(backend, codec, k, planes):
    """Three row tiles (the last one ragged) whose K is shared by up to eight CTAs, evenly or not, and one that is
    just not worth it (2560, 1 plane): a half tile and one more token, a full tile and one more, three tiles.
    Sampled rows against the oracle; the parts are added in a fixed order, so a second run gives the same bits."""
    import torch
    from gpu_common import oracle_rows, product_only, sample_rows
    n = 300
    prod = product_only(n, k, planes, seed=k)
    rows = sample_rows(n)
    orac, resident = oracle_rows(prod, rows), backend.upload_salt_v2(prod, codec)
    backend.reserve(resident, 300)
    for m in (65, 128, 129, 300):
        x = make_activations(m, k, seed=m, bf16=True)
        x_dev = torch.from_numpy(x).cuda().to(torch.bfloat16)
        y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
        dump = torch.zeros(m, n, k // 128, planes, dtype=torch.int32, device="cuda")
        backend.forward_dev(resident, x_dev, y, a8=True, acc_dump=dump)
        torch.cuda.synchronize()
        backend.check()
        want, want_dump, _ = orc.a8_linear(orac, x, dump=True)
        at = torch.from_numpy(rows).cuda()
        assert np.array_equal(dump[:, at].cpu().numpy(), want_dump[..., :planes]), m
        assert rel_l2(y[:, at].cpu().numpy(), want) <= 1e-5, m
        outputs_follow_without_the_dump(backend, resident, x_dev, y)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [24, 200])
@pytest.mark.parametrize("dtype", ["bf16", "f32", "int8"])
def test_unaligned_activations_in_front_of_the_tensor_cores(backend, m, dtype):
    """The quantisation pre-pass reads eight activations per load where the rows start on 16-byte
    boundaries, and one by one elsewhere: a pointer one element past a boundary gives the same bits."""
    import torch
    n, k = 80, 768
    prod, orac = uniform_pair(n, k, 3, seed=13)
    resident = backend.upload_salt_v2(prod, SaltV2Codec.B3)
    backend.reserve(resident, m)
    t = {"bf16": torch.bfloat16, "f32": torch.float32, "int8": torch.int8}[dtype]
    x = make_activations(m, k, seed=4, bf16=dtype == "bf16")
    q, s = orc.quantize_act_int8(x, m, k)
    values = torch.from_numpy(np.asarray(q, np.float32).reshape(m, k) if dtype == "int8" else x).cuda().to(t)
    scale = torch.from_numpy(np.asarray(s, np.float32)).cuda() if dtype == "int8" else None
    flat = torch.zeros(m * k + 16, dtype=t, device="cuda")
    outs = []
    for start in (0, 1):
        shifted = flat[start:start + m * k].view(m, k)
        shifted.copy_(values)
        assert (shifted.data_ptr() % 16 == 0) == (start == 0)
        y = torch.full((m, n), float("nan"), dtype=torch.float32, device="cuda")
        backend.forward_dev(resident, shifted, y, a8=True, act_scale=scale)
        torch.cuda.synchronize()
        backend.check()
        outs.append(y)
    assert torch.equal(outs[0], outs[1])
    assert rel_l2(outs[1].cpu().numpy(), orc.a8_linear(orac, x, dump=False)[0]) <= 1e-5


@pytest.mark.gpu
@pytest.mark.parametrize("group", [64, 128])
@pytest.mark.parametrize("n,k", [(9, 37), (11, 31 * 64 + 1), (17, 32 * 64 - 1), (5, 33 * 128 + 3), (8, 64 * 128 + 5)])
def test_exact_kernel_where_its_chunks_of_segments_end(backend, group, n, k):
    """Rows whose scale-group segments just fill, just exceed and several times exceed the 32 segments
    that are staged at a time, with every offset of a row inside its group: the oracle's bits."""
    from tritium_b200.format import SaltV2Tensor
    rng = np.random.default_rng(n * k + group)
    tiles, tail = -(-n * k // 256), n * k % 256
    trits = np.zeros((tiles, 3, 256), np.int8)
    trits[:, :2] = rng.integers(-1, 2, (tiles, 2, 256), dtype=np.int8)
    trits[-1, :, tail:] = 0
    gpt = 256 // group
    scales = np.zeros((tiles, 3, 4), np.uint16)
    scales[:, :2, :gpt] = (0.02 * np.abs(rng.standard_normal((tiles, 2, gpt))) + 1e-3).astype(np.float16).view(np.uint16)
    scales[-1, :, -(-tail // group):] = 0
    prod = SaltV2Tensor("w", n, k, np.full(tiles, 2, np.uint8), trits, scales, group)
    orac = orc.Tensor(n, k, group, prod.plane_count, prod.trits, prod.scales)
    resident = backend.upload_salt_v2(prod, SaltV2Codec.B3)
    for m in (1, 3, 4, 5):
        x = make_activations(m, k, seed=m)
        got = backend.salt_v2_forward_exact(resident, x, m).output
        assert np.array_equal(got.view(np.uint32), orc.matmul(orac, x).view(np.uint32)), m


F32_MAX = float(np.finfo(np.float32).max)


@pytest.mark.gpu
@pytest.mark.parametrize("group", [64, 128])
@pytest.mark.parametrize("what", ["element", "scale", "running_sum"])
@pytest.mark.parametrize("m,token", [(1, 0), (3, 1), (6, 5)])
def test_exact_overflow_names_the_row_and_column_of_the_reference(backend, group, what, m, token):
    """One row and one token leave the finite range, far behind the first 32 scale groups: at an element
    in the middle of a segment, where a segment's sum meets its scale, or where the running sum takes the
    second of two large contributions.  The message names what the oracle names."""
    from tritium_b200.format import SaltV2Tensor
    rng = np.random.default_rng(group)
    n, k, row = 5, 40 * group + 7, 3
    tiles, tail, gpt = -(-n * k // 256), n * k % 256, 256 // group
    trits = np.zeros((tiles, 3, 256), np.int8)
    trits[:, :2] = rng.integers(-1, 2, (tiles, 2, 256), dtype=np.int8)
    scales = np.zeros((tiles, 3, 4), np.uint16)
    scales[:, :2, :gpt] = (0.02 * np.abs(rng.standard_normal((tiles, 2, gpt))) + 1e-3).astype(np.float16).view(np.uint16)
    first = 36 * group + group // 2
    at = [first + i for i in range(6)] if what != "running_sum" else [first, first + group]
    for r in range(n):           # the columns in question count in one row only
        for c in at:
            tile, local = divmod(r * k + c, 256)
            trits[tile, :, local] = (1, 0, 0) if r == row else 0
            if r == row and what != "element":
                scales[tile, 0, local // group] = 0x7BFF if what == "scale" else 0x3C00
    trits[-1, :, tail:] = 0
    scales[-1, :, -(-tail // group):] = 0
    prod = SaltV2Tensor("w", n, k, np.full(tiles, 2, np.uint8), trits, scales, group)
    orac = orc.Tensor(n, k, group, prod.plane_count, prod.trits, prod.scales)
    resident = backend.upload_salt_v2(prod, SaltV2Codec.B3)
    x = make_activations(m, k, seed=m)
    x[token, at] = {"element": F32_MAX / 3, "scale": F32_MAX / 1000, "running_sum": F32_MAX / 4 * 3}[what]
    with pytest.raises(orc.OracleError) as e:
        orc.matvec(orac, x[token])
    assert e.value.row == row and e.value.column > 33 * group
    with pytest.raises(errors.InvalidInput, match=f"output row {e.value.row} became non-finite at column {e.value.column}$"):
        backend.salt_v2_forward_exact(resident, x, m)


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [float("inf"), float("nan")], ids=["inf", "nan"])
def test_exact_kernel_leaves_out_zero_trits_of_nonfinite_activations(backend, bad):
    """Device pointers, bit-exact route: an activation that is not finite is reported, and it reaches only the
    outputs of rows whose trits there are not all zero, and only those of its own token."""
    import torch
    n, k, m, token, column = 24, 33 * 64 + 5, 4, 2, 32 * 64 + 9
    from tritium_b200.format import SaltV2Tensor
    rng = np.random.default_rng(5)
    tiles = -(-n * k // 256)
    trits = np.zeros((tiles, 3, 256), np.int8)
    trits[:, :2] = rng.integers(-1, 2, (tiles, 2, 256), dtype=np.int8)
    scales = np.zeros((tiles, 3, 4), np.uint16)
    scales[:, :2] = (0.02 * np.abs(rng.standard_normal((tiles, 2, 4))) + 1e-3).astype(np.float16).view(np.uint16)
    tail = n * k % 256
    trits[-1, :, tail:] = 0
    scales[-1, :, -(-tail // 64):] = 0
    prod = SaltV2Tensor("w", n, k, np.full(tiles, 2, np.uint8), trits, scales, 64)
    resident = backend.upload_salt_v2(prod, SaltV2Codec.B3)
    where = np.arange(n) * k + column
    reached = trits[where // 256, :, where % 256].any(axis=1)
    assert reached.any() and not reached.all()
    x = make_activations(m, k, seed=1)
    clean = x.copy()
    clean[token, column] = 0
    x[token, column] = bad
    want = orc.matmul(orc.Tensor(n, k, 64, prod.plane_count, prod.trits, prod.scales), clean)
    y = torch.full((m, n), 7.0, dtype=torch.float32, device="cuda")
    backend.forward_dev(resident, torch.from_numpy(x).cuda(), y, a8=False, flags=_lib.TB_FWD_EXACT)
    torch.cuda.synchronize()
    with pytest.raises(errors.InvalidInput, match="non-finite"):
        backend.check()
    got, same = y.cpu().numpy(), np.ones((m, n), bool)
    same[token, reached] = False
    assert np.array_equal(got.view(np.uint32)[same], want.view(np.uint32)[same])
    assert not np.isfinite(got[~same]).any()


@pytest.mark.parametrize("m", [1, 40])
def test_host_outputs_keep_their_memory(m):
    """Outputs of host calls lie in pinned buffers that are used again once the array is gone: arrays that are kept
    hold their values through later calls and through the end of the backend, and a failing call gives none away."""
    from tritium_b200 import B200Backend
    b = B200Backend(0)
    n, k = 2304, 512
    prod, orac = uniform_pair(n, k, 2, seed=5)
    resident = b.upload_salt_v2(prod, SaltV2Codec.B3)
    xs = [make_activations(m, k, seed=i, bf16=True) for i in range(4)]
    kept = [b.salt_v2_forward_fast(resident, x, m).output for x in xs]
    for x in xs:
        b.salt_v2_forward_fast(resident, x, m)          # dropped at once
        b.linear_forward_a8(resident, x, m)
    with pytest.raises(errors.InvalidInput):
        b.salt_v2_forward_exact(resident, np.full((m, k), np.nan, np.float32), m)
    exact = b.salt_v2_forward_exact(resident, xs[0], m).output
    tail = kept[1][:, 7:]                               # a view alone keeps the buffer
    want = [orc.matmul(orac, x) for x in xs]
    del kept[1]
    b.salt_v2_forward_fast(resident, xs[3], m)
    resident.free()
    b.close()
    assert rel_l2(tail, want[1][:, 7:]) <= 1e-5
    for got, i in zip(kept, (0, 2, 3)):
        assert rel_l2(got, want[i]) <= 1e-5 and got.flags.writeable and got.shape == (m, n)
    assert np.array_equal(exact.view(np.uint32), want[0].view(np.uint32))


@pytest.mark.parametrize("k", [768, 2560])
@pytest.mark.parametrize("m", [5, 8])
def test_five_to_eight_tokens_with_and_without_reserved_scratch(k, m):
    """Device calls of five to eight tokens take the tensor cores where scratch for them is reserved and two decode
    passes where it is not (nothing is allocated then: the call can be captured).  Both against the oracle, with a
    norm and a residual too."""
    import torch
    from tritium_b200 import B200Backend
    n = 300
    prod, orac = uniform_pair(n, k, 2, seed=k)
    x = make_activations(m, k, seed=m, bf16=True)
    want, want_acc, _ = orc.a8_linear(orac, x, dump=True)
    weight = (1 + 0.1 * np.random.default_rng(3).standard_normal(k)).astype(np.float32)
    residual = torch.randn(m, n, device="cuda")
    xd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(weight).cuda()
    normed = orc.a8_linear(orac, orc.rmsnorm(x, weight, 1e-6), dump=False)[0]
    for reserved in (False, True):
        b = B200Backend(0)
        resident = b.upload_salt_v2(prod, SaltV2Codec.B3)
        if reserved:
            b.reserve(resident, m)
        y, dump = torch.zeros(m, n, device="cuda"), torch.zeros(m, n, k // 128, 2, dtype=torch.int32, device="cuda")
        y2, y3 = torch.zeros_like(y), torch.zeros_like(y)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            b.forward_dev(resident, xd, y, acc_dump=dump)
        graph.replay()
        b.norm_linear_forward_dev(resident, xd, y2, norm_weight=wd, eps=1e-6)
        b.norm_linear_forward_dev(resident, xd, y3, norm_weight=wd, eps=1e-6, residual=residual)
        b.check()
        assert np.array_equal(dump.cpu().numpy(), want_acc[..., :2])
        assert rel_l2(y.cpu().numpy(), want) <= 1e-5 and rel_l2(y2.cpu().numpy(), normed) <= 1e-5
        assert torch.equal(y3, residual + y2)
        del graph
        resident.free()
        b.close()


def test_graphs_outlive_later_reservations_and_calls():
    """Captured calls on the backend's scratch (five and eight tokens, norm in front of prepared tables, fp32 activations, a
    layout without a fast kernel) give the same bits after larger reservations and host calls, with whatever those
    freed filled with ones."""
    import torch
    from tritium_b200 import B200Backend
    b = B200Backend(0)
    small, _ = uniform_pair(300, 2560, 2, seed=1)
    large, _ = uniform_pair(1500, 8448, 1, seed=2)
    rng = np.random.default_rng(3)
    scales = np.full((60, 3, 4), np.float16(0.05).view(np.uint16))
    ragged = SaltV2Tensor("w", 40, 384, np.full(60, 3, np.uint8), rng.integers(-1, 2, (60, 3, 256)).astype(np.int8), scales, 64)
    w, wl, wr = (b.upload_salt_v2(t, SaltV2Codec.B3) for t in (small, large, ragged))
    b.reserve(w, 8)
    weight = {k: torch.rand(k, device="cuda") + 0.5 for k in (2560, 8448)}
    calls = []
    for wt, n, k, m in ((w, 300, 2560, 5), (w, 300, 2560, 8), (wl, 1500, 8448, 1), (w, 300, 2560, 2), (wr, 40, 384, 3)):
        calls.append((wt, torch.randn(m, k, device="cuda"), torch.zeros(m, n, device="cuda"), k))

    def run(i):
        wt, x, y, k = calls[i]
        if i in (1, 2):
            b.norm_linear_forward_dev(wt, x, y, norm_weight=weight[k], eps=1e-6)
        else:
            b.forward_dev(wt, x, y, a8=i != 3)

    graphs, first = [], []
    for i in range(len(calls)):
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            run(i)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run(i)
        graph.replay()
        torch.cuda.synchronize()
        graphs.append(graph)
        first.append(calls[i][2].clone())
        assert first[-1].abs().sum() > 0
    b.check()
    b.reserve(wl, 2048)
    b.linear_forward_a8(wl, np.ones((8, 8448), np.float32), 8)
    b.salt_v2_forward_fast(wl, np.ones((64, 8448), np.float32), 64)
    b.linear_forward_a8(wr, np.ones((200, 384), np.float32), 200)
    torch.cuda.synchronize()
    filler = [torch.ones(1 << 20, device="cuda") for _ in range(64)]
    for (_, _, y, _), graph, want in zip(calls, graphs, first):
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)
    b.check()
    assert all(bool((f == 1).all()) for f in filler)
    graphs.clear()
    for h in (w, wl, wr):
        h.free()
    b.close()


def device_receipt(backend, resident, x, y, flags=0):
    """Receipt of one device call: kernel 1 decode, 2 tensor cores."""
    import ctypes as C
    import torch
    args = _lib.ForwardArgs()
    args.x, args.x_dtype, args.m = x.data_ptr(), _lib.TB_F32, x.shape[0]
    args.y, args.y_dtype, args.flags = y.data_ptr(), _lib.TB_F32, _lib.TB_FWD_A8 | flags
    args.stream = _lib.stream_handle(torch.cuda.current_stream())
    r = _lib.Receipt()
    assert backend._L.tb_linear_forward_dev(backend._h, resident._h, C.byref(args), C.byref(r)) == 0
    return r


@pytest.mark.parametrize("codec", [SaltV2Codec.B3, SaltV2Codec.D2])
@pytest.mark.parametrize("n,k,planes,tensor_cores", [(4096, 768, 1, False), (2048, 1024, 2, False), (2049, 1024, 2, True), (300, 1280, 2, True),
                                                     (18944, 1792, 3, True), (18945, 1792, 3, None), (18945, 1536, 3, True), (23937, 1792, 3, True),
                                                     (18945, 6144, 2, None), (18945, 5888, 2, True)])
def test_kernel_of_five_to_eight_tokens_follows_the_tensors_own_reservation(codec, n, k, planes, tensor_cores):
    """The kernel of a call of five to eight tokens depends on the tensor and on what was reserved for it: not on other
    tensors' reservations, host calls or launch flags.  None: only B3 keeps the decode passes (a second wave of row
    tiles that is nearly empty).  An unrelated reservation changes no bit."""
    import torch
    from gpu_common import product_only
    from tritium_b200 import B200Backend
    b = B200Backend(0)
    w = b.upload_salt_v2(product_only(n, k, planes, seed=1), codec)
    other = b.upload_salt_v2(product_only(512, 8192, 2, seed=2), codec)
    if tensor_cores is None:
        tensor_cores = codec != SaltV2Codec.B3
    x, y = torch.randn(8, k, device="cuda"), torch.zeros(8, n, device="cuda")
    assert device_receipt(b, w, x, y).kernel == 1
    before = y.clone()
    assert device_receipt(b, w, x[:6], y[:6]).kernel == 1
    before_six = y[:6].clone()                              # passes of four and two tokens, where eight take four and four
    b.reserve(other, 2048)
    b.linear_forward_a8(w, np.ones((64, k), np.float32), 64)
    assert device_receipt(b, w, x, y).kernel == 1 and torch.equal(y, before)
    b.reserve(w, 6)
    assert device_receipt(b, w, x, y).kernel == 1 and torch.equal(y, before)          # eight tokens are not reserved
    for m in (5, 6):
        for flags in (0, _lib.TB_FWD_PDL):
            assert device_receipt(b, w, x[:m], y[:m], flags).kernel == (2 if tensor_cores else 1)
    assert device_receipt(b, w, x[:6], y[:6], _lib.TB_FWD_FORCE_DECODE).kernel == 1
    assert torch.equal(y[:6], before_six)
    assert device_receipt(b, w, x[:4], y[:4]).kernel == 1
    assert device_receipt(b, w, torch.zeros(9, k, device="cuda"), torch.zeros(9, n, device="cuda")).kernel == 2
    b.check()
    for h in (w, other):
        h.free()
    b.close()


@pytest.mark.parametrize("codec,k,m,launches", [(SaltV2Codec.D2, 3072, 1, 1), (SaltV2Codec.D2, 3328, 1, 2), (SaltV2Codec.D2, 1536, 2, 1),
                                                (SaltV2Codec.D2, 1792, 2, 2), (SaltV2Codec.D2, 768, 4, 1), (SaltV2Codec.D2, 1024, 3, 2),
                                                (SaltV2Codec.B3, 8192, 1, 1), (SaltV2Codec.B3, 8448, 1, 2), (SaltV2Codec.B3, 4096, 2, 1),
                                                (SaltV2Codec.B3, 4352, 2, 2), (SaltV2Codec.B3, 1024, 3, 1), (SaltV2Codec.B3, 1280, 4, 2)])
def test_tables_on_both_sides_of_the_builders_limit(backend, codec, k, m, launches):
    """The largest tables that the decode kernel builds itself (one launch; D2 12 pairs, B3 32, with the four-token
    layout 16) and the smallest that the preparation kernel builds (two), each against the oracle."""
    import torch
    prod, _ = uniform_pair(20, k, 1, seed=k + m)
    resident = backend.upload_salt_v2(prod, codec)
    y = torch.zeros(m, 20, device="cuda")
    assert device_receipt(backend, resident, torch.zeros(m, k, device="cuda"), y).launches == launches
    test_activation_tables_where_their_passes_end(backend, codec, k, m)
