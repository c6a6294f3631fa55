"""Calls of the packed ternary linear layer that a user of this library has it do, with their inputs
and the exact results, for timing and for comparison.

Five kinds of call, each through the public Python entry points:

  linear   one linear on device tensors (``forward_dev``): decode, batched decode and prefill;
  layers   the four linears of decoder layers with their fused steps (``norm_linear_forward_dev``),
           recorded once in a CUDA graph and replayed, as a decode loop does;
  stack    layers of one shape that read the same host buffer (``LinearStack.forward_host``);
  fast     fp32 activations from host memory (``salt_v2_forward_fast``);
  exact    the bit-exact entry point from host memory (``salt_v2_forward_exact``), any layout.

Weights are made on the GPU from the seed (trits with the densities of the benchmark: dense first
plane, 10 % and 3 % in the residual planes) and uploaded as packed arenas.
"""
from __future__ import annotations

import numpy as np
import torch

from tritium_b200 import B200Backend, SaltV2Codec, SaltV2Tensor
from tritium_b200 import _lib
from tritium_b200.backend import LinearStack

DENSITY = (0.66, 0.10, 0.03)       # share of nonzero trits of plane 0, 1, 2
PLANE_SCALE = (1.0, 0.3, 0.1)      # scale of a plane relative to the first one's
PLANE_BYTES = {"b3": 52, "d2": 64}
NORM_EPS = 1e-6

_backend = None


def backend() -> B200Backend:
    """One backend per process, as a program that serves a model keeps."""
    global _backend
    if _backend is None:
        _backend = B200Backend(0)
    return _backend


# ---------------------------------------------------------------------------------------- cases
def listed():
    return [
        # the attention output projection of a 2B-class decoder at one token: the smallest call, all latency
        dict(name="o_2b_m1", kind="linear", n=2560, k=2560, planes=1, codec="b3", m=1, x="bf16", y="bf16"),
        # gate and up projection of a 27B-class decoder at one token: one long weight stream
        dict(name="gateup_27b_m1", kind="linear", n=34816, k=5120, planes=2, codec="b3", m=1, x="bf16", y="bf16"),
        # QKV of the 27B-class decoder for four sequences, weights in the 2-bit codec
        dict(name="qkv_27b_d2_m4", kind="linear", n=7168, k=5120, planes=2, codec="d2", m=4, x="bf16", y="f32"),
        # down projection of the 27B-class decoder for sixteen sequences: long rows
        dict(name="down_27b_m16", kind="linear", n=5120, k=17408, planes=2, codec="b3", m=16, x="bf16", y="bf16"),
        # gate and up projection of the 2B-class decoder for 64 sequences
        dict(name="gateup_2b_m64", kind="linear", n=13824, k=2560, planes=1, codec="b3", m=64, x="bf16", y="bf16"),
        # a short prompt through one FFN projection of the 2B-class decoder
        dict(name="ffn_2b_m512", kind="linear", n=6912, k=2560, planes=1, codec="b3", m=512, x="bf16", y="bf16"),
        # a prompt through the three-plane FFN projection: the benchmark's prefill
        dict(name="ffn_3p_m2048", kind="linear", n=6912, k=2560, planes=3, codec="b3", m=2048, x="bf16", y="bf16"),
        # a long prompt through the 27B-class gate and up projection: the largest call
        dict(name="gateup_27b_m4096", kind="linear", n=34816, k=5120, planes=2, codec="b3", m=4096, x="bf16", y="bf16"),
        # a decode step of the 2B-class decoder: norm + QKV, O + residual, norm + gate/up, gate + down + residual
        dict(name="layers_2b_m1", kind="layers", hidden=2560, qkv=3840, ffn=6912, planes=1, codec="b3", m=1, layers=8),
        # the benchmark's decode: layer copies that exceed L2, one host buffer in, every output out
        dict(name="stack_3p_m1", kind="stack", n=6912, k=2560, planes=3, codec="b3", m=1, layers=26),
        # fp32 activations for a 1.7B-class FFN projection, host buffers in and out
        dict(name="fast_1p_m32", kind="fast", n=8192, k=2048, planes=1, codec="b3", m=32),
        # the bit-exact entry point on a ragged matrix with groups of 64 (rows straddle tiles)
        dict(name="exact_ragged_m4", kind="exact", n=2500, k=1900, planes=2, codec="b3", group=64, m=4),
    ]


def _log(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    kind = rng.choice(["linear"] * 6 + ["layers", "stack", "fast", "exact"])
    codec = rng.choice(["b3", "b3", "d2"])
    planes = rng.choice([1, 2, 3])
    if kind == "linear":
        # tokens over the three regimes (a few, a batch, a prompt), widths over the decoders' range, odd row counts too
        m = int(_log(rng, *rng.choice([(1, 9), (9, 65), (65, 4097)])))
        n, k = int(_log(rng, 512, 34817)), 256 * int(_log(rng, 2, 69))
        while 2.0 * m * n * k * planes > 2.9e12 or n * k * planes > 34816 * 5120 * 2:
            n = max(512, n // 2)
        n += rng.choice([0, 0, 1, 5]) if rng.random() < 0.5 else -n % 64
        return dict(kind=kind, n=n, k=k, planes=planes, codec=codec, m=m, x=rng.choice(["bf16", "bf16", "f32"]), y=rng.choice(["bf16", "bf16", "f32"]))
    if kind == "layers":
        hidden = 256 * int(_log(rng, 4, 21))
        return dict(kind=kind, hidden=hidden, qkv=hidden + 128 * rng.randrange(2, 13), ffn=256 * int(_log(rng, 8, 69)), planes=rng.choice([1, 2]),
                    codec=codec, m=rng.choice([1, 1, 2, 3, 4, 8]), layers=rng.randrange(2, 9))
    if kind == "stack":
        return dict(kind=kind, n=16 * int(_log(rng, 64, 433)), k=256 * int(_log(rng, 4, 21)), planes=planes, codec=codec, m=rng.choice([1, 1, 2, 4]),
                    layers=rng.randrange(4, 27))
    if kind == "fast":
        return dict(kind=kind, n=int(_log(rng, 512, 13825)), k=256 * int(_log(rng, 4, 28)), planes=planes, codec=codec, m=int(_log(rng, 1, 129)))
    return dict(kind=kind, n=int(_log(rng, 512, 4097)), k=int(_log(rng, 512, 4097)), planes=rng.choice([1, 2]), codec=codec,
                group=rng.choice([64, 128]), m=int(_log(rng, 1, 17)))


# ---------------------------------------------------------------------------------------- weights and activations
def _generator(seed, what):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1_000_003 + what) & 0x7FFFFFFF)
    return g


def make_weight(n, k, planes, group, g):
    """Trits int8 [tiles, planes, 256] and f16 scales [tiles, planes, 256 / group] of the row-major coefficients cut into tiles."""
    tiles, gpt = -(-n * k // 256), 256 // group
    trits = torch.empty(tiles, planes, 256, dtype=torch.int8, device="cuda")
    for p in range(planes):
        for at in range(0, tiles, 1 << 18):   # in parts, so that the random numbers stay small beside the card
            u = torch.rand(min(1 << 18, tiles - at), 256, generator=g, device="cuda")
            trits[at:at + u.shape[0], p] = (u < DENSITY[p]).to(torch.int8) - 2 * (u < DENSITY[p] / 2).to(torch.int8)
    base = 0.02 * torch.randn(tiles, 1, gpt, generator=g, device="cuda").abs() + 1e-3
    scales = (base * torch.tensor(PLANE_SCALE[:planes], device="cuda").view(1, planes, 1)).to(torch.float16)
    return trits, scales


def pack(trits, codec):
    """Packed bytes [tiles, planes, 52 or 64]; digit = trit + 1, padding digits are zero trits."""
    tiles, planes, _ = trits.shape
    if codec == "d2":
        d = (trits + 1).view(tiles, planes, 64, 4)
        return (d[..., 0] | (d[..., 1] << 2) | (d[..., 2] << 4) | (d[..., 3] << 6)).view(torch.uint8)
    d = torch.ones(tiles, planes, 260, dtype=torch.uint8, device="cuda")
    d[..., :256] = (trits + 1).view(torch.uint8)
    d = d.view(tiles, planes, 52, 5)
    return d[..., 0] + 3 * (d[..., 1] + 3 * (d[..., 2] + 3 * (d[..., 3] + 3 * d[..., 4])))


def upload(n, k, planes, codec, group, trits, scales):
    b, c = backend(), SaltV2Codec.B3 if codec == "b3" else SaltV2Codec.D2
    if n * k % 256 == 0:
        tiles, code = n * k // 256, planes - 1
        pmap = np.full(tiles // 4, code * 0x55, np.uint8)
        terminal = sum(code << (2 * i) for i in range(tiles % 4))
        return b.upload_salt_v2_arenas(c, group, n, k, pack(trits, codec).reshape(-1).cpu().numpy(), scales.reshape(-1).cpu().numpy().view(np.uint16),
                                       pmap, terminal)
    tiles, tail = trits.shape[0], n * k % 256   # the last tile is short: the dense host form packs it
    t = np.zeros((tiles, 3, 256), np.int8)
    s = np.zeros((tiles, 3, 4), np.uint16)
    t[:, :planes] = trits.cpu().numpy()
    t[-1, :, tail:] = 0
    s[:, :planes, : 256 // group] = scales.cpu().numpy().view(np.uint16)
    s[-1, :, -(-tail // group):] = 0
    return b.upload_salt_v2(SaltV2Tensor("w", n, k, np.full(tiles, planes, np.uint8), t, s, group), c)


def dense64(n, k, trits, scales):
    """The matrix [n, k] that the packed planes stand for, in 64 bits."""
    tiles, planes, gpt = scales.shape
    w = torch.zeros(tiles, 256, dtype=torch.float64, device="cuda")
    for p in range(planes):
        w += trits[:, p].double() * scales[:, p].double().repeat_interleave(256 // gpt, dim=1)
    return w.view(-1)[: n * k].view(n, k)


def make_x(m, k, g):
    """N(0, 1) activations; 0.1 % of the channels are twenty times as large."""
    x = torch.randn(m, k, generator=g, device="cuda")
    x[:, torch.randperm(k, generator=g, device="cuda")[: round(0.001 * k)]] *= 20
    return x


DTYPE = {"bf16": torch.bfloat16, "f32": torch.float32}


def _layer_shapes(c):
    return [(c["qkv"], c["hidden"]), (c["hidden"], c["hidden"]), (2 * c["ffn"], c["hidden"]), (c["hidden"], c["ffn"])]


def _layer_inputs(c, li, seed):
    """Inputs of the four linears of layer `li`: (x, norm weight, residual, up) each."""
    g, m, h = _generator(seed, 5000 + li), c["m"], c["hidden"]
    norm = lambda: 1 + 0.1 * torch.randn(h, generator=g, device="cuda")  # noqa: E731
    res = lambda: torch.randn(m, h, generator=g, device="cuda")  # noqa: E731
    return [(make_x(m, h, g), norm(), None, None), (make_x(m, h, g).bfloat16(), None, res(), None), (make_x(m, h, g), norm(), None, None),
            (make_x(m, c["ffn"], g), None, res(), torch.randn(m, c["ffn"], generator=g, device="cuda"))]


# ---------------------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    c, b, kind = case, backend(), case["kind"]
    if kind == "linear":
        w = upload(c["n"], c["k"], c["planes"], c["codec"], 128, *make_weight(c["n"], c["k"], c["planes"], 128, _generator(seed, 1)))
        b.reserve(w, c["m"])
        return dict(kind=kind, w=w, x=make_x(c["m"], c["k"], _generator(seed, 2)).to(DTYPE[c["x"]]),
                    y=torch.empty(c["m"], c["n"], dtype=DTYPE[c["y"]], device="cuda"))
    if kind == "layers":
        calls = []
        for li in range(c["layers"]):
            for (n, k), (x, norm, res, up), i in zip(_layer_shapes(c), _layer_inputs(c, li, seed), range(4)):
                w = upload(n, k, c["planes"], c["codec"], 128, *make_weight(n, k, c["planes"], 128, _generator(seed, 10 + 4 * li + i)))
                b.reserve(w, c["m"])
                calls.append((w, x, torch.empty(c["m"], n, device="cuda"), norm, res, up))

        def step():
            for w, x, y, norm, res, up in calls:
                b.norm_linear_forward_dev(w, x, y, norm_weight=norm, eps=NORM_EPS if norm is not None else 0.0, residual=res, relu2_up=up,
                                          flags=_lib.TB_FWD_PDL)

        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            step()
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            step()
        return dict(kind=kind, graph=graph, calls=calls, y=[call[2] for call in calls])
    if kind == "stack":
        ws = [upload(c["n"], c["k"], c["planes"], c["codec"], 128, *make_weight(c["n"], c["k"], c["planes"], 128, _generator(seed, 10 + i)))
              for i in range(c["layers"])]
        x = make_x(c["m"], c["k"], _generator(seed, 2)).bfloat16()
        return dict(kind=kind, stack=LinearStack(b, ws, [False] * c["layers"], c["m"]), x=x.cpu().view(torch.int16).numpy().view(np.uint16), m=c["m"])
    group = c.get("group", 128)
    w = upload(c["n"], c["k"], c["planes"], c["codec"], group, *make_weight(c["n"], c["k"], c["planes"], group, _generator(seed, 1)))
    return dict(kind=kind, w=w, x=make_x(c["m"], c["k"], _generator(seed, 2)).cpu().numpy(), m=c["m"])


def run(state):
    b, kind = backend(), state["kind"]
    if kind == "linear":
        b.forward_dev(state["w"], state["x"], state["y"])
        return state["y"]
    if kind == "layers":
        state["graph"].replay()
        return state["y"]
    if kind == "stack":
        # bf16 bit patterns as the entry point returns them, read as numbers
        return torch.from_numpy(state["stack"].forward_host(state["x"], state["m"], x_is_bf16=True).view(np.int16)).view(torch.bfloat16)
    if kind == "fast":
        return b.salt_v2_forward_fast(state["w"], state["x"], state["m"]).output
    return b.salt_v2_forward_exact(state["w"], state["x"], state["m"]).output


# ---------------------------------------------------------------------------------------- bounds and results
def _weight_bytes(n, k, planes, codec, group=128):
    coeffs = n * k
    packed = -(-coeffs // 256) * PLANE_BYTES[codec] * planes
    return packed + -(-coeffs // group) * planes * 2 + 2 * (coeffs // 256) // 8


def work(case):
    c, kind = case, case["kind"]
    size = {"bf16": 2, "f32": 4}
    if kind == "layers":
        total, flops = 0, 0
        for i, (n, k) in enumerate(_layer_shapes(c)):
            # inputs: x (bf16 for the second linear, fp32 else), norm weight, residual, the up projection
            total += _weight_bytes(n, k, c["planes"], c["codec"]) + c["m"] * n * 4 + c["m"] * k * (2 if i == 1 else 4)
            total += (k * 4 if i in (0, 2) else c["m"] * n * 4) + (c["m"] * k * 4 if i == 3 else 0)
            flops += 2 * c["m"] * n * k * c["planes"]
        return dict(bytes=total * c["layers"], flops=flops * c["layers"])
    layers = c.get("layers", 1)
    xs, ys = (size[c["x"]], size[c["y"]]) if kind == "linear" else (2, 2) if kind == "stack" else (4, 4)
    each = _weight_bytes(c["n"], c["k"], c["planes"], c["codec"], c.get("group", 128)) + c["m"] * c["n"] * ys
    return dict(bytes=layers * each + c["m"] * c["k"] * xs, flops=2 * layers * c["m"] * c["n"] * c["k"] * c["planes"])


def tolerance(case):
    if case["kind"] == "exact":
        return "exact"                     # the order of the sums is part of the contract
    if case["kind"] == "stack" or case.get("y") == "bf16":
        return {"rel": 6e-3}               # one rounding to bf16: 1.65e-3 against 64 bits
    if case["kind"] == "layers":
        # A norm or gate that rounds differently moves single int8 codes by one step of 127
        return {"rel": 1e-3}
    return {"rel": 1e-6}                   # fp32 sums of exact integer group sums: up to 2.5e-7 against 64 bits


def _quantised(x):
    """The int8 codes (quantize_act_int8: absmax per token, fp32 arithmetic, ties to even) and the token scales, in 64 bits."""
    x = x.float()
    gamma = x.abs().amax(dim=1, keepdim=True)
    q = torch.clamp(torch.round(x * torch.where(gamma > 0, 127.0 / gamma, torch.zeros_like(gamma))), -128, 127)
    return q.double(), gamma.double() / 127


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "layers":
        out = []
        for li in range(c["layers"]):
            for (n, k), (x, norm, res, up), i in zip(_layer_shapes(c), _layer_inputs(c, li, seed), range(4)):
                if norm is not None:
                    inv = 1 / torch.sqrt(x.double().square().mean(dim=1, keepdim=True) + NORM_EPS)
                    x = (x * inv.float()) * norm
                if up is not None:
                    x = (x.clamp(min=0) * x.clamp(min=0)) * up
                q, a = _quantised(x)
                y = q @ dense64(n, k, *make_weight(n, k, c["planes"], 128, _generator(seed, 10 + 4 * li + i))).T * a
                out.append(y + res.double() if res is not None else y)
        return out
    x = make_x(c["m"], c["k"], _generator(seed, 2))
    if kind == "linear":
        q, a = _quantised(x.to(DTYPE[c["x"]]))
        return q @ dense64(c["n"], c["k"], *make_weight(c["n"], c["k"], c["planes"], 128, _generator(seed, 1))).T * a
    if kind == "stack":
        q, a = _quantised(x.bfloat16())
        return torch.stack([q @ dense64(c["n"], c["k"], *make_weight(c["n"], c["k"], c["planes"], 128, _generator(seed, 10 + i))).T * a
                            for i in range(c["layers"])])
    return x.double() @ dense64(c["n"], c["k"], *make_weight(c["n"], c["k"], c["planes"], c.get("group", 128), _generator(seed, 1))).T
