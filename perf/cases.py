"""Performance cases of the block-scaled FP8 GEMM: the calls a program that uses this library makes, over the range it
makes them.

`listed()` gives the named cases, `draw(rng)` one more of the same ranges; `prepare` builds what a program holds before
the call, `run` is one pass through the public entry points, `work` the bytes and operations a pass cannot do without,
`tolerance` how far two correct implementations of the same precision may differ.

Every case has an "op":
  gemm      C = gemm(A, B, a_scale, b_scale) on operands that are already fp8: run-time dispatch, no forced kernel.  With
            n_total set, the call computes the columns [n0, n0 + N) of a wider problem (one GPU's shard).
  linear    a linear layer's forward pass: quantize_rowwise on the activations, then gemm with weights that were
            quantised once, when the model was loaded
  quantize  quantize_rowwise or quantize_block alone (activations of a layer, weights at load time)
  reencode  e4m3fnuz bytes already on the device -> e4m3fn (loading operands of the other dialect)
  host      HostContext.gemm: operands in pinned host memory in, C in pinned host memory out
"""
import math

import torch

import fp8_quant_matmul_b200 as f

DEV = "cuda"
# No drawn case costs more than the largest listed one (2 * 6144 * 4608 * 7168 operations).
MAX_FLOPS = 2.0 * 6144 * 4608 * 7168


def listed():
    return [
        # decode: a handful of tokens against one weight matrix; latency, and the bytes of the weights
        {"name": "gemm_decode_16x7168x2304", "op": "gemm", "M": 16, "N": 7168, "K": 2304},
        # the benchmark's first configuration: few tiles, long K (K has to be cut to fill the GPU)
        {"name": "gemm_1024x1536x7168", "op": "gemm", "M": 1024, "N": 1536, "K": 7168},
        # short K with few rows: a low-rank up-projection of a small batch, a few microseconds of work
        {"name": "gemm_1024x7168x256", "op": "gemm", "M": 1024, "N": 7168, "K": 256},
        # the same projection for a large batch: nearly all of the bytes are the output
        {"name": "gemm_6144x7168x256", "op": "gemm", "M": 6144, "N": 7168, "K": 256},
        # the benchmark's compute-bound shape, and the largest case
        {"name": "gemm_6144x4608x7168", "op": "gemm", "M": 6144, "N": 4608, "K": 7168},
        # ragged: no dimension fills its last tile (a batch of sequences of uneven length, an odd layer width)
        {"name": "gemm_ragged_2064x1552x3200", "op": "gemm", "M": 2064, "N": 1552, "K": 3200},
        # one GPU's eighth of a wide problem partitioned by columns; the shard begins inside a 128-column scale block
        {"name": "gemm_shard_16384x576x7168", "op": "gemm", "M": 16384, "N": 576, "K": 7168, "n0": 1728, "n_total": 4608},
        # a linear layer while decoding: bf16 activations of 32 tokens
        {"name": "linear_32x4096x2048_bf16", "op": "linear", "M": 32, "N": 4096, "K": 2048, "bf16": True},
        # a linear layer in prefill: bf16 activations of a few thousand tokens
        {"name": "linear_4096x4608x7168_bf16", "op": "linear", "M": 4096, "N": 4608, "K": 7168, "bf16": True},
        # weights quantised once at load time, from fp32
        {"name": "quantize_block_4608x7168", "op": "quantize", "kind": "block", "M": 4608, "K": 7168, "bf16": False},
        # weights stored in the other fp8 dialect, brought over at load time
        {"name": "reencode_7168x2304", "op": "reencode", "M": 7168, "K": 2304},
        # operands and result in host memory
        {"name": "host_1024x3072x1536", "op": "host", "M": 1024, "N": 3072, "K": 1536},
    ]


def _log_multiple(rng, lo, hi, step):
    """A multiple of `step` in [lo, hi], spread over the logarithm of its value."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, int(round(v / step)) * step))


def draw(rng):
    op = rng.choice(["gemm"] * 6 + ["linear"] * 2 + ["quantize", "reencode", "host"])
    while True:
        M = _log_multiple(rng, 16, 16384, 16)
        N = _log_multiple(rng, 64, 7168, 16)
        K = _log_multiple(rng, 128, 7168, 128)
        if op == "reencode":
            return {"op": op, "M": _log_multiple(rng, 128, 7168, 16), "K": _log_multiple(rng, 128, 7168, 128)}
        if op == "quantize":
            return {"op": op, "kind": rng.choice(["block", "rowwise"]), "M": min(M, 7168), "K": K,
                    "bf16": rng.random() < 0.5}
        if 2.0 * M * N * K > MAX_FLOPS:
            continue
        if op == "host":
            if M * K + N * K + 2 * M * N > 64 << 20:      # what a synchronous call from host memory is used for
                continue
            return {"op": op, "M": M, "N": N, "K": K}
        if op == "linear":
            return {"op": op, "M": M, "N": N, "K": K, "bf16": rng.random() < 0.7}
        case = {"op": op, "M": M, "N": N, "K": K}
        if rng.random() < 0.2:                            # a column shard of one of 2, 4 or 8 GPUs
            world = rng.choice([2, 4, 8])
            N = max(64, N // 64 * 64)
            if N * world <= 8192:
                case.update(N=N, n0=N * rng.randrange(world), n_total=N * world)
        return case


# ---------------------------------------------------------------- inputs -----------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _fp8(g, n):
    """N(0,1) rounded to e4m3fn, magnitudes below 2^-6 flushed to +0: the benchmark's element distribution, made of the
    values that both fp8 dialects hold."""
    q = torch.randn(n, generator=g, device=DEV).to(torch.float8_e4m3fn).view(torch.uint8)
    return torch.where((q & 0x7F) < 8, torch.zeros_like(q), q)


def _scales(g, n):
    return torch.rand(n, generator=g, device=DEV) * 0.99 + 0.01


def _activations(g, M, K, bf16):
    """Activations of a layer: normal, with the spread between channels that makes per-block scales worth having."""
    x = torch.randn(M, K, generator=g, device=DEV)
    x *= torch.exp(torch.randn(K, generator=g, device=DEV))
    return x.to(torch.bfloat16) if bf16 else x


def _weights(g, N, K, bf16=False):
    w = torch.randn(N, K, generator=g, device=DEV) * (K ** -0.5)
    return w.to(torch.bfloat16) if bf16 else w


def _operands(g, case):
    """fp8 operands and their scales, in the operator's layouts."""
    M, N, K = case["M"], case["N"], case["K"]
    n_total = case.get("n_total") or N
    return {"A": _fp8(g, M * K), "B": _fp8(g, N * K), "a_scale": _scales(g, M * (K // 128)),
            "b_scale": _scales(g, (n_total + 127) // 128 * (K // 128))}


def prepare(case, seed):
    g = _gen(seed)
    op, M, K = case["op"], case["M"], case["K"]
    state = {"case": case}
    if op == "gemm":
        state.update(_operands(g, case), n0=case.get("n0") or 0, n_total=case.get("n_total") or case["N"])
    elif op == "linear":
        Wq, Ws = f.quantize_block(_weights(g, case["N"], K, case["bf16"]))
        state.update(X=_activations(g, M, K, case["bf16"]), Wq=Wq, Ws=Ws)
    elif op == "quantize":
        state["X"] = _weights(g, M, K, case["bf16"]) if case["kind"] == "block" else _activations(g, M, K, case["bf16"])
    elif op == "reencode":
        # the same values in e4m3fnuz: the byte is 8 higher, zero stays zero
        q = _fp8(g, M * K)
        state["src"] = torch.where(q == 0, q, q + 8)
    else:
        # operands and result in the program's own pinned buffers, as numpy arrays; the context is kept between calls
        N = case["N"]
        state["ctx"] = f.HostContext(M, N, K)
        state["C_host"] = torch.empty(M, N, dtype=torch.bfloat16, pin_memory=True)
        state["C"] = state["C_host"].view(torch.int16).numpy()
        for name, values in _operands(g, case).items():
            state[name] = values.cpu().pin_memory().numpy()
    return state


def run(state):
    case = state["case"]
    op, M, K = case["op"], case["M"], case["K"]
    if op == "gemm":
        return f.gemm(state["A"], state["B"], state["a_scale"], state["b_scale"], M=M, N=case["N"], K=K, n0=state["n0"],
                      n_total=state["n_total"])
    if op == "linear":
        q, s = f.quantize_rowwise(state["X"])
        return f.gemm(q, state["Wq"], s, state["Ws"], M=M, N=case["N"], K=K)
    if op == "quantize":
        return f.quantize_block(state["X"]) if case["kind"] == "block" else f.quantize_rowwise(state["X"])
    if op == "reencode":
        return f.fnuz_to_fn_device(state["src"])
    state["ctx"].gemm(state["C"], state["A"], state["B"], state["a_scale"], state["b_scale"], M, case["N"], K)
    return state["C_host"]


def work(case):
    op, M, K = case["op"], case["M"], case["K"]
    if op == "reencode":
        return {"bytes": 2.0 * M * K, "flops": 0.0}
    if op == "quantize":
        scales = M * (K // 128) if case["kind"] == "rowwise" else (M + 127) // 128 * (K // 128)
        return {"bytes": M * K * (2.0 if case["bf16"] else 4.0) + M * K + 4.0 * scales, "flops": 0.0}
    N = case["N"]
    bytes_ = float(N * K + 4 * (N + 127) // 128 * (K // 128) + 2 * M * N)
    if op == "linear":      # activations in; their fp8 form is an intermediate
        bytes_ += M * K * (2.0 if case["bf16"] else 4.0)
    else:
        bytes_ += M * K + 4.0 * M * (K // 128)
    return {"bytes": bytes_, "flops": 2.0 * M * N * K}


def tolerance(case):
    # Quantisers and the re-encoding are defined bit for bit.
    if case["op"] in ("quantize", "reencode"):
        return "exact"
    # bf16 results of fp32 sums.  The rounding to bf16 alone is 1.66e-3 (2-norm) and 3.9e-3 at most (against float64);
    # four times that.
    return {"rel": 6.6e-3, "max": 1.6e-2}


# ------------------------------------------------------- the same results in 64 bits ------------------------------
def _quantized(X, rows_per_group):
    """X in groups of rows_per_group rows x 128 columns: the fp8 values and the inverse scale of every group, both as
    float64.  The quantisation is defined in fp32: scale = (1 / absmax) * 448, value = e4m3(x * scale)."""
    R, K = X.shape
    pad = -R % rows_per_group
    x = torch.nn.functional.pad(X.float(), (0, 0, 0, pad)).view((R + pad) // rows_per_group, rows_per_group, K // 128, 128)
    scale = x.abs().amax(dim=(1, 3), keepdim=True).clamp(min=1e-12).reciprocal() * 448.0
    q = (x * scale).clamp(-448.0, 448.0).to(torch.float8_e4m3fn).double().view(R + pad, K)[:R]
    return q, (1.0 / scale).double().view(-1, K // 128)


def _blockwise_product(A, B, a_scale, b_scale):
    """A [M, K], B [N, K] with scales per row (or column) and 128 k: [M, K / 128], [N, K / 128].  All float64."""
    return (A * a_scale.repeat_interleave(128, 1)) @ (B * b_scale.repeat_interleave(128, 1)).T


def exact(case, seed):
    g = _gen(seed)
    op, M, K = case["op"], case["M"], case["K"]
    if op == "reencode":                                  # bytes and a count
        return None
    if op == "quantize":                                  # bytes, and the inverse scales
        X = _weights(g, M, K, case["bf16"]) if case["kind"] == "block" else _activations(g, M, K, case["bf16"])
        _, inv = _quantized(X, 128 if case["kind"] == "block" else 1)
        return None, inv.T.contiguous().flatten()
    N = case["N"]
    if op == "linear":
        Bv, bs = _quantized(_weights(g, N, K, case["bf16"]), 128)
        Av, as_ = _quantized(_activations(g, M, K, case["bf16"]), 1)
        return _blockwise_product(Av, Bv, as_, bs.repeat_interleave(128, 0)[:N])
    t = _operands(g, case)
    n0 = case.get("n0") or 0
    A = t["A"].view(torch.float8_e4m3fn).double().view(K, M).T
    B = t["B"].view(torch.float8_e4m3fn).double().view(K, N).T
    bs = t["b_scale"].double().view(K // 128, -1).T.repeat_interleave(128, 0)[n0:n0 + N]
    C = _blockwise_product(A, B, t["a_scale"].double().view(K // 128, M).T, bs)
    return C if op == "gemm" else C.cpu()
