"""Performance cases of the operator surface: the OFT product, its other algebraic order, and the plain GEMMs.

Sizes come from the configurations, the tests and the benchmark of this repository; the small and ragged ones are
generic.  All inputs are seeded and made on the GPU; outputs are written to a buffer that the caller keeps, as a
program that calls these C-style entry points does.
"""
import torch

from cute_mma_b200 import ops

_DEV = "cuda"


def listed():
    return [
        # A finetuned 4096 x 4096 projection in a decode step: a handful of tokens, the weight is read once.
        {"name": "oft_decode", "op": "oft", "m": 8, "n": 4096, "k": 4096, "b": 64, "group": 4096},
        # The CPU oracle's configuration: a small layer, where launches and latency count.
        {"name": "oft_small", "op": "oft", "m": 512, "n": 1024, "k": 1024, "b": 32, "group": 1024},
        # A prompt of odd length through an up-projection: ragged in M, N not a power of two.
        {"name": "oft_prompt_ragged", "op": "oft", "m": 3001, "n": 11008, "k": 4096, "b": 32, "group": 11008},
        # The reference's own benchmark point: a rotation per group of 256 columns, 8 x 8 blocks.
        {"name": "oft_groups", "op": "oft", "m": 8192, "n": 8192, "k": 8192, "b": 8, "group": 256},
        # The projection configuration: 16384 tokens of a training or prefill batch.
        {"name": "oft_projection", "op": "oft", "m": 16384, "n": 4096, "k": 4096, "b": 64, "group": 4096},
        # The large configuration on one GPU, the benchmark's default workload.
        {"name": "oft_large", "op": "oft", "m": 65536, "n": 28672, "k": 8192, "b": 128, "group": 28672},
        # Rotation folded into the weight inside the call (a weight that changes every step), a medium batch.
        {"name": "oft_a_rw", "op": "a_rw", "m": 2048, "n": 4096, "k": 4096, "b": 64, "group": 4096},
        # The smallest calls: a ragged half GEMM of a few tiles.
        {"name": "gemm_half_tn_tiny", "op": "gemm", "type": "half", "layout": "TN", "m": 200, "n": 328, "k": 136},
        # An ordinary float (TF32) GEMM that does not fill the GPU.
        {"name": "gemm_float_tn_small", "op": "gemm", "type": "float", "layout": "TN", "m": 640, "n": 1280, "k": 1024},
        # The float (TF32) configuration.
        {"name": "gemm_float_nt", "op": "gemm", "type": "float", "layout": "NT", "m": 4096, "n": 4096, "k": 4096},
        # The half configuration.
        {"name": "gemm_half_tn", "op": "gemm", "type": "half", "layout": "TN", "m": 8192, "n": 8192, "k": 8192},
        # A weight gradient of a backward pass: both operands token-major, long K, half in, float out, the loss scale taken out.
        {"name": "gemm_half_nt_wgrad", "op": "wgrad", "m": 4096, "n": 4096, "k": 16384},
    ]


def _log_int(rng, lo, hi):
    """Spread over the logarithm of [lo, hi]."""
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    op = rng.choice(["oft", "oft", "oft", "gemm", "gemm", "wgrad", "a_rw"])
    if op in ("oft", "a_rw"):
        b = rng.choice([8, 16, 32, 64, 128])
        m = _log_int(rng, 1, 65536 if op == "oft" else 16384)
        n = _log_int(rng, 256, 28672)
        k = b * max(1, _log_int(rng, 256, 8192) // b)
        kind = rng.random()
        if kind < 0.25:  # several N-groups, each with a rotation of its own
            group = rng.choice([256, 512] if b == 128 else [128, 256, 512])
            n = group * max(1, n // group)
        else:  # one rotation for all of N; half of these widths as models have them
            n = 64 * max(4, n // 64) if kind < 0.65 else n
            group = n
        return {"op": op, "m": m, "n": n, "k": k, "b": b, "group": group}
    if op == "gemm":
        return {"op": op, "type": rng.choice(["half", "float"]), "layout": rng.choice(["TN", "NT"]), "m": _log_int(rng, 64, 8192),
                "n": _log_int(rng, 64, 8192), "k": _log_int(rng, 64, 8192)}
    return {"op": op, "m": 8 * _log_int(rng, 32, 1376), "n": 8 * _log_int(rng, 32, 1024), "k": _log_int(rng, 512, 16384)}


def _up8(x):
    return (x + 7) // 8 * 8


def _matrix(rows, cols, gen, sigma, dtype):
    """[rows][ld] with rows padded to a multiple of 8 elements, N(0, sigma)."""
    return torch.randn((rows, _up8(cols)), generator=gen, device=_DEV, dtype=dtype) * sigma


def _rotations(groups, k, b, gen):
    """Stored R of Cayley-transformed skew-symmetric blocks: (I - S)(I + S)^-1, S with entries of N(0, 0.01), as the
    projection configuration makes them.  [groups * b][k], every block transposed."""
    s = torch.randn((groups * (k // b), b, b), generator=gen, device=_DEV) * 0.01
    s = torch.triu(s, 1)
    s = s - s.transpose(1, 2)
    eye = torch.eye(b, device=_DEV)
    r = torch.linalg.solve(eye + s, eye - s)  # (I + S)^-1 and (I - S) commute
    return r.reshape(groups, k // b, b, b).permute(0, 3, 1, 2).reshape(groups * b, k).half().contiguous()


def prepare(case, seed):
    gen = torch.Generator(device=_DEV)
    gen.manual_seed(seed)
    m, n, k = case["m"], case["n"], case["k"]
    st = {"case": case, "lib": ops.load_library()}
    if case["op"] in ("oft", "a_rw"):  # activations of N(0, 1), weights of N(0, 0.02)
        st["A"] = _matrix(m, k, gen, 1.0, torch.float16)
        st["B"] = _matrix(n, k, gen, 0.02, torch.float16)
        st["R"] = _rotations(n // case["group"], k, case["b"], gen)
        st["C"] = torch.empty((m, n), device=_DEV, dtype=torch.float16)
        return st
    if case["op"] == "wgrad":  # A(i, l), B(j, l) stored with i, j contiguous: [k][m], [k][n]; C column-major
        st["A"] = _matrix(k, m, gen, 1.0, torch.float16)
        st["B"] = _matrix(k, n, gen, 0.5, torch.float16)
        st["C"] = torch.empty((n, m), device=_DEV, dtype=torch.float32)
        return st
    dtype = torch.float16 if case["type"] == "half" else torch.float32
    shape_a, shape_b = ((m, k), (n, k)) if case["layout"] == "TN" else ((k, m), (k, n))
    st["A"] = _matrix(*shape_a, gen, 1.0, dtype)
    st["B"] = _matrix(*shape_b, gen, 1.0, dtype)
    st["C"] = torch.empty((n, m), device=_DEV, dtype=dtype)
    return st


def run(state):
    c, A, B, C = state["case"], state["A"], state["B"], state["C"]
    m, n, k, ld_a, ld_b = c["m"], c["n"], c["k"], A.stride(0), B.stride(0)
    stream = torch.cuda.current_stream()
    if c["op"] == "oft":
        ops.oft_tn(m, n, k, A, ld_a, B, ld_b, state["R"], k, C, n, stream, group_size=c["group"], reconn_sz=c["b"], lib=state["lib"])
    elif c["op"] == "a_rw":
        ops.oft_tn_a_rw(m, n, k, A, ld_a, B, ld_b, state["R"], k, C, n, stream, group_size=c["group"], reconn_sz=c["b"], lib=state["lib"])
    elif c["op"] == "wgrad":
        ops.gemm_ex("N", "T", m, n, k, 1.0 / 128, A, ld_a, B, ld_b, 0.0, C, m, stream, in_type=ops.F16, out_type=ops.F32, lib=state["lib"])
    else:
        gemm = ops.gemm_tn if c["layout"] == "TN" else ops.gemm_nt
        gemm(m, n, k, A, ld_a, B, ld_b, C, m, stream, dtype=c["type"], lib=state["lib"])
    return C


def work(case):
    m, n, k = case["m"], case["n"], case["k"]
    flops = 2 * m * n * k
    size_in = 4 if case.get("type") == "float" else 2
    size_out = 4 if case.get("type") == "float" or case["op"] == "wgrad" else 2
    moved = (m + n) * k * size_in + m * n * size_out
    if case["op"] in ("oft", "a_rw"):
        groups = n // case["group"]
        flops += 2 * k * case["b"] * (groups * m if case["op"] == "oft" else n)  # the rotation of X per group, or of W
        moved += groups * case["b"] * k * 2
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    # About four times what was measured against the same product in 64 bits (X.R, or R.W, rounded to half as the
    # operator does; float operands cut to TF32).  Half results: one rounding of the result and one of the rotated
    # operand, 2.1e-4 and at most 5.7e-4 of the larger of value and root mean square.  Float results: the tensor
    # cores' 32-bit accumulation, an error that grows with K: 9.6e-6 at K 4096 (float operands), 1.9e-5 at K 16384
    # (half operands).
    if case["op"] == "wgrad":
        return {"rel": 5e-6 * max(1.0, case["k"] / 1024)}
    if case.get("type") == "float":
        return {"rel": 1e-5 * max(1.0, case["k"] / 1024)}
    return {"rel": 8e-4, "max": 2.5e-3}
