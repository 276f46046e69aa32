"""C = alpha * A.B^T + beta * C with beta != 0 on each of the plain GEMM's kernels: the bits of the epilogue's arithmetic at the
edges of its blocks of columns, and no wait per column."""
import contextlib

import pytest

torch = pytest.importorskip("torch")

from cute_mma_b200 import ops  # noqa: E402

pytestmark = pytest.mark.gpu

KERNELS = {"small": {"small_tiles": 1}, "pair": {"small_tiles": 0, "gemm_wide": 0}, "wide": {"small_tiles": 0, "gemm_wide": 1}}


def operands(m, n, k, layout, dtype, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    up8 = lambda x: (x + 7) // 8 * 8
    shapes = ((m, up8(k)), (n, up8(k))) if layout == "TN" else ((k, up8(m)), (k, up8(n)))
    return [torch.randn(s, device="cuda", generator=gen).to(dtype) for s in shapes]


def product(lib, layout, m, n, k, alpha, A, B, beta, C):
    ops.gemm_ex(layout[0], layout[1], m, n, k, alpha, A, A.stride(0), B, B.stride(0), beta, C, C.stride(0),
                in_type=ops.F16 if A.dtype is torch.float16 else ops.TF32, out_type=ops.F16 if C.dtype is torch.float16 else ops.F32, lib=lib)


# columns around the blocks of 16 and 32 that are read together, rows and columns around the tiles
@pytest.mark.parametrize("m,n", [(1, 1), (130, 15), (127, 16), (128, 17), (33, 31), (256, 32), (257, 33), (300, 129), (200, 512), (515, 801)])
@pytest.mark.parametrize("kind", ["half-half", "half-float", "float-float"])
@pytest.mark.parametrize("kernel", KERNELS)
def test_bits(lib, pair_build, kernel, kind, m, n):
    """alpha and beta are powers of two, so that the result is the 32-bit sum of two values that are known to the bit."""
    if not pair_build and kernel != "pair":
        pytest.skip("the single-CTA build has one kernel")
    t_in, t_out = (torch.float16 if t == "half" else torch.float32 for t in kind.split("-"))
    alpha, beta, k = 0.25, 0.5, 264
    for layout in ("TN", "NT"):
        A, B = operands(m, n, k, layout, t_in, m + n)
        sums = torch.empty((n, m), device="cuda")
        before = torch.randn((n, m + 3), device="cuda").to(t_out)
        C = before.clone()
        with contextlib.ExitStack() as options:
            for name, value in {"small_split": 1, **KERNELS[kernel]}.items():
                options.enter_context(ops.option(name, value, lib))
            product(lib, layout, m, n, k, 1.0, A, B, 0.0, sums)
            product(lib, layout, m, n, k, alpha, A, B, beta, C)
        assert ops.device_status(lib)[0] == 0
        assert torch.equal(C[:, :m], (alpha * sums + beta * before[:, :m].float()).to(t_out))
        assert torch.equal(C[:, m:], before[:, m:])


def us(call, reps=20):
    call()
    best = float("inf")
    for _ in range(5):
        a, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda._sleep(500000)  # the launches are queued behind it: host time does not count
        a.record()
        for _ in range(reps):
            call()
        e.record()
        e.synchronize()
        best = min(best, a.elapsed_time(e) * 1e3 / reps)
    return best


# columns of one warp in one round of tiles of 2304 x 2048 (pair tiles 72, of 128 x 128 288, wide ones all cut in halves)
@pytest.mark.parametrize("kernel,columns", [("small", 64), ("pair", 256), ("wide", 128)])
@pytest.mark.parametrize("kind", ["half-half", "half-float", "float-float"])
def test_columns_do_not_wait_for_one_another(lib, pair_build, kernel, columns, kind):
    """A load from L2 takes 0.25 us at least.  One after the other a warp's columns add that much each; the bound is 0.1."""
    if not pair_build:
        pytest.skip("about the kernels of the CTA-pair build")
    m, n, k = 2304, 2048, 512
    t_in, t_out = (torch.float16 if t == "half" else torch.float32 for t in kind.split("-"))
    A, B = operands(m, n, k, "TN", t_in, 1)
    C = torch.zeros((n, m), device="cuda", dtype=t_out)
    with contextlib.ExitStack() as options:
        for name, value in KERNELS[kernel].items():
            options.enter_context(ops.option(name, value, lib))
        plain, added = (us(lambda: product(lib, "TN", m, n, k, 1.0, A, B, beta, C)) for beta in (0.0, 0.5))
    assert added - plain <= 0.1 * columns, (plain, added)
