"""Plain GEMM on 256 x 512 pair tiles (gemm2w_kernel): the bits of the 256 x 256 pair tiles, which the other GEMM tests pin,
and the product itself in 64 bits."""
import pytest

torch = pytest.importorskip("torch")

from cute_mma_b200 import ops  # noqa: E402

pytestmark = pytest.mark.gpu

# (m, n, k): least K of the kernel (4 steps of 64 halves), two halves of one tile, a last half of one column, odd numbers of 256-column
# tiles, all of them single halves on 74 pairs; then whole tiles, with single halves behind them, and a part-filled round of whole
# tiles whose free pairs take two halves each.  (Whole tiles of least K and cut tiles: test_wide_schedule.py.)
SHAPES = [(256, 512, 256), (256, 512, 200), (129, 257, 1024), (300, 700, 520), (1000, 2000, 640), (2304, 4352, 264), (5000, 9000, 328), (20000, 1100, 264)]
KINDS = [("half", "half", "TN", 1.0, 0.0), ("half", "half", "NT", 1.0, 0.0), ("half", "float", "NT", 1 / 128, 0.0), ("half", "half", "TN", 0.5, 2.0),
         ("float", "float", "TN", 1.0, 0.0), ("float", "float", "NT", 1.0, 0.0)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("kind", KINDS, ids=lambda k: "-".join(map(str, k[:3])) + ("-beta" if k[4] else ""))
def test_wide_tiles_have_the_bits_of_pair_tiles(shape, kind):
    m, n, k = shape
    t_in, t_out, layout, alpha, beta = kind
    dt, od = (torch.float16 if t == "half" else torch.float32 for t in (t_in, t_out))
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    up8 = lambda x: (x + 7) // 8 * 8
    rows_a, rows_b, cols_a, cols_b = (m, n, k, k) if layout == "TN" else (k, k, m, n)
    A = torch.randn((rows_a, up8(cols_a)), device="cuda", generator=gen).to(dt)
    B = torch.randn((rows_b, up8(cols_b)), device="cuda", generator=gen).to(dt)
    A[:, cols_a:], B[:, cols_b:] = float("nan"), float("nan")  # padding is never read into a sum
    ld = m + 5
    before = torch.randn((n, ld), device="cuda", generator=gen).to(od)
    got = []
    for wide in (0, 1):
        C = before.clone()
        with ops.option("gemm_wide", wide), ops.option("small_tiles", 0):
            ops.gemm_ex(layout[0], layout[1], m, n, k, alpha, A, A.stride(0), B, B.stride(0), beta, C, ld,
                        in_type=ops.F16 if t_in == "half" else ops.TF32, out_type=ops.F16 if t_out == "half" else ops.F32)
        assert ops.device_status()[0] == 0
        got.append(C)
    assert torch.equal(got[0], got[1])
    assert torch.equal(got[1][:, m:], before[:, m:])
    # a few rows of C in 64 bits, operands cut to TF32 where the tensor core does; the 32-bit sums of k products of N(0, 1)
    # stray by less than k * 2^-24 of their mean magnitude sqrt(k), the result's rounding adds half an ulp
    cut = lambda x: (x.view(torch.int32) & -8192).view(torch.float32) if t_in == "float" else x
    mat = lambda x, cols: (cut(x[:, :cols].contiguous()) if layout == "TN" else cut(x[:, :cols].contiguous()).t()).double()
    pick = torch.tensor(sorted({0, m // 2, m - 1}), device="cuda")
    want = alpha * mat(A, cols_a)[pick] @ mat(B, cols_b).t() + beta * before.t()[pick].double()
    have = got[1].t()[pick].double()
    scale = (k ** 0.5 + 1) * (k * 2.0 ** -24 + 2.0 ** -23) + want.abs() * (2.0 ** -11 if od is torch.float16 else 2.0 ** -24) + 2.0 ** -24
    assert ((have - want).abs() <= 8 * scale).all()
