"""Where the OFT product runs as rotation pass + GEMM by the library's own choice: either side of its lines, every route
returns the same bits."""
import pytest

torch = pytest.importorskip("torch")

from cute_mma_b200 import inputs, ops  # noqa: E402

pytestmark = pytest.mark.gpu

# few rows of any block edge and one round of tiles; more rows and more tiles than SM pairs; the same with 128 x 128 blocks or
# with one round of tiles stays on the ring; few N tiles only with short K
CASES = [(300, 4096, 768, 64, "two_pass"), (1023, 4352, 1024, 128, "two_pass"), (1024, 4352, 1024, 128, "fused_ring"),
         (2304, 2560, 1024, 32, "two_pass"), (1792, 2560, 1024, 32, "fused_ring"), (5000, 1280, 1032, 8, "two_pass"),
         (5000, 1024, 1032, 8, "fused_tmem"), (9000, 640, 512, 16, "two_pass"), (9000, 640, 576, 16, "fused_tmem")]


@pytest.mark.parametrize("m,n,k,b,route", CASES)
def test_bits_do_not_depend_on_the_choice(lib, cuda, pair_build, m, n, k, b, route):
    if not pair_build:
        pytest.skip("the single-CTA build has one route")
    gen = torch.Generator(device=cuda).manual_seed(m)
    A = torch.randn((m, k), generator=gen, device=cuda).half()
    B = (torch.randn((n, k), generator=gen, device=cuda) * 0.02).half()
    R = torch.from_numpy(inputs.pack_r(inputs.blocks_qr(1, k // b, b, 5))).to(cuda)
    got = []
    for forced in (0, 1):
        C = torch.full((m + 1, n), -7.0, device=cuda, dtype=torch.float16)
        with ops.option("oft_route", forced, lib), ops.option("small_tiles", 0, lib):
            assert forced or ops.oft_route(m, n, k, reconn_sz=b, lib=lib) == route
            ops.oft_tn(m, n, k, A, k, B, k, R, k, C, n, reconn_sz=b, lib=lib)
        assert ops.device_status(lib)[0] == 0
        assert (C[m] == -7.0).all()
        got.append(C.view(torch.int16))
    assert torch.equal(got[0], got[1])


# several groups: two launches each, so only where the other routes launch group by group as well; route 1 takes narrow ones
# together, whatever their rows (few, and enough for each group to fill the GPU)
GROUPS = [(300, 3840, 1024, 64, "fused_tmem", 1280), (520, 1536, 512, 32, "fused_tmem", 768), (2900, 3584, 768, 16, "fused_tmem", 1792),
          (300, 1536, 512, 128, "fused_tmem", 768), (300, 4096, 1024, 64, "two_pass", 2048), (2700, 4096, 1024, 32, "two_pass", 2048),
          (300, 2560, 1024, 128, "two_pass", 1280)]


@pytest.mark.parametrize("m,n,k,b,route,group", GROUPS)
def test_several_groups(lib, cuda, pair_build, m, n, k, b, route, group):
    if not pair_build:
        pytest.skip("the single-CTA build has one route")
    gen = torch.Generator(device=cuda).manual_seed(m)
    A = torch.randn((m, k), generator=gen, device=cuda).half()
    B = (torch.randn((n, k), generator=gen, device=cuda) * 0.02).half()
    R = torch.from_numpy(inputs.pack_r(inputs.blocks_qr(n // group, k // b, b, 5))).to(cuda)
    got = []
    for forced in (0, 1):
        C = torch.full((m + 1, n), -7.0, device=cuda, dtype=torch.float16)
        with ops.option("oft_route", forced, lib), ops.option("small_tiles", 0, lib):
            assert forced or ops.oft_route(m, n, k, group_size=group, reconn_sz=b, lib=lib) == route
            ops.oft_tn(m, n, k, A, k, B, k, R, k, C, n, group_size=group, reconn_sz=b, lib=lib)
        assert ops.device_status(lib)[0] == 0
        assert (C[m] == -7.0).all()
        got.append(C.view(torch.int16))
    assert torch.equal(got[0], got[1])
