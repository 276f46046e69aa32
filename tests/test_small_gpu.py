"""small_kernel (problems of up to about one 128 x 128 tile per SM) at the edges of its tiles, its pieces along K and its
rotation buffers, against the routes it replaces (bit for bit where K is not cut) and against fp64."""
import numpy as np
import pytest

from _util import GRAPH_MEM_ALLOC, graph_node_types, make_oft_case, truth_ok
from cute_mma_b200 import ops
from oracle import oracle

pytestmark = pytest.mark.gpu


def _oft(lib, cuda, A, R, B, m, n, k, b, gs, ldc, shift, **opts):
    """C[m, n] with rows ldc apart and its base `shift` elements past an aligned address; canaries around it."""
    import contextlib
    import torch

    dA, dB, dR = (torch.from_numpy(x).to(cuda) for x in (A, B, R))
    buf = torch.full(((m + 1) * ldc + shift,), -7.0, dtype=torch.float16, device=cuda)
    with contextlib.ExitStack() as es:
        for name, v in opts.items():
            es.enter_context(ops.option(name, v, lib))
        ops.oft_tn(m, n, k, dA, k, dB, k, dR, k, buf.data_ptr() + 2 * shift, ldc, group_size=gs, reconn_sz=b, lib=lib)
        path = ops.oft_plan(m, n, k, group_size=gs, reconn_sz=b, lib=lib)["path"]
    assert ops.device_status(lib)[0] == 0
    out = buf.cpu().numpy()
    rows = out[shift:].reshape(m + 1, ldc)
    assert np.all(out[:shift] == -7.0) and np.all(rows[m] == -7.0) and np.all(rows[:m, n:] == -7.0)
    return rows[:m, :n].copy(), path


# rows at the edges of the 16-column granule, of a warp's 32 rows, of the three-buffer limit (64) and of a tile (128)
@pytest.mark.parametrize("m,n,k,b,gs,pad,shift", [
    (1, 256, 64, 64, None, 0, 0), (16, 300, 1024, 32, None, 4, 0), (17, 129, 1040, 16, None, 3, 1), (33, 512, 2048, 128, 256, 0, 0),
    (64, 384, 1152, 64, 128, 8, 4), (65, 640, 1280, 128, None, 1, 0), (128, 127, 2056, 8, None, 0, 1), (129, 1000, 896, 32, None, 0, 0),
    (257, 512, 8192, 128, 512, 0, 0), (300, 1280, 1344, 8, 256, 2, 0)])
def test_small_oft_matches_the_other_route_and_truth(lib, cuda, pair_build, m, n, k, b, gs, pad, shift):
    if not pair_build:
        pytest.skip("the single-CTA build has one route")
    A, R, B = make_oft_case(m, n, k, b, gs, seed=91, xdist="normal", wsigma=0.05)
    args = (lib, cuda, A, R, B, m, n, k, b, gs, n + pad, shift)
    got, _ = _oft(*args)
    forced, path = _oft(*args, oft_route=5)
    assert path == "fused_small" and np.array_equal(forced.view(np.uint16), got.view(np.uint16))  # the library's own choice
    groups, g_sz = (1, n) if gs is None else (n // gs, gs)
    truth = oracle.oft_f64(A, R, B, m, g_sz, groups, k, b, round_xr=True)
    assert truth_ok(got, truth)[0] == 0
    tmem, path = _oft(*args, oft_route=1)
    assert path == "fused_tmem"
    whole, _ = _oft(*args, oft_route=5, gemm_split=0)  # K in one piece: the same sums in the same order
    assert np.array_equal(whole.view(np.uint16), tmem.view(np.uint16))
    for split in (2, 3, 8):  # pieces of unequal length; one rounding of C, so at most a step of fp16 apart
        cut, _ = _oft(*args, small_split=split)
        d = np.abs(cut.astype(np.float64) - whole.astype(np.float64))
        assert np.all(d <= 2.0 ** -10 * (np.abs(whole.astype(np.float64)) + 1.0)), (split, float(d.max()))


@pytest.mark.parametrize("layout", ["TN", "NT"])
@pytest.mark.parametrize("in_type,out_type", [(0, 0), (0, 1), (2, 1)])
@pytest.mark.parametrize("m,n,k,alpha,beta,pad", [(1, 8, 8, 1.0, 0.0, 0), (129, 72, 1032, 1.0, 0.0, 1), (264, 136, 2048, 0.5, -0.25, 4), (120, 1000, 523, 1.0, 0.0, 3)])
def test_small_gemm_matches_the_pair_kernel(lib, cuda, pair_build, layout, in_type, out_type, m, n, k, alpha, beta, pad):
    if not pair_build:
        pytest.skip("the small-problem kernel belongs to the CTA-pair build")
    import torch

    g = torch.Generator(device=cuda).manual_seed(92)
    up8 = lambda x: (x + 7) // 8 * 8
    tin, tout = (torch.float16 if in_type == 0 else torch.float32), (torch.float16 if out_type == 0 else torch.float32)
    sa, sb = ((m, up8(k)), (n, up8(k))) if layout == "TN" else ((k, up8(m)), (k, up8(n)))
    A, B = (torch.randn(s, generator=g, device=cuda).to(tin) for s in (sa, sb))
    c0 = torch.randn((n + 1, m + pad), generator=g, device=cuda).to(tout)

    def run(**opts):
        C = c0.clone()
        import contextlib
        with contextlib.ExitStack() as es:
            for name, v in opts.items():
                es.enter_context(ops.option(name, v, lib))
            ops.gemm_ex(*layout, m, n, k, alpha, A, sa[1], B, sb[1], beta, C, m + pad, in_type=in_type, out_type=out_type, lib=lib)
        assert ops.device_status(lib)[0] == 0
        assert torch.equal(C[n], c0[n]) and torch.equal(C[:, m:], c0[:, m:])
        return C[:n, :m]

    pair = run(small_tiles=0, gemm_split=0)
    assert torch.equal(run(gemm_split=0), pair)
    # cut along K: fp32 sums in another order, |error| <= K 2^-24 sum |a b| and one rounding of the result
    bound = 4 * k ** 0.5 * 2.0 ** -23 + (2.0 ** -10 if out_type == 0 else 0)
    scale = pair.double().abs() + abs(alpha) * k ** 0.5
    for opts in ({}, {"small_split": 2}, {"small_split": 5}):
        assert bool(((run(**opts).double() - pair.double()).abs() <= bound * scale).all()), opts


def test_small_products_chained_on_two_streams(lib, cuda, pair_build):
    """Launches that may start their prologue under the one before them: a chain in which every product reads what the
    last one wrote, on two streams at once and under graph capture, gives the bits of the same chain with a
    synchronisation after every launch."""
    if not pair_build:
        pytest.skip("the small-problem kernel belongs to the CTA-pair build")
    import torch

    n = k = 1024
    g = torch.Generator(device=cuda).manual_seed(93)
    W = (torch.randn((n, k), generator=g, device=cuda) / 32).half()
    x0 = torch.randn((24, k), generator=g, device=cuda).half()

    def chain(bufs, stream, wait=False):
        for i in range(6):  # row-major [24][n]: the column-major n x 24 result of W . X^T
            ops.gemm_tn(n, 24, k, W, k, bufs[i], k, bufs[i + 1], n, stream, lib=lib)
            if wait:
                torch.cuda.synchronize()

    new = lambda: [x0.clone()] + [torch.zeros_like(x0) for _ in range(6)]
    want = new()
    chain(want, torch.cuda.current_stream(), wait=True)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    b1, b2, b3 = new(), new(), new()
    torch.cuda.synchronize()
    for _ in range(3):
        chain(b1, s1)
        chain(b2, s2)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        chain(b3, torch.cuda.current_stream())
    graph.replay()
    torch.cuda.synchronize()
    assert ops.device_status(lib)[0] == 0
    for b in (b1, b2, b3):
        assert torch.equal(b[6], want[6])


@pytest.mark.parametrize("m,n,k,b,gs,want", [
    (33000, 65, 4096, 64, None, 2),       # one group, unaligned rows: rotation pass in two chunks of X.R
    (2300, 2300, 192, 64, None, 1),       # aligned (n % 4 == 0 but ldC padded to 8), short K, few N tiles
    (2304, 2303, 448, 32, None, 2),       # unaligned, more than two 128 x 128 tiles per SM
    (4400, 4104, 320, 8, None, 2),        # aligned, K below 1024 and more tiles than SM pairs
    (2176, 2048, 136, 8, None, 1),        # two tiles per SM, little to do: the small-problem kernel
    (4608, 4096, 576, 64, 2048, 2),       # two wide groups
    (3, 65536, 448, 64, None, 2),         # few rows, a very wide group: the passes' GEMM is the small-problem kernel's
    (1, 40001, 1536, 32, None, 2),
    (1100, 1500, 8192, 128, None, 2)])    # a GEMM that would be cut by itself
def test_choice_between_the_routes_is_invisible(lib, cuda, pair_build, m, n, k, b, gs, want):
    """Shapes either side of the lines between the small-problem kernel, the rotation pass + GEMM and the fused kernels:
    the library's choice has the bits of the kernel that forms X.R per N tile, with aligned and unaligned rows of C."""
    if not pair_build:
        pytest.skip("the single-CTA build has one route")
    import torch
    from cute_mma_b200 import inputs

    g = torch.Generator(device=cuda).manual_seed(94)
    X = torch.randn((m, k), generator=g, device=cuda).half()
    W = (torch.randn((n, k), generator=g, device=cuda) * 0.02).half()
    groups = 1 if gs is None else n // gs
    R = torch.from_numpy(inputs.pack_r(inputs.blocks_qr(groups, k // b, b, 94))).to(cuda)

    def run(ldc, **opts):
        C = torch.full((m + 1, ldc), -7.0, dtype=torch.float16, device=cuda)
        import contextlib
        with contextlib.ExitStack() as es:
            for name, v in opts.items():
                es.enter_context(ops.option(name, v, lib))
            ops.oft_tn(m, n, k, X, k, W, k, R, k, C, ldc, group_size=gs, reconn_sz=b, lib=lib)
        assert ops.device_status(lib)[0] == 0
        assert bool((C[m] == -7.0).all()) and bool((C[:m, n:] == -7.0).all())
        return C[:m, :n]

    path = ops.oft_plan(m, n, k, group_size=gs, reconn_sz=b, lib=lib)["path"]
    if n % 8 == 0 or want == 2:
        assert path == {1: "fused_tmem", 2: "two_pass"}[want]
    want_bits = run((n + 7) // 8 * 8, oft_route=1).contiguous().view(torch.int16)
    for ldc in ((n + 7) // 8 * 8, n + (3 if n % 8 == 0 else 0)):
        assert torch.equal(run(ldc).contiguous().view(torch.int16), want_bits), ldc


def test_dependent_launches_of_the_other_kernels(lib, cuda, pair_build):
    """The same for the pair GEMM, the kernel that keeps X.R in tensor memory and the rotation pass: every product reads
    what the last one wrote, and scratch from the pool is handed on between calls."""
    if not pair_build:
        pytest.skip("the pair kernels belong to the CTA-pair build")
    import torch
    from cute_mma_b200 import inputs

    m, d, b = 1400, 2048, 64  # 11 x 16 tiles of 128 x 128
    g = torch.Generator(device=cuda).manual_seed(96)
    W = (torch.randn((d, d), generator=g, device=cuda) / 45).half()
    R = torch.from_numpy(inputs.pack_r(inputs.blocks_qr(1, d // b, b, 96))).to(cuda)
    x0 = torch.randn((m, d), generator=g, device=cuda).half()

    def chain(bufs, stream, wait=False):
        for i in range(6):
            if i % 3 == 0:
                ops.gemm_tn(d, m, d, W, d, bufs[i], d, bufs[i + 1], d, stream, lib=lib)
            elif i % 3 == 1:
                ops.oft_tn_two_pass(m, d, d, bufs[i], d, W, d, R, d, bufs[i + 1], d, stream, reconn_sz=b, lib=lib)
            else:
                ops.oft_tn_a_rw(m, d, d, bufs[i], d, W, d, R, d, bufs[i + 1], d, stream, reconn_sz=b, lib=lib)
            ops.oft_tn(m, 768, d, bufs[i + 1], d, W, d, R, d, bufs[7 + i], 768, stream, reconn_sz=b, lib=lib)
            if wait:
                torch.cuda.synchronize()

    new = lambda: [x0.clone()] + [torch.zeros_like(x0) for _ in range(6)] + [torch.zeros((m, 768), dtype=torch.float16, device=cuda) for _ in range(6)]
    want = new()
    chain(want, torch.cuda.current_stream(), wait=True)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    b1, b2 = new(), new()
    torch.cuda.synchronize()
    for _ in range(3):
        chain(b1, s1)
        chain(b2, s2)
    torch.cuda.synchronize()
    assert ops.device_status(lib)[0] == 0
    for got in (b1, b2):
        assert all(torch.equal(x, y) for x, y in zip(got, want))


def test_rows_of_x_longer_than_a_megabyte(lib, cuda, pair_build):
    """K above 524288: the plan answers, and a call with unaligned rows of C has the bits of the kernel that forms X.R
    per N tile."""
    import torch

    b, k = 64, 524288 + 64
    assert ops.oft_plan(4096, 256, k, reconn_sz=b, lib=lib)["path"] in ("fused_tmem", "fused_ring")
    assert ops.oft_plan(4096, 4096, k, reconn_sz=b, lib=lib)["kernel_launches"] >= 1
    if not pair_build:
        return
    m, n = 300, 257
    g = torch.Generator(device=cuda).manual_seed(98)
    X = torch.randn((m, k), generator=g, device=cuda).half()
    W = (torch.randn((n, k), generator=g, device=cuda) * 0.02).half()
    R = (torch.randn((b, k), generator=g, device=cuda) * 0.1).half()

    def run(**opts):
        import contextlib
        C = torch.full((m + 1, n), -7.0, dtype=torch.float16, device=cuda)
        with contextlib.ExitStack() as es:
            for name, v in opts.items():
                es.enter_context(ops.option(name, v, lib))
            ops.oft_tn(m, n, k, X, k, W, k, R, k, C, n, reconn_sz=b, lib=lib)
        assert ops.device_status(lib)[0] == 0
        return C.view(torch.int16)

    assert torch.equal(run(small_tiles=0), run(oft_route=1))


@pytest.mark.parametrize("layout", ["TN", "NT"])
@pytest.mark.parametrize("in_type,out_type,alpha,beta", [(0, 0, 0.5, 0.0), (0, 1, 1.0 / 128, 0.0), (2, 1, -4.0, 0.0), (2, 1, 1.0, -0.25), (0, 1, 0.5, 1.0)])
def test_scaled_products_have_the_sums_of_the_bare_one(lib, cuda, pair_build, layout, in_type, out_type, alpha, beta):
    """What the header says of products scaled by alpha or beta, on a shape whose K is cut into pieces: the fp32 sums are
    those of the bare product, scaled once (alpha is a power of two, so that step is exact), and the option gemm_split = 0
    keeps K whole, with the bits of the pair kernel."""
    if not pair_build:
        pytest.skip("the single-CTA build never cuts K")
    import torch

    m, n, k = 264, 136, 2048
    g = torch.Generator(device=cuda).manual_seed(97)
    tin = torch.float16 if in_type == 0 else torch.float32
    sa, sb = ((m, k), (n, k)) if layout == "TN" else ((k, m), (k, n))
    A, B = (torch.randn(s, generator=g, device=cuda).to(tin) for s in (sa, sb))
    c0 = torch.randn((n, m), generator=g, device=cuda)

    def run(a, be, out=out_type, **opts):
        import contextlib
        C = c0.to(torch.float16 if out == 0 else torch.float32, copy=True)
        with contextlib.ExitStack() as es:
            for name, v in opts.items():
                es.enter_context(ops.option(name, v, lib))
            ops.gemm_ex(*layout, m, n, k, a, A, sa[1], B, sb[1], be, C, m, in_type=in_type, out_type=out, lib=lib)
        assert ops.device_status(lib)[0] == 0
        return C

    sums = run(1.0, 0.0, out=1)
    assert not torch.equal(sums, run(1.0, 0.0, out=1, gemm_split=0))  # K is cut
    got = run(alpha, beta)
    if beta == 0.0:
        assert torch.equal(got, (alpha * sums).to(got.dtype))
    else:  # one or two roundings of fp32
        want, terms = alpha * sums.double() + beta * c0.double(), (alpha * sums.double()).abs() + (beta * c0.double()).abs()
        assert bool(((got.double() - want).abs() <= 2.0 ** -23 * terms).all())
    assert torch.equal(run(alpha, beta, gemm_split=0), run(alpha, beta, small_tiles=0, gemm_split=0))


@pytest.mark.parametrize("k", [512, 2048])
def test_wide_groups_that_no_kernel_takes_stay_refused(lib, cuda, pair_build, k):
    """A group that is neither all of N nor a multiple or divisor of the N tile is refused whatever K is."""
    if not pair_build:
        pytest.skip("the single-CTA build has one route")
    import torch

    m, gs, b = 4000, 2056, 64
    n = 2 * gs
    X, W, R, C = (torch.zeros(s, dtype=torch.float16, device=cuda) for s in ((m, k), (n, k), (2 * b, k), (m, n)))
    with pytest.raises(ops.Error) as e:
        ops.oft_tn(m, n, k, X, k, W, k, R, k, C, n, group_size=gs, reconn_sz=b, lib=lib)
    assert e.value.code == ops.EUNSUPPORTED and "group_size" in e.value.message


def test_route_names_the_kernel_that_runs(lib, cuda, pair_build):
    """oft_plan reports small problems as fused_tmem (X.R formed per tile, no scratch), oft_route by their own name; both
    agree elsewhere, and rows of C off 16-byte boundaries count."""
    if not pair_build:
        pytest.skip("the single-CTA build has one route")
    assert ops.oft_plan(8, 4096, 4096, reconn_sz=64, lib=lib) == {"path": "fused_tmem", "kernel_launches": 1}
    assert ops.oft_route(8, 4096, 4096, reconn_sz=64, lib=lib) == "fused_small"
    with ops.option("small_tiles", 0, lib):
        assert ops.oft_route(8, 1024, 4096, reconn_sz=64, lib=lib) == "fused_tmem"
    for m, n, k, b, gs in ((16384, 4096, 4096, 64, None), (8192, 8192, 8192, 8, 256), (65536, 28672, 8192, 128, None), (6503, 7008, 512, 64, None)):
        assert ops.oft_route(m, n, k, group_size=gs, reconn_sz=b, lib=lib) == ops.oft_plan(m, n, k, group_size=gs, reconn_sz=b, lib=lib)["path"]
    assert ops.oft_route(16384, 4096, 4096, reconn_sz=64, c_aligned=False, lib=lib) == "two_pass"
    for route, name in ops.ROUTES.items():
        with ops.option("oft_route", route, lib):
            assert ops.oft_route(384, 2048, 512, reconn_sz=64, lib=lib) == name
    with pytest.raises(ops.Error) as e:
        ops.oft_route(8, 4096, 4100, reconn_sz=64, lib=lib)
    assert e.value.code == ops.EINVAL


@pytest.mark.parametrize("m,n,k,b", [(5000, 1473, 576, 64), (4000, 647, 1152, 128)])
def test_narrow_unaligned_products_are_captured_without_scratch(lib, cuda, pair_build, m, n, k, b):
    """Rows of C that are not 16-byte aligned, a narrow group: the rotation pass + GEMM outside of a capture, the kernel
    that needs no scratch inside (a graph with allocation nodes could be no child graph or conditional body); the same
    bits."""
    if not pair_build:
        pytest.skip("the single-CTA build has one route")
    import torch

    g = torch.Generator(device=cuda).manual_seed(99)
    X = torch.randn((m, k), generator=g, device=cuda).half()
    W = (torch.randn((n, k), generator=g, device=cuda) * 0.02).half()
    R = (torch.randn((b, k), generator=g, device=cuda) * 0.1).half()
    C = torch.zeros((m, n), dtype=torch.float16, device=cuda)

    def call():
        ops.oft_tn(m, n, k, X, k, W, k, R, k, C, n, torch.cuda.current_stream(), reconn_sz=b, lib=lib)

    call()
    torch.cuda.synchronize()
    want = C.clone()
    assert GRAPH_MEM_ALLOC not in graph_node_types(call)
    C.zero_()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    graph.replay()
    torch.cuda.synchronize()
    assert ops.device_status(lib)[0] == 0
    assert torch.equal(C.view(torch.int16), want.view(torch.int16))


def test_dependent_launch_behind_two_streams(lib, cuda, pair_build):
    """A product whose operands come from two streams joined by an event, run and captured: the launch that may start
    early waits for both producers."""
    if not pair_build:
        pytest.skip("the single-CTA build has no dependent launches")
    import torch

    m, n, k = 24, 1024, 1024
    g = torch.Generator(device=cuda).manual_seed(100)
    W0 = (torch.randn((n, k), generator=g, device=cuda) / 32).half()
    X0 = torch.randn((m, k), generator=g, device=cuda).half()
    big = torch.randn((4096, 4096), generator=g, device=cuda)
    want = torch.empty((m, n), dtype=torch.float16, device=cuda)
    ops.gemm_tn(n, m, k, W0, k, X0, k, want, n, lib=lib)
    torch.cuda.synchronize()
    W, X, C = torch.zeros_like(W0), torch.zeros_like(X0), torch.zeros_like(want)
    side, scratch = torch.cuda.Stream(), torch.zeros_like(big)

    def step():
        main = torch.cuda.current_stream()
        side.wait_stream(main)
        with torch.cuda.stream(side):
            for _ in range(3):
                torch.add(big, big, out=scratch)  # keeps the side stream busy in front of the copy
            W.copy_(W0)
        X.copy_(X0)
        main.wait_stream(side)
        ops.gemm_tn(n, m, k, W, k, X, k, C, n, main, lib=lib)

    def check():
        torch.cuda.synchronize()
        assert ops.device_status(lib)[0] == 0
        assert torch.equal(C, want)
        W.zero_(), X.zero_(), C.zero_()

    s = torch.cuda.Stream()
    for _ in range(3):
        with torch.cuda.stream(s):
            step()
        check()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    for _ in range(3):
        graph.replay()
        check()
