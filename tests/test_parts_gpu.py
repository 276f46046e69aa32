"""Parts of one product (row chunks, slabs of N, several destinations) have the bits of a single call on the whole of it,
also where the library cuts K into pieces: it then does so by the whole product's sizes."""
import types

import numpy as np
import pytest

from _util import GRAPH_KERNEL, GRAPH_MEMCPY, graph_node_types, make_oft_case
from cute_mma_b200 import ops, sharded

pytestmark = pytest.mark.gpu


def _operands(cuda, m, n, k, b, gs, seed):
    import torch

    A, R, B = make_oft_case(m, n, k, b, gs, seed=seed, xdist="normal", wsigma=0.05)
    return (A, R, B), tuple(torch.from_numpy(x).to(cuda) for x in (A, R, B))


def _whole(lib, cuda, dA, dR, dB, m, n, k, b, gs, ldc=None):
    import torch

    C = torch.empty((m, ldc or n), dtype=torch.float16, device=cuda)
    ops.oft_tn(m, n, k, dA, k, dB, k, dR, k, C, ldc or n, group_size=gs, reconn_sz=b, lib=lib)
    assert ops.device_status(lib)[0] == 0
    return C[:, :n].contiguous().view(torch.int16)


# K long enough to be cut: the whole in one piece and its parts in several, the other way round, groups of which only a
# slab is one group of its own width, unaligned rows of C
CASES = [(4096, 512, 4096, 64, None), (1024, 1024, 2048, 128, None), (300, 1536, 1280, 32, 256), (128, 512, 1024, 16, 64), (2304, 509, 1024, 8, None)]


@pytest.mark.parametrize("m,n,k,b,gs", CASES)
def test_slabs_and_row_chunks_have_the_bits_of_the_whole(lib, cuda, pair_build, m, n, k, b, gs):
    if not pair_build:
        pytest.skip("the single-CTA build never cuts K")
    import torch

    _, (dA, dR, dB) = _operands(cuda, m, n, k, b, gs, 101)
    want = _whole(lib, cuda, dA, dR, dB, m, n, k, b, gs)
    g = n if gs is None else gs
    for world in (2, 8):
        got = torch.empty((m, n), dtype=torch.float16, device=cuda)
        for r in range(world):
            n0, n1 = ops.shard_range(n, g, world, r, lib=lib)
            R_slab = dR if gs is None else dR[n0 // g * b:]
            sharded.oft_tn_slab(m, n, k, dA, k, dB[n0:], k, R_slab, k, got[:, n0:], n, n0, n1, group_size=gs, reconn_sz=b, lib=lib)
        assert ops.device_status(lib)[0] == 0
        assert torch.equal(got.view(torch.int16), want), world
    Bs, Rs, Cs, got = [], [], [], torch.empty((m, n), dtype=torch.float16, device=cuda)
    for r in range(3):  # the C entry point for several devices, every slab on this one
        n0, _ = ops.shard_range(n, g, 3, r, lib=lib)
        Bs.append(dB[n0:]); Cs.append(got[:, n0:]); Rs.append(dR if gs is None else dR[n0 // g * b:])
    ops.oft_tn_sharded(m, n, k, [0] * 3, [dA] * 3, k, Bs, k, Rs, k, Cs, n, group_size=gs, reconn_sz=b, lib=lib)
    assert ops.device_status(lib)[0] == 0
    assert torch.equal(got.view(torch.int16), want)


@pytest.mark.parametrize("m,n,k,b,gs", CASES)
def test_host_paths_have_the_bits_of_the_whole(lib, cuda, pair_build, m, n, k, b, gs):
    """The C entry point on host buffers (2048 rows a chunk) and HostSlabRunner (eight chunks) on one rank."""
    if not pair_build:
        pytest.skip("the single-CTA build never cuts K")
    import torch

    (A, R, B), (dA, dR, dB) = _operands(cuda, m, n, k, b, gs, 102)
    want = _whole(lib, cuda, dA, dR, dB, m, n, k, b, gs).cpu().numpy()
    hC = np.zeros((m, n), np.float16)
    ops.oft_tn_host(m, n, k, A, k, B, k, R, k, hC, n, group_size=gs, reconn_sz=b, lib=lib)
    assert np.array_equal(hC.view(np.int16), want)
    runner = sharded.HostSlabRunner(m, n, k, 0, n, group_size=gs, reconn_sz=b, world=1, rank=0, device=cuda, lib=lib)
    hY = torch.zeros((m, n), dtype=torch.float16)
    runner(torch.from_numpy(A), torch.from_numpy(B), torch.from_numpy(R), hY)
    assert ops.device_status(lib)[0] == 0
    assert np.array_equal(hY.numpy().view(np.int16), want)


@pytest.mark.parametrize("mode", ["copy_engines", "stores"])
def test_slab_with_overlapped_all_gather_has_the_bits_of_the_whole(lib, cuda, pair_build, mode):
    """SlabProductAllGather as rank 1 of 2 with the peer's buffer on this GPU (its constructor, which maps real peers,
    left out)."""
    if not pair_build:
        pytest.skip("the single-CTA build never cuts K")
    import torch

    m, n, k, b = 1024, 1024, 2048, 64
    _, (dA, dR, dB) = _operands(cuda, m, n, k, b, None, 103)
    want = _whole(lib, cuda, dA, dR, dB, m, n, k, b, None)
    ag = object.__new__(sharded.SlabProductAllGather)
    mine, peer = (torch.zeros((2, m, n // 2), dtype=torch.float16, device=cuda) for _ in range(2))
    ag.torch, ag.dist = torch, types.SimpleNamespace(barrier=lambda: None)
    ag.mode, ag.world, ag.rank = mode, 2, 1
    ag.m, ag.n_total, ag.k, ag.n_loc, ag.b, ag.lib, ag.device = m, n, k, n // 2, b, lib, torch.device("cuda", 0)
    ag.y_all, ag.peer_views = mine, [peer, mine]
    ag.copy_streams, ag.chunk_rows = [torch.cuda.Stream()], 256
    ag(dA, dB[n // 2:], dR)
    assert ops.device_status(lib)[0] == 0
    for buf in (mine, peer):
        assert torch.equal(buf[1].view(torch.int16), want[:, n // 2:]) and not bool(buf[0].any())


# wide group of few rows, K cut / whole; narrow; odd ldC and an 8-byte base that not every destination has
@pytest.mark.parametrize("m,n,k,b,gs,pad", [(16, 4096, 4096, 64, None, 0), (16, 2304, 320, 32, None, 8), (200, 640, 1024, 128, None, 8), (130, 2055, 1088, 16, None, 3),
                                            (33, 512, 1024, 8, 256, 0)])
def test_small_gather_is_one_launch_with_the_bits_of_the_plain_call(lib, cuda, pair_build, m, n, k, b, gs, pad):
    """Small problems store to all destinations from the kernel, as the wide groups of the shared-X.R kernel do: no copy
    follows the launch."""
    if not pair_build:
        pytest.skip("the single-CTA build copies")
    import torch

    _, (dA, dR, dB) = _operands(cuda, m, n, k, b, gs, 104)
    want = _whole(lib, cuda, dA, dR, dB, m, n, k, b, gs)
    ldc = n + pad
    for shift in (0, 2):  # elements by which the second destination's base is off a 16-byte boundary
        bufs = [torch.full(((m + 1) * ldc + 2,), -7.0, dtype=torch.float16, device=cuda) for _ in range(3)]
        dsts = [x.data_ptr() + (2 * shift if i == 1 else 0) for i, x in enumerate(bufs)]

        def call():
            ops.oft_tn_gather(m, n, k, dA, k, dB, k, dR, k, dsts, ldc, torch.cuda.current_stream(), group_size=gs, reconn_sz=b, lib=lib)

        call()
        assert ops.device_status(lib)[0] == 0
        for i, x in enumerate(bufs):
            off = shift if i == 1 else 0
            rows = x[off: off + (m + 1) * ldc].view(m + 1, ldc)
            assert torch.equal(rows[:m, :n].contiguous().view(torch.int16), want), (shift, i)
            assert bool((rows[m] == -7.0).all()) and bool((rows[:m, n:] == -7.0).all()) and bool((x[:off] == -7.0).all())
        kinds = graph_node_types(call)
        assert GRAPH_MEMCPY not in kinds and kinds.count(GRAPH_KERNEL) == (2 if b == 8 else 1)  # 8 x 8 blocks: R is expanded first
