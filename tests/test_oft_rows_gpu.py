"""Row-major stores of the fused OFT kernels when rows of C are not 16-byte aligned: every parity of base, leading
dimension and width, against the aligned stores of the same kernel, bit for bit."""
import numpy as np
import pytest

from _util import make_oft_case
from cute_mma_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("route,b,gs", [(1, 64, None), (1, 16, 128), (1, 128, None), (3, 64, None), (3, 128, None)])
@pytest.mark.parametrize("m,n,pad,shift", [(300, 512, 1, 0), (300, 512, 2, 1), (129, 512, 4, 3), (300, 511, 0, 0), (33, 577, 0, 1), (257, 258, 3, 0), (65, 319, 2, 2)])
def test_unaligned_rows_of_c(lib, cuda, pair_build, route, b, gs, m, n, pad, shift):
    if not pair_build:
        pytest.skip("the single-CTA build stores one row per lane")
    import torch

    if gs is not None:
        n = (n + gs - 1) // gs * gs
    k = 256
    A, R, B = make_oft_case(m, n, k, b, gs, seed=95, xdist="normal", wsigma=0.05)
    dA, dB, dR = (torch.from_numpy(x).to(cuda) for x in (A, B, R))

    def run(ldc, shift):
        buf = torch.full(((m + 1) * ldc + shift,), -7.0, dtype=torch.float16, device=cuda)
        with ops.option("oft_route", route, lib):
            ops.oft_tn(m, n, k, dA, k, dB, k, dR, k, buf.data_ptr() + 2 * shift, ldc, group_size=gs, reconn_sz=b, lib=lib)
        assert ops.device_status(lib)[0] == 0
        out = buf.cpu().numpy()
        rows = out[shift:].reshape(m + 1, ldc)
        assert np.all(out[:shift] == -7.0) and np.all(rows[m] == -7.0) and np.all(rows[:m, n:] == -7.0)
        return rows[:m, :n].copy()

    want = run((n + 7) // 8 * 8, 0)
    assert np.array_equal(run(n + pad, shift).view(np.uint16), want.view(np.uint16))
