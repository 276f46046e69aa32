import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); run with -m gpu")


@pytest.fixture(scope="session")
def lib():
    """The CUDA library through the C ABI.  Built in-tree; never falls back to anything else."""
    from cute_mma_b200 import build, ops

    build.build()
    return ops.load_library()


@pytest.fixture(scope="session")
def cuda():
    import torch

    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    torch.cuda.set_device(0)
    return torch.device("cuda:0")


@pytest.fixture(scope="session")
def pair_build(lib):
    """True when the library was built with CTA pairs (ctas = 2, the default); a few features exist only there."""
    from cute_mma_b200 import ops

    return ops.kernel_info(lib)["oft"]["ctas"] == 2


@pytest.fixture(params=[-1, 0], ids=["chosen", "no_small_kernel"])
def small_tiles(request, lib):
    """The library's own choice of kernel, then the same test without the kernel for small problems, which otherwise takes
    almost every shape a test can afford."""
    from cute_mma_b200 import ops

    with ops.option("small_tiles", request.param, lib):
        yield request.param


@pytest.fixture(autouse=True)
def room_in_the_tensor_cache(request):
    """test_zz_no_alloc compares the driver's free memory around calls that also clone a 1 MB tensor: torch's cache must
    hold room for it whatever ran before, or the difference it sees is torch's own new segment."""
    if request.module.__name__ == "test_zz_no_alloc":
        import torch

        spare = [torch.empty(1 << 20, dtype=torch.uint8, device="cuda") for _ in range(16)]
        del spare
    yield
