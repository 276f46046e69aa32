"""The plain GEMM's choice between its kernels, by time, where a rule that counts too little picks the slower one: the library's
choice against the kernels that the rule decides between, forced, in turns."""
import contextlib

import pytest

torch = pytest.importorskip("torch")

from cute_mma_b200 import ops  # noqa: E402
from test_beta_gpu import KERNELS, operands, product, us  # noqa: E402

pytestmark = pytest.mark.gpu


# narrow tiles of many K steps, whose 128 rows cost as much as their columns
@pytest.mark.parametrize("m,n,k,kind,layout", [(7016, 272, 2536, "half-half", "TN"), (12601, 169, 2532, "half-float", "TN"), (33475, 147, 2919, "half-half", "TN"),
                                               (11929, 175, 5739, "half-half", "TN"), (15189, 145, 2601, "float-float", "NT")])
def test_choice_is_the_faster_kernel(lib, pair_build, m, n, k, kind, layout):
    """Within 6 % of the fastest; one kernel's best times of two sets of runs differ by up to 2 %."""
    if not pair_build:
        pytest.skip("the single-CTA build has one kernel")
    t_in, t_out = (torch.float16 if t == "half" else torch.float32 for t in kind.split("-"))
    A, B = operands(m, n, k, layout, t_in, 1)
    C = torch.zeros((n, m), device="cuda", dtype=t_out)
    best = {}
    for _ in range(3):
        for name, forced in {"choice": {}, "small": KERNELS["small"], "pair": KERNELS["pair"]}.items():
            with contextlib.ExitStack() as options:
                for option, value in forced.items():
                    options.enter_context(ops.option(option, value, lib))
                best[name] = min(best.get(name, 1e30), us(lambda: product(lib, layout, m, n, k, 1.0, A, B, 0.0, C)))
    assert best["choice"] <= 1.06 * min(best.values()), best
