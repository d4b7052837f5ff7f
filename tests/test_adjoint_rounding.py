"""The parameter gradients divide and take roots with correct rounding, as the
projection they are the adjoint of does: the gradient kernels' source uses no
hardware estimate in place of them."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ESTIMATES = r"\.approx|\brsqrtf\b|__fdividef|__fsqrt_r[^n]|__frcp_r[^n]|__expf|__logf"


def test_no_estimates_in_the_gradient_kernels():
    with open(os.path.join(ROOT, "rustscan_b200", "csrc", "k_backward.cu")) as fh:
        code = re.sub(r"//[^\n]*", "", fh.read())
    assert not re.findall(ESTIMATES, code)
