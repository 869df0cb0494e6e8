"""Two-SM work items of at most 128 token rows, whose pipeline has nine stages instead of six: the longest list decides."""
import pytest

from tests import test_gpu_pair_items as pair_items

pytestmark = pytest.mark.gpu

SHORT = [128, 1, 96, 127, 65, 33, 128, 64, 97, 128, 2, 126]
LONGEST_129 = SHORT[:-1] + [129]
FEW = [128]


@pytest.mark.parametrize("rows", [SHORT, LONGEST_129, FEW], ids=["short", "one-row-more", "one-item"])
@pytest.mark.parametrize("kind", ["w8a8", "w8a16", "bf16"])
def test_against_one_sm_kernel(cuda_device, kind, rows):
    pair_items.test_against_one_sm_kernel(cuda_device, kind, rows)
