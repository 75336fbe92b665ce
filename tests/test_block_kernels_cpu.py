"""What the block kernels refuse, as far as that can be seen without a GPU."""
import re

import pytest
import torch

from polyrl_b200.ops import build
from polyrl_b200.ops import functional as OF


@pytest.mark.parametrize("blk,off", [(5, 0), (-6, 0), (0, 4), (0, -5)])
def test_gather_outside_the_cache(blk, off):
    """The general path raises.  The kernel fails an assertion, which ends the process's context: it is only looked for in the source."""
    kc = torch.zeros(5, 2, 4, 8)
    with pytest.raises(IndexError):
        OF.gather_cached(kc, kc, torch.tensor([0, blk]), torch.tensor([1, off]))
    body = (build.CSRC / "elementwise.cu").read_text().split("gather_pages_kernel(", 1)[1].split("\n}\n", 1)[0]
    guard, loads = body.index("assert(b >= 0 && b < pages && o >= 0 && o < page"), body.index("ld_nc_v4(kc")
    assert guard < loads and not any(re.search("NDEBUG", f) for f in build.NVCC_FLAGS)
