"""Forward of CLUSTENWF in 16 bits on either side of the line between its two kernels (csrc/wf_direct.cu): m * ic up to 96 with 64 channels, up to 48 with
more, and 32 merge rows per SM (74 x 64 on 148 SMs)."""
import pytest
import torch

import workloads
from helpers import TOL, rel_err
from oracle import formula

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bfloat16", "float16"])
@pytest.mark.parametrize("kind", ["model", "outside"])
@pytest.mark.parametrize("n_out", [63, 64, 65])
@pytest.mark.parametrize("m,ic,c", [(48, 1, 64), (48, 1, 128), (40, 1, 192), (48, 2, 64), (48, 2, 128), (24, 2, 128), (24, 4, 64), (24, 4, 128), (48, 4, 64),
                                    (13, 4, 64), (13, 4, 128), (1, 1, 64)])
def test_either_side(lib, m, ic, c, n_out, kind, dtype):
    from clusten import ops
    b, n = 74, 203
    if kind == "model":
        idx = workloads.select_rows(workloads.make_index("model" if m % 8 == 0 else "shared", b, n, m, 20, DEV), n_out, 21)
    else:
        idx = torch.randint(-3, n + 3, (b, n_out, m), generator=torch.Generator(device=DEV).manual_seed(22), device=DEV)
    w, feat, _ = workloads.merge_operands(b, n_out, n, m, ic, c, dtype, 23, DEV)
    got, stored = ops.wf_forward(w, feat, idx), ops.wf_forward(w, feat, idx, row_order=False)
    assert got.shape == (b, n_out, ic, c) and torch.equal(got, stored)
    for e in (0, 40, b - 1):
        one = slice(e, e + 1)
        ok = ((idx[one] >= 0) & (idx[one] < n)).double().unsqueeze(3)     # an index outside contributes nothing
        assert rel_err(got[one], formula.wf(w[one].double() * ok, feat[one].double(), idx[one].clamp(0, n - 1))) <= TOL[dtype]
