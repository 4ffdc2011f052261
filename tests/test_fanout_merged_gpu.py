"""Fan-outs whose matrices share a launch, and dispatches that form their own fragments, against one dispatch per matrix."""
import numpy as np
import pytest
import torch

import ctox_llm_b200 as ctox
from ctox_llm_b200 import native as N
from ctox_llm_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [ctox.Q4B64, ctox.Q2B64])
@pytest.mark.parametrize("columns", [64, 320, 1024, 2112, 5120])
@pytest.mark.parametrize("rows", [(33,), (1024, 64, 64), (700, 5000), (2048, 31, 400, 128), (300, 200, 100, 64, 50)])
def test_fanout_equals_single_dispatches(rows, columns, dtype):
    """One, two, four and more than four matrices, tiny ones among them (fewer units than warps); 1, 4, 5, 8 and 16 positions;
    the input at an odd offset, so that its rows cannot be read four values at a time. Only the order in which pieces of a
    32-bit sum are added differs: 2e-6 of the row's norm."""
    be = ctox.B200Backend(0)
    s_in = synthetic.recovery_scales_f16(columns, 3, 1)
    mats = [be.prepare_fused_matvec(ctox.FusedMatVec(dtype, synthetic.packed_weights(dtype, r, columns, 5 + i), r, columns, None, s_in=s_in,
                                                     s_out=synthetic.recovery_scales_f16(r, 9, i))) for i, r in enumerate(rows)]
    g = torch.Generator(device="cuda").manual_seed(columns)
    for positions, offset, kind in ((1, 0, torch.float32), (4, 1, torch.bfloat16), (5, 0, torch.bfloat16), (8, 1, torch.float32), (16, 0, torch.float32)):
        flat = torch.randn(positions * columns + 8, device="cuda", generator=g).to(kind)
        x = flat[offset:offset + positions * columns]
        code = N.F32 if kind == torch.float32 else N.BF16
        together = [torch.zeros(positions, r, device="cuda") for r in rows]
        alone = [torch.zeros(positions, r, device="cuda") for r in rows]
        torch.cuda.synchronize()
        be.fanout_dispatch_device(mats, x.data_ptr(), code, positions, columns, [y.data_ptr() for y in together], list(rows))
        for m, y, r in zip(mats, alone, rows):
            m.dispatch_device(x.data_ptr(), code, positions, columns, y.data_ptr(), r)
        torch.cuda.synchronize()
        for a, b in zip(together, alone):
            a, b = a.double().cpu().numpy(), b.double().cpu().numpy()
            assert b.any() and np.all(np.linalg.norm(a - b, axis=1) <= 2e-6 * np.linalg.norm(b, axis=1))
    be.close()
