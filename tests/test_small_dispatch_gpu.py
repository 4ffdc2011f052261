"""Dispatches whose CTAs take whole row pairs and write the outputs themselves, at the edges of what they take: column slices of 1 to 8
super-tiles, ragged rows, as many CTAs as SMs and one more (which takes the split over all warps), several positions, fan-outs."""
import numpy as np
import pytest

import ctox_llm_b200 as ctox
from ctox_llm_b200 import synthetic
from gpu_util import rel_l2, to_oracle_op

pytestmark = pytest.mark.gpu
Q2, Q4 = ctox.Q2B64, ctox.Q4B64


@pytest.mark.parametrize("dtype,rows,columns,positions", [
    (Q4, [1024], 1024, 1), (Q2, [33], 64, 1), (Q4, [1], 256, 8), (Q2, [300], 320, 4), (Q4, [161], 768, 2), (Q2, [95], 1280, 1),
    (Q4, [64], 1536, 1), (Q2, [129], 2048, 1), (Q4, [130], 512, 4), (Q2, [18944], 1024, 1), (Q2, [18945], 1024, 1),
    (Q4, [512, 31, 100], 512, 3), (Q2, [40, 700, 1, 65], 1024, 2), (Q4, [300, 300], 2304, 1)])
def test_outputs(orc, dtype, rows, columns, positions):
    import torch
    be = ctox.B200Backend(0)
    s_in = synthetic.recovery_scales_f16(columns, 5, 1)
    ops = [ctox.FusedMatVec(dtype, synthetic.packed_weights(dtype, n, columns, i), n, columns, None, s_in=s_in,
                            s_out=synthetic.recovery_scales_f16(n, i, 2), bias=synthetic.bias(n, i),
                            activation=ctox.ACT_SILU if i % 2 else ctox.ACT_IDENTITY) for i, n in enumerate(rows)]
    mats = [be.prepare_fused_matvec(op) for op in ops]
    x = synthetic.activations(columns, 3, positions=positions).reshape(positions, columns)
    xd = torch.from_numpy(x).cuda()
    ys = [torch.full((positions, n + 3), -7.0, device="cuda") for n in rows]  # a stride of its own
    torch.cuda.synchronize()
    if len(mats) == 1:
        mats[0].dispatch_device(xd.data_ptr(), ctox.F32, positions, columns, ys[0].data_ptr(), rows[0] + 3)
    else:
        be.fanout_dispatch_device(mats, xd.data_ptr(), ctox.F32, positions, columns, [y.data_ptr() for y in ys], [n + 3 for n in rows])
    be.synchronize()
    for op, n, y in zip(ops, rows, ys):
        y = y.cpu().numpy()
        assert np.all(y[:, n:] == -7.0)
        for m in range(positions):
            o = to_oracle_op(orc, op)
            o.input = x[m]
            assert rel_l2(y[m, :n], orc.fused_matvec(o)) <= 5e-5  # the bound of test_matvec_gpu.py
    for m in mats:
        m.destroy()
    assert be.allocated_bytes() == 0
    be.close()
