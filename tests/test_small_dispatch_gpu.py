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


@pytest.mark.parametrize("rows,columns,positions,shift", [
    ([1024], 1024, 1, 0), ([1024], 1024, 2, 0), ([256], 256, 8, 0), ([700], 512, 1, -300), ([40], 2048, 1, 2000), ([4096], 4096, 1, 0),
    ([18945], 1024, 1, -9000), ([512, 256, 100], 512, 2, 100)])
def test_outputs_over_the_activations(orc, rows, columns, positions, shift):
    """The first matrix writes where the activations lie (from `shift` values behind their start): launches whose CTAs read all of them
    and write outputs keep away from such calls, and only from those."""
    import torch
    be = ctox.B200Backend(0)
    s_in = synthetic.recovery_scales_f16(columns, 5, 1)
    ops = [ctox.FusedMatVec(Q4, synthetic.packed_weights(Q4, n, columns, i), n, columns, None, s_in=s_in,
                            s_out=synthetic.recovery_scales_f16(n, i, 2)) for i, n in enumerate(rows)]
    mats = [be.prepare_fused_matvec(op) for op in ops]
    x = synthetic.activations(columns, 3, positions=positions).reshape(positions, columns)
    stride = max(columns, rows[0])
    memory = torch.empty(positions * stride + 2 * abs(shift), device="cuda")
    x_at = abs(shift)
    others = [torch.empty(positions, n, device="cuda") for n in rows[1:]]
    apart = torch.empty(positions, stride, device="cuda")

    def dispatch(y_ptr):
        memory.zero_()
        memory[x_at:x_at + positions * stride].view(positions, stride)[:, :columns] = torch.from_numpy(x).cuda()
        torch.cuda.synchronize()
        before = be.kernel_launches()
        xp = memory.data_ptr() + 4 * x_at
        if len(mats) == 1:
            mats[0].dispatch_device(xp, ctox.F32, positions, stride, y_ptr, stride)
        else:
            be.fanout_dispatch_device(mats, xp, ctox.F32, positions, stride, [y_ptr] + [y.data_ptr() for y in others], [stride] + rows[1:])
        be.synchronize()
        return be.kernel_launches() - before

    want = []
    for op in ops:
        o = to_oracle_op(orc, op)
        want.append([])
        for m in range(positions):
            o.input = x[m]
            want[-1].append(orc.fused_matvec(o))
    closed = dispatch(apart.data_ptr()) == 1
    assert closed == (columns <= 2048 and rows[0] < 18945)
    over = x_at + shift
    for _ in range(20):
        assert dispatch(memory.data_ptr() + 4 * over) >= 2
        got = [memory[over:over + positions * stride].view(positions, stride).cpu().numpy()] + [y.cpu().numpy() for y in others]
        for w, n, y in zip(want, rows, got):
            for m in range(positions):
                assert rel_l2(y[m, :n], w[m]) <= 5e-5  # as above
    for m in mats:
        m.destroy()
    be.close()


@pytest.mark.parametrize("dtype,rows,columns,positions", [
    (Q4, 15000, 3584, 2), (Q4, 15000, 3584, 4), (Q2, 15000, 3584, 4), (Q2, 17408, 4096, 1), (Q2, 24000, 4096, 1), (Q4, 5120, 17408, 3)])
def test_either_side_of_the_eight_warp_form(orc, dtype, rows, columns, positions):
    """Dispatches of one matrix with eight warps per CTA and, beyond a work per warp that depends on the positions, with sixteen."""
    test_outputs(orc, dtype, [rows], columns, positions)
