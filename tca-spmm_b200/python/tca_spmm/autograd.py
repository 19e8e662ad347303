"""torch.autograd wrapper of the SpMM and its adjoints -- a gradient harness.

    Y = spmm(plan, vals, B)

computes Y = A B with A the plan's sparsity pattern carrying `vals` (one
value per nonzero, in the CSR order the plan was built from). Backward:
    d vals = SDDMM(dY, B) on A's pattern   (tca_sddmm)
    d B    = A^T dY                         (tca_spmm_t)
Both accumulate in FP32; dY is rounded to FP16 (the kernels' input type)."""
from __future__ import annotations

import torch

from . import Plan


class SpMMFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, vals, B, plan: Plan, out_dtype):
        v16 = vals.detach().to(torch.float16).contiguous()
        B16 = B.detach().to(torch.float16).contiguous()
        plan.update_values(v16)
        ctx.values_version = plan.values_version()
        Y = plan.spmm(B16, out_dtype=out_dtype)
        ctx.plan = plan
        ctx.save_for_backward(v16, B16)
        ctx.vals_dtype, ctx.B_dtype = vals.dtype, B.dtype
        return Y

    @staticmethod
    def backward(ctx, dY):
        v16, B16 = ctx.saved_tensors
        plan = ctx.plan
        dY16 = dY.to(torch.float16).contiguous()
        d_vals = d_B = None
        # the pattern's values as they were in forward: another forward may have
        # replaced them, or may before a capture of this backward is replayed
        if ctx.needs_input_grad[1] and (ctx.values_version == 0 or plan.values_version() != ctx.values_version or
                                        torch.cuda.is_current_stream_capturing()):
            plan.update_values(v16)
        # gradients in the inputs' types: FP32 sums, rounded once by the kernel that forms them
        direct = (torch.float16, torch.float32)
        if ctx.needs_input_grad[0]:
            out = ctx.vals_dtype if ctx.vals_dtype in direct else torch.float32
            d_vals = plan.sddmm(dY16, B16, out_dtype=out).to(ctx.vals_dtype)
        if ctx.needs_input_grad[1]:
            out = ctx.B_dtype if ctx.B_dtype in direct else torch.float32
            d_B = plan.spmm_t(dY16, out_dtype=out).to(ctx.B_dtype)
        return d_vals, d_B, None, None


def spmm(plan: Plan, vals, B, out_dtype=torch.float32):
    """Differentiable Y = A(vals) @ B on the plan's pattern."""
    return SpMMFunction.apply(vals, B, plan, out_dtype)
