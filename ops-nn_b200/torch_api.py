"""torch-tensor entry points with the signatures of the torch-npu plugin functions that sit on top of these operators in the
reference's stack (`torch_npu.npu_quant_matmul`, `torch_npu.npu_weight_quant_batchmatmul`; call forms as exercised by
matmul/weight_quant_batch_matmul_v2/tests/assets/wqbmmv2_e2e_golden.py:196-275 of the reference). They take CUDA tensors,
allocate the output and the workspace from torch's allocator, and run the aclnn two-phase call on the current stream. Transposed weights
are passed the torch way, as `.t()` views: the library reads the strides, nothing is copied."""
from . import aclnn as _aclnn


def _torch():
    import torch

    return torch


def npu_quant_matmul(x1, x2, scale, *, offset=None, pertoken_scale=None, bias=None, output_dtype=None, group_sizes=None,
                     x1_dtype=None, x2_dtype=None, scale_dtype=None, pertoken_scale_dtype=None):
    """aclnnQuantMatmulV5 behind the torch-npu signature. x1 (.., m, k), x2 (.., k, n) (or a transposed view of (n, k));
    `scale` is x2's scale (per-tensor/-channel, per-block, or e8m0), `pertoken_scale` x1's; `group_sizes` = [gm, gn, gk].
    `x1_dtype` / `x2_dtype` / `scale_dtype` / `pertoken_scale_dtype` name the element type of tensors torch cannot type itself
    (e.g. "float4_e2m1" over uint8 storage, "float8_e8m0" scales); the logical last dim of a 4-bit tensor is twice its
    storage. output_dtype defaults to torch.int8 like the plugin (requantised output needs a packed int64 scale)."""
    group = 0
    if group_sizes is not None:
        gm, gn, gk = (list(group_sizes) + [0, 0, 0])[:3]
        group = (int(gm) << 32) | (int(gn) << 16) | int(gk)
    if output_dtype is None:
        output_dtype = _torch().int8
    return _aclnn.native().npu_quant_matmul(x1, x2, scale, offset, pertoken_scale, bias, output_dtype, group, x1_dtype, x2_dtype, scale_dtype,
                                            pertoken_scale_dtype)


def npu_weight_quant_batchmatmul(x, weight, antiquant_scale, antiquant_offset=None, quant_scale=None, quant_offset=None,
                                 bias=None, antiquant_group_size=0, inner_precise=0, weight_dtype=None):
    """aclnnWeightQuantBatchMatmulV3 behind the torch-npu signature. x (m, k) bf16/fp16; weight (k, n) int8, or int32 words of
    eight int4 values (k, n / 8), or a `.t()` view of the (n, k) storage; scale/offset (n,), (1, n) or (k / group, n).
    quant_scale / quant_offset (int8 output) are not implemented and must be None."""
    if quant_scale is not None or quant_offset is not None:
        raise NotImplementedError("quant_scale / quant_offset (int8 output) are not implemented")
    return _aclnn.native().npu_weight_quant_batchmatmul(x, weight, antiquant_scale, antiquant_offset, bias, antiquant_group_size, inner_precise,
                                                        weight_dtype)
