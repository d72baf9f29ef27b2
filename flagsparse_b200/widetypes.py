"""float16, bfloat16, complex64 and complex128 values: operands of the kernels that take them.

The reference's base paths take these four value types by computing in a wider real type and casting back:
half precisions run its float32 kernel on `data.to(float32)` and `x.to(float32)` and round the result
(src/flagsparse/sparse_operations/spmv_csr.py:496-535, spmm_csr.py:525-560 of the reference), complex values run a
kernel over the interleaved real view (spmv_csr.py:123-155, 536-554; spmm_csr.py:138-195).  On the GPU the entry points
hand matrix and dense operand to fsb_spmv_csr_stored / fsb_spmm_csr_stored as they are (2 bytes per half-precision
value, interleaved pairs for complex values; sums in float32, one rounding).  `dense_dtype` is the type that the C entry
points fsb_spmv_csr_wide / fsb_spmm_csr_wide take their dense operand and result in: float32 for the half precisions
(the caller widens the one and rounds the other), the caller's type for complex values.
"""

import torch

HALF_DTYPES = (torch.float16, torch.bfloat16)
COMPLEX_DTYPES = (torch.complex64, torch.complex128)
WIDE_DTYPES = HALF_DTYPES + COMPLEX_DTYPES


def dense_dtype(dtype):
    """Type of the dense operand and of the result as the kernel sees them, for matrix values of `dtype`."""
    if dtype in HALF_DTYPES:
        return torch.float32
    if dtype in COMPLEX_DTYPES:
        return dtype
    raise TypeError(f"{dtype} has kernels of its own")
