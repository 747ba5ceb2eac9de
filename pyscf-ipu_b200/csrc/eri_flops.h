// Generated by eri_flops_count.cu from eri_su.cuh: arithmetic of one primitive quartet of the
// float32 ERI kernels per class (bra slice type, ket pair type) = (0,0) (0,1) (1,1) (0,2) (1,2) (2,2)
// (flops: +, -, *, /; special: sqrt, exp, erf, reciprocal square root), and of the ket's polynomial
// per bra slice and ket primitive, constants folded as the compiler folds them.
#pragma once
static const int B2_ERI_FLOPS[6] = {22, 46, 118, 77, 243, 372};
static const int B2_ERI_SPECIAL[6] = {3, 2, 2, 2, 2, 2};
static const int B2_ERI_KET_FLOPS[6] = {1, 13, 52, 94, 376, 376};
