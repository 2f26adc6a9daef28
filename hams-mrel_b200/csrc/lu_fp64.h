// lu_fp64.h -- complex128 LU and solve of the plain form (lu_fp64.cu).
#pragma once
#include <cublas_v2.h>
#include <cuda_runtime.h>

// Most rows whose panels the factorisation can hold (16 blocks of a cluster, a
// row per thread); larger systems are the caller's to factor otherwise.
constexpr int kZluMaxRows = 16 * 512;

// Ints of workspace zlu_solve needs.
size_t zlu_work_ints();

// 0 if device dev can run the factorisation of order n.
int zlu_supported(int n);

// X (n x nrhs, ld n) <- A^-1 X; A (n x n, ld n) is overwritten by its factors
// (partial pivoting in 16-column panels, rows ordered by pivot).  info[0]
// receives 1 + the first column with a zero pivot, or stays at 0.  evf, if not
// null, is recorded after the last column is factored (the forward substitution
// is part of the factorisation).  Returns 0, 1 on a CUDA error, or 10 + a
// cuBLAS status.
int zlu_solve(cudaStream_t st, cublasHandle_t blas, int n, int nrhs, double2* A, double2* X, int* info, int* work,
              cudaEvent_t evf, long long* launches, long long* lib_calls);
