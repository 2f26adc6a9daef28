// lu_fp64.h -- complex128 LU and solve of the plain form (lu_fp64.cu).
#pragma once
#include <cublas_v2.h>
#include <cuda_runtime.h>

// Most rows whose panels the factorisation can hold (16 blocks of a cluster, a
// row per thread); larger systems are the caller's to factor otherwise.
constexpr int kZluMaxRows = 16 * 512;

// Ints of workspace zlu_solve needs for batch systems.
size_t zlu_work_ints(int batch);

// 0 if the current device can run the factorisation of order n.
int zlu_supported(int n);

// X (n x nrhs, ld n) <- A^-1 X for batch systems of order n, sa and sx elements
// apart (at most 65,535); A (n x n, ld n) is overwritten by its factors (partial pivoting
// in 16-column panels, rows ordered by pivot).  info[0] receives 1 + a column
// with a zero pivot, the first one of a single system, or stays at 0.  evf, if
// not null, is recorded after the last column is factored (the forward
// substitution is part of the factorisation).  Returns 0, 1 on a CUDA error (left as
// the thread's last error), or 10 + a cuBLAS status.
int zlu_solve(cudaStream_t st, cublasHandle_t blas, int batch, int n, int nrhs, double2* A, size_t sa, double2* X,
              size_t sx, int* info, int* work, cudaEvent_t evf, long long* launches, long long* lib_calls);
