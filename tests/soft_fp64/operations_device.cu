// Applies an operation of operations.h to n pairs on the device (tests/test_soft_operations.py).
#include <cuda_runtime.h>

#include "operations.h"

static __global__ void apply(int op, const double *a, const double *b, double *out, unsigned char *left, long long n) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    bool l;
    out[i] = soft_cases::operation(op, a[i], b[i], l);
    left[i] = l;
}

// Device pointers; 0 or a CUDA error.
extern "C" int soft_operations_device(int op, const double *a, const double *b, double *out, unsigned char *left,
                                      long long n) {
    apply<<<(unsigned)((n + 255) / 256), 256>>>(op, a, b, out, left, n);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
