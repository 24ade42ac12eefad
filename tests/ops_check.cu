// Device evaluation of single operations of the library's arithmetic headers
// for tests/test_gpu_ops.py: operand rows in, result rows out, beside the
// compiler's own operations where a comparison needs them.
#include "adjoint_math.h"
#include "euler_math.cuh"

#include <cuda_runtime.h>

namespace {

struct Arcp {  // 1/b and the compiler's
    static constexpr int in = 1, out = 2;
    static __device__ void f(const double *x, double *r)
    {
        r[0] = cfd::adj::arcp(x[0]);
        r[1] = 1.0 / x[0];
    }
};
struct Asqrt {
    static constexpr int in = 1, out = 2;
    static __device__ void f(const double *x, double *r)
    {
        r[0] = cfd::adj::asqrt(x[0]);
        r[1] = sqrt(x[0]);
    }
};
struct Wcns5Adj {  // five stencil values and the result's adjoint
    static constexpr int in = 6, out = 5;
    static __device__ void f(const double *x, double *r)
    {
        for (int i = 0; i < 5; i++) r[i] = 0.0;
        cfd::adj::wcns5_adj(x, x[5], r);
    }
};
struct FaceVjp {  // six cells' cons and the adjoint of the flux, along x
    static constexpr int in = 28, out = 24;
    static __device__ void f(const double *x, double *r)
    {
        double U[6][4], Ub[6][4] = {};
        for (int j = 0; j < 24; j++) U[j / 4][j % 4] = x[j];
        cfd::adj::face_vjp<0>(U, x + 24, Ub);
        for (int j = 0; j < 24; j++) r[j] = Ub[j / 4][j % 4];
    }
};

// operands a and b, b > 0: branch-free a/b, 1/b, sqrt(b), each followed by
// whether it was taken and by the compiler's
struct Spec {
    static constexpr int in = 2, out = 9;
    static __device__ void f(const double *x, double *r)
    {
        cfd::OpsSpec q, y, s;
        r[0] = q.div(x[0], x[1]);
        r[1] = q.ok;
        r[2] = x[0] / x[1];
        r[3] = y.rcp(x[1]);
        r[4] = y.ok;
        r[5] = 1.0 / x[1];
        r[6] = s.sqrt(x[1]);
        r[7] = s.ok;
        r[8] = sqrt(x[1]);
    }
};
struct DivSum {  // a / b for a sum of weights b >= 1, whether it was taken, the compiler's
    static constexpr int in = 2, out = 3;
    static __device__ void f(const double *x, double *r)
    {
        cfd::OpsSpec o;
        r[0] = o.div_sum(x[0], x[1]);
        r[1] = o.ok;
        r[2] = x[0] / x[1];
    }
};
struct Wenoz {  // five stencil values: WENO-Z, whether the branch-free path took them, by the compiler's operations
    static constexpr int in = 5, out = 3;
    static __device__ void f(const double *x, double *r)
    {
        cfd::OpsSpec o;
        cfd::OpsIeee i;
        r[0] = cfd::inter5<cfd::FAM_WENOZ>(x[0], x[1], x[2], x[3], x[4], 0.0, 0.0, o);
        r[1] = o.ok;
        r[2] = cfd::inter5<cfd::FAM_WENOZ>(x[0], x[1], x[2], x[3], x[4], 0.0, 0.0, i);
    }
};
#if defined(CFD_FAST)
struct Rsqrt {
    static constexpr int in = 1, out = 2;
    static __device__ void f(const double *x, double *r)
    {
        cfd::OpsSpec o;
        r[0] = o.rsqrt(x[0]);
        r[1] = o.ok;
    }
};
struct Wcns5Pair {  // a field's six values: both face states, whether the fast path took them
    static constexpr int in = 6, out = 3;
    static __device__ void f(const double *x, double *r)
    {
        cfd::OpsSpec o;
        cfd::wcns5_pair(x, r[0], r[1], o);
        r[2] = o.ok;
    }
};
#endif

template <class OP>
__global__ void each(const double *x, double *r, long n)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        OP::f(x + i * OP::in, r + i * OP::out);
}

template <class OP>
int run(const double *x, double *r, long n)
{
    double *dx = nullptr, *dr = nullptr;
    cudaError_t e = cudaMalloc(&dx, sizeof(double) * OP::in * n);
    if (e == cudaSuccess) e = cudaMalloc(&dr, sizeof(double) * OP::out * n);
    if (e == cudaSuccess) e = cudaMemcpy(dx, x, sizeof(double) * OP::in * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        each<OP><<<148 * 4, 128>>>(dx, dr, n);
        e = cudaMemcpy(r, dr, sizeof(double) * OP::out * n, cudaMemcpyDeviceToHost);
    }
    cudaFree(dx);
    cudaFree(dr);
    return (int)e;
}

} // namespace

extern "C" {
int ops_div_sum(const double *x, double *r, long n) { return run<DivSum>(x, r, n); }
int ops_wenoz(const double *x, double *r, long n) { return run<Wenoz>(x, r, n); }
int ops_spec(const double *x, double *r, long n) { return run<Spec>(x, r, n); }
int ops_arcp(const double *x, double *r, long n) { return run<Arcp>(x, r, n); }
int ops_asqrt(const double *x, double *r, long n) { return run<Asqrt>(x, r, n); }
int ops_wcns5_adj(const double *x, double *r, long n) { return run<Wcns5Adj>(x, r, n); }
#if defined(CFD_FAST)
int ops_rsqrt(const double *x, double *r, long n) { return run<Rsqrt>(x, r, n); }
int ops_wcns5_pair(const double *x, double *r, long n) { return run<Wcns5Pair>(x, r, n); }
#endif
int ops_face_vjp(const double *x, double *r, long n) { return run<FaceVjp>(x, r, n); }
}
