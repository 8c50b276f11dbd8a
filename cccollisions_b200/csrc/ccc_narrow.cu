// ccc_narrow.cu — the continuous narrow phase (k_ccd_narrow) and the solver's test hooks.
//
// This translation unit alone is compiled with nvcc's default multiply-add contraction
// (-fmad=true), as the reference extension is: the solver calls CUDA's pow, whose result on
// rare arguments depends on that setting (pow(g, 2.0) in the cubic's h differs by an ulp on
// about 6 in a million arguments under -fmad=false, which moved a root near t = 0 of a nearly
// coplanar sub-test).  The solver's other CUDA functions (cbrt, acos, cos, sin, cbrtf,
// rsqrt, rsqrtf) gave the same bits under both settings on 2^28 arguments each.  Every
// operation of this library's own reached from here rounds as written under either setting:
// products that feed sums are explicitly rounded (mulrn / addrn / subrn, ccc_mul / ccc_add /
// ccc_sub) or operands of explicit fused multiply-adds (fmaT / ccc_fma), which are never
// fused further.  The rest of the library is compiled with -fmad=false.
#define CCC_NARROW_TU
#include "../../include/ccc_b200.h"
#include "ccc_kernels.cuh"
#include "ccc_engine.cuh"
#include "ccc_runtime.cuh"

namespace ccc {

// the combinations the library launches: (type, mode, sink, math library, source, batch)
#define CCC_NARROW_INSTANCE(T, MODE, SINK, LIB, SRC, BM)                                                           \
    template cudaError_t launch_ccd_narrow<T, MODE, SINK, LIB, SRC, BM>(int, cudaStream_t, const CcdArgs<T>&,        \
                                                                           const SINK&);                              \
    template cudaError_t prepare_ccd_narrow<T, MODE, SINK, LIB, SRC, BM>();
#define CCC_NARROW_TYPES(MODE, SINK, SRC, BM)                                                                      \
    CCC_NARROW_INSTANCE(float, MODE, SINK<float>, LIB_REFERENCE, SRC, BM)                                           \
    CCC_NARROW_INSTANCE(double, MODE, SINK<double>, LIB_REFERENCE, SRC, BM)                                         \
    CCC_NARROW_INSTANCE(float, MODE, SINK<float>, LIB_PORTABLE, SRC, BM)                                            \
    CCC_NARROW_INSTANCE(double, MODE, SINK<double>, LIB_PORTABLE, SRC, BM)
#define CCC_CONTACT_TYPES(SINK)                                                                                    \
    template cudaError_t launch_ccd_contacts<float, SINK<float>, LIB_REFERENCE>(int, cudaStream_t,                  \
                                                                                   const CcdArgs<float>&,            \
                                                                                   const SINK<float>&);               \
    template cudaError_t launch_ccd_contacts<double, SINK<double>, LIB_REFERENCE>(int, cudaStream_t,                \
                                                                                     const CcdArgs<double>&,         \
                                                                                     const SINK<double>&);            \
    template cudaError_t launch_ccd_contacts<float, SINK<float>, LIB_PORTABLE>(int, cudaStream_t,                   \
                                                                                  const CcdArgs<float>&,             \
                                                                                  const SINK<float>&);                \
    template cudaError_t launch_ccd_contacts<double, SINK<double>, LIB_PORTABLE>(int, cudaStream_t,                 \
                                                                                    const CcdArgs<double>&,          \
                                                                                    const SINK<double>&);
// the reference-format operations (pairs and masks from the candidate buffer), batches of 256
CCC_NARROW_TYPES(CCD_ROWS, CornerSink, SRC_PACKED, 1)
CCC_NARROW_TYPES(CCD_IMPULSES, CornerSink, SRC_PACKED, 1)
CCC_CONTACT_TYPES(CornerSink)
// the resident engine's collision step (shared sub-tests), batches of 256 or 512, and its
// impulse loop
CCC_NARROW_TYPES(CCD_ROWS, CornerSink, SRC_STAGED, 1)
CCC_NARROW_TYPES(CCD_ROWS, CornerSink, SRC_STAGED, 2)
CCC_NARROW_TYPES(CCD_IMPULSES, LoopSink, SRC_STAGED, 1)
CCC_CONTACT_TYPES(LoopSink)

// Element-wise evaluation of the solver's arithmetic building blocks, for tests that compare
// them bit for bit with the CPU oracle and against CUDA's own elementary functions.
// op 0 cbrt, 1 acos, 2 cos, 3 sin, 4 certified product (in: x0, x1, k, y; out: r0, r1),
// 5 solve_cubic (in: a, b, c, d; out: three roots), 6 CUDA cbrt, 7 CUDA acos, 8 CUDA cos,
// 9 CUDA sin, 10 the solver prefix of a, b, c, d without its short cuts (out: f, g, h), 11 the
// solver's divisions by 3 and by 27, 12 CUDA sincos (out: sine, cosine).  in has 4 doubles per
// element, out 3.
static __global__ void k_debug_math(int op, const double* __restrict__ in, double* __restrict__ out, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* a = in + 4 * i;
    double* o = out + 3 * i;
    o[0] = o[1] = o[2] = 0.0;
    switch (op) {
        case 0: o[0] = ccc_cbrt(a[0]); break;
        case 1: o[0] = ccc_acos(a[0]); break;
        case 2: o[0] = ccc_cos(a[0]); break;
        case 3: o[0] = ccc_sin(a[0]); break;
        case 4: {
            ccc_dd d = ccc_certmul(a[0], a[1], (int)a[2], a[3]);
            o[0] = d.hi;
            o[1] = d.lo;
            break;
        }
        case 5: solve_cubic<double, LIB_PORTABLE>(a[0], a[1], a[2], a[3], o); break;
        case 6: o[0] = cbrt(a[0]); break;
        case 7: o[0] = acos(a[0]); break;
        case 8: o[0] = cos(a[0]); break;
        case 9: o[0] = sin(a[0]); break;
        case 10: {
            // the solver prefix without its short cuts (certified products, divisions)
            const double A = a[0], B = a[1], C = a[2], D = a[3];
            auto cube = [](double x) {
                const ccc_dd sq = ccc_certmul(x, 0.0, 1, x);
                return ccc_certmul(sq.hi, sq.lo, 2, x).hi;
            };
            const double f = ((3.0 * C / A) - ((B * B) / (A * A))) / 3.0;
            const double g = (2 * cube(B) / cube(A) - (B * C * 9) / ccc_certmul(A, 0.0, 1, A).hi + 27.0 * D / A) / 27.0;
            o[0] = f;
            o[1] = g;
            o[2] = addrn(mulrn(mulrn(g, g), 0.25), cube(f) / 27.0);
            break;
        }
        case 11:
            o[0] = div_const<3>(a[0]);
            o[1] = div_const<27>(a[0]);
            break;
        case 12: sincos(a[0], &o[0], &o[1]); break;
        default: break;
    }
}

// Stages of the continuous narrow phase on caller tetrahedra (v0..v3, dv0..dv3 = 24
// doubles per element), for tests against the reference's own kernels and the oracle.
// op 0: cubic coefficients -> 4 doubles; op 1: cubic solve (in: 4 coefficients) -> 3
// roots; op 2: root filter (in: tet, type, root) -> 1.0 / 0.0; op 3: contact kinematics
// (in: tet, type, root, 4 masses) -> normal (3), normal velocity, mass pair (2); op 4: solver
// prefix (in: 4 coefficients) -> class, g, h; op 5: early end of a cubic (in: 4 coefficients) ->
// cubic_misses and the solver's roots in [0, 1], in double and in single precision; op 6: early
// ends of a sub-test (in: tet, type) -> cubic_misses, roots_fail, the solver's roots in [0, 1]
// and those of them that pass the filter, in double and in single precision.
// lib selects the elementary functions (MathLib).
template <class T> __device__ __forceinline__ int debug_roots(int lib, const T cf[4], T r[3]) {
    if (lib == LIB_REFERENCE) solve_cubic<T, LIB_REFERENCE>((double)cf[0], (double)cf[1], (double)cf[2], (double)cf[3], r);
    else solve_cubic<T, LIB_PORTABLE>((double)cf[0], (double)cf[1], (double)cf[2], (double)cf[3], r);
    int n = 0;
    for (int s = 0; s < 3; ++s) n += r[s] >= 0 && r[s] <= 1;
    return n;
}
template <class T> __device__ __noinline__ void debug_cubic_end(int lib, const double* a, double* o) {
    const T cf[4] = {(T)a[0], (T)a[1], (T)a[2], (T)a[3]};
    T r[3];
    o[0] = cubic_misses<T>((double)cf[0], (double)cf[1], (double)cf[2], (double)cf[3]);
    o[1] = debug_roots(lib, cf, r);
}
template <class T> __device__ __noinline__ void debug_subtest_end(int lib, const MTet<double>& t, int k, double* o) {
    MTet<T> m;
    for (int p = 0; p < 4; ++p) {
        m.v[p] = mk<T>((T)t.v[p].x, (T)t.v[p].y, (T)t.v[p].z);
        m.dv[p] = mk<T>((T)t.dv[p].x, (T)t.dv[p].y, (T)t.dv[p].z);
    }
    T cf[4], r[3];
    cubic_coeffs(m, cf);
    o[0] = cubic_misses<T>((double)cf[0], (double)cf[1], (double)cf[2], (double)cf[3]);
    o[1] = roots_fail(m, k, cf);
    o[2] = debug_roots(lib, cf, r);
    int pass = 0;
    for (int s = 0; s < 3; ++s) pass += r[s] >= 0 && r[s] <= 1 && ccd_filter(m, k, r[s]);
    o[3] = pass;
}
static __global__ void k_debug_stage(int op, int lib, const double* __restrict__ in, int in_stride,
                              double* __restrict__ out, int out_stride, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double* a = in + (long long)i * in_stride;
    double* o = out + (long long)i * out_stride;
    MTet<double> t;
    if (op != 1 && op != 4 && op != 5) {
        for (int p = 0; p < 4; ++p) {
            t.v[p] = mk<double>(a[3 * p], a[3 * p + 1], a[3 * p + 2]);
            t.dv[p] = mk<double>(a[12 + 3 * p], a[12 + 3 * p + 1], a[12 + 3 * p + 2]);
        }
    }
    if (op == 0) {
        cubic_coeffs(t, o);
    } else if (op == 1) {
        if (lib == LIB_REFERENCE) solve_cubic<double, LIB_REFERENCE>(a[0], a[1], a[2], a[3], o);
        else solve_cubic<double, LIB_PORTABLE>(a[0], a[1], a[2], a[3], o);
    } else if (op == 2) {
        o[0] = ccd_filter(t, (int)a[24], a[25]) ? 1.0 : 0.0;
    } else if (op == 4) {
        double g, h;
        const int cls = lib == LIB_REFERENCE ? cubic_prefix<LIB_REFERENCE>(a[0], a[1], a[2], a[3], g, h)
                                             : cubic_prefix<LIB_PORTABLE>(a[0], a[1], a[2], a[3], g, h);
        o[0] = cls;
        o[1] = g;
        o[2] = h;
    } else if (op == 5) {
        debug_cubic_end<double>(lib, a, o);
        debug_cubic_end<float>(lib, a, o + 2);
    } else if (op == 6) {
        debug_subtest_end<double>(lib, t, (int)a[24], o);
        debug_subtest_end<float>(lib, t, (int)a[24], o + 4);
    } else if (op == 3) {
        double q[4] = {a[26], a[27], a[28], a[29]};
        Contact<double> ct = lib == LIB_REFERENCE ? contact<double, LIB_REFERENCE>(t, (int)a[24], a[25], q)
                                                  : contact<double, LIB_PORTABLE>(t, (int)a[24], a[25], q);
        o[0] = ct.n.x; o[1] = ct.n.y; o[2] = ct.n.z; o[3] = ct.vn; o[4] = ct.m0; o[5] = ct.m1;
    }
}


cudaError_t launch_debug_math(int op, const double* in, double* out, int n, cudaStream_t s) {
    k_debug_math<<<grid_for(n, 128), 128, 0, s>>>(op, in, out, n);
    return cudaGetLastError();
}

cudaError_t launch_debug_stage(int op, int lib, const double* in, int in_stride, double* out, int out_stride, int n,
                               cudaStream_t s) {
    k_debug_stage<<<grid_for(n, 128), 128, 0, s>>>(op, lib, in, in_stride, out, out_stride, n);
    return cudaGetLastError();
}

}  // namespace ccc
