// kernels.cuh -- sm_103a kernels of the Multigrid Monte Carlo step.
//
// Data layout (every level): padded lexicographic arrays with shared ghost
// rows/planes, see Geometry in setup.h.  A point with 0-based interior
// coordinates (a, b, c) lives at P = (c+1) sz + (b+1) sy + (a+1); ghosts are
// zero, so stencil loads need no boundary tests.
//
// Kernels (one V-cycle at level l uses them in this order):
//   k_sweep_rb_vec      one colour of the red-black SOR sweep of the 7-point
//                       level, FP32, 8-point spans with float4 loads/stores
//   k_sweep_rb_pass     the same, one point per thread (FP64, parity)
//   k_sweep_row_pair    two colours of the 8-colour (2D: 4-colour) SOR sweep of
//                       a 27-point (9-point) level; k_sweep_row_sym: the same
//                       for FP64 chains' symmetric stencils
//   k_sweep_c27_pass    one colour of it, for rows too long for a CTA
//   k_sweep_wavefront   lexicographic SOR sweep as a hyperplane wavefront
//                       (one CTA; parity mode)
//   k_bt_partial        partial sums of y = B^T x, the low-rank noise
//   k_lr_correct        the m x m solve and x += C z over the rows of C = M^{-1} B
//   k_lr_z              the solve alone, for k_lr_correct on large m or supports
//   k_bt_full           y = B^T x in one launch (k_bt_sum: from partial sums)
//   k_resid_restrict_tma    f_c = R (f - A_0 x), TMA tiles (fused residual
//                           + restriction; _tiled / plain variants otherwise)
//   k_resid_restrict_sym    the same for FP64 chains' symmetric stencils
//   k_resid_restrict_point  the same, one coarse point per thread
//   k_resid_Bq          f_c -= B_c Sigma^{-1} y (k_add_Bq: elsewhere)
//   k_prolong_add       x += alpha P x_c
//   k_chol_gemv_*       coarse-level Cholesky sample (k_chol_subst: parity)
//   k_step_end          observables z = b^T x, step counter
// Host conversions: k_unpack / k_unpack2 / k_pack; adjoint helpers: k_axpy,
// k_adj_update, k_add_Bz; deterministic solver (FP64 loop around the noise-free
// cycle): k_solve_resid, k_solve_update, k_solve_gather; parameter adjoint:
// k_pgrad_stencil, k_pgrad_combine, k_coarse_normals, k_pgrad_coarse_phi,
// k_pgrad_coarse_sigma, k_accum_sum; building blocks: k_apply_stencil; the
// low-rank Cholesky sampler: k_chol_tri, k_chol_step, k_chol_step_t, k_chol_qt,
// k_chol_v / k_chol_t / k_chol_w, k_chol_add.
#pragma once

#include <cstdint>
#include <cuda.h>  // CUtensorMap (type only; the driver entry point is resolved at run time)
#include <cuda_runtime.h>
#include <type_traits>

namespace mgmc {

typedef long long i64;
typedef unsigned long long u64;

// Programmatic dependent launch: wait until the previous kernel on the
// stream has completed and its writes are visible (a kernel launched with
// the programmatic-serialization attribute may start once every CTA of its
// predecessor has let it, with pdl_trigger or by its exit).  Without the
// attribute this is a no-op.
//
// The rules of every kernel that waits:
// - It waits before it lets the next one start.  Then "the kernel before has
//   completed" holds for all kernels before that one too.
// - Before the wait it writes nothing outside its CTA and reads only what no
//   launch of the step writes: operators, factors, index lists, and the step
//   counter, which the step's last launch advances.  One exception: the
//   correction reads the state before its wait (k_lr_correct says why it may).
// - Memory that a launch of the step writes carries no __restrict__ and is not
//   read by ld.global.nc or __ldg: a compiler may move loads of memory promised
//   to be constant, or private to a pointer, above the wait.
__device__ __forceinline__ void pdl_begin() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Let the next kernel on the stream start its CTAs now (they still wait in
// pdl_begin until this grid has completed), so that its noise and independent
// loads overlap this one.  For grids that leave room: the waiting CTAs hold SM
// slots, and after the wait of every kernel, whatever its grid, it made the
// 256^3 step 1.8 % slower.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Both, for a kernel between two sweeps: a grid of at most two CTAs per SM
// lets the next kernel start at once (it draws its noise and loads what does
// not depend on this one meanwhile; see k_chol_gemv_lower for what it gave);
// a larger one needs the SM slots.
constexpr unsigned PDL_SMALL_GRID = 304;
__device__ __forceinline__ void pdl_begin_trigger() {
    pdl_begin();
    if (gridDim.x * gridDim.y * gridDim.z <= PDL_SMALL_GRID) pdl_trigger();
}

// ------------------------------------------------------------- geometry
struct Grid3 {
    int N0, N1, N2;  // interior vertices per direction
    i64 sy, sz;      // padded strides
    int pdl = 0;     // kernels on this level take part in programmatic dependent launch
    __host__ __device__ i64 pad(int a, int b, int c) const { return (i64)(c + 1) * sz + (i64)(b + 1) * sy + (a + 1); }
    __host__ __device__ i64 compact(int a, int b, int c) const { return ((i64)c * N1 + b) * N0 + a; }
};

template <typename T>
struct StencilArg {
    T w[27];  // (dz+1)*9 + (dy+1)*3 + (dx+1)
    T diag;   // w[13]
    T omega;
    T sd;         // sqrt(diag (2 - omega) / omega): noise scale (sor_sampler.cc:20-27)
    T omega_diag; // omega / diag
    T tmo;        // 2 - omega (per-point noise scales of variable stencils)
};

// Per-point stencil of a level with variable coefficients.  VAR == 1: w[P]
// (padded index) is the centre weight, the other weights are the constant
// ones of StencilArg; VAR == 2: w[k * stride + P] is weight k.  VAR == 0:
// the constant StencilArg alone.
template <typename T>
struct VarField {
    const T *w;
    i64 stride;
};

template <typename T, int VAR>
__device__ __forceinline__ T vweight(const StencilArg<T> &s, const VarField<T> &vf, i64 P, int k) {
    if (VAR == 2) return vf.w[(i64)k * vf.stride + P];
    if (VAR == 1 && k == 13) return vf.w[P];
    return s.w[k];
}

// ---------------------------------------------------------------- noise
enum { NOISE_NONE = 0, NOISE_PHILOX = 1, NOISE_INJECTED = 2 };
enum { PURPOSE_POINT = 0, PURPOSE_LOWRANK = 1, PURPOSE_COARSE = 2, PURPOSE_EXACT = 3, PURPOSE_CHOLESKY = 4 };

struct NoiseArgs {
    const double *buf;   // injected: normals for this consumer, index = vertex / column
    u64 seed;            // Philox key
    const u64 *d_step;   // device step counter
    unsigned invocation; // position of this noise consumer inside one step
    unsigned level;
};

// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, "Parallel random numbers: as
// easy as 1, 2, 3", SC'11): 10 rounds of the 4x32 bijection with the
// published multipliers and Weyl key increments.
__device__ __forceinline__ uint4 philox4x32_10(uint4 ctr, uint2 key) {
    const unsigned M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
    const unsigned W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        unsigned lo0 = M0 * ctr.x, hi0 = __umulhi(M0, ctr.x);
        unsigned lo1 = M1 * ctr.z, hi1 = __umulhi(M1, ctr.z);
        ctr = make_uint4(hi1 ^ ctr.y ^ key.x, lo1, hi0 ^ ctr.w ^ key.y, lo0);
        key.x += W0;
        key.y += W1;
    }
    return ctr;
}

// Two Box-Muller pairs in FP32 (Box & Muller 1958) with the SFU
// approximations of log2, reciprocal square root and sine/cosine (absolute
// error of order 1e-6 per normal).  u1 is in (0, 1]: the product of a
// value <= 2^32 with 2^-32 plus 2^-33 rounds to at most 1.0f, so -log2(u1)
// is never negative; the angle lies in [-pi, pi), the accurate range of the
// fast sine and cosine.
__device__ __forceinline__ float4 normals4(uint4 r) {
    const float two_m32 = 2.3283064365386963e-10f;  // 2^-32
    const float two_m33 = 1.1641532182693481e-10f;  // 2^-33
    const float m2ln2 = -1.3862943611198906f;       // -2 ln 2
    const float twopi = 6.283185307179586f;
    float u1a = __fmaf_rn(__uint2float_rn(r.x), two_m32, two_m33);
    float u1b = __fmaf_rn(__uint2float_rn(r.z), two_m32, two_m33);
    float qa = fmaxf(m2ln2 * __log2f(u1a), 1e-30f);
    float qb = fmaxf(m2ln2 * __log2f(u1b), 1e-30f);
    float ra = qa * rsqrtf(qa), rb = qb * rsqrtf(qb);
    float sa, ca, sb, cb;
    __sincosf(__fmaf_rn(__uint2float_rz(r.y), two_m32, -0.5f) * twopi, &sa, &ca);
    __sincosf(__fmaf_rn(__uint2float_rz(r.w), two_m32, -0.5f) * twopi, &sb, &cb);
    return make_float4(ra * ca, ra * sa, rb * cb, rb * sb);
}

__device__ __forceinline__ float pick(float4 v, int lane) {
    return lane == 0 ? v.x : (lane == 1 ? v.y : (lane == 2 ? v.z : v.w));
}

__device__ __forceinline__ uint4 noise_ctr(const NoiseArgs &nz, unsigned x, unsigned purpose, unsigned low) {
    u64 sc = (*nz.d_step) * 4096ull + nz.invocation;
    return make_uint4(x, (purpose << 24) | (nz.level << 8) | low, (unsigned)sc, (unsigned)(sc >> 32));
}

__device__ __forceinline__ uint2 noise_key(const NoiseArgs &nz) {
    return make_uint2((unsigned)nz.seed, (unsigned)(nz.seed >> 32));
}

// Normals of the 4 points of x-parity (a & 1) inside the 8-point x-group
// a >> 3 of row (b, c): lane (a & 7) >> 1.
__device__ __forceinline__ float4 point_normals(const NoiseArgs &nz, const Grid3 &g, int a, int b, int c) {
    unsigned G0 = (unsigned)((g.N0 + 7) >> 3);
    unsigned grp = (unsigned)(((u64)c * g.N1 + b) * G0 + (a >> 3));
    return normals4(philox4x32_10(noise_ctr(nz, grp, PURPOSE_POINT, a & 1), noise_key(nz)));
}

// a float that is zero or normal as a double, by its bits (the conversion
// instruction would take the FP64 unit)
__device__ __forceinline__ double widen(float v) {
    const unsigned u = __float_as_uint(v), m = u & 0x7fffffffu;
    const unsigned hi = (u & 0x80000000u) | (m < 0x00800000u ? 0u : (m >> 3) + 0x38000000u);
    return __hiloint2double((int)hi, m < 0x00800000u ? 0 : (int)(u << 29));
}
__device__ __forceinline__ double to_double(double v) { return v; }
__device__ __forceinline__ double to_double(float v) {  // widen, for any value
    const unsigned m = __float_as_uint(v) & 0x7fffffffu;
    return m - 0x00800000u < 0x7f000000u || m == 0u ? widen(v) : (double)v;
}

// ------------------------------------------------------- exact arithmetic
// Parity kernels evaluate the reference's expressions with one rounding per
// operation (no FMA contraction), as the reference's compiled CPU code does.
template <bool EXACT>
struct Ar;
template <>
struct Ar<true> {
    static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
};
template <>
struct Ar<false> {
    template <typename T>
    static __device__ __forceinline__ T mul(T a, T b) { return a * b; }
    template <typename T>
    static __device__ __forceinline__ T add(T a, T b) { return a + b; }
    template <typename T>
    static __device__ __forceinline__ T sub(T a, T b) { return a - b; }
};

// One SOR point update (sor_smoother.cc:66-76 with the noisy right hand
// side of sor_sampler.cc:42-46):
//   c = sd * xi + f;  res = sum_k w_k x_k (ascending index, diagonal
//   included);  x += omega * (c - res) / diag.
// Row P of A_0 x: sum_k w_k x_k in ascending index order, diagonal
// included, with the neighbour (dz, dy, dx) of P read through xa(dz, dy, dx)
// (global memory or values loaded beforehand: the same arithmetic either way).
template <typename T, int NPT, bool EXACT, int VAR, typename XA>
__device__ __forceinline__ T stencil_row_acc(const XA &xa, const StencilArg<T> &s, i64 P, const VarField<T> &vf) {
    typedef Ar<EXACT> A;
    T res = T(0);
    if (NPT == 7) {
        const int ks[7] = {4, 10, 12, 13, 14, 16, 22};
        const int dzs[7] = {-1, 0, 0, 0, 0, 0, 1}, dys[7] = {0, -1, 0, 0, 0, 1, 0}, dxs[7] = {0, 0, -1, 0, 1, 0, 0};
#pragma unroll
        for (int q = 0; q < 7; ++q) res = A::add(res, A::mul(vweight<T, VAR>(s, vf, P, ks[q]), xa(dzs[q], dys[q], dxs[q])));
    } else {
        constexpr int ZLO = NPT == 9 ? 0 : -1, ZHI = NPT == 9 ? 0 : 1;  // a 2D level has no neighbours in z
#pragma unroll
        for (int dz = ZLO; dz <= ZHI; ++dz)
#pragma unroll
            for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
                for (int dx = -1; dx <= 1; ++dx)
                    res = A::add(res, A::mul(vweight<T, VAR>(s, vf, P, (dz + 1) * 9 + (dy + 1) * 3 + (dx + 1)),
                                             xa(dz, dy, dx)));
    }
    return res;
}

template <typename T, int NPT, bool EXACT, int VAR = 0>
__device__ __forceinline__ T stencil_row(const T *x, const Grid3 &g, const StencilArg<T> &s, i64 P,
                                         const VarField<T> &vf = VarField<T>{nullptr, 0}) {
    return stencil_row_acc<T, NPT, EXACT, VAR>(
        [&](int dz, int dy, int dx) { return x[P + dz * g.sz + dy * g.sy + dx]; }, s, P, vf);
}

// The updated value of point P from its neighbours (xa), old value xo and
// right hand side fv.  With a variable stencil (VAR != 0) the diagonal, the
// noise scale sqrt(d (2 - omega) / omega) and omega / d are formed per
// point, in the oracle's operation order on the parity path.
template <typename T, int NPT, bool EXACT, int VAR, typename XA>
__device__ __forceinline__ T sor_value(const XA &xa, T xo, T fv, const StencilArg<T> &s, i64 P, bool noisy, T xi,
                                       const VarField<T> &vf) {
    typedef Ar<EXACT> A;
    const T res = stencil_row_acc<T, NPT, EXACT, VAR>(xa, s, P, vf);
    T cval = fv;
    if (VAR == 0) {
        if (noisy) cval = A::add(A::mul(s.sd, xi), cval);
        if (EXACT) return A::add(xo, A::mul(s.omega, A::sub(cval, res)) / s.diag);
        return xo + s.omega_diag * (cval - res);
    }
    const T d = vweight<T, VAR>(s, vf, P, 13);
    if (noisy) {
        const T sd = sqrt(A::mul(d, s.tmo) / s.omega);
        cval = A::add(A::mul(sd, xi), cval);
    }
    if (EXACT) return A::add(xo, A::mul(s.omega, A::sub(cval, res)) / d);
    return xo + (s.omega / d) * (cval - res);
}

template <typename T, int NPT, bool EXACT, int VAR = 0>
__device__ __forceinline__ void sor_point(T *x, const T *f, const Grid3 &g,
                                          const StencilArg<T> &s, i64 P, bool noisy, T xi,
                                          const VarField<T> &vf = VarField<T>{nullptr, 0}) {
    x[P] = sor_value<T, NPT, EXACT, VAR>([&](int dz, int dy, int dx) { return x[P + dz * g.sz + dy * g.sy + dx]; },
                                         x[P], f[P], s, P, noisy, xi, vf);
}

// Constant stencil with equal weights at +-dx, +-dy, +-dz: wc[|dz| * 4 +
// |dy| * 2 + |dx|] is the weight of a class.
struct SymWeights {
    double wc[8];
    double sd, od, om1;  // noise scale, omega / d, 1 - omega (kernels' UNIT: omega = 1, om1 = 0)
};

// With omega = 1 a point's new value does not need its old one.  A non-finite
// old value still has to stay (x + (omega / d)(c - A x) keeps it, and an
// observable reports it), so v becomes NaN there: by its bits, without an FP64
// instruction.
__device__ __forceinline__ double keep_nonfinite(double v, double old) {
    const bool bad = (__double2hiint(old) & 0x7ff00000) == 0x7ff00000;
    return __hiloint2double(bad ? 0x7ff80000 : __double2hiint(v), __double2loint(v));
}

// ------------------------------------------------- red-black SOR sweep
// Noise of a 7-point level: the normals of the 4 points of one x-parity in
// the 8-aligned group of padded positions P = a + 1 in [8q, 8q + 8) of row
// (b, c) come from one Philox block, lane (P & 7) >> 1.
__device__ __forceinline__ float4 fine_normals(const NoiseArgs &nz, const Grid3 &g, int P, int b, int c) {
    const unsigned G0 = (unsigned)((g.N0 + 1) >> 3) + 1u;
    const unsigned grp = (unsigned)(((u64)c * g.N1 + b) * G0 + (P >> 3));
    return normals4(philox4x32_10(noise_ctr(nz, grp, PURPOSE_POINT, P & 1), noise_key(nz)));
}

// One colour of a red-black sweep of an axis-only (7-point) level, one
// thread per point of the colour.  A CTA is blockDim.x points along x times
// blockDim.y rows (b) of one plane c (sweep_block() picks the shape so that
// no thread idles on short rows); each warp load reads a contiguous span.
// `reverse` walks the planes from the top so that the second colour finds
// the data the first colour touched last in L2.
constexpr int RBP_THREADS = 256;

// CTA shape for `count` work items along x: the smallest power of two
// >= count (at least 8, at most RBP_THREADS) along x, the rest along y.
__host__ __forceinline__ dim3 sweep_block(int count) {
    int tx = 8;
    while (tx < count && tx < RBP_THREADS) tx *= 2;
    return dim3(tx, RBP_THREADS / tx, 1);
}

// The normals are drawn before the wait for the launch before, and with
// `trigger` the next launch starts early (see k_sweep_row_pair).
template <typename T, bool EXACT, int NOISE, int VAR = 0>
__global__ void __launch_bounds__(RBP_THREADS) k_sweep_rb_pass(T *x, const T *f, Grid3 g, StencilArg<T> s, int colour,
                                                               int reverse, NoiseArgs nz, VarField<T> vf, int trigger) {
    const int b = blockIdx.y * blockDim.y + threadIdx.y;
    const int c = reverse ? g.N2 - 1 - (int)blockIdx.z : (int)blockIdx.z;
    const int p = (colour + b + c) & 1;
    const int a = 2 * (blockIdx.x * blockDim.x + threadIdx.x) + p;
    T xi = T(0);
    if (NOISE == NOISE_PHILOX) xi = (T)pick(fine_normals(nz, g, a + 1, b, c), ((a + 1) & 7) >> 1);
    if (g.pdl) pdl_begin();
    if (trigger) pdl_trigger();
    if (a >= g.N0 || b >= g.N1) return;
    if (NOISE == NOISE_INJECTED) xi = (T)nz.buf[g.compact(a, b, c)];
    sor_point<T, 7, EXACT, VAR>(x, f, g, s, g.pad(a, b, c), NOISE != NOISE_NONE, xi, vf);
}

// The same colour pass for FP64 chains whose constant axis stencil has equal
// weights at +-1 (Level::sym): 8 FP64 instructions per point (6 in 2D) instead
// of 11, since the FP64 unit is what it waits for (see k_sweep_row_sym): the
// neighbours are added in pairs, the diagonal drops out of
// x'' = (1 - omega) x + (omega / d)(sd xi + f - sum over the neighbours), and
// the normal is widened by its bits.
template <bool D3, int NOISE, bool UNIT>
__global__ void __launch_bounds__(RBP_THREADS) k_sweep_rb_sym(double *x, const double *f, Grid3 g, SymWeights w,
                                                              int colour, int reverse, NoiseArgs nz, int trigger) {
    const int b = blockIdx.y * blockDim.y + threadIdx.y;
    const int c = reverse ? g.N2 - 1 - (int)blockIdx.z : (int)blockIdx.z;
    const int p = (colour + b + c) & 1;
    const int a = 2 * (blockIdx.x * blockDim.x + threadIdx.x) + p;
    double xi = 0.0;
    if (NOISE == NOISE_PHILOX) xi = widen(pick(fine_normals(nz, g, a + 1, b, c), ((a + 1) & 7) >> 1));
    if (g.pdl) pdl_begin();
    if (trigger) pdl_trigger();
    if (a >= g.N0 || b >= g.N1) return;
    double *q = x + g.pad(a, b, c);
    double cv = f[g.pad(a, b, c)];
    const double old = *q;
    const double sx = q[-1] + q[1], sy = q[-g.sy] + q[g.sy], sz = D3 ? q[-g.sz] + q[g.sz] : 0.0;
    if (NOISE != NOISE_NONE) cv = fma(w.sd, xi, cv);
    if (D3) cv = fma(-w.wc[4], sz, cv);
    cv = fma(-w.wc[2], sy, cv);
    cv = fma(-w.wc[1], sx, cv);
    *q = UNIT ? keep_nonfinite(w.od * cv, old) : fma(w.od, cv, w.om1 * old);
}

// 256-bit vector access (sm_100 and later): 8 floats at a 32-byte aligned
// address in one instruction.  ld8 reads through L1 (x is written in the
// same pass); read-once streams use ld8_stream below.
__device__ __forceinline__ void ld8(const float *p, float *v) {
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p)
                 : "memory");
}
// Read-once streams (f and the centre field of the fine sweep): no L1
// allocation, and first in line for L2 eviction, so that the L2 keeps x --
// which the next colour pass reads again -- rather than f, which it does
// not.  (Measured at 256^3: 53.3 -> 49.7 us per two-pass sweep.)  An earlier
// launch may have written f: ordinary loads, kept behind the wait by the
// clobber, not loads of memory that is constant while the kernel runs.
__device__ __forceinline__ unsigned long long l2_evict_first_policy() {
    unsigned long long p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ float4 ld4_stream(const float *p, unsigned long long pol) {
    float4 r;
    asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v4.f32 {%0,%1,%2,%3}, [%4], %5;"
                 : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
                 : "l"(p), "l"(pol)
                 : "memory");
    return r;
}
__device__ __forceinline__ void ld8_stream(const float *p, float *v, unsigned long long pol) {
    asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8], %9;"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ void st8(float *p, const float *v) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]),
                 "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}

// FP32 variant with vector loads (rows padded to a multiple of 4 floats): a
// thread owns the 8 padded positions [8q, 8q + 8) of a row, loads them and
// the matching spans of the four neighbouring rows and f as float4, draws
// one Philox block for its 4 points of the colour and stores those 4 points.
// VD: a per-point centre weight field vd (same padded layout), loaded as a
// fifth pair of float4 spans.  V8 (rows a multiple of 8 floats): every span
// is one 256-bit access instead of two float4 ones, which halves the L1
// wavefronts of the loads (a warp's 32-byte spans are contiguous).  FS (with
// V8): f comes from fsc, the colour's half of f split by colour
// (k_split_colours), so the pass reads one float4 of f per span -- only the
// values it uses -- instead of the whole span.
// The body, with the CTA coordinates (bx, by, bz) passed in: the solo
// kernel below and the batched kernel (k_sweep_rb_vec_batch) run the same
// arithmetic.
// EARLY (levels in programmatic dependent launch): the normals are drawn before
// the wait for the launch before, and the next launch starts early.
template <int NOISE, bool VD, bool V8, bool FS, bool EARLY>
__device__ __forceinline__ void sweep_rb_vec_body(float *x, const float *f, const Grid3 &g,
                                                  const StencilArg<float> &s, int colour, int reverse,
                                                  const NoiseArgs &nz, const float *__restrict__ vd,
                                                  const float *fsc, int bx, int by, int bz) {
    const int b = by * blockDim.y + threadIdx.y;
    const int c = reverse ? g.N2 - 1 - bz : bz;
    const int q = bx * blockDim.x + threadIdx.x;
    const int ngrp = (g.N0 + 8) >> 3;
    const int P0 = 8 * q;
    // points of the colour: padded P with (P - 1 + b + c) & 1 == colour; the
    // two parities get separate code so that every register index is static
    const int j0 = (colour + b + c + 1) & 1;  // first local index j (P = P0 + j) of the colour
    float4 nrm = make_float4(0.f, 0.f, 0.f, 0.f);
    if (EARLY) {
        if (NOISE == NOISE_PHILOX) nrm = fine_normals(nz, g, P0 + j0, b, c);
        pdl_begin();
        pdl_trigger();
    }
    if (q >= ngrp || b >= g.N1) return;
    const i64 rb = (i64)(c + 1) * g.sz + (i64)(b + 1) * g.sy;
    const float4 *xr = reinterpret_cast<const float4 *>(x + rb + P0);
    const float4 *xn = reinterpret_cast<const float4 *>(x + rb - g.sy + P0);
    const float4 *xs_ = reinterpret_cast<const float4 *>(x + rb + g.sy + P0);
    const float4 *xd = reinterpret_cast<const float4 *>(x + rb - g.sz + P0);
    const float4 *xu = reinterpret_cast<const float4 *>(x + rb + g.sz + P0);
    const float4 *fr = reinterpret_cast<const float4 *>(f + rb + P0);
    float v[10], ym[8], yp[8], zm[8], zp[8], fv[8], dv[8];
    const unsigned long long pol_stream = V8 ? l2_evict_first_policy() : 0ull;
    if (VD) {
        if (V8) {
            ld8_stream(vd + rb + P0, dv, pol_stream);
        } else {
            const float4 *dr = reinterpret_cast<const float4 *>(vd + rb + P0);
            const float4 d0 = dr[0], d1 = dr[1];
            dv[0] = d0.x; dv[1] = d0.y; dv[2] = d0.z; dv[3] = d0.w; dv[4] = d1.x; dv[5] = d1.y; dv[6] = d1.z; dv[7] = d1.w;
        }
    }
    if (V8) {
        v[0] = P0 > 0 ? x[rb + P0 - 1] : 0.f;
        ld8(x + rb + P0, v + 1);
        v[9] = x[rb + P0 + 8];
        ld8(x + rb - g.sy + P0, ym);
        ld8(x + rb + g.sy + P0, yp);
        ld8(x + rb - g.sz + P0, zm);
        ld8(x + rb + g.sz + P0, zp);
        if (FS) {
            const float4 fq = ld4_stream(fsc + ((rb + P0) >> 1), pol_stream);
            if (j0 == 0) {
                fv[0] = fq.x; fv[2] = fq.y; fv[4] = fq.z; fv[6] = fq.w;
            } else {
                fv[1] = fq.x; fv[3] = fq.y; fv[5] = fq.z; fv[7] = fq.w;
            }
        } else {
            ld8_stream(f + rb + P0, fv, pol_stream);
        }
    } else {
        const float4 a0 = xr[0], a1 = xr[1];
        v[0] = P0 > 0 ? x[rb + P0 - 1] : 0.f;  // P0 - 1 is a ghost column for q = 0 (read 0 directly)
        v[1] = a0.x; v[2] = a0.y; v[3] = a0.z; v[4] = a0.w;
        v[5] = a1.x; v[6] = a1.y; v[7] = a1.z; v[8] = a1.w;
        v[9] = x[rb + P0 + 8];
        const float4 n0 = xn[0], n1 = xn[1], s0 = xs_[0], s1 = xs_[1], d0 = xd[0], d1 = xd[1], u0 = xu[0], u1 = xu[1];
        const float4 f0 = fr[0], f1 = fr[1];
        ym[0] = n0.x; ym[1] = n0.y; ym[2] = n0.z; ym[3] = n0.w; ym[4] = n1.x; ym[5] = n1.y; ym[6] = n1.z; ym[7] = n1.w;
        yp[0] = s0.x; yp[1] = s0.y; yp[2] = s0.z; yp[3] = s0.w; yp[4] = s1.x; yp[5] = s1.y; yp[6] = s1.z; yp[7] = s1.w;
        zm[0] = d0.x; zm[1] = d0.y; zm[2] = d0.z; zm[3] = d0.w; zm[4] = d1.x; zm[5] = d1.y; zm[6] = d1.z; zm[7] = d1.w;
        zp[0] = u0.x; zp[1] = u0.y; zp[2] = u0.z; zp[3] = u0.w; zp[4] = u1.x; zp[5] = u1.y; zp[6] = u1.z; zp[7] = u1.w;
        fv[0] = f0.x; fv[1] = f0.y; fv[2] = f0.z; fv[3] = f0.w; fv[4] = f1.x; fv[5] = f1.y; fv[6] = f1.z; fv[7] = f1.w;
    }
    if (!EARLY && NOISE == NOISE_PHILOX) nrm = fine_normals(nz, g, P0 + j0, b, c);
    auto upd = [&](int j, int k) {
        const int a = P0 + j - 1;
        if (a < 0 || a >= g.N0) return;
        float xi = 0.f;
        if (NOISE == NOISE_PHILOX) xi = pick(nrm, k);
        if (NOISE == NOISE_INJECTED) xi = (float)nz.buf[g.compact(a, b, c)];
        const float dg = VD ? dv[j] : s.w[13];
        float res = s.w[4] * zm[j];
        res = fmaf(s.w[10], ym[j], res);
        res = fmaf(s.w[12], v[j], res);
        res = fmaf(dg, v[j + 1], res);
        res = fmaf(s.w[14], v[j + 2], res);
        res = fmaf(s.w[16], yp[j], res);
        res = fmaf(s.w[22], zp[j], res);
        float cval = fv[j];
        const float sd = VD ? sqrtf(dg * s.tmo / s.omega) : s.sd;
        if (NOISE != NOISE_NONE) cval = fmaf(sd, xi, cval);
        const float od = VD ? s.omega / dg : s.omega_diag;
        v[j + 1] = v[j + 1] + od * (cval - res);  // neighbours are of the other colour
    };
    if (j0 == 0) {
        upd(0, 0);
        upd(2, 1);
        upd(4, 2);
        upd(6, 3);
    } else {
        upd(1, 0);
        upd(3, 1);
        upd(5, 2);
        upd(7, 3);
    }
    // Whole 8-position spans go back as two float4 stores (full sectors
    // instead of one partial sector per point); the other colour's values
    // are rewritten unchanged -- no thread writes them in this pass.  A span
    // that reaches past its row (short rows only) stores its second half
    // point by point.
    if (V8 && P0 + 8 <= g.sy) {
        st8(x + rb + P0, v + 1);
        return;
    }
    float4 *xo = reinterpret_cast<float4 *>(x + rb + P0);
    xo[0] = make_float4(v[1], v[2], v[3], v[4]);
    if (P0 + 8 <= g.sy) {
        xo[1] = make_float4(v[5], v[6], v[7], v[8]);
    } else {
#pragma unroll
        for (int j = 4; j < 8; ++j) {
            const int a = P0 + j - 1;
            if (((j - j0) & 1) == 0 && a >= 0 && a < g.N0) x[rb + P0 + j] = v[j + 1];
        }
    }
}

template <int NOISE, bool VD, bool V8, bool FS, bool EARLY>
__global__ void __launch_bounds__(RBP_THREADS) k_sweep_rb_vec(float *x, const float *f,
                                                              Grid3 g, StencilArg<float> s, int colour, int reverse,
                                                              NoiseArgs nz, const float *__restrict__ vd,
                                                              const float *fsc) {
    sweep_rb_vec_body<NOISE, VD, V8, FS, EARLY>(x, f, g, s, colour, reverse, nz, vd, fsc, blockIdx.x, blockIdx.y, blockIdx.z);
}

// Level 0's f split by colour for the FP32 fine sweep: the value of point
// (a, b, c) of colour k = (a + b + c) & 1 at fs[k * half + (P >> 1)], P its
// padded index.  With even row and plane pitches, the two points P = 2i,
// 2i + 1 of a row have different colours, so each colour's half holds one
// value per pair, and a span [8q, 8q + 8) of a row maps to one float4.
__global__ void __launch_bounds__(256) k_split_colours(const float *__restrict__ f, float *__restrict__ fs, i64 half,
                                                       Grid3 g) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y, c = blockIdx.z;
    if (a >= g.N0) return;
    const i64 P = g.pad(a, b, c);
    fs[(i64)((a + b + c) & 1) * half + (P >> 1)] = f[P];
}

// One colour of an 8-colour (27-point) sweep, one thread per point (colour
// index (a & 1) | (b & 1) << 1 | (c & 1) << 2).
template <typename T, bool EXACT, int NOISE, int VAR>
__device__ __forceinline__ void sweep_c27_body(T *x, const T *f, const Grid3 &g,
                                               const StencilArg<T> &s, int colour, const NoiseArgs &nz,
                                               const VarField<T> &vf, int bx, int by, int bz) {
    const int pa = colour & 1, pb = (colour >> 1) & 1, pc = (colour >> 2) & 1;
    const int a = 2 * (bx * blockDim.x + threadIdx.x) + pa;
    const int b = 2 * (by * blockDim.y + threadIdx.y) + pb, c = 2 * bz + pc;
    if (b >= g.N1 || c >= g.N2) return;
    T xi = T(0);
    if (NOISE == NOISE_PHILOX) xi = (T)pick(point_normals(nz, g, a, b, c), (a & 7) >> 1);
    if (a >= g.N0) return;
    if (NOISE == NOISE_INJECTED) xi = (T)nz.buf[g.compact(a, b, c)];
    const i64 P = g.pad(a, b, c);
    if (sizeof(T) == 4 && (g.sy & 1) == 0 && (g.sz & 1) == 0) {
        // FP32, even pitches: the points of a colour share the parity of P,
        // and each of the nine rows of the stencil is one aligned pair load
        // plus one single load (the threads of a warp, two points apart, then
        // read whole sectors); the same values in the same order as
        // sor_point.  (Measured at 256^3: FP32 step 0.766 -> 0.759 ms; the
        // FP64 chain was 0.4 % slower with 16-byte pairs and keeps sor_point.)
        typedef typename std::conditional<sizeof(T) == 4, float2, double2>::type T2;
        const bool odd = (P & 1) != 0;
        T v[27];
#pragma unroll
        for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
            for (int dy = -1; dy <= 1; ++dy) {
                const T *r = x + P + dz * g.sz + dy * g.sy;
                const int k = (dz + 1) * 9 + (dy + 1) * 3;
                if (odd) {
                    const T2 q = *reinterpret_cast<const T2 *>(r - 1);
                    v[k] = q.x;
                    v[k + 1] = q.y;
                    v[k + 2] = r[1];
                } else {
                    const T2 q = *reinterpret_cast<const T2 *>(r);
                    v[k] = r[-1];
                    v[k + 1] = q.x;
                    v[k + 2] = q.y;
                }
            }
        x[P] = sor_value<T, 27, EXACT, VAR>([&](int dz, int dy, int dx) { return v[(dz + 1) * 9 + (dy + 1) * 3 + dx + 1]; },
                                            v[13], f[P], s, P, NOISE != NOISE_NONE, xi, vf);
        return;
    }
    sor_point<T, 27, EXACT, VAR>(x, f, g, s, P, NOISE != NOISE_NONE, xi, vf);
}

template <typename T, bool EXACT, int NOISE, int VAR = 0>
__global__ void __launch_bounds__(RBP_THREADS) k_sweep_c27_pass(T *x, const T *f, Grid3 g,
                                                                StencilArg<T> s, int colour, NoiseArgs nz,
                                                                VarField<T> vf) {
    if (g.pdl) pdl_begin();
    sweep_c27_body<T, EXACT, NOISE, VAR>(x, f, g, s, colour, nz, vf, blockIdx.x, blockIdx.y, blockIdx.z);
}

// ------------------------------------------- two colours of a row per launch
// The colours of a 27-point (9-point in 2D) level come in pairs that share
// the parities of b and c and differ in the parity of a.  A point of the
// second colour of a pair has neighbours of the first one in its own row
// only, so a CTA that owns whole rows runs both colours of the pair: the
// rows around are read once for both, and a sweep takes half the launches.
// The update of every point, the order of its sum included, is that of the
// one-colour pass.
//
// What bounds it: on levels of up to 63^3 points the round trip of one
// dependent launch (parameters, one L2 load, the sum, one store), above that
// the L2 traffic.  The normals do not depend on the launch before, so they
// are drawn before the wait for it (`wait`), and with `trigger` the next
// launch's CTAs start, and draw theirs, while this one's loads are in flight.
// (GB300, a whole sweep with Philox noise in a graph of dependent launches,
// one-colour passes -> row pairs: FP32 127^3 31.5 -> 14.9 us, 63^3 15.4 ->
// 6.2, 31^3 14.1 -> 5.9; FP64 31^3 22.3 -> 13.0, 15^3 20.8 -> 12.7; FP32 rows
// of 255, 383 and 511 points, 64 x 64 of them: 22.6 -> 11.3, 27.7 -> 16.4, 31.8
// -> 17.3.  FP64 levels above 2^18 points that add weight by weight choose at
// set-up: see autotune_sweeps.)
//
// Thread t of a row owns the points 2t and 2t + 1: the four positions 2t ..
// 2t + 3 of the nine (three) rows around, two aligned pair loads each where
// the pitches are even.  One Philox block holds the normals of four points
// of one parity of a group of eight, so of the four threads of a group the
// even ones draw the even points' block, the odd ones the odd points', and
// neighbours swap.
constexpr int ROW_PAIR_THREADS = 256;                 // most threads of a CTA
constexpr int ROW_PAIR_MAX_N0 = 2 * ROW_PAIR_THREADS; // longest row a CTA can own

template <typename T>
struct Pair;
template <>
struct Pair<float> {
    typedef float2 type;
};
template <>
struct Pair<double> {
    typedef double2 type;
};

template <typename T, int NPT, bool EXACT, int NOISE, int VAR>
__device__ __forceinline__ void sweep_row_pair_body(T *x, const T *f, const Grid3 &g,
                                                    const StencilArg<T> &s, int pb, int pc, int odd_first,
                                                    const NoiseArgs &nz, const VarField<T> &vf, int by, int bz,
                                                    T *sh, bool wait, bool trigger) {
    constexpr int NR = NPT == 9 ? 3 : 9;  // rows of the stencil
    const int t = threadIdx.x, a0 = 2 * t;
    const int b = 2 * (by * blockDim.y + threadIdx.y) + pb, c = 2 * bz + pc;
    const bool row_in = b < g.N1 && c < g.N2;
    const bool in0 = row_in && a0 < g.N0, in1 = row_in && a0 + 1 < g.N0;
    T xi0 = T(0), xi1 = T(0);
    if (NOISE == NOISE_PHILOX) {  // point_normals of the two points
        const unsigned G0 = (unsigned)((g.N0 + 7) >> 3);
        const unsigned grp = (unsigned)(((u64)c * g.N1 + b) * G0 + (t >> 2));
        const float4 r = normals4(philox4x32_10(noise_ctr(nz, grp, PURPOSE_POINT, t & 1), noise_key(nz)));
        const float own = pick(r, t & 3), other = __shfl_xor_sync(0xffffffffu, pick(r, (t & 3) ^ 1), 1);
        xi0 = (T)((t & 1) ? other : own);
        xi1 = (T)((t & 1) ? own : other);
    }
    if (wait) pdl_begin();
    if (trigger) pdl_trigger();
    const i64 P = g.pad(a0, b, c);
    if (NOISE == NOISE_INJECTED) {
        if (in0) xi0 = (T)nz.buf[g.compact(a0, b, c)];
        if (in1) xi1 = (T)nz.buf[g.compact(a0 + 1, b, c)];
    }
    T v[NR][4], f0 = T(0), f1 = T(0);
    if (in0) {
        f0 = f[P];
        if (in1) f1 = f[P + 1];
        const bool even = (g.sy & 1) == 0 && (g.sz & 1) == 0;  // then P - 1 is even too
        typedef typename Pair<T>::type T2;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const T *q = x + P - 1 + (NR == 9 ? (r / 3 - 1) * g.sz : 0) + (r % 3 - 1) * g.sy;
            if (even) {
                const T2 u = *reinterpret_cast<const T2 *>(q), w = *reinterpret_cast<const T2 *>(q + 2);
                v[r][0] = u.x;
                v[r][1] = u.y;
                v[r][2] = w.x;
                v[r][3] = w.y;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) v[r][j] = j < 3 || in1 ? q[j] : T(0);
            }
        }
    }
    constexpr int OWN = NR / 2;
    auto updated = [&](int o, T fv, T xi) {  // point 2t + o
        return sor_value<T, NPT, EXACT, VAR>(
            [&](int dz, int dy, int dx) { return v[(NR == 9 ? (dz + 1) * 3 : 0) + dy + 1][1 + o + dx]; }, v[OWN][1 + o],
            fv, s, P + o, NOISE != NOISE_NONE, xi, vf);
    };
    // the first colour's new values reach the neighbouring threads through
    // shared memory (one slot per thread and row, one more at the row's end)
    T *row = sh + threadIdx.y * (blockDim.x + 1);
    if (!odd_first) {
        T n = T(0);
        if (in0) x[P] = n = v[OWN][1] = updated(0, f0, xi0);
        row[t] = n;
        if (t == 0) row[blockDim.x] = T(0);
        __syncthreads();
        v[OWN][3] = row[t + 1];
        if (in1) x[P + 1] = updated(1, f1, xi1);
    } else {
        T n = T(0);
        if (in1) x[P + 1] = n = v[OWN][2] = updated(1, f1, xi1);
        row[t + 1] = n;
        if (t == 0) row[0] = T(0);
        __syncthreads();
        v[OWN][0] = row[t];
        if (in0) x[P] = updated(0, f0, xi0);
    }
}

template <typename T, int NPT, bool EXACT, int NOISE, int VAR>
__global__ void __launch_bounds__(ROW_PAIR_THREADS)
    k_sweep_row_pair(T *x, const T *f, Grid3 g, StencilArg<T> s, int pb, int pc, int odd_first,
                     NoiseArgs nz, VarField<T> vf, int trigger) {
    extern __shared__ __align__(16) unsigned char row_sm[];
    sweep_row_pair_body<T, NPT, EXACT, NOISE, VAR>(x, f, g, s, pb, pc, odd_first, nz, vf, blockIdx.y, blockIdx.z,
                                                   reinterpret_cast<T *>(row_sm), g.pdl != 0, trigger != 0);
}

// The same pair of colours for FP64 chains whose constant stencil has equal
// weights at +-dx, +-dy, +-dz (Level::sym).  GB300 issues about two FP64
// operations per clock per SM -- one instruction of a warp holds the FP64
// unit of its SM partition for 64 clocks -- so the count of FP64
// instructions is what a launch takes.  The rows around are first added by
// class (|dy|, |dz|), each sum is shared with the two neighbours in x, and
// the diagonal term drops out of x + (omega / d)(c - sum):
//   x'' = (1 - omega) x + (omega / d)(sd xi + f - sum over the neighbours),
// 21 FP64 instructions per point instead of 30 (8 instead of 30 in 2D, where
// the one-colour pass also multiplied the zero weights of the planes above
// and below).  One thread per point: a warp per 32 points spreads a small
// level over more FP64 units than two points per thread do.
constexpr int ROW_SYM_THREADS = 512;  // most threads of a CTA, and the longest row

template <int NPT, int NOISE, bool UNIT>
__global__ void __launch_bounds__(ROW_SYM_THREADS)
    k_sweep_row_sym(double *x, const double *f, Grid3 g, SymWeights w, int pb, int pc,
                    int odd_first, NoiseArgs nz, int trigger) {
    constexpr int NC = NPT == 9 ? 1 : 3;  // classes beside the own row
    extern __shared__ __align__(16) unsigned char row_sm[];
    const int a = threadIdx.x;
    const int b = 2 * (blockIdx.y * blockDim.y + threadIdx.y) + pb, c = 2 * blockIdx.z + pc;
    const bool in = a < g.N0 && b < g.N1 && c < g.N2;
    double xi = 0.0;
    if (NOISE == NOISE_PHILOX) xi = widen(pick(point_normals(nz, g, a, b, c), (a & 7) >> 1));
    if (g.pdl) pdl_begin();
    if (trigger) pdl_trigger();
    const i64 P = g.pad(a, b, c);
    // position a + 1 of the class rows; positions 0 and N0 + 1 are ghosts
    const int pitch = blockDim.x + 2;
    double *row = reinterpret_cast<double *>(row_sm) + threadIdx.y * (NC + 1) * pitch + 1 + a;
    double s[NC + 1], cv = 0.0;
#pragma unroll
    for (int k = 0; k <= NC; ++k) s[k] = 0.0;
    if (in) {
        const double *q = x + P;
        s[0] = q[0];
        s[1] = q[-g.sy] + q[g.sy];
        if (NPT == 27) {
            s[2] = q[-g.sz] + q[g.sz];
            s[3] = (q[-g.sz - g.sy] + q[-g.sz + g.sy]) + (q[g.sz - g.sy] + q[g.sz + g.sy]);
        }
        cv = f[P];
    }
#pragma unroll
    for (int k = 0; k <= NC; ++k) {
        row[k * pitch] = s[k];
        if (a == 0) row[k * pitch - 1] = 0.0;
        if (a == blockDim.x - 1) row[k * pitch + 1] = 0.0;
    }
    __syncthreads();
    if (NOISE != NOISE_NONE) cv = fma(w.sd, xi, cv);
#pragma unroll
    for (int k = 1; k <= NC; ++k) {
        cv = fma(-w.wc[2 * k], s[k], cv);
        cv = fma(-w.wc[2 * k + 1], row[k * pitch - 1] + row[k * pitch + 1], cv);
    }
    const double keep = UNIT ? 0.0 : w.om1 * s[0];
    // own row: the first colour, then the second one from its new values
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if ((a & 1) == (h ^ odd_first)) {
            const double c1 = fma(-w.wc[1], row[-1] + row[1], cv);
            const double v = UNIT ? keep_nonfinite(w.od * c1, s[0]) : fma(w.od, c1, keep);
            if (h == 0) row[0] = v;
            if (in) x[P] = v;
            if (h == 0 && !in) row[0] = 0.0;
        }
        if (h == 0) __syncthreads();
    }
}

// ------------------------------------------------ lexicographic wavefront
// Lexicographic order as hyperplanes t = a + hb b + hc c: every neighbour
// that precedes a point lexicographically lies on an earlier hyperplane
// ((1,1,1) for axis stencils, (1,2,4) for 27-point stencils), points on one
// hyperplane are independent.  One CTA, one __syncthreads per hyperplane.
template <typename T, int NPT, bool EXACT, int NOISE>
__global__ void __launch_bounds__(1024) k_sweep_wavefront(T *x, const T *f, Grid3 g,
                                                           StencilArg<T> s, int forward, int hb, int hc, NoiseArgs nz) {
    if (g.pdl) pdl_begin();
    const int tmax = (g.N0 - 1) + hb * (g.N1 - 1) + hc * (g.N2 - 1);
    const int npair = g.N1 * g.N2;
    for (int step = 0; step <= tmax; ++step) {
        const int t = forward ? step : tmax - step;
        for (int pr = threadIdx.x; pr < npair; pr += blockDim.x) {
            int b = pr % g.N1, c = pr / g.N1;
            int a = t - hb * b - hc * c;
            if (a < 0 || a >= g.N0) continue;
            T xi = T(0);
            if (NOISE == NOISE_PHILOX) xi = (T)pick(point_normals(nz, g, a, b, c), (a & 7) >> 1);
            if (NOISE == NOISE_INJECTED) xi = (T)nz.buf[g.compact(a, b, c)];
            sor_point<T, NPT, EXACT>(x, f, g, s, g.pad(a, b, c), NOISE != NOISE_NONE, xi);
        }
        __syncthreads();
    }
}

// ----------------------------------------------------------- reductions
template <int NT>
__device__ __forceinline__ double block_sum(double v, double *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = v;
    __syncthreads();
    v = (threadIdx.x < NT / 32) ? sh[threadIdx.x] : 0.0;
    if (w == 0) {  // the sum of NT / 32 values, in lane 0
#pragma unroll
        for (int o = NT / 64; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    __syncthreads();
    return v;  // valid in thread 0
}

// block_sum over the 256 threads of a two-dimensional CTA
__device__ __forceinline__ double block_sum_2d(double v, double *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int t = threadIdx.y * blockDim.x + threadIdx.x;
    if ((t & 31) == 0) sh[t >> 5] = v;
    __syncthreads();
    v = t < 8 ? sh[t] : 0.0;
    if (t < 32) {
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    return v;  // valid in thread 0
}

// ------------------------------------------------ float-float arithmetic
// An unevaluated sum hi + lo of two FP32 numbers carries about 48
// significant bits.  GB300 issues about two FP64 FMAs per clock per SM
// against 128 FP32 ones, so the FP32 chain forms the cross-thread sums of
// B^T x and the low-rank m x m product in this arithmetic instead of FP64.
// Error-free transformations: TwoSum (Knuth, TAOCP vol. 2, 4.2.2), Fast
// TwoSum (Dekker 1971) and TwoProd with an FMA (Ogita, Rump, Oishi,
// "Accurate sum and dot product", SIAM J. Sci. Comput. 26, 2005).  The _rn
// intrinsics keep the compiler from contracting a product and a sum into one
// FMA, which would break the transformations.
struct ff32 {
    float hi, lo;
};

__device__ __forceinline__ ff32 two_sum(float a, float b) {  // s + e == a + b exactly
    const float s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ ff32 fast_two_sum(float a, float b) {  // exact when |a| >= |b| or a == 0
    const float s = __fadd_rn(a, b);
    return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
// (a.hi + a.lo) + (b.hi + b.lo): both parts summed with TwoSum, then
// renormalised twice (accurate under cancellation).  Symmetric in a and b
// bit for bit, since TwoSum's error term is the exact error.
__device__ __forceinline__ ff32 ff_add(ff32 a, ff32 b) {
    ff32 s = two_sum(a.hi, b.hi);
    const ff32 t = two_sum(a.lo, b.lo);
    s = fast_two_sum(s.hi, __fadd_rn(s.lo, t.hi));
    return fast_two_sum(s.hi, __fadd_rn(s.lo, t.lo));
}
// (a.hi + a.lo) (b.hi + b.lo) without the a.lo b.lo term
__device__ __forceinline__ ff32 ff_mul(ff32 a, ff32 b) {
    const float p = __fmul_rn(a.hi, b.hi);
    float e = __fmaf_rn(a.hi, b.hi, -p);
    e = __fmaf_rn(a.hi, b.lo, e);
    e = __fmaf_rn(a.lo, b.hi, e);
    return fast_two_sum(p, e);
}
__device__ __forceinline__ ff32 ff_neg(ff32 a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ ff32 ff_of(float2 v) { return {v.x, v.y}; }
__device__ __forceinline__ double ff_to_double(ff32 a) { return (double)a.hi + (double)a.lo; }
__device__ __forceinline__ float ff_to_float(ff32 a) { return __fadd_rn(a.hi, a.lo); }

// A sum of products of a thread.  FP32 values: the products and the sum with
// their rounding errors (exact products, TwoSum), so that a sum whose terms
// cancel keeps the bits of its result.  FP64: one FMA per term.
template <typename T>
struct ProductSum {
    T hi = T(0), lo = T(0);
    __device__ __forceinline__ void add(T w, T v) {
        if constexpr (sizeof(T) == 4) {
            const float p = __fmul_rn(w, v);
            const ff32 s = two_sum(hi, p);
            lo = __fadd_rn(lo, __fadd_rn(s.lo, __fmaf_rn(w, v, -p)));
            hi = s.hi;
        } else {
            hi = fma(w, v, hi);
        }
    }
    __device__ __forceinline__ double value() const { return sizeof(T) == 4 ? (double)hi + (double)lo : (double)hi; }
};

// block_sum's shuffle tree in float-float; the result is valid in thread 0
template <int NT>
__device__ __forceinline__ ff32 block_sum_ff(ff32 v, float2 *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v = ff_add(v, ff32{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)});
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) sh[w] = make_float2(v.hi, v.lo);
    __syncthreads();
    v = (threadIdx.x < NT / 32) ? ff_of(sh[threadIdx.x]) : ff32{0.f, 0.f};
    if (w == 0) {
#pragma unroll
        for (int o = NT / 64; o > 0; o >>= 1)
            v = ff_add(v, ff32{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)});
    }
    __syncthreads();
    return v;
}

// Low-rank arguments of one level and sweep direction.
struct LowRankArg {
    int m;
    const i64 *Bptr;    // m+1, CSC of B
    const unsigned *Bidx;  // padded indices (levels below 2^32 padded points)
    const double *Bval;
    const double *SinvT; // m x m, S^{-1} = (Sigma + B^T M^{-1} B)^{-1}, transposed (column q contiguous)
    const double *sigma_sqrt; // Sigma^{1/2}
    double *y;          // m scratch: B^T x
    const float *Bvalf; // B values rounded to FP32 (FP32 chain)
    double *part;       // m x P scratch: partial sums of B^T x (the FP32 chain
                        // stores float-float pairs, float2, in the same slots)
    unsigned *counter;  // CTA counter of k_bt_full (reset by its last CTA)
    void *w;                     // m scratch: Sigma^{1/2} xi' (double, or float2 for the FP32 chain)
    double *zpub;                // where the solve leaves z (null: nowhere)
    void *zv;                    // m scratch: z of k_lr_z in the chain's type
    const float2 *SinvT_ff;      // SinvT as float-float pairs (FP32 chain)
    const float2 *sigma_sqrt_ff; // Sigma^{1/2} as float-float pairs (FP32 chain)
};

// Partial sums of y_j = sum_i B_ij x_i: gridDim.y CTAs per column j, CTA p
// writing part[j * P + p].  Each thread issues eight index/value loads, then
// the eight gathers of x, before it accumulates them in entry order; the
// per-thread sums are in the state's precision (FP32 products for the FP32
// chain) and are combined across the CTA in FP64, or in float-float for the
// FP32 chain (stored as a float2 in the slot).  B does not change, so a
// thread's first index/value loads are issued before the wait for the
// kernel that wrote x (`wait`: the caller has not waited yet).
template <typename T>
__device__ __forceinline__ void bt_partial_cta(const T *x, const LowRankArg &lr, double *sh, int j, int p, int P) {
    const i64 e0 = lr.Bptr[j], e1 = lr.Bptr[j + 1];
    const i64 len = P == 1 ? e1 - e0 : (e1 - e0 + P - 1) / P;
    const i64 lo = e0 + p * len, hi = min(e1, lo + len);
    T tacc = T(0);
    i64 idx[8];
    T val[8];
    auto load = [&](i64 e) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const i64 ee = e + 256 * k;
            idx[k] = ee < hi ? (i64)lr.Bidx[ee] : -1;
            val[k] = ee < hi ? (sizeof(T) == 4 ? (T)lr.Bvalf[ee] : (T)lr.Bval[ee]) : T(0);
        }
    };
    i64 e = lo + threadIdx.x;
    load(e);
    pdl_begin();
    pdl_trigger();  // the correction's rows, S^{-1} and normals load meanwhile
    // eight index/value loads, then the eight gathers, in flight at once;
    // the products are added in entry order
    for (; e < hi; e += 8 * 256) {
        T xv[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) xv[k] = idx[k] >= 0 ? x[idx[k]] : T(0);
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (idx[k] >= 0) tacc += val[k] * xv[k];
        if (e + 8 * 256 < hi) load(e + 8 * 256);
    }
    if (sizeof(T) == 4) {
        const ff32 acc = block_sum_ff<256>(ff32{(float)tacc, 0.f}, reinterpret_cast<float2 *>(sh));
        if (threadIdx.x == 0) reinterpret_cast<float2 *>(lr.part)[j * P + p] = make_float2(acc.hi, acc.lo);
    } else {
        const double acc = block_sum<256>((double)tacc, sh);
        if (threadIdx.x == 0) lr.part[j * P + p] = acc;
    }
}

// Also the low-rank noise Sigma^{1/2} xi' of the column (lr.w, unless null),
// drawn before the wait by a thread that has little else to do.
template <typename T, int NOISE>
__device__ __forceinline__ void bt_partial_body(const T *x, const LowRankArg &lr, const NoiseArgs &nz, int j, int p, int P) {
    __shared__ double sh[32];
    const bool draws = lr.w && p == 0 && threadIdx.x == 255;
    float xif = 0.f;
    if (draws && NOISE == NOISE_PHILOX)
        xif = pick(normals4(philox4x32_10(noise_ctr(nz, (unsigned)(j >> 2), PURPOSE_LOWRANK, 0), noise_key(nz))), j & 3);
    bt_partial_cta<T>(x, lr, sh, j, p, P);
    if (draws) {
        if constexpr (sizeof(T) == 4) {
            const ff32 w = ff_mul(ff_of(lr.sigma_sqrt_ff[j]), ff32{NOISE == NOISE_INJECTED ? (float)nz.buf[j] : xif, 0.f});
            static_cast<float2 *>(lr.w)[j] = make_float2(w.hi, w.lo);
        } else {
            static_cast<double *>(lr.w)[j] = lr.sigma_sqrt[j] * (NOISE == NOISE_INJECTED ? nz.buf[j] : widen(xif));
        }
    }
}

template <typename T, int NOISE>
__global__ void __launch_bounds__(256) k_bt_partial(const T *x, LowRankArg lr, NoiseArgs nz) {
    bt_partial_body<T, NOISE>(x, lr, nz, blockIdx.x, blockIdx.y, gridDim.y);
}

// One CTA: y_k = sum_p part[k * P + p] (fixed order, so the result does not
// depend on block timing), in float-float for the FP32 chain
template <typename T>
__device__ __forceinline__ void bt_sum_cta(const LowRankArg &lr, int P) {
    for (int k = threadIdx.x; k < lr.m; k += blockDim.x) {
        if constexpr (sizeof(T) == 4) {
            const float2 *part = reinterpret_cast<const float2 *>(lr.part) + (i64)k * P;
            ff32 t{0.f, 0.f};
            for (int p0 = 0; p0 < P; p0 += 8) {
                float2 pp[8];
#pragma unroll
                for (int r = 0; r < 8; ++r) pp[r] = p0 + r < P ? __ldcg(part + p0 + r) : make_float2(0.f, 0.f);
#pragma unroll
                for (int r = 0; r < 8; ++r)
                    if (p0 + r < P) t = ff_add(t, ff_of(pp[r]));
            }
            lr.y[k] = ff_to_double(t);
        } else {
            double t = 0.0;
            for (int p0 = 0; p0 < P; p0 += 8) {
                double pp[8];
#pragma unroll
                for (int r = 0; r < 8; ++r) pp[r] = p0 + r < P ? __ldcg(lr.part + (i64)k * P + p0 + r) : 0.0;
#pragma unroll
                for (int r = 0; r < 8; ++r)
                    if (p0 + r < P) t += pp[r];
            }
            lr.y[k] = t;
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(256) k_bt_sum(LowRankArg lr, int P) {
    pdl_begin();
    bt_sum_cta<T>(lr, P);
}

// y = B^T x in one launch: the last CTA to finish (block counter, reset by
// that CTA) adds the partial sums in k_bt_sum's order.  The thread that wrote
// the CTA's partial sum counts it with an acquire-release atomic, which orders
// that write before the count and, in the last CTA, the other CTAs' sums
// before the barrier after which its threads read them.
template <typename T>
__global__ void __launch_bounds__(256) k_bt_full(const T *x, LowRankArg lr) {
    __shared__ double sh[32];
    __shared__ bool last;
    bt_partial_cta<T>(x, lr, sh, blockIdx.x, blockIdx.y, gridDim.y);
    if (threadIdx.x == 0) {
        unsigned prev;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(prev) : "l"(lr.counter) : "memory");
        last = prev == gridDim.x * gridDim.y - 1u;
        if (last) *lr.counter = 0u;
    }
    __syncthreads();
    if (last) bt_sum_cta<T>(lr, gridDim.y);
}

// Support rows of C = M^{-1} B as x += C z reads them: the rows with one
// entry -- nearly all, since the measurement balls rarely overlap -- as
// (row, column, value) triples, the others in CSR form.  Padded row indices
// are 32-bit (levels of fewer than 2^32 padded points).
struct CorrRows {
    i64 n1 = 0, nm = 0;            // rows with one entry / with several
    const unsigned *r1 = nullptr;  // n1 padded row indices
    const int *c1 = nullptr;       // their columns
    const void *v1 = nullptr;      // their values (type T)
    const unsigned *rm = nullptr;  // nm padded row indices
    const int *pm = nullptr;       // nm + 1 offsets into cm / vm
    const int *cm = nullptr;
    const void *vm = nullptr;
};

// Four single-entry rows of a thread, r0 + j stride (j < 4) of the n rows from
// `base` on: row index, column, value and state loaded together, before the wait
// (the state through L2: see k_lr_correct); the update adds the product to zero,
// then to the state, as a multi-entry row's (FP64: one FMA).
template <typename T>
struct CorrQuad {
    unsigned row[4];
    int col[4];
    T val[4], xv[4];
    __device__ __forceinline__ void load(const T *x, const CorrRows &C, i64 base, int r0, int stride, int n) {
        const unsigned *r1 = C.r1 + base;
        const int *c1 = C.c1 + base;
        const T *v1 = static_cast<const T *>(C.v1) + base;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = r0 + j * stride;
            const bool ok = r < n;
            row[j] = ok ? r1[r] : 0u;
            col[j] = ok ? c1[r] : 0;
            val[j] = ok ? v1[r] : T(0);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            xv[j] = r0 + j * stride < n ? __ldcg(x + row[j]) : T(0);
    }
    template <typename ZT>
    __device__ __forceinline__ void apply(T *x, int r0, int stride, int n, const ZT *z) const {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (r0 + j * stride >= n) continue;
            if (sizeof(T) == 4) {
                T acc = T(0);
                acc += val[j] * (T)z[col[j]];
                x[row[j]] = xv[j] + acc;
            } else {  // one FP64 instruction instead of two
                x[row[j]] = fma(val[j], (T)z[col[j]], xv[j]);
            }
        }
    }
};

// One multi-entry row r (two entries at least) with its row index, entry
// range, first PF entries and state loaded together, before the wait; its
// products are added to zero in entry order, then to the state.
template <typename T, int PF>
struct CorrMulti {
    unsigned row;
    int e0, e1, col[PF];
    T val[PF], xv;
    __device__ __forceinline__ void load(const T *x, const CorrRows &C, i64 r) {
        const T *vm = static_cast<const T *>(C.vm);
        row = C.rm[r];
        e0 = C.pm[r];
        e1 = C.pm[r + 1];
#pragma unroll
        for (int k = 0; k < PF; ++k)
            if (k < 2 || e0 + k < e1) {
                col[k] = C.cm[e0 + k];
                val[k] = vm[e0 + k];
            }
        xv = __ldcg(x + row);
    }
    template <typename ZT>
    __device__ __forceinline__ void apply(T *x, const CorrRows &C, const ZT *z) const {
        const T *vm = static_cast<const T *>(C.vm);
        T acc = T(0);
#pragma unroll
        for (int k = 0; k < PF; ++k)
            if (k < 2 || e0 + k < e1) acc += val[k] * (T)z[col[k]];
#pragma unroll 4
        for (int e = e0 + PF; e < e1; ++e) acc += vm[e] * (T)z[C.cm[e]];
        x[row] = xv + acc;
    }
};

// Low-rank solve and correction in one launch, x += C z with
// z = S^{-1}(Sigma^{1/2} xi' - y).  A CTA takes a run of rows of C (single- or
// multi-entry ones, both sorted by column).  MODE 0, up to LRC_MAX_M columns
// and mostly single-entry rows: it forms the z of the columns of its own rows
// only, their products one per thread.  MODE 1, the same where columns overlap
// throughout (coarse levels): all of z, S^{-1} loaded before the wait.  MODE 2,
// more columns, or overlapping ones on more CTAs than should repeat the solve:
// z comes from a launch of its own (k_lr_z).  The FP32 chain forms every z_k of
// modes 0 and 1 in the same order wherever it is formed (256 / m groups of
// terms per column, two alternating sums in a group), so all CTAs and the
// batched kernels agree bit for bit.
//
// What bounds it is the chain of dependent loads and sums behind the launch
// that gathered x, so everything that does not depend on it -- the rows of C
// with the state they correct, S^{-1} -- is loaded before the wait, while
// k_bt_partial gathers (it lets this kernel start once the sweep has
// completed, so the state is final; it is read through L2, the level at which
// the sweep's writes are visible), and few registers keep all CTAs of a large
// support resident.  (Gather and correction behind a short launch, the
// kernels before -> these: FP64 m = 32, 8,000 rows 7.5 -> 4.5 us, 54,000 rows
// 9.4 -> 6.0; FP32 m = 64, 19,000 rows 7.1 -> 4.4, 256,000 rows 9.6 -> 4.8.)
constexpr int LRC_MAX_M = 64, LRC_MAX_COLS = 16;  // columns of S^{-1} in modes 0 and 1, and of a CTA's rows in mode 0

struct CorrJob {
    i64 r0;          // first row (a level may have more than 2^31 single-entry rows)
    int n;           // rows
    int multi;       // of the multi-entry rows
    int c0, nc;      // their columns: cols[c0 .. c0 + nc)
};
// in the list of columns: the first CTA that has the column
constexpr int CORR_OWNER = 1 << 30;

// u = Sigma^{1/2} xi' - y, the partial sums of y in order (a CTA of 256 threads)
template <typename T, typename V>
__device__ __forceinline__ void lr_rhs(const LowRankArg &lr, int P, V *u) {
    for (int k = threadIdx.x; k < lr.m; k += 256) {
        const V *part = reinterpret_cast<const V *>(lr.part) + (i64)k * P;
        const V w = __ldcg(static_cast<const V *>(lr.w) + k);
        if constexpr (sizeof(T) == 4) {
            ff32 t{0.f, 0.f};
            for (int p0 = 0; p0 < P; p0 += 4) {
                float2 pp[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) pp[r] = p0 + r < P ? __ldcg(part + p0 + r) : make_float2(0.f, 0.f);
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (p0 + r < P) t = ff_add(t, ff_of(pp[r]));
            }
            const ff32 uk = ff_add(ff_of(w), ff_neg(t));
            u[k] = make_float2(uk.hi, uk.lo);
        } else {
            double t = 0.0;
            for (int p0 = 0; p0 < P; p0 += 4) {
                double pp[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) pp[r] = p0 + r < P ? __ldcg(part + p0 + r) : 0.0;
                t += (pp[0] + pp[1]) + (pp[2] + pp[3]);
            }
            u[k] = w - t;
        }
    }
}

// z = S^{-1} u, LRZ_COLS values per CTA: a lane per column, warp w the terms w,
// w + 8, ..., the warps' sums added in order.  The first LRZ_PF of a thread's
// entries of S^{-1} are loaded before the wait.
constexpr int LRZ_COLS = 32, LRZ_PF = 16;
template <typename T>
__device__ __forceinline__ void lr_z_body(const LowRankArg &lr, int P, int tile, double *dyn) {
    typedef typename std::conditional<sizeof(T) == 4, float2, double>::type V;  // FP32 chain: float-float
    const int m = lr.m, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, k = tile * LRZ_COLS + lane;
    V *u = reinterpret_cast<V *>(dyn), *pr = u + m;
    const V *Sinv;
    if constexpr (sizeof(T) == 4)
        Sinv = lr.SinvT_ff;
    else
        Sinv = lr.SinvT;
    Sinv += k;
    auto entry = [&](int c) {  // zero beyond the m terms and columns
        if constexpr (sizeof(T) == 4)
            return c < m && k < m ? __ldg(Sinv + (i64)c * m) : make_float2(0.f, 0.f);
        else
            return c < m && k < m ? __ldg(Sinv + (i64)c * m) : 0.0;
    };
    V first[LRZ_PF];
#pragma unroll
    for (int i = 0; i < LRZ_PF; ++i) first[i] = entry(warp + 8 * i);
    pdl_begin();
    pdl_trigger();
    lr_rhs<T>(lr, P, u);
    __syncthreads();
    if constexpr (sizeof(T) == 4) {
        ff32 t[2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
        for (int i = 0; i < LRZ_PF; ++i)
            if (warp + 8 * i < m) t[i & 1] = ff_add(t[i & 1], ff_mul(ff_of(first[i]), ff_of(u[warp + 8 * i])));
        for (int c0 = warp + 8 * LRZ_PF; c0 < m; c0 += 64) {
            float2 s[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) s[i] = entry(c0 + 8 * i);
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (c0 + 8 * i < m) t[i & 1] = ff_add(t[i & 1], ff_mul(ff_of(s[i]), ff_of(u[c0 + 8 * i])));
        }
        const ff32 a = ff_add(t[0], t[1]);
        pr[warp * 32 + lane] = make_float2(a.hi, a.lo);
        __syncthreads();
        if (warp > 0 || k >= m) return;
        ff32 z{0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 8; ++i) z = ff_add(z, ff_of(pr[i * 32 + lane]));
        static_cast<float *>(lr.zv)[k] = ff_to_float(z);
        if (lr.zpub) lr.zpub[k] = ff_to_double(z);
    } else {
        double t[2] = {0.0, 0.0};
#pragma unroll
        for (int i = 0; i < LRZ_PF; ++i)
            if (warp + 8 * i < m) t[i & 1] = fma(first[i], u[warp + 8 * i], t[i & 1]);
        for (int c0 = warp + 8 * LRZ_PF; c0 < m; c0 += 64) {
            double s[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) s[i] = entry(c0 + 8 * i);
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (c0 + 8 * i < m) t[i & 1] = fma(s[i], u[c0 + 8 * i], t[i & 1]);
        }
        pr[warp * 32 + lane] = t[0] + t[1];
        __syncthreads();
        if (warp > 0 || k >= m) return;
        double z = 0.0;
#pragma unroll
        for (int i = 0; i < 8; ++i) z += pr[i * 32 + lane];
        static_cast<double *>(lr.zv)[k] = z;
        if (lr.zpub) lr.zpub[k] = z;
    }
}

template <typename T>
__global__ void __launch_bounds__(256) k_lr_z(LowRankArg lr, int P) {
    extern __shared__ double dyn[];
    lr_z_body<T>(lr, P, blockIdx.x, dyn);
}

// PF entries of a multi-entry row are loaded ahead: 8 in k_lr_correct's mode 1
// (coarse rows have many: 2D 768 x 480 FP64 step 2.5 % faster than with 2, 3D
// 128^3 1.3 %), 2 in the batch, whose CTAs need the registers to be resident
// (20 chains: 2.5 % slower with 8).
template <typename T, int MODE, int NQ, int PF = 2>
__device__ __forceinline__ void lr_correct_body(T *x, const LowRankArg &lr, int P, const CorrRows &C, const CorrJob &jb,
                                                const int *__restrict__ jobcols, bool first, double *dyn) {
    typedef typename std::conditional<sizeof(T) == 4, float2, double>::type V;  // FP32 chain: float-float
    const int m = lr.m, tid = threadIdx.x;
    V *u = reinterpret_cast<V *>(dyn), *pr = u + m;
    T *zs = MODE == 2 ? reinterpret_cast<T *>(dyn) : reinterpret_cast<T *>(pr + (MODE ? 256 : 64 * 8));
    const V *Sinv;
    if constexpr (sizeof(T) == 4)
        Sinv = lr.SinvT_ff;
    else
        Sinv = lr.SinvT;
    CorrQuad<T> q[NQ];
    CorrMulti<T, PF> mr;
    if (jb.multi) {
        if (tid < jb.n) mr.load(x, C, jb.r0 + tid);
    } else {
#pragma unroll
        for (int i = 0; i < NQ; ++i)
            if (tid + 1024 * i < jb.n) q[i].load(x, C, jb.r0, tid + 1024 * i, 256, jb.n);
    }
    // terms of a column in groups g = 0 .. tpr - 1: columns g, g + tpr, ... of S^{-1}
    const int tpr = MODE == 2 ? 1 : 256 / m, groups = min(tpr, m);
    const int g = MODE == 1 ? tid / m : 0, kk = tid - g * m, cnt = g < groups ? (m - g + tpr - 1) / tpr : 0;
    const int warp = tid >> 5, lane = tid & 31;
    V pv[MODE == 1 ? 16 : 4];
    int kcol[2] = {0, 0};
    if (MODE == 0) {  // warp w takes the columns w and w + 8, lanes l and l + 32 their terms
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (warp + 8 * i >= jb.nc) break;
            kcol[i] = jobcols[jb.c0 + warp + 8 * i];
            const int k = kcol[i] & ~CORR_OWNER;
            if (lane < m) pv[2 * i] = __ldg(Sinv + lane * m + k);
            if (lane + 32 < m) pv[2 * i + 1] = __ldg(Sinv + (lane + 32) * m + k);
        }
    }
    if (MODE == 1) {
#pragma unroll
        for (int i = 0; i < (MODE == 1 ? 16 : 0); ++i)
            if (i < cnt) pv[i] = __ldg(Sinv + (g + i * tpr) * m + kk);
    }
    pdl_begin();
    pdl_trigger();
    if constexpr (MODE == 2) {
        for (int k = tid; k < m; k += 256) zs[k] = __ldcg(static_cast<const T *>(lr.zv) + k);
    } else {
        lr_rhs<T>(lr, P, u);
    }
    __syncthreads();
    if constexpr (MODE == 0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (warp + 8 * i >= jb.nc) break;
            if constexpr (sizeof(T) == 4) {
                // products, the two sums of each group (lane 2 g + h: h of
                // group g; 2 groups <= 32), then z_k over the groups
                V *p = pr + 64 * warp;
                const ff32 v0 = lane < m ? ff_mul(ff_of(pv[2 * i]), ff_of(u[lane])) : ff32{0.f, 0.f};
                const ff32 v1 = lane + 32 < m ? ff_mul(ff_of(pv[2 * i + 1]), ff_of(u[lane + 32])) : ff32{0.f, 0.f};
                p[lane] = make_float2(v0.hi, v0.lo);
                p[lane + 32] = make_float2(v1.hi, v1.lo);
                __syncwarp();
                ff32 a{0.f, 0.f};
                if (lane < 2 * groups)
                    for (int c = (lane >> 1) + (lane & 1) * tpr; c < m; c += 2 * tpr) a = ff_add(a, ff_of(p[c]));
                a = ff_add(a, ff32{__shfl_xor_sync(0xffffffffu, a.hi, 1), __shfl_xor_sync(0xffffffffu, a.lo, 1)});
                ff32 zk{0.f, 0.f};
                for (int h = 0; h < groups; ++h)
                    zk = ff_add(zk, ff32{__shfl_sync(0xffffffffu, a.hi, 2 * h), __shfl_sync(0xffffffffu, a.lo, 2 * h)});
                if (lane == 0) {
                    zs[kcol[i] & ~CORR_OWNER] = ff_to_float(zk);
                    if (lr.zpub && (kcol[i] & CORR_OWNER)) lr.zpub[kcol[i] & ~CORR_OWNER] = ff_to_double(zk);
                }
                __syncwarp();
            } else {
                double a = lane < m ? pv[2 * i] * u[lane] : 0.0;
                if (lane + 32 < m) a = fma(pv[2 * i + 1], u[lane + 32], a);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
                if (lane == 0) {
                    zs[kcol[i] & ~CORR_OWNER] = a;
                    if (lr.zpub && (kcol[i] & CORR_OWNER)) lr.zpub[kcol[i] & ~CORR_OWNER] = a;
                }
            }
        }
        __syncthreads();
    } else if constexpr (MODE == 1) {  // every CTA forms all of z
        if (g < groups) {
            if constexpr (sizeof(T) == 4) {
                ff32 t0{0.f, 0.f}, t1{0.f, 0.f};
#pragma unroll
                for (int i = 0; i < 16; i += 2) {
                    if (i < cnt) t0 = ff_add(t0, ff_mul(ff_of(pv[i]), ff_of(u[g + i * tpr])));
                    if (i + 1 < cnt) t1 = ff_add(t1, ff_mul(ff_of(pv[i + 1]), ff_of(u[g + (i + 1) * tpr])));
                }
                const ff32 v = ff_add(t0, t1);
                pr[g * m + kk] = make_float2(v.hi, v.lo);
            } else {
                double t0 = 0.0, t1 = 0.0;
#pragma unroll
                for (int i = 0; i < 16; i += 2) {
                    if (i < cnt) t0 = fma(pv[i], u[g + i * tpr], t0);
                    if (i + 1 < cnt) t1 = fma(pv[i + 1], u[g + (i + 1) * tpr], t1);
                }
                pr[g * m + kk] = t0 + t1;
            }
        }
        __syncthreads();
        if (tid < m) {
            if constexpr (sizeof(T) == 4) {
                ff32 zk{0.f, 0.f};
                for (int h = 0; h < groups; ++h) zk = ff_add(zk, ff_of(pr[h * m + tid]));
                zs[tid] = ff_to_float(zk);
                if (lr.zpub && first) lr.zpub[tid] = ff_to_double(zk);
            } else {
                double zk = 0.0;
                for (int h = 0; h < groups; ++h) zk += pr[h * m + tid];
                zs[tid] = zk;
                if (lr.zpub && first) lr.zpub[tid] = zk;
            }
        }
        __syncthreads();
    }
    if (jb.multi) {
        if (tid < jb.n) mr.apply(x, C, zs);
        if (MODE == 2)  // large supports: up to 1024 rows per CTA
            for (int r = tid + 256; r < jb.n; r += 256) {
                mr.load(x, C, jb.r0 + r);
                mr.apply(x, C, zs);
            }
    } else {
#pragma unroll
        for (int i = 0; i < NQ; ++i)
            if (tid + 1024 * i < jb.n) q[i].apply(x, tid + 1024 * i, 256, jb.n, zs);
    }
}

template <typename T, int MODE, int NQ>
__global__ void __launch_bounds__(256, MODE == 1 || NQ > 1 ? 2 : 4)
    k_lr_correct(T *x, LowRankArg lr, int P, CorrRows C, const CorrJob *__restrict__ jobs, const int *__restrict__ jobcols) {
    extern __shared__ double dyn[];
    lr_correct_body<T, MODE, NQ, MODE == 1 ? 8 : 2>(x, lr, P, C, jobs[blockIdx.x], jobcols, blockIdx.x == 0, dyn);
}

// dst -= B_c Sigma^{-1} y over the rows of the coarse level's B, y from the
// partial sums of k_bt_partial: the low-rank term of a residual-restriction
// (k_add_Bq's arithmetic).  The rows are known before the wait; dst was
// written by the kernel before k_bt_partial.  base (not null): dst = base -
// ... instead, base one value per row.
template <typename T>
__device__ __forceinline__ void resid_Bq_body(T *dst, i64 nrows, const i64 *__restrict__ rows, const i64 *__restrict__ ptr,
                                              const int *__restrict__ col, const double *__restrict__ val,
                                              const double *lrpart, int m, int P, const double *__restrict__ sigma_inv,
                                              i64 r, double *qs, const T *base = nullptr) {
    i64 row = 0, e0 = 0, e1 = 0;
    double v0 = 0.0;
    int c0 = 0;
    if (r < nrows) {
        row = rows[r];
        e0 = ptr[r];
        e1 = ptr[r + 1];
        v0 = val[e0];
        c0 = col[e0];
    }
    const double si = threadIdx.x < m ? sigma_inv[threadIdx.x] : 0.0;
    pdl_begin();
    pdl_trigger();
    const T d = r < nrows ? (base ? base[r] : dst[row]) : T(0);
    for (int k = threadIdx.x; k < m; k += 256) {
        double y = 0.0;
        if constexpr (sizeof(T) == 4) {
            const float2 *part = reinterpret_cast<const float2 *>(lrpart) + (i64)k * P;
            ff32 t{0.f, 0.f};
            for (int p = 0; p < P; ++p) t = ff_add(t, ff_of(__ldcg(part + p)));
            y = ff_to_double(t);
        } else {
            for (int p = 0; p < P; ++p) y += __ldcg(lrpart + (i64)k * P + p);
        }
        qs[k] = y * (k == (int)threadIdx.x ? si : sigma_inv[k]);
    }
    __syncthreads();
    if (r >= nrows) return;
    double acc = v0 * qs[c0];
    for (i64 e = e0 + 1; e < e1; ++e) acc += val[e] * qs[col[e]];
    dst[row] = d + (T)(-1.0 * acc);
}

template <typename T>
__global__ void __launch_bounds__(256)
    k_resid_Bq(T *dst, i64 nrows, const i64 *__restrict__ rows, const i64 *__restrict__ ptr, const int *__restrict__ col,
               const double *__restrict__ val, const double *lrpart, int m, int P, const double *__restrict__ sigma_inv,
               const T *base) {
    extern __shared__ double qs[];
    resid_Bq_body<T>(dst, nrows, rows, ptr, col, val, lrpart, m, P, sigma_inv, (i64)blockIdx.x * 256 + threadIdx.x, qs,
                     base);
}

// ------------------------------------------------- residual + restriction
// f_c(P_c) = sum_{a in {-1,0,1}^d} r(a) (f - A_0 x)(2 i_c + a),
// r(a) = prod {1/2, 1, 1/2}: IntergridOperator::restrict
// (intergrid_operator.hh:74-88) of the residual f - A_0 x
// (multigridmc_sampler.cc:124-126), with the stencil part of A.
//
// One coarse row segment of RRS_TX points per CTA: a thread forms one residual
// of its 33 x 3 x 3 fine footprint (33 x 3 in 2D), then one thread per coarse
// point adds its taps in ascending order.  Rows of residuals are shared by
// neighbouring CTAs' footprints, that is formed 9/4 times, but a level has
// enough CTAs: one thread per coarse point, which formed its 27 residuals one
// after the other, left all but a few SMs idle on the coarse levels (27-point
// fields, FP32: 77 us for 15^3 coarse points, 73 for 7^3 under ncu).  ZERO:
// the restriction of f alone.
constexpr int RRS_TX = 16, RRS_FW = 2 * RRS_TX + 1, RRS_THREADS = 320;  // >= 33 * 9

template <typename T, int NPT, int VAR, bool ZERO>
__global__ void __launch_bounds__(RRS_THREADS) k_resid_restrict(const T *x, const T *f, T *fc, T *xc, Grid3 gf, Grid3 gc,
                                                                StencilArg<T> s, int dim, VarField<T> vf) {
    if (gf.pdl) pdl_begin_trigger();
    __shared__ T res[9 * RRS_FW];
    const int ca0 = blockIdx.x * RRS_TX, cb = blockIdx.y, cc = blockIdx.z;
    const int nr = dim > 2 ? 9 : dim > 1 ? 3 : 1;  // rows of the footprint
    const int row = threadIdx.x / RRS_FW, la = threadIdx.x - row * RRS_FW;
    if (row < nr) {
        const int a = 2 * ca0 + la, b = dim > 1 ? 2 * cb + row % 3 : 0, c = dim > 2 ? 2 * cc + row / 3 : 0;
        T v = T(0);
        if (a < gf.N0) {
            const i64 P = gf.pad(a, b, c);
            v = ZERO ? f[P] : f[P] - stencil_row<T, NPT, false, VAR>(x, gf, s, P, vf);
        }
        res[threadIdx.x] = v;
    }
    __syncthreads();
    const int ca = ca0 + (int)threadIdx.x;
    if (threadIdx.x >= RRS_TX || ca >= gc.N0) return;
    T acc = T(0);
    for (int r = 0; r < nr; ++r)
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            const T wr = T((ax == 1 ? 1.0 : 0.5) * (dim > 1 && r % 3 != 1 ? 0.5 : 1.0) * (dim > 2 && r / 3 != 1 ? 0.5 : 1.0));
            acc += wr * res[r * RRS_FW + 2 * threadIdx.x + ax];
        }
    const i64 Pc = gc.pad(ca, dim > 1 ? cb : 0, dim > 2 ? cc : 0);
    fc[Pc] = acc;
    if (xc) xc[Pc] = T(0);  // the coarse sample starts from zero
}

// The same with one thread per coarse point, for levels with enough of them
// (restrict_by_point has the line and both sides' times): every residual is
// formed 27/8 (2D 9/4) times instead of 9/4 (3/2), but no CTA is a mere row
// segment, of whose threads one to three tenths work in 2D and 1D.
template <typename T, int NPT, int VAR>
__global__ void __launch_bounds__(256) k_resid_restrict_point(const T *x, const T *f, T *fc, T *xc, Grid3 gf, Grid3 gc,
                                                              StencilArg<T> s, int dim, VarField<T> vf) {
    if (gf.pdl) pdl_begin_trigger();
    const i64 t = (i64)blockIdx.x * 256 + threadIdx.x;
    if (t >= (i64)gc.N0 * gc.N1 * gc.N2) return;
    const int a = (int)(t % gc.N0), b = (int)(t / gc.N0 % gc.N1), c = (int)(t / ((i64)gc.N0 * gc.N1));
    const int hy = dim > 1, hz = dim > 2;  // half widths of the footprint
    T acc = T(0);
    for (int z = -hz; z <= hz; ++z)
        for (int y = -hy; y <= hy; ++y) {
            const i64 row = gf.pad(2 * a + 1, hy ? 2 * b + 1 + y : 0, hz ? 2 * c + 1 + z : 0);
#pragma unroll
            for (int q = -1; q <= 1; ++q) {
                const T wr = T((q ? 0.5 : 1.0) * (y ? 0.5 : 1.0) * (z ? 0.5 : 1.0));
                acc += wr * (f[row + q] - stencil_row<T, NPT, false, VAR>(x, gf, s, row + q, vf));
            }
        }
    const i64 Pc = gc.pad(a, hy ? b : 0, hz ? c : 0);
    fc[Pc] = acc;
    if (xc) xc[Pc] = T(0);  // the coarse sample starts from zero
}

// 3D-tiled variant: a CTA owns RR_TX x RR_TY x RR_TZ coarse points.  It
// stages the x values of the tile's fine footprint plus a one-point halo in
// shared memory (all loads issued at once), computes each fine residual of
// the footprint once and restricts.
constexpr int RR_TX = 16, RR_TY = 4, RR_TZ = 4;
constexpr int RR_FW = 2 * RR_TX + 1, RR_FH = 2 * RR_TY + 1, RR_FD = 2 * RR_TZ + 1;  // residual footprint, 33 x 9 x 9
constexpr int RR_XW = RR_FW + 2, RR_XH = RR_FH + 2, RR_XD = RR_FD + 2;             // x with halo
constexpr int RR_THREADS = 320;  // >= RR_FW * RR_FH = 297 footprint columns and RR_TX * RR_TY * RR_TZ = 256 coarse points
constexpr int RR_RZ = RR_TZ * RR_FH * RR_FW;  // z-restricted residuals of a tile

// The arithmetic of one tile, x (footprint plus halo) in shared memory with
// row pitch XP (footprint point (la, lb, lc) at ((lc + 1) RR_XH + lb + 1) XP
// + la + 1), f through fv(la, lb, lc).  Thread t < 297 takes the column
// (la, lb) of the footprint -- warp lb the first 32 columns of row lb, so
// that a warp's shared-memory loads are one contiguous run (no bank
// conflicts), and the tenth warp the last column of every row: the 9
// residuals along z stay in registers (the x loads of a 7-point column slide
// along z) and are restricted in z, r_z = r(2 cz) / 2 + r(2 cz + 1) +
// r(2 cz + 2) / 2, into rz.  Then thread t < 256 takes one coarse point: the
// 3 x 3 in-plane taps of rz with the weights (1/2, 1, 1/2) in y and x.  The
// product of those weights is the trilinear restriction of
// intergrid_operator.hh:74-88.
template <typename T, int NPT, int XP, typename FV>
__device__ __forceinline__ void rr_tile_compute(const T *xs, const FV &fv, T *rz, T *fc,
                                                T *xc, const Grid3 &gf, const Grid3 &gc,
                                                const StencilArg<T> &s, int ca0, int cb0, int cc0) {
    constexpr int SY = XP, SZ = XP * RR_XH;
    const int fa0 = 2 * ca0, fb0 = 2 * cb0, fz0 = 2 * cc0;
    constexpr int RW = RR_FW - 1;  // 32 columns of a row per warp
    for (int t = threadIdx.x; t < RR_FW * RR_FH; t += blockDim.x) {
        const int lb = t < RW * RR_FH ? t / RW : t - RW * RR_FH;
        const int la = t < RW * RR_FH ? t - lb * RW : RW;
        const bool col_in = fa0 + la < gf.N0 && fb0 + lb < gf.N1;
        const T *xq = xs + (lb + 1) * SY + (la + 1);
        // r_z(cz) = (r(2 cz) / 2 + r(2 cz + 1)) + r(2 cz + 2) / 2, formed as
        // the residuals come, so that only two of them are live at a time
        T rprev = T(0), part = T(0);
#pragma unroll
        for (int lc = 0; lc < RR_FD; ++lc) {
            T v = T(0);
            if (col_in && fz0 + lc < gf.N2) {
                const int q = (lc + 1) * SZ;
                T res;
                if (NPT == 7) {
                    res = s.w[4] * xq[q - SZ] + s.w[10] * xq[q - SY] + s.w[12] * xq[q - 1] + s.w[13] * xq[q] +
                          s.w[14] * xq[q + 1] + s.w[16] * xq[q + SY] + s.w[22] * xq[q + SZ];
                } else {
                    res = T(0);
#pragma unroll
                    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
                        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
                            for (int dx = -1; dx <= 1; ++dx)
                                res += s.w[(dz + 1) * 9 + (dy + 1) * 3 + (dx + 1)] * xq[q + dz * SZ + dy * SY + dx];
                }
                v = fv(la, lb, lc) - res;
            }
            if (lc & 1) {
                part = T(0.5) * rprev + v;
            } else {
                if (lc > 0) rz[((lc / 2 - 1) * RR_FH + lb) * RR_FW + la] = part + T(0.5) * v;
                rprev = v;
            }
        }
    }
    __syncthreads();
    if (threadIdx.x >= RR_TX * RR_TY * RR_TZ) return;
    const int la = threadIdx.x % RR_TX, lb = (threadIdx.x / RR_TX) % RR_TY, lc = threadIdx.x / (RR_TX * RR_TY);
    const int ca = ca0 + la, cb = cb0 + lb, cc = cc0 + lc;
    if (ca >= gc.N0 || cb >= gc.N1 || cc >= gc.N2) return;
    T acc = T(0);
#pragma unroll
    for (int ay = 0; ay < 3; ++ay)
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            const T wr = T((ax == 1 ? 1.0 : 0.5) * (ay == 1 ? 1.0 : 0.5));
            acc += wr * rz[(lc * RR_FH + 2 * lb + ay) * RR_FW + 2 * la + ax];
        }
    fc[gc.pad(ca, cb, cc)] = acc;
    if (xc) xc[gc.pad(ca, cb, cc)] = T(0);  // the coarse sample starts from zero
}

template <typename T>
constexpr size_t rr_smem_bytes() {
    return sizeof(T) * (RR_XW * RR_XH * RR_XD + RR_RZ);
}

template <typename T, int NPT>
__device__ __forceinline__ void resid_restrict_tiled_body(const T *x, const T *f,
                                                          T *fc, T *xc, const Grid3 &gf,
                                                          const Grid3 &gc, const StencilArg<T> &s, unsigned char *smem,
                                                          int bx, int by, int bz) {
    T *xs = reinterpret_cast<T *>(smem);  // [RR_XD][RR_XH][RR_XW]
    T *rz = xs + RR_XW * RR_XH * RR_XD;   // [RR_TZ][RR_FH][RR_FW]
    const int ca0 = bx * RR_TX, cb0 = by * RR_TY, cc0 = bz * RR_TZ;
    // fine 0-based origin of the footprint: the centre of coarse ca0 is fine
    // 2 ca0 + 1, its lower neighbour 2 ca0
    const int fa0 = 2 * ca0, fb0 = 2 * cb0, fz0 = 2 * cc0;
    // one warp per row of the box (no index divisions per element; a row is
    // one contiguous run of x)
    const int lane = threadIdx.x & 31;
    for (int row = threadIdx.x >> 5; row < RR_XH * RR_XD; row += RR_THREADS / 32) {
        const int lb = row % RR_XH, lc = row / RR_XH;
        const int gb = fb0 - 1 + lb, gz = fz0 - 1 + lc;
        const bool rin = gb >= 0 && gb < gf.N1 && gz >= 0 && gz < gf.N2;
        const T *xr = x + (rin ? gf.pad(fa0 - 1, gb, gz) : 0);
        for (int la = lane; la < RR_XW; la += 32) {
            const int ga = fa0 - 1 + la;
            xs[row * RR_XW + la] = rin && ga >= 0 && ga < gf.N0 ? xr[la] : T(0);
        }
    }
    __syncthreads();
    rr_tile_compute<T, NPT, RR_XW>(
        xs, [&](int la, int lb, int lc) { return f[gf.pad(fa0 + la, fb0 + lb, fz0 + lc)]; }, rz, fc, xc, gf, gc, s,
        ca0, cb0, cc0);
}

template <typename T, int NPT>
__global__ void __launch_bounds__(RR_THREADS) k_resid_restrict_tiled(const T *x, const T *f,
                                                                      T *fc, T *xc, Grid3 gf, Grid3 gc,
                                                                      StencilArg<T> s) {
    if (gf.pdl) pdl_begin_trigger();
    extern __shared__ __align__(16) unsigned char rr_smem[];
    resid_restrict_tiled_body<T, NPT>(x, f, fc, xc, gf, gc, s, rr_smem, blockIdx.x, blockIdx.y, blockIdx.z);
}

// ---------------------------------------------- bulk tensor copies (TMA)
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// 3D tiled copy of the tensor map's box at element coordinates (x, y, z)
// into shared memory; completion is counted on `bar` in bytes.
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z,
                                            unsigned long long *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<u64>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ u64 global_ns() {
    u64 t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Wait for phase `parity` of `bar`, giving up after limit_ns nanoseconds.
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long *bar, unsigned parity, u64 limit_ns) {
    const u64 t0 = global_ns();
    while (!mbar_try_wait(bar, parity))
        if (global_ns() - t0 > limit_ns) return false;
    return true;
}

constexpr u64 TILE_WAIT_NS = 200000000ull;  // 0.2 s: a tile copy that has not landed by then is reported
constexpr unsigned ERR_TILE_TIMEOUT = 2u;    // error bit: a tile copy wait ran out

// TMA variant of the residual-restriction (rows of x and f that are
// multiples of 16 bytes): thread 0 issues two 3D bulk tensor copies of the
// padded arrays -- x over the footprint plus a one-point halo, f over the
// footprint -- with rows widened to RR_BW elements (the copy's x coordinate
// 2 * 16 * blockIdx.x stays 16-byte aligned); points outside the arrays read
// as zero, like the ghost layer.  Then rr_tile_compute.
constexpr int RR_BW = 36;

template <typename T>
__host__ __device__ constexpr size_t rr_tma_xbytes() {
    return (sizeof(T) * RR_BW * RR_XH * RR_XD + 127) / 128 * 128;
}
template <typename T>
__host__ __device__ constexpr size_t rr_tma_fbytes() {
    return (sizeof(T) * RR_BW * RR_FH * RR_FD + 15) / 16 * 16;
}
template <typename T>
__host__ __device__ constexpr size_t rr_tma_smem_bytes() {
    return rr_tma_xbytes<T>() + rr_tma_fbytes<T>() + sizeof(T) * RR_RZ;
}

// The arithmetic of one tile once its x and f boxes are in shared memory
// (rr_tile_compute; the f box's footprint point (la, lb, lc) at
// (lc RR_FH + lb) RR_BW + la + 1).
template <typename T, int NPT>
__device__ __forceinline__ void resid_restrict_tile(const T *xs, const T *fs, T *rz, T *fc,
                                                    T *xc, const Grid3 &gf, const Grid3 &gc,
                                                    const StencilArg<T> &s, int ca0, int cb0, int cc0) {
    rr_tile_compute<T, NPT, RR_BW>(
        xs, [&](int la, int lb, int lc) { return fs[(lc * RR_FH + lb) * RR_BW + la + 1]; }, rz, fc, xc, gf, gc, s,
        ca0, cb0, cc0);
}

template <typename T, int NPT>
__global__ void __launch_bounds__(RR_THREADS) k_resid_restrict_tma(const __grid_constant__ CUtensorMap xmap,
                                                                   const __grid_constant__ CUtensorMap fmap,
                                                                   T *fc, T *xc, Grid3 gf, Grid3 gc,
                                                                   StencilArg<T> s, unsigned *err) {
    if (gf.pdl) pdl_begin_trigger();
    extern __shared__ __align__(1024) unsigned char rr_tma_smem[];
    __shared__ unsigned long long bar;
    T *xs = reinterpret_cast<T *>(rr_tma_smem);                      // [RR_XD][RR_XH][RR_BW]
    T *fs = reinterpret_cast<T *>(rr_tma_smem + rr_tma_xbytes<T>()); // [RR_FD][RR_FH][RR_BW]
    T *rz = reinterpret_cast<T *>(rr_tma_smem + rr_tma_xbytes<T>() + rr_tma_fbytes<T>());
    const int ca0 = blockIdx.x * RR_TX, cb0 = blockIdx.y * RR_TY, cc0 = blockIdx.z * RR_TZ;
    const int fa0 = 2 * ca0, fb0 = 2 * cb0, fz0 = 2 * cc0;
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        mbar_expect_tx(&bar, (unsigned)(sizeof(T) * RR_BW * (RR_XH * RR_XD + RR_FH * RR_FD)));
        // padded coordinates: fine vertex a sits at a + 1
        tma_load_3d(xs, &xmap, fa0, fb0, fz0, &bar);         // fine (fa0-1, fb0-1, fz0-1) ...
        tma_load_3d(fs, &fmap, fa0, fb0 + 1, fz0 + 1, &bar); // fine (fa0-1, fb0, fz0) ...
    }
    const bool ok = mbar_wait_bounded(&bar, 0, TILE_WAIT_NS);
    if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) atomicOr_system(err, ERR_TILE_TIMEOUT);
        mbar_wait_bounded(&bar, 0, TILE_WAIT_NS);  // let copies in flight land before the CTA exits
        return;
    }
    resid_restrict_tile<T, NPT>(xs, fs, rz, fc, xc, gf, gc, s, ca0, cb0, cc0);
}

// FP64 residual-restriction of a level whose constant stencil has equal
// weights at +-dx, +-dy, +-dz (Level::sym; NPT 27 or 7 in 3D, 9 or 5 in 2D).
// The FP64 unit takes two operations per clock per SM (k_sweep_row_sym), so
// the sums are arranged for few of them: with E the sum of the two
// neighbours along a direction, A_0 is a sum of w_ijk E_x^i E_y^j E_z^k
// (i, j, k in {0, 1}) and the restriction a product of one-dimensional ones,
// so R A_0 is the sum of w_ijk (R E^i)_x (R E^j)_y (R E^k)_z with the
// one-dimensional rows R = (1/2, 1, 1/2) and R E = (1/2, 1, 1, 1, 1/2)
// about the coarse point.  Each direction is applied at the resolution that
// the ones before it left: 5 operations for both rows per column and coarse
// plane, 10 per coarse row, 7 per coarse point, against 27 per fine point
// and halo point for the residuals themselves.
//
// Thread t of a row owns the fine column a = x0 + t of one coarse row and
// plane (25 values of x and 9 of f in 3D, all loads in flight together); only
// the last direction, x, goes through shared memory.  Rows that fit a CTA are
// taken whole (x0 = 0), longer ones in windows of blockDim.x columns that
// overlap by three.  Two coarse rows per thread, or two to eight coarse planes
// sliding through registers, load less and were slower on every level but one
// (31^3 fine points, 27-point: 3.9 us, 6.0 with two rows, 6.5 with two planes;
// 127^3, 7-point: 46.8, 50.5 with both; 63^3: 11.2, 10.2 with two rows): they
// leave fewer warps for the FP64 units.  Measured in graphs of dependent
// launches; residuals formed point by point in shared-memory tiles
// (k_resid_restrict_tma) took 27 us on 31^3 and 63^3, 64 us on 127^3 under
// ncu, where this kernel takes 5.5, 13 and 50.
template <int NPT>
__global__ void __launch_bounds__(256)
    k_resid_restrict_sym(const double *x, const double *f, double *fc, double *xc, Grid3 gf, Grid3 gc, SymWeights w,
                         int whole) {
    if (gf.pdl) pdl_begin_trigger();
    constexpr bool D3 = NPT == 27 || NPT == 7, FULL = NPT == 27 || NPT == 9;
    constexpr int NPX = D3 ? 5 : 1, NPF = D3 ? 3 : 1;  // planes of x and f
    extern __shared__ __align__(16) unsigned char rr_sym_sm[];
    const int txc = whole ? gc.N0 : ((int)blockDim.x - 3) / 2;
    const int ca0 = blockIdx.x * txc, x0 = whole ? 0 : 2 * ca0 - 1;
    const int a = x0 + (int)threadIdx.x;
    const int cb = blockIdx.y * blockDim.y + threadIdx.y, cc = D3 ? blockIdx.z : 0;
    const bool col_in = a >= 0 && a < gf.N0;
    // G and Q: blockDim.x + 4 values each, two zeros at either end
    const int pitch = blockDim.x + 4;
    double *sm = reinterpret_cast<double *>(rr_sym_sm) + threadIdx.y * 2 * pitch;
    if (threadIdx.x < 2) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            sm[q * pitch + threadIdx.x] = 0.0;
            sm[q * pitch + blockDim.x + 2 + threadIdx.x] = 0.0;
        }
    }
    auto at = [&](const double *v, int b, int c) {  // zero outside the lattice
        return col_in && b >= 0 && b < gf.N1 && c >= 0 && c < gf.N2 ? v[gf.pad(a, b, c)] : 0.0;
    };
    auto r1 = [](const double *q) { return fma(0.5, q[0] + q[2], q[1]); };                  // R
    auto re = [](const double *q) { return fma(0.5, q[0] + q[4], (q[1] + q[3]) + q[2]); };  // R E
    double xv[5][NPX], fv[3][NPF];
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int p = 0; p < NPX; ++p) xv[r][p] = at(x, 2 * cb - 1 + r, D3 ? 2 * cc - 1 + p : 0);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int p = 0; p < NPF; ++p) fv[r][p] = at(f, 2 * cb + r, D3 ? 2 * cc + p : 0);
    double z0[5], z1[5], zf[3];  // (R)_z x, (R E)_z x, (R)_z f
#pragma unroll
    for (int r = 0; r < 5; ++r) {
        z0[r] = D3 ? r1(xv[r] + NPX / 2 - D3) : xv[r][0];
        z1[r] = D3 ? re(xv[r]) : 0.0;
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) zf[r] = D3 ? r1(fv[r]) : fv[r][0];
    const double y0z0 = r1(z0 + 1), y1z0 = re(z0);
    double P = fma(w.wc[2], y1z0, w.wc[0] * y0z0), Q = w.wc[1] * y0z0;
    if (FULL) Q = fma(w.wc[3], y1z0, Q);
    if (D3) {
        const double y0z1 = r1(z1 + 1);
        P = fma(w.wc[4], y0z1, P);
        if (FULL) {
            const double y1z1 = re(z1);
            P = fma(w.wc[6], y1z1, P);
            Q = fma(w.wc[5], y0z1, Q);
            Q = fma(w.wc[7], y1z1, Q);
        }
    }
    sm[2 + threadIdx.x] = r1(zf) - P;
    sm[pitch + 2 + threadIdx.x] = Q;
    __syncthreads();
    const int ca = ca0 + (int)threadIdx.x;
    if ((int)threadIdx.x < txc && ca < gc.N0 && cb < gc.N1) {
        const double *g = sm + 2 + (2 * ca + 1 - x0), *q = g + pitch;
        const i64 Pc = gc.pad(ca, cb, cc);
        fc[Pc] = r1(g - 1) - re(q - 2);
        if (xc) xc[Pc] = 0.0;  // the coarse sample starts from zero
    }
}

// dst[row] += sign * sum_e B_e y_{col_e} / Sigma_{col_e} over the rows of B
// (row-compressed): the B Sigma^{-1} B^T x part of A x.
template <typename T>
__global__ void __launch_bounds__(256) k_add_Bq(T *dst, i64 nrows, const i64 *__restrict__ rows,
                                                 const i64 *__restrict__ ptr, const int *__restrict__ col,
                                                 const double *__restrict__ val, const double *y,
                                                 const double *__restrict__ sigma_inv, double sign) {
    pdl_begin();
    for (i64 r = (i64)blockIdx.x * blockDim.x + threadIdx.x; r < nrows; r += (i64)gridDim.x * blockDim.x) {
        double acc = 0.0;
        for (i64 e = ptr[r]; e < ptr[r + 1]; ++e) acc += val[e] * (y[col[e]] * sigma_inv[col[e]]);
        dst[rows[r]] += (T)(sign * acc);
    }
}

// --------------------------------------------------------- prolongation
// x += alpha P x_c (intergrid_operator.hh:106-120): every fine vertex
// gathers its <= 2^d coarse parents, weight 1 (even coordinate) or 1/2 for
// each of the two parents (odd coordinate).
//
// A thread owns the 2^d fine vertices of a coarse cell.  FP64: the sums of the
// parents direction by direction, 12 additions in 3D, and one FMA per vertex
// with alpha times the weight (the sums parent by parent, with the weights as
// run-time values, took over 80 FP64 instructions; k_sweep_row_sym says why
// their number counts).  FP32 adds the parents in their order.
// On 127^3, FP64, under ncu: 24.4 -> 16.5 us, of which the FP64 unit 10.
template <typename T, int DIM>
__device__ __forceinline__ void prolong_add_body(T *x, const T *xc, const Grid3 &gf,
                                                 const Grid3 &gc, T alpha, int bx, int by, int bz_from_top) {
    // coarse cell (i, j, k), 0 <= i <= Nc0 etc., owns the fine vertices with
    // 1-based coordinates 2 i + {0, 1} (those inside the interior); its
    // corners are the coarse vertices i, i+1 (1-based, ghosts are zero)
    // planes from the top: the residual-restriction before ends there, and
    // the sweep after starts at the bottom, which this kernel writes last
    // (both find their first planes in L2)
    constexpr int NY = DIM > 1 ? 2 : 1, NZ = DIM > 2 ? 2 : 1;
    const int i = bx * blockDim.x + threadIdx.x;
    const int j = DIM > 1 ? by : 0, k = DIM > 2 ? bz_from_top : 0;
    if (i > gc.N0) return;
    const i64 Pc = (i64)(DIM > 2 ? k : 1) * gc.sz + (i64)(DIM > 1 ? j : 1) * gc.sy + i;
    const i64 Pf = (i64)(DIM > 2 ? 2 * k : 1) * gf.sz + (i64)(DIM > 1 ? 2 * j : 1) * gf.sy + 2 * i;
    T v[NZ][NY][2], xv[NZ][NY][2];
    bool in[NZ][NY][2];
#pragma unroll
    for (int z = 0; z < NZ; ++z)
#pragma unroll
        for (int y = 0; y < NY; ++y)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                v[z][y][q] = xc[Pc + z * gc.sz + y * gc.sy + q];
                const int fk = DIM > 2 ? 2 * k + z : 1, fj = DIM > 1 ? 2 * j + y : 1, fi = 2 * i + q;
                in[z][y][q] = fk >= 1 && fk <= gf.N2 && fj >= 1 && fj <= gf.N1 && fi >= 1 && fi <= gf.N0;
                xv[z][y][q] = in[z][y][q] ? x[Pf + z * gf.sz + y * gf.sy + q] : T(0);
            }
    if constexpr (sizeof(T) == 8) {
        const T a[4] = {alpha, T(0.5) * alpha, T(0.25) * alpha, T(0.125) * alpha};
#pragma unroll
        for (int z = 0; z < NZ; ++z)
#pragma unroll
            for (int y = 0; y < NY; ++y) v[z][y][1] += v[z][y][0];
        if (DIM > 1) {
#pragma unroll
            for (int z = 0; z < NZ; ++z)
#pragma unroll
                for (int q = 0; q < 2; ++q) v[z][NY - 1][q] += v[z][0][q];
        }
        if (DIM > 2) {
#pragma unroll
            for (int y = 0; y < NY; ++y)
#pragma unroll
                for (int q = 0; q < 2; ++q) v[NZ - 1][y][q] += v[0][y][q];
        }
#pragma unroll
        for (int z = 0; z < NZ; ++z)
#pragma unroll
            for (int y = 0; y < NY; ++y)
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    if (in[z][y][q]) x[Pf + z * gf.sz + y * gf.sy + q] = fma(a[z + y + q], v[z][y][q], xv[z][y][q]);
    } else {
#pragma unroll
        for (int oz = 0; oz < NZ; ++oz)
#pragma unroll
            for (int oy = 0; oy < NY; ++oy)
#pragma unroll
                for (int ox = 0; ox < 2; ++ox) {
                    // even coordinate: the vertex itself; odd: half of each neighbour
                    const T w = (oz ? T(0.5) : T(1)) * (oy ? T(0.5) : T(1)) * (ox ? T(0.5) : T(1));
                    T acc = T(0);
#pragma unroll
                    for (int dz = 0; dz <= oz; ++dz)
#pragma unroll
                        for (int dy = 0; dy <= oy; ++dy)
#pragma unroll
                            for (int dx = 0; dx <= ox; ++dx) acc += w * v[dz][dy][dx];
                    if (in[oz][oy][ox]) x[Pf + oz * gf.sz + oy * gf.sy + ox] = xv[oz][oy][ox] + alpha * acc;
                }
    }
}

template <typename T, int DIM>
__global__ void __launch_bounds__(128) k_prolong_add(T *x, const T *xc, Grid3 gf, Grid3 gc,
                                                      T alpha) {
    if (gf.pdl) pdl_begin_trigger();
    prolong_add_body<T, DIM>(x, xc, gf, gc, alpha, blockIdx.x, blockIdx.y, (int)(gridDim.z - 1 - blockIdx.z));
}

// ----------------------------------------------------- stencil apply
// y = A_0 x (LinearOperator::apply without the low-rank term).
template <typename T, int VAR = 0>
__global__ void __launch_bounds__(256) k_apply_stencil(const T *__restrict__ x, T *__restrict__ y, Grid3 g,
                                                        StencilArg<T> s, VarField<T> vf) {
    i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    i64 n = (i64)g.N0 * g.N1 * g.N2;
    if (t >= n) return;
    int a = (int)(t % g.N0), b = (int)((t / g.N0) % g.N1), c = (int)(t / ((i64)g.N0 * g.N1));
    i64 P = g.pad(a, b, c);
    T res = T(0);
    for (int dz = -1; dz <= 1; ++dz)
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx)
                res += vweight<T, VAR>(s, vf, P, (dz + 1) * 9 + (dy + 1) * 3 + (dx + 1)) * x[P + dz * g.sz + dy * g.sy + dx];
    y[P] = res;
}

// ---------------------------------------------------- layout conversion
template <typename T>
__global__ void __launch_bounds__(256) k_unpack(const double *__restrict__ src, T *__restrict__ dst, Grid3 g) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y, c = blockIdx.z;
    if (a >= g.N0) return;
    dst[g.pad(a, b, c)] = (T)src[((i64)c * g.N1 + b) * g.N0 + a];
}

// Both inputs of Sampler::apply in one pass (two independent read streams
// per thread).
template <typename T>
__global__ void __launch_bounds__(256) k_unpack2(const double *__restrict__ f_src, const double *__restrict__ x_src,
                                                 T *__restrict__ f_dst, T *__restrict__ x_dst, Grid3 g) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y, c = blockIdx.z;
    if (a >= g.N0) return;
    const i64 i = ((i64)c * g.N1 + b) * g.N0 + a, P = g.pad(a, b, c);
    const double fv = f_src[i], xv = x_src[i];
    f_dst[P] = (T)fv;
    x_dst[P] = (T)xv;
}

template <typename T>
__global__ void __launch_bounds__(256) k_pack(const T *__restrict__ src, double *__restrict__ dst, Grid3 g) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x, b = blockIdx.y, c = blockIdx.z;
    if (a >= g.N0) return;
    dst[((i64)c * g.N1 + b) * g.N0 + a] = (double)src[g.pad(a, b, c)];
}

// ------------------------------------------------- coarse Cholesky sample
// CholeskySampler::apply (cholesky_sampler.hh:52-66) with the dense
// natural-order factor Q = L L^T: g = L^{-1} f, x = L^{-T} (xi + g).
// Parity form: column-oriented substitution in one CTA (same operation
// order as the oracle, one rounding per operation).
template <typename T, int NOISE>
__global__ void __launch_bounds__(1024) k_chol_subst(const T *f, T *x, Grid3 g,
                                                      const double *__restrict__ L, double *gv,
                                                      NoiseArgs nz) {
    if (g.pdl) pdl_begin();
    const i64 n = (i64)g.N0 * g.N1 * g.N2;
    for (i64 i = threadIdx.x; i < n; i += blockDim.x) {
        int a = (int)(i % g.N0), b = (int)((i / g.N0) % g.N1), c = (int)(i / ((i64)g.N0 * g.N1));
        gv[i] = (double)f[g.pad(a, b, c)];
    }
    __syncthreads();
    __shared__ double piv;
    for (i64 i = 0; i < n; ++i) {  // forward: L g = f
        if (threadIdx.x == 0) {
            piv = gv[i] / L[i * n + i];
            gv[i] = piv;
        }
        __syncthreads();
        const double p = piv;
        for (i64 k = i + 1 + threadIdx.x; k < n; k += blockDim.x) gv[k] = __dsub_rn(gv[k], __dmul_rn(L[k * n + i], p));
        __syncthreads();
    }
    for (i64 i = threadIdx.x; i < n; i += blockDim.x) {  // xi + g
        double xi = 0.0;
        if (NOISE == NOISE_INJECTED) xi = nz.buf[i];
        if (NOISE == NOISE_PHILOX) {
            float4 r = normals4(philox4x32_10(noise_ctr(nz, (unsigned)(i >> 2), PURPOSE_COARSE, 0), noise_key(nz)));
            xi = (double)pick(r, (int)(i & 3));
        }
        gv[i] = __dadd_rn(xi, gv[i]);
    }
    __syncthreads();
    for (i64 i = n - 1; i >= 0; --i) {  // backward: L^T x = xi + g
        if (threadIdx.x == 0) {
            piv = gv[i] / L[i * n + i];
            gv[i] = piv;
        }
        __syncthreads();
        const double p = piv;
        for (i64 k = threadIdx.x; k < i; k += blockDim.x) gv[k] = __dsub_rn(gv[k], __dmul_rn(L[i * n + k], p));
        __syncthreads();
    }
    for (i64 i = threadIdx.x; i < n; i += blockDim.x) {
        int a = (int)(i % g.N0), b = (int)((i / g.N0) % g.N1), c = (int)(i / ((i64)g.N0 * g.N1));
        x[g.pad(a, b, c)] = (T)gv[i];
    }
}

// Throughput form with the explicit inverse factor Linv = L^{-1}, stored
// row-major in the matrix type MT (double for the FP64 chain, float for the
// FP32 chain) with a leading dimension ld that is a multiple of 16 bytes and
// explicit zeros outside the triangle (and in columns n..ld-1), so that rows
// are read in aligned 16-byte vectors and a vector that straddles the
// diagonal multiplies zeros.  One warp per row; rows i and n-1-i go to
// neighbouring warps, so that every CTA gets the same number of non-zeros.
template <typename MT>
struct Vec16;
template <>
struct Vec16<float> {
    typedef float4 type;
    static constexpr int N = 4;
    static __device__ __forceinline__ float dot(float4 a, const float *v) {
        return a.x * v[0] + a.y * v[1] + a.z * v[2] + a.w * v[3];
    }
};
template <>
struct Vec16<double> {
    typedef double2 type;
    static constexpr int N = 2;
    static __device__ __forceinline__ double dot(double2 a, const double *v) { return a.x * v[0] + a.y * v[1]; }
};

// A warp's row, vectors q0 .. q1 - 1: sum of row . vs, lanes strided, four
// vectors in flight.  The first four of a lane are loaded by load(), which a
// kernel calls before it waits for vs.
template <typename MT>
struct WarpRow {
    typedef typename Vec16<MT>::type V;
    static constexpr int NV = Vec16<MT>::N;
    const V *r;
    int q, q1;
    V first[4];
    __device__ __forceinline__ void load(const MT *__restrict__ row, int q0, int end, int lane) {
        r = reinterpret_cast<const V *>(row);
        q = q0 + lane;
        q1 = end;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (q + 32 * k < q1) first[k] = __ldg(r + q + 32 * k);
    }
    __device__ __forceinline__ MT dot(const MT *vs) const {
        MT a0 = MT(0), a1 = MT(0), a2 = MT(0), a3 = MT(0);
        int p = q;
        if (p + 96 < q1) {
            a0 += Vec16<MT>::dot(first[0], vs + NV * p);
            a1 += Vec16<MT>::dot(first[1], vs + NV * (p + 32));
            a2 += Vec16<MT>::dot(first[2], vs + NV * (p + 64));
            a3 += Vec16<MT>::dot(first[3], vs + NV * (p + 96));
            p += 128;
            for (; p + 96 < q1; p += 128) {
                V v0 = __ldg(r + p), v1 = __ldg(r + p + 32), v2 = __ldg(r + p + 64), v3 = __ldg(r + p + 96);
                a0 += Vec16<MT>::dot(v0, vs + NV * p);
                a1 += Vec16<MT>::dot(v1, vs + NV * (p + 32));
                a2 += Vec16<MT>::dot(v2, vs + NV * (p + 64));
                a3 += Vec16<MT>::dot(v3, vs + NV * (p + 96));
            }
            for (; p < q1; p += 32) a0 += Vec16<MT>::dot(__ldg(r + p), vs + NV * p);
        } else {
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (p + 32 * k < q1) a0 += Vec16<MT>::dot(first[k], vs + NV * (p + 32 * k));
        }
        MT acc = (a0 + a1) + (a2 + a3);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        return acc;
    }
};

// v = xi + Linv f (row i: vectors 0 .. i / NV), one warp per row: row, noise
// and addresses before the wait for f.
template <typename T, typename MT, int NOISE>
__device__ __forceinline__ void chol_gemv_lower_body(const T *f, const Grid3 &g, const MT *__restrict__ Linv,
                                                     int ld, MT *v, const NoiseArgs &nz, bool wait,
                                                     unsigned char *chol_sm, int bx) {
    MT *fs = reinterpret_cast<MT *>(chol_sm);
    const int n = g.N0 * g.N1 * g.N2;
    constexpr int NV = Vec16<MT>::N;
    const int lane = threadIdx.x & 31, ii = bx * 8 + (threadIdx.x >> 5);
    const int i = (ii & 1) ? n - 1 - (ii >> 1) : (ii >> 1);
    WarpRow<MT> row;
    MT xi = MT(0);
    if (ii < n) {
        row.load(Linv + (i64)i * ld, 0, i / NV + 1, lane);
        if (NOISE == NOISE_PHILOX) {
            const float4 r = normals4(philox4x32_10(noise_ctr(nz, (unsigned)(i >> 2), PURPOSE_COARSE, 0), noise_key(nz)));
            if constexpr (sizeof(MT) == 4)
                xi = pick(r, i & 3);
            else
                xi = widen(pick(r, i & 3));
        }
    }
    // k / N0 and t / N1 by multiplication with 2^32 / d rounded up (k d < 2^32:
    // a coarse level has at most 12,000 unknowns): 14 of them stand between
    // the wait and the product on 15^3 unknowns (17.1 -> 14.7 us under ncu)
    const u64 r0 = 0xffffffffull / (unsigned)g.N0 + 1, r1 = 0xffffffffull / (unsigned)g.N1 + 1;
    auto padded = [&](int k) {
        const int t = (int)((unsigned)k * r0 >> 32), c = (int)((unsigned)t * r1 >> 32);
        return g.pad(k - t * g.N0, t - c * g.N1, c);
    };
    const i64 P0 = (int)threadIdx.x < n ? padded(threadIdx.x) : 0;
    if (wait) pdl_begin_trigger();
#pragma unroll 4
    for (int k = threadIdx.x; k < ld; k += 256) fs[k] = k < n ? (MT)f[k < 256 ? P0 : padded(k)] : MT(0);
    __syncthreads();
    if (ii >= n) return;
    const MT acc = row.dot(fs);
    if (lane == 0) v[i] = (NOISE == NOISE_INJECTED ? (MT)nz.buf[i] : xi) + acc;
}

// (With the row and the noise loaded and drawn after the wait, and no early
// start here, in the residual-restriction and in the prolongation, whole
// steps were slower: 2D 64 x 64 FP64 59.0 us, now 56.4; 3D 32^3 FP64 128 ->
// 122 us; 96x48x80 27-point FP32 258 -> 240 us.)
template <typename T, typename MT, int NOISE>
__global__ void __launch_bounds__(256) k_chol_gemv_lower(const T *f, Grid3 g, const MT *__restrict__ Linv,
                                                          int ld, MT *v, NoiseArgs nz) {
    extern __shared__ __align__(16) unsigned char chol_sm[];
    chol_gemv_lower_body<T, MT, NOISE>(f, g, Linv, ld, v, nz, g.pdl != 0, chol_sm, blockIdx.x);
}

// ... x = Linv^T v (row j of Linv^T: vectors j / NV .. ld / NV - 1).
template <typename T, typename MT>
__device__ __forceinline__ void chol_gemv_upper_body(const MT *v, const Grid3 &g,
                                                     const MT *__restrict__ LinvT, int ld, T *x, bool wait,
                                                     unsigned char *chol_sm, int bx) {
    MT *vs = reinterpret_cast<MT *>(chol_sm);
    const int n = g.N0 * g.N1 * g.N2;
    constexpr int NV = Vec16<MT>::N;
    const int lane = threadIdx.x & 31, jj = bx * 8 + (threadIdx.x >> 5);
    const int j = (jj & 1) ? n - 1 - (jj >> 1) : (jj >> 1);
    WarpRow<MT> row;
    i64 P = 0;
    if (jj < n) {
        row.load(LinvT + (i64)j * ld, j / NV, ld / NV, lane);
        const int a = j % g.N0, t = j / g.N0;
        P = g.pad(a, t % g.N1, t / g.N1);
    }
    if (wait) pdl_begin_trigger();
    for (int i = threadIdx.x; i < ld; i += 256) vs[i] = i < n ? v[i] : MT(0);
    __syncthreads();
    if (jj >= n) return;
    const MT acc = row.dot(vs);
    if (lane == 0) x[P] = (T)acc;
}

template <typename T, typename MT>
__global__ void __launch_bounds__(256) k_chol_gemv_upper(const MT *v, Grid3 g,
                                                          const MT *__restrict__ LinvT, int ld, T *x) {
    extern __shared__ __align__(16) unsigned char chol_sm[];
    chol_gemv_upper_body<T, MT>(v, g, LinvT, ld, x, g.pdl != 0, chol_sm, blockIdx.x);
}

// ------------------------------------------------------------- adjoint
// y += alpha x over whole padded arrays (ghosts are zero in both).
template <typename T>
__global__ void __launch_bounds__(256) k_axpy(T *__restrict__ y, const T *__restrict__ x, T alpha, i64 n) {
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) y[i] += alpha * x[i];
}

// a -= A_0 u, b += u (b may be null) and `zero` = 0 (the work vector of the
// next transposed sweep, may be null) over the interior, in one pass.  A_0 u
// cancels most of a (u is about A_0^{-1} a): FP32 forms the difference without
// intermediate roundings.
template <typename T, int NPT, int VAR>
__global__ void __launch_bounds__(256) k_adj_update(const T *u, T *a, T *b, T *zero, Grid3 g, StencilArg<T> s, VarField<T> vf) {
    if (g.pdl) pdl_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= g.N0 || j >= g.N1) return;
    const i64 P = g.pad(i, j, blockIdx.z);
    constexpr int NZ = NPT == 9 ? 1 : 3;
    ProductSum<T> sum[NZ];  // by planes: three sums in flight
#pragma unroll
    for (int z = 0; z < NZ; ++z) {
        const int dz = NZ == 1 ? 0 : z - 1;
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx) {
                if (NPT == 7 && (dz != 0) + (dy != 0) + (dx != 0) > 1) continue;
                sum[z].add(vweight<T, VAR>(s, vf, P, (dz + 1) * 9 + (dy + 1) * 3 + dx + 1), u[P + dz * g.sz + dy * g.sy + dx]);
            }
    }
    if constexpr (sizeof(T) == 4) {
        ff32 t{sum[0].hi, sum[0].lo};
#pragma unroll
        for (int z = 1; z < NZ; ++z) t = ff_add(t, ff32{sum[z].hi, sum[z].lo});
        a[P] = ff_to_float(ff_add(ff32{a[P], 0.f}, ff_neg(t)));
    } else {
        a[P] -= NZ == 1 ? sum[0].hi : (sum[0].hi + sum[NZ - 1].hi) + sum[NZ / 2].hi;
    }
    if (b) b[P] += u[P];
    if (zero) zero[P] = T(0);
}

// dst[row] += sum_e B_e z_{col_e} over the rows of B
template <typename T>
__global__ void __launch_bounds__(256) k_add_Bz(T *dst, i64 nrows, const i64 *__restrict__ rows, const i64 *__restrict__ ptr,
                                                const int *__restrict__ col, const double *__restrict__ val, const double *z) {
    pdl_begin();
    const i64 r = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nrows) return;
    double acc = 0.0;
    for (i64 e = ptr[r]; e < ptr[r + 1]; ++e) acc += val[e] * z[col[e]];
    dst[rows[r]] += (T)acc;
}

// ------------------------------------------------- deterministic solver
// One iteration of LoopSolver::apply (loop_solver.cc:24-42) keeps the
// iterate x, the right hand side b and the residual r in FP64 on level 0,
// whatever the type T of the hierarchy that applies the multigrid
// preconditioner: with an FP32 hierarchy the loop is iterative refinement
// and still converges to FP64 accuracy.
//
// r = b - A_0 x over the interior in FP64, with everything an iteration does
// with it: |r|^2 (the partial sums of the CTAs, added in their order by the
// CTA that finishes last, so the norm is reproducible; it goes to page-locked
// host memory), the preconditioner's right hand side f = (T) r, its split by
// colour (fs, may be null: k_split_colours' layout) and its zero initial
// state (multigrid_preconditioner.cc:76).  b has B Sigma^{-1} B^T x
// subtracted already (k_resid_Bq with k_solve_gather's values).  r itself is
// not stored.
//
// A warp takes segments of SOLVE_SEG points of a row, its lanes consecutive
// ones (CTAs of 256 threads along a row left half of the threads of 127
// points idle), at most four CTAs per SM (one segment per warp: 48 us, the
// reduction at the end of a CTA is FP64 work too).  Bound by the FP64 unit: 9
// instructions a point of a 7-point stencil, 31 us at 127^3.  Measured there
// under ncu: 42 us; 71 us for the residual (35), the right hand side with the
// partial sums of the norm (19), their sum (6) and the split (11) in four
// launches.
constexpr int SOLVE_SEG = 128;
template <typename T, int NPT, int VAR = 0>
__global__ void __launch_bounds__(256) k_solve_resid(const double *__restrict__ x, const double *__restrict__ b,
                                                     T *__restrict__ f, T *__restrict__ px, float *__restrict__ fs,
                                                     i64 fhalf, Grid3 g, StencilArg<double> s, VarField<double> vf,
                                                     double *part, unsigned *counter, double *norm) {
    __shared__ double sh[32];
    __shared__ bool last;
    const int nseg = (g.N0 + SOLVE_SEG - 1) / SOLVE_SEG;
    const i64 ntask = (i64)g.N1 * g.N2 * nseg;
    double acc = 0.0;
    for (i64 task = (i64)blockIdx.x * 8 + (threadIdx.x >> 5); task < ntask; task += (i64)gridDim.x * 8) {
        const i64 row = task / nseg;
        const int bb = (int)(row % g.N1), c = (int)(row / g.N1);
        const int a0 = (int)(task - row * nseg) * SOLVE_SEG + (threadIdx.x & 31);
        const i64 P0 = g.pad(a0, bb, c);
#pragma unroll(NPT == 7 ? SOLVE_SEG / 32 : 1)
        for (int q = 0; q < SOLVE_SEG / 32; ++q) {
            const i64 P = P0 + 32 * q;
            if (a0 + 32 * q >= g.N0) break;
            double v = b[P];
#pragma unroll
            for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
                for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
                    for (int dx = -1; dx <= 1; ++dx) {
                        if (NPT == 7 && (dz != 0) + (dy != 0) + (dx != 0) > 1) continue;
                        v = fma(-vweight<double, VAR>(s, vf, P, (dz + 1) * 9 + (dy + 1) * 3 + dx + 1),
                                x[P + dz * g.sz + dy * g.sy + dx], v);
                    }
            acc = fma(v, v, acc);
            const T fv = (T)v;
            f[P] = fv;
            px[P] = T(0);
            if (sizeof(T) == 4 && fs) fs[(i64)((a0 + 32 * q + bb + c) & 1) * fhalf + (P >> 1)] = (float)fv;
        }
    }
    acc = block_sum<256>(acc, sh);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = acc;
        unsigned prev;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(prev) : "l"(counter) : "memory");
        last = prev == gridDim.x - 1u;
        if (last) *counter = 0u;
    }
    __syncthreads();
    if (!last) return;
    acc = 0.0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += 256) acc += __ldcg(part + i);
    acc = block_sum<256>(acc, sh);
    if (threadIdx.x == 0) *norm = acc;
}

// dst[r] = src[rows[r]]
__global__ void __launch_bounds__(256) k_solve_gather(double *__restrict__ dst, const double *__restrict__ src,
                                                      const i64 *__restrict__ rows, i64 nrows) {
    const i64 r = (i64)blockIdx.x * 256 + threadIdx.x;
    if (r < nrows) dst[r] = src[rows[r]];
}

// x += P r: the preconditioner's result (type T) added to the FP64 iterate
// over whole padded arrays (ghosts are zero in both), four entries per
// thread.
template <typename T>
__global__ void __launch_bounds__(256) k_solve_update(double *__restrict__ x, const T *__restrict__ dx, i64 n) {
    typedef typename std::conditional<sizeof(T) == 4, float2, double2>::type T2;
    const i64 i = 4 * ((i64)blockIdx.x * 256 + threadIdx.x);
    if (i + 3 < n) {
        double2 *xv = reinterpret_cast<double2 *>(x + i);
        const T2 *dv = reinterpret_cast<const T2 *>(dx + i);
        const double2 a = xv[0], b = xv[1];
        const T2 d = dv[0], e = dv[1];
        xv[0] = make_double2(a.x + to_double(d.x), a.y + to_double(d.y));
        xv[1] = make_double2(b.x + to_double(e.x), b.y + to_double(e.y));
    } else {
        for (i64 k = i; k < n; ++k) x[k] += to_double(dx[k]);
    }
}

// ------------------------------------------------------ exact sampler
// A draw eta ~ N(0, A_0) for a symmetric stencil with non-positive
// off-diagonal weights and a non-negative diagonal surplus
// c_0 = w_c - sum_k |w_k|:  x^T A_0 x = c_0 |x|^2 + sum over edges (p, q) of
// c_k (x_q - x_p)^2, one edge per pair of stencil neighbours in each of the
// 13 directions k of positive linear offset, c_k = -w_k, and one boundary
// edge (outside value zero) wherever a neighbour lies outside the lattice
// (which keeps the diagonal of the Dirichlet operator).  So
//   eta_p = sqrt(c_0) xi_p + sum_k sqrt(c_k) (xi_{k, p - o_k} - xi_{k, p}),
// with independent normals xi on the points and on the edges (edge (r, r +
// o_k) keyed by its lower end r, which may be a ghost position).  Philox
// keys: the sampler's seed; counter (edge or point id, purpose EXACT,
// direction k in the level byte, the step counter).  b += eta.
struct EdgeWeights {
    double c0;        // sqrt(c_0)
    double ck[13];    // sqrt(c_k) for the directions of positive offset
    int off[13][3];   // (dx, dy, dz) of direction k
};

__device__ __forceinline__ double exact_normal(const NoiseArgs &nz, int k, unsigned id) {
    NoiseArgs a = nz;
    a.level = (unsigned)k;
    return (double)normals4(philox4x32_10(noise_ctr(a, id, PURPOSE_EXACT, 0), noise_key(a))).x;
}

// cdiag (may be null): per-point centre weights, c_0 = cdiag[P] - offsum.
template <int NPT>
__global__ void __launch_bounds__(256) k_prior_perturbation(double *__restrict__ b, Grid3 g, EdgeWeights ew,
                                                            NoiseArgs nz, const double *__restrict__ cdiag,
                                                            double offsum) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x, bb = blockIdx.y, c = blockIdx.z;
    if (a >= g.N0) return;
    // ids over positions (-1 .. N) in every direction
    const unsigned X = (unsigned)g.N0 + 2u, Y = (unsigned)g.N1 + 2u;
    auto id = [&](int pa, int pb, int pc) { return ((unsigned)(pc + 1) * Y + (unsigned)(pb + 1)) * X + (unsigned)(pa + 1); };
    const double c0 = cdiag ? sqrt(fmax(cdiag[g.pad(a, bb, c)] - offsum, 0.0)) : ew.c0;
    double eta = c0 * exact_normal(nz, 0, id(a, bb, c));
#pragma unroll
    for (int k = 0; k < 13; ++k) {
        const int dx = ew.off[k][0], dy = ew.off[k][1], dz = ew.off[k][2];
        if (NPT == 7 && (dx != 0) + (dy != 0) + (dz != 0) > 1) continue;
        if (ew.ck[k] == 0.0) continue;
        eta += ew.ck[k] * (exact_normal(nz, k + 1, id(a - dx, bb - dy, c - dz)) - exact_normal(nz, k + 1, id(a, bb, c)));
    }
    b[g.pad(a, bb, c)] += eta;
}

// y_j = Sigma_j^{1/2} xi_j with m more normals (direction byte 14), so that
// k_add_Bq (which divides by Sigma) adds B Sigma^{-1/2} xi: the low-rank
// part of eta ~ N(0, A_0 + B Sigma^{-1} B^T).
__global__ void __launch_bounds__(256) k_lowrank_perturbation(NoiseArgs nz, const double *__restrict__ sigma_sqrt, int m,
                                                              double *__restrict__ y) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= m) return;
    y[j] = sigma_sqrt[j] * exact_normal(nz, 14, (unsigned)j);
}

// ------------------------------------------------ parameter adjoint
// Derivatives of one step (noise fixed) with respect to the fine stencil's
// centre weight s (for the FD prior, s = h^d kappa^2 + const, so
// d/dkappa^2 = h^d d/ds) and to log Sigma_k.  A sweep is
// x'' = x + M_f^{-1}(c - A x) with M_f = M + B Sigma^{-1} B^T,
// M = D / omega + (A_0's part before the point in the sweep order) and
// c = f + sd xi + B Sigma^{-1/2} xi'; with u = M_f^{-T} x-bar'' it adds
//   u^T dc - u^T dN x - u^T dM_f x''   (N = A_0 - M)
// to the gradient.  dA_0/ds on level l is the Galerkin stencil E_l of the
// unit centre weight; the noise part c - f = M x'' + N x + B Sigma^{-1} B^T x''
// - f is rebuilt from the sweep's input and output states, so the point
// normals need not be stored.
// Colour of interior point (a, b, c) in the multicolour order (2 colours:
// parity of a + b + c; 2^dim colours: one parity bit per direction).
__device__ __forceinline__ int point_colour(int ncol, int a, int b, int c) {
    return ncol == 2 ? ((a + b + c) & 1) : ((a & 1) | ((b & 1) << 1) | ((c & 1) << 2));
}

// An event's sum over the level's points p, one partial sum per CTA:
//   sum_p u_p [sum_{q before p} c_pq v_q + sum_{q after p} c_pq w_q
//              + cv v_p + cw w_p + cf f_p]
// over the off-diagonal neighbours q (the 6 axis neighbours of a 7-point
// level, or all), "before" in the order of the sweep of direction `forward`:
// by linear index for the lexicographic order (ncol = 0), by colour otherwise.
// A sweep (v = its output, w = its input; kd = dsd/ds / sd = E_c / (2 A_c))
// has c = kd A - E, cv = kd A_c / omega - E_c / omega,
// cw = kd A_c (1 - 1/omega) - E_c (1 - 1/omega), cf = -kd; -u^T dA v has
// v = w, c = -E, cw = -E_c.  The neighbour sums are FP64 ones, or those of
// ProductSum over FP32 values; the u_p-weighted sum is FP64.  One weight per
// neighbour instead of one each for the products with A and E (and one sum
// instead of eight): 30 FP64 instructions per point instead of 75, on a unit
// that takes two per clock.
template <typename T>
struct PgradWeights {
    T c[27];
    double cv, cw, cf;
};

template <typename T, int NPT>
__global__ void __launch_bounds__(256) k_pgrad_stencil(const T *u, const T *v, const T *w, const T *f, Grid3 g,
                                                       PgradWeights<T> pw, int ncol, int forward, double *part) {
    __shared__ double sh[32];
    const int nrows = g.N1 * g.N2;
    double acc = 0.0;
    for (int row = blockIdx.x * blockDim.y + threadIdx.y; row < nrows; row += gridDim.x * blockDim.y) {
        const int bb = row % g.N1, c = row / g.N1;
        for (int a = threadIdx.x; a < g.N0; a += blockDim.x) {
            const i64 P = g.pad(a, bb, c);
            const T up = u[P];
            if (up == T(0)) continue;
            const int cp = ncol ? point_colour(ncol, a, bb, c) : 0;
            ProductSum<T> sum[3];  // by planes
#pragma unroll
            for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
                for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
                    for (int dx = -1; dx <= 1; ++dx) {
                        const int nzo = (dx != 0) + (dy != 0) + (dz != 0);
                        if (nzo == 0 || (NPT == 7 && nzo > 1) || (NPT == 9 && dz != 0)) continue;
                        bool before;
                        if (ncol == 0) {
                            const bool lower = dz < 0 || (dz == 0 && (dy < 0 || (dy == 0 && dx < 0)));
                            before = forward ? lower : !lower;
                        } else {
                            const int cq = point_colour(ncol, a + dx, bb + dy, c + dz);
                            before = forward ? cq < cp : cq > cp;
                        }
                        sum[dz + 1].add(pw.c[(dz + 1) * 9 + (dy + 1) * 3 + (dx + 1)],
                                        (before ? v : w)[P + dz * g.sz + dy * g.sy + dx]);
                    }
            const double own = fma(pw.cv, (double)v[P], fma(pw.cw, (double)w[P], pw.cf * (double)f[P]));
            acc = fma((double)up, ((sum[0].value() + sum[2].value()) + sum[1].value()) + own, acc);
        }
    }
    acc = block_sum_2d(acc, sh);
    if (threadIdx.x == 0 && threadIdx.y == 0) part[blockIdx.x] = acc;
}

// Adds one event's contribution to the gradients (one CTA): S = the sum of the
// np partial sums of k_pgrad_stencil, Bu = B^T u (a vector, or -Sigma z of the
// low-rank solve whose result u is: then Bu_k = -Sigma_k z_k), Bv = B^T v from
// the P partial sums of k_bt_partial, and xi' the sweep's low-rank normals:
// sweep (kd != 0):
//   g_s += S + kd [sum_k Bu_k Bv_k / Sigma_k - sum_k Bu_k xi'_k / Sigma_k^{1/2}]
//   g_k += Bu_k (Bv_k / Sigma_k - xi'_k / (2 Sigma_k^{1/2}))
// -u^T dA v (kd = 0; the residual f - A x with u = P f_c-bar, and the coarse
// mean Q^{-1} f with u = Q^{-1} x-bar):
//   g_s += S;   g_k += Bu_k Bv_k / Sigma_k
template <typename T, int NOISE>
__global__ void __launch_bounds__(256) k_pgrad_combine(const double *part, int np, const double *Bu, int from_z,
                                                       const double *bv_part, int P, NoiseArgs nz,
                                                       const double *__restrict__ sigma_inv,
                                                       const double *__restrict__ sigma_sqrt, int m, double kd, double *g_s,
                                                       double *g_sig) {
    __shared__ double sh[32];
    double acc = 0.0;
    for (int i = threadIdx.x; i < np; i += blockDim.x) acc += part[i];
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
        double bv = 0.0;
        for (int p = 0; p < P; ++p) {
            if constexpr (sizeof(T) == 4)
                bv += ff_to_double(ff_of(reinterpret_cast<const float2 *>(bv_part)[(i64)k * P + p]));
            else
                bv += bv_part[(i64)k * P + p];
        }
        const double sq = sigma_sqrt[k], si = sigma_inv[k], bu = from_z ? -(sq * sq) * Bu[k] : Bu[k], q = bu * bv * si;
        if (kd != 0.0) {
            double xi = 0.0;
            if (NOISE == NOISE_PHILOX)
                xi = (double)pick(normals4(philox4x32_10(noise_ctr(nz, (unsigned)(k >> 2), PURPOSE_LOWRANK, 0), noise_key(nz))), k & 3);
            if (NOISE == NOISE_INJECTED) xi = nz.buf[k];
            const double r = bu * xi / sq;
            acc += kd * (q - r);
            g_sig[k] += q - 0.5 * r;
        } else {
            g_sig[k] += q;
        }
    }
    acc = block_sum<256>(acc, sh);
    if (threadIdx.x == 0) *g_s += acc;
}

// The n coarse normals of the Cholesky sample, compact.
template <int NOISE>
__global__ void __launch_bounds__(256) k_coarse_normals(NoiseArgs nz, int n, double *__restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double xi = 0.0;
    if (NOISE == NOISE_PHILOX) {
        float4 r = normals4(philox4x32_10(noise_ctr(nz, (unsigned)(i >> 2), PURPOSE_COARSE, 0), noise_key(nz)));
        xi = (double)pick(r, i & 3);
    }
    if (NOISE == NOISE_INJECTED) xi = nz.buf[i];
    out[i] = xi;
}

// The coarse Cholesky sample x = Q^{-1} f + L^{-T} xi, Q = L L^T: with
// dL = L Phi(L^{-1} dQ L^{-T}), Phi(X) = strict lower part + half the
// diagonal, x-bar^T dx = -w1^T dQ mu - xi^T Phi(L^{-1} dQ L^{-T}) w2
// (mu = Q^{-1} f, w1 = Q^{-1} x-bar, w2 = L^{-1} x-bar).
//
// s-term: part[blockIdx.x] = sum over its rows i of xi_i (Phi(X_E) w2)_i,
// X_E = L^{-1} E_c L^{-T} stored like the inverse factor (row-major, ld a
// multiple of 16 bytes, zeros above the diagonal); one warp per row.
template <typename MT>
__global__ void __launch_bounds__(256) k_pgrad_coarse_phi(const MT *__restrict__ Phi, int ld,
                                                          const MT *__restrict__ w2, const double *__restrict__ xi,
                                                          int n, double *__restrict__ part) {
    extern __shared__ __align__(16) unsigned char chol_sm[];
    __shared__ double sh[32];
    MT *ws = reinterpret_cast<MT *>(chol_sm);
    for (int i = threadIdx.x; i < ld; i += blockDim.x) ws[i] = i < n ? w2[i] : MT(0);
    __syncthreads();
    constexpr int NV = Vec16<MT>::N;
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * (blockDim.x >> 5);
    double acc = 0.0;
    for (int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
        WarpRow<MT> row;
        row.load(Phi + (i64)i * ld, 0, i / NV + 1, lane);
        const MT r = row.dot(ws);
        if (lane == 0) acc += xi[i] * (double)r;
    }
    acc = block_sum<256>(acc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

// *target += scale * sum(part[0 .. np))
__global__ void __launch_bounds__(256) k_accum_sum(const double *__restrict__ part, int np, double scale,
                                                   double *__restrict__ target) {
    __shared__ double sh[32];
    double acc = 0.0;
    for (int i = threadIdx.x; i < np; i += blockDim.x) acc += part[i];
    acc = block_sum<256>(acc, sh);
    if (threadIdx.x == 0) *target += scale * acc;
}

// log Sigma_k term of the coarse sample's L^{-T} xi part (dQ = -b_k b_k^T /
// Sigma_k, u = L^{-1} b_k, column k of U):
//   g_k += (1 / Sigma_k) sum_j u_j w2_j (sum_{i > j} u_i xi_i + u_j xi_j / 2).
// One CTA per k; the suffix sums run over chunks of 256 indices from the
// end, a block scan inside each chunk.
template <typename MT>
__global__ void __launch_bounds__(256) k_pgrad_coarse_sigma(const double *__restrict__ U, const MT *__restrict__ w2,
                                                            const double *__restrict__ xi,
                                                            const double *__restrict__ sigma_inv,
                                                            double *__restrict__ g_sig, int n) {
    __shared__ double wsum[8];
    __shared__ double sh[32];
    __shared__ double carry;
    const int k = blockIdx.x;
    const double *u = U + (i64)k * n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0.0;
    __syncthreads();
    double acc = 0.0;
    for (int base = ((n - 1) / 256) * 256; base >= 0; base -= 256) {
        const int j = base + threadIdx.x;
        const double uj = j < n ? u[j] : 0.0, xj = j < n ? xi[j] : 0.0, wj = j < n ? (double)w2[j] : 0.0;
        const double v = uj * xj;
        double incl = v;  // sum over the lanes at or above this one
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double t = __shfl_down_sync(0xffffffffu, incl, o);
            if (lane + o < 32) incl += t;
        }
        if (lane == 0) wsum[warp] = incl;
        __syncthreads();
        double above = 0.0;
        for (int q = warp + 1; q < 8; ++q) above += wsum[q];
        acc += wj * uj * (carry + above + (incl - v) + 0.5 * v);
        __syncthreads();
        if (threadIdx.x == 0) {
            double tot = 0.0;
            for (int q = 0; q < 8; ++q) tot += wsum[q];
            carry += tot;
        }
        __syncthreads();
    }
    acc = block_sum<256>(acc, sh);
    if (threadIdx.x == 0) g_sig[k] += sigma_inv[k] * acc;
}

// ------------------------------------------------------------ step end
// Observables z_p = b_p^T x of measure_sampling_time (sampling_time.cc:40):
// CTA (p, q), q < split, sums its share of probe p's entries
// bptr[p]..bptr[p+1] into part[p split + q]; the last CTA to finish adds the
// shares in order, stores z_p at obs[k * nprobe + p] for step k while
// k < capacity (a non-finite value raises the error flag) and advances the
// observation count and the step counter that keys the Philox streams.  Runs
// after every other kernel of the step.  The entries do not depend on the
// step: a CTA's first 1024 are loaded before the wait.  (The central ball of
// 256^3, 8,700 entries: one CTA took 18.6 us under ncu, its loads one after
// the other and its sums on one SM's FP64 unit; nine CTAs 7.)
struct StepEnd {
    int nprobe, split;
    const i64 *bptr, *bidx;
    const double *bval;
    double *part, *obs;
    i64 capacity;
    u64 *obs_count, *d_step;
    unsigned *err, *done;
};
constexpr int STEP_END_ENTRIES = 1024, STEP_END_MAX_SPLIT = 16;


template <typename T>
__device__ __forceinline__ void step_end_body(const T *x, const StepEnd &e, int cta, int nblocks) {
    __shared__ double sh[32];
    __shared__ bool last;
    const int p = e.split ? cta / e.split : 0, q = cta - p * e.split;
    const bool mine = p < e.nprobe;
    i64 lo = 0, hi = 0, idx[4];
    double val[4];
    if (mine) {
        const i64 b0 = e.bptr[p], b1 = e.bptr[p + 1], len = (b1 - b0 + e.split - 1) / e.split;
        lo = b0 + q * len + threadIdx.x;
        hi = min(b1, b0 + (q + 1) * len);
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (lo + 256 * t < hi) {
                idx[t] = e.bidx[lo + 256 * t];
                val[t] = e.bval[lo + 256 * t];
            }
    }
    pdl_begin();
    if (mine) {
        double acc = 0.0;
        T xv[4];
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (lo + 256 * t < hi) xv[t] = x[idx[t]];
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (lo + 256 * t < hi) acc = fma(val[t], to_double(xv[t]), acc);
#pragma unroll 4
        for (i64 i = lo + STEP_END_ENTRIES; i < hi; i += 256) acc = fma(e.bval[i], to_double(x[e.bidx[i]]), acc);
        acc = block_sum<256>(acc, sh);
        if (threadIdx.x == 0) e.part[cta] = acc;
    }
    if (threadIdx.x == 0) {
        unsigned prev;  // publishes the partial sum; in the last CTA, makes the others visible
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(prev) : "l"(e.done) : "memory");
        last = prev == (unsigned)nblocks - 1u;
    }
    __syncthreads();
    if (!last) return;
    if (e.nprobe > 0) {
        const u64 k = *e.obs_count;
        for (int r = threadIdx.x; r < e.nprobe; r += blockDim.x) {
            double z = 0.0;
            for (int t = 0; t < e.split; ++t) z += __ldcg(e.part + (i64)r * e.split + t);
            if ((i64)k < e.capacity) e.obs[k * e.nprobe + r] = z;
            if (!isfinite(z)) atomicOr_system(e.err, 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (e.nprobe > 0) *e.obs_count += 1ull;
        *e.d_step += 1ull;
        *e.done = 0u;
    }
}

template <typename T>
__global__ void __launch_bounds__(256) k_step_end(const T *x, StepEnd e) {
    step_end_body<T>(x, e, blockIdx.x, gridDim.x);
}

// ------------------------------------------- low-rank Cholesky sampler
// The block solves with L (blocks D_k = L_kk^{-1}, O_k = L_{k,k-1} of p x p)
//   g_k = D_k (f_k - O_k g_{k-1}) = D_k f_k - E_k g_{k-1},      E_k = D_k O_k
//   x_k = D_k^T (xi_k - O_{k+1}^T x_{k+1}) = D_k^T xi_k - G_k x_{k+1},
//                                                   G_k = D_k^T O_{k+1}^T
// are a product of all triangular blocks at once (k_chol_tri) and a chain of
// one dense product per block (k_chol_step): half the dependent launches of
// the form with two products per block, and every product reads rows.
// Vectors are stored by blocks of ld doubles (p, padded with zeros to a
// multiple of 4), matrices with rows of ld.  D_k and D_k^T share one symmetric
// array: row i holds row i of D_k up to the diagonal and row i of D_k^T from
// there on.  Where E and G do not fit, the chain keeps O and runs the first
// form, one block at a time (k_chol_step with O_k, k_chol_step_t, k_chol_tri).

// y_k = A_k v_k for all blocks k = blockIdx.y, A_k the lower or (UPPER: columns
// j >= i) the upper triangle of the stored block.  A warp takes the rows i and
// p - 1 - i, together one full row, and reduces both sums in five steps instead
// of ten: FP64 instructions, two per clock per SM, bound it.
template <bool UPPER>
__global__ void __launch_bounds__(256) k_chol_tri(const double *__restrict__ A, int p, int ld, const double *v, double *y) {
    const int lane = threadIdx.x & 31, i = blockIdx.x * 8 + (threadIdx.x >> 5), k = blockIdx.y;
    pdl_begin();
    if (i >= (p + 1) / 2) return;
    const int i2 = p - 1 - i;
    const double2 *vk = reinterpret_cast<const double2 *>(v + (i64)k * ld);
    auto row_sum = [&](int r) {
        const double2 *a = reinterpret_cast<const double2 *>(A + ((i64)k * p + r) * ld);
        const int q0 = UPPER ? r / 2 : 0, q1 = UPPER ? ld / 2 : r / 2 + 1;
        // the pair at the diagonal, a lane's first (UPPER) or last one, may hold a value of the other triangle
        const int qd = UPPER == (r & 1) ? r / 2 : -1;
        double s0 = 0.0, s1 = 0.0;
        int q = q0 + lane;
        for (; q + 96 < q1; q += 128) {
            double2 av[4], vv[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) av[t] = __ldcs(a + q + 32 * t);
            if (UPPER && q == qd) av[0].x = 0.0;
            if (!UPPER && q + 96 == qd) av[3].y = 0.0;
#pragma unroll
            for (int t = 0; t < 4; ++t) vv[t] = vk[q + 32 * t];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                s0 = fma(av[t].x, vv[t].x, s0);
                s1 = fma(av[t].y, vv[t].y, s1);
            }
        }
        for (; q < q1; q += 32) {
            double2 av = __ldcs(a + q);
            const double2 vv = vk[q];
            if (q == qd) (UPPER ? av.x : av.y) = 0.0;
            s0 = fma(av.x, vv.x, s0);
            s1 = fma(av.y, vv.y, s1);
        }
        return s0 + s1;
    };
    const double a0 = row_sum(i), a1 = i2 == i ? 0.0 : row_sum(i2);
    const double give = lane < 16 ? a1 : a0;  // lanes 0-15 reduce row i, 16-31 row i2
    double s = (lane < 16 ? a0 : a1) + __shfl_xor_sync(0xffffffffu, give, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) y[(i64)k * ld + i] = s;
    if (lane == 16 && i2 != i) y[(i64)k * ld + i2] = s;
}

// One link of the chain: y -= A v, A p x p dense, one warp per row.  The row
// does not depend on the launch before, so its first 1024 values are in
// registers before the wait, and the next link starts at once to load its own:
// what is left between two links is the read of v, 30 FP64 multiplications and
// five additions.  (32^3 cells, p = 961: a sample of 425 us is a chain of 60
// links beside the triangular and low-rank products, 5 to 6 us each.)
__global__ void __launch_bounds__(256, 2) k_chol_step(const double *__restrict__ A, int p, int ld, const double *v, double *y) {
    const int lane = threadIdx.x & 31, row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), n2 = ld / 2;
    const double2 *a = reinterpret_cast<const double2 *>(A + (i64)min(row, p - 1) * ld);
    const double2 *vv = reinterpret_cast<const double2 *>(v);
    double2 av[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) av[t] = lane + 32 * t < n2 ? __ldcs(a + lane + 32 * t) : make_double2(0.0, 0.0);
    pdl_begin();
    pdl_trigger();
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (256 * h >= n2) break;
        double2 w[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) w[t] = lane + 32 * (8 * h + t) < n2 ? vv[lane + 32 * (8 * h + t)] : make_double2(0.0, 0.0);
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            if (32 * (8 * h + t) >= n2) break;
            s0 = fma(av[8 * h + t].x, w[t].x, s0);
            s1 = fma(av[8 * h + t].y, w[t].y, s1);
        }
    }
    for (int q = lane + 512; q < n2; q += 128) {
        double2 b[4], w[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const bool in = q + 32 * t < n2;
            b[t] = in ? __ldcs(a + q + 32 * t) : make_double2(0.0, 0.0);
            w[t] = in ? vv[q + 32 * t] : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            s0 = fma(b[t].x, w[t].x, s0);
            s1 = fma(b[t].y, w[t].y, s1);
        }
    }
    double s = s0 + s1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0 && row < p) y[row] -= s;
}

// y -= A^T v, A p x p dense: a CTA takes 32 columns, its warps every eighth row.
__global__ void __launch_bounds__(256) k_chol_step_t(const double *__restrict__ A, int p, int ld, const double *v, double *y) {
    __shared__ double sh[8][32];
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5, j = blockIdx.x * 32 + l;
    pdl_begin();
    double t = 0.0;
    if (j < p) {
#pragma unroll 4
        for (int i = w; i < p; i += 8) t = fma(A[(i64)i * ld + j], v[i], t);
    }
    sh[w][l] = t;
    __syncthreads();
    if (w == 0 && j < p) {
        t = 0.0;
#pragma unroll
        for (int i = 0; i < 8; ++i) t += sh[i][l];
        y[j] -= t;
    }
}

// Low-rank part, xi += g + Q (W^T - Id) Q^T g, then xi += Q (W - Id) Q^T xi:
// each a product with Q^T (k_chol_qt), an m x m one (k_chol_v, or k_chol_t and
// k_chol_w) and one with Q
// (k_chol_add).  Q^T xi is formed from the updated xi although W^T Q^T g +
// Q^T xi would save a pass over Q: W is small where the measurements are
// accurate, and only the product with the rounded xi damps its rounding too
// (16^3 posterior against the oracle: 1.1e-12 instead of below 1e-12).
//
// Partial sums of Q^T v over CHOL_QT_ROWS rows per CTA: part[cta * m + j].
constexpr int CHOL_QT_ROWS = 128;
__global__ void __launch_bounds__(256) k_chol_qt(const double *__restrict__ Q, i64 rows, int m, const double *v,
                                                 double *part) {
    __shared__ double sh[8][32];
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    pdl_begin();
    pdl_trigger();
    const i64 r0 = (i64)blockIdx.x * CHOL_QT_ROWS, r1 = min(rows, r0 + CHOL_QT_ROWS);
    for (int j0 = 0; j0 < m; j0 += 32) {
        const int j = j0 + l;
        double t = 0.0;
        if (j < m) {
#pragma unroll 4
            for (i64 r = r0 + w; r < r1; r += 8) t = fma(Q[r * m + j], v[r], t);
        }
        sh[w][l] = t;
        __syncthreads();
        if (w == 0 && j < m) {
            double a = 0.0;
#pragma unroll
            for (int i = 0; i < 8; ++i) a += sh[i][l];
            part[(i64)blockIdx.x * m + j] = a;
        }
        __syncthreads();
    }
}

// t = the sum of the parts and v = (W - Id) t (TRANSPOSE: (W^T - Id) t) in one
// CTA, eight lanes per sum, for up to CHOL_V_COLS columns; more take k_chol_t
// and k_chol_w, whose CTAs share the m^2 terms.  (A sample of 16^3 cells, both
// products in one CTA and in two launches each: 8 columns 103 and 105 us, 32 109
// and 109, 64 124 and 120, 128 163 and 145; of 24^3 with 1000: 2085 and 1027.)
constexpr int CHOL_V_COLS = 32;
template <bool TRANSPOSE>
__global__ void __launch_bounds__(8 * CHOL_V_COLS) k_chol_v(const double *part, int nparts, int m, const double *__restrict__ W,
                                                 double *v) {
    __shared__ double ts[CHOL_V_COLS];
    pdl_begin();
    pdl_trigger();
    const int l = threadIdx.x & 7, c = threadIdx.x >> 3;
    auto over8 = [](double a) {
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        return a;
    };
    double a = 0.0;
    if (c < m) {
#pragma unroll 4
        for (int i = l; i < nparts; i += 8) a += part[(i64)i * m + c];
    }
    a = over8(a);
    if (l == 0 && c < m) ts[c] = a;
    __syncthreads();
    a = 0.0;
    if (c < m)
        for (int k = l; k < m; k += 8)
            a = fma((TRANSPOSE ? W[(i64)k * m + c] : W[(i64)c * m + k]) - (k == c ? 1.0 : 0.0), ts[k], a);
    a = over8(a);
    if (l == 0 && c < m) v[c] = a;
}

// the sum over the warps of a CTA of 256 threads, lane by lane, in warp 0
__device__ __forceinline__ double sum_over_warps(double a) {
    __shared__ double sh[8][32];
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    sh[w][l] = a;
    __syncthreads();
    a = 0.0;
    if (w == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) a += sh[i][l];
    }
    return a;
}

// t = the sum of the parts, 32 columns per CTA
__global__ void __launch_bounds__(256) k_chol_t(const double *part, int nparts, int m, double *t) {
    pdl_begin();
    pdl_trigger();
    const int c = blockIdx.x * 32 + (threadIdx.x & 31);
    double a = 0.0;
    if (c < m) {
#pragma unroll 4
        for (int i = threadIdx.x >> 5; i < nparts; i += 8) a += part[(i64)i * m + c];
    }
    a = sum_over_warps(a);
    if (threadIdx.x < 32 && c < m) t[c] = a;
}

// v = (W - Id) t, a warp per row and 8 rows per CTA, or (TRANSPOSE) (W^T - Id) t,
// 32 columns per CTA, its warps every eighth row
template <bool TRANSPOSE>
__global__ void __launch_bounds__(256) k_chol_w(const double *__restrict__ W, int m, const double *t, double *v) {
    pdl_begin();
    pdl_trigger();
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    double a = 0.0;
    if (TRANSPOSE) {
        const int c = blockIdx.x * 32 + l;
        if (c < m) {
#pragma unroll 4
            for (int k = w; k < m; k += 8) a = fma(W[(i64)k * m + c] - (k == c ? 1.0 : 0.0), t[k], a);
        }
        a = sum_over_warps(a);
        if (w == 0 && c < m) v[c] = a;
    } else {
        const int c = blockIdx.x * 8 + w;
        if (c < m) {
#pragma unroll 4
            for (int k = l; k < m; k += 32) a = fma(W[(i64)c * m + k] - (k == c ? 1.0 : 0.0), t[k], a);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (l == 0 && c < m) v[c] = a;
    }
}

// xi += Q v (ADD_G: + g), one thread per row, v in shared memory unless WIDE
// (more columns than it takes)
constexpr int CHOL_STAGE_M = 28672;
template <bool ADD_G, bool WIDE>
__global__ void __launch_bounds__(128) k_chol_add(double *xi, const double *g, const double *__restrict__ Q, i64 rows, int m,
                                                  const double *v) {
    extern __shared__ double v_sm[];
    const double *vs = WIDE ? v : v_sm;
    pdl_begin();
    pdl_trigger();
    if (!WIDE) {
        for (int j = threadIdx.x; j < m; j += blockDim.x) v_sm[j] = v[j];
        __syncthreads();
    }
    const i64 r = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    double a0 = 0.0, a1 = 0.0;
    const double *q = Q + r * m;
    int j = 0;
    for (; j + 3 < m; j += 4) {
        const double q0 = q[j], q1 = q[j + 1], q2 = q[j + 2], q3 = q[j + 3];
        a0 = fma(q0, vs[j], a0);
        a1 = fma(q1, vs[j + 1], a1);
        a0 = fma(q2, vs[j + 2], a0);
        a1 = fma(q3, vs[j + 3], a1);
    }
    for (; j < m; ++j) a0 = fma(q[j], vs[j], a0);
    a0 += a1;
    if (ADD_G) a0 += g[r];
    xi[r] += a0;
}

// xi_i ~ N(0, 1): Philox (counter: vertex group i / 4, purpose
// PURPOSE_CHOLESKY, the sampler's step counter) or the injected normals, into
// blocks of ld (zeros behind the p values of a block)
template <int NOISE>
__global__ void __launch_bounds__(256) k_cholesky_normals(NoiseArgs nz, int nb, int p, int ld, double *xi) {
    const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    const int k = (int)(t / ld), j = (int)(t - (i64)k * ld);
    if (k >= nb) return;
    const i64 i = (i64)k * p + j;
    double v = 0.0;
    if (j < p) {
        if (NOISE == NOISE_INJECTED)
            v = nz.buf[i];
        else
            v = (double)pick(normals4(philox4x32_10(noise_ctr(nz, (unsigned)(i >> 2), PURPOSE_CHOLESKY, 0), noise_key(nz))),
                             (int)(i & 3));
    }
    xi[t] = v;
}

// compact vectors of nb p values to and from blocks of ld
__global__ void __launch_bounds__(256) k_chol_pad(const double *__restrict__ src, double *__restrict__ dst, int nb, int p, int ld) {
    const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    const int k = (int)(t / ld), j = (int)(t - (i64)k * ld);
    if (k < nb) dst[t] = j < p ? src[(i64)k * p + j] : 0.0;
}
__global__ void __launch_bounds__(256) k_chol_unpad(const double *__restrict__ src, double *__restrict__ dst, int nb, int p, int ld) {
    const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    const int k = (int)(t / ld), j = (int)(t - (i64)k * ld);
    if (k < nb && j < p) dst[(i64)k * p + j] = src[t];
}

// Set-up: C_k(i, j) = sum_l A_k(i, l) B_k(l, j), p x p each, A_k the lower or
// (UPPER) the upper triangle of a block of S, B_k through strides (B_k(l, j) at
// k bs + l bl + j bj); tiles of 64 x 64, 4 x 4 per thread.
template <bool UPPER>
__global__ void __launch_bounds__(256) k_chol_gemm(const double *__restrict__ S, i64 mat, int ld, const double *__restrict__ B,
                                                   i64 bs, i64 bl, i64 bj, double *__restrict__ C, int p) {
    __shared__ double At[16][64 + 1], Bt[16][64 + 1];
    S += blockIdx.z * mat;
    B += blockIdx.z * bs;
    C += blockIdx.z * mat;
    const int i0 = blockIdx.y * 64, j0 = blockIdx.x * 64, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double acc[4][4] = {};
    const int l1 = UPPER ? p : min(p, i0 + 64);
    for (int l0 = UPPER ? i0 : 0; l0 < l1; l0 += 16) {
        for (int t = threadIdx.x; t < 16 * 64; t += 256) {
            const int la = t & 15, i = i0 + (t >> 4), l = l0 + la;
            At[la][t >> 4] = i < p && l < p && (UPPER ? l >= i : l <= i) ? S[(i64)i * ld + l] : 0.0;
            // the index with the unit stride runs over the threads
            const int lb = bl == 1 ? t & 15 : t >> 6, jb = bl == 1 ? t >> 4 : t & 63;
            Bt[lb][jb] = j0 + jb < p && l0 + lb < p ? B[(l0 + lb) * bl + (j0 + jb) * bj] : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int l = 0; l < 16; ++l)
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) acc[a][b] = fma(At[l][ty + 16 * a], Bt[l][tx + 16 * b], acc[a][b]);
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (i0 + ty + 16 * a < p && j0 + tx + 16 * b < p) C[(i64)(i0 + ty + 16 * a) * ld + j0 + tx + 16 * b] = acc[a][b];
}

// the upper triangles of blocks of p rows of ld from the lower ones
__global__ void __launch_bounds__(256) k_chol_mirror(double *S, int p, int ld) {
    __shared__ double tile[32][33];
    S += (i64)blockIdx.z * p * ld;
    const int i0 = blockIdx.y * 32, j0 = blockIdx.x * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    if (i0 < j0) return;
    for (int r = ty; r < 32; r += 8)
        if (i0 + r < p && j0 + tx < p) tile[r][tx] = S[(i64)(i0 + r) * ld + j0 + tx];
    __syncthreads();
    for (int r = ty; r < 32; r += 8)
        if (i0 + tx < p && i0 + tx > j0 + r) S[(i64)(j0 + r) * ld + i0 + tx] = tile[tx][r];
}

__global__ void k_counter_advance(u64 *step) {
    pdl_begin();
    *step += 1ull;
}

// ------------------------------------------------------- batched chains
// Chains of one lattice geometry stepped together (FP32-mixed chains with
// Philox noise): every launch of the step covers all chains of the group --
// blockIdx.z (or blockIdx.y) picks the chain for the regular work, a job
// table for the ragged low-rank work -- and each chain keeps its own arrays,
// stencils, low-rank data, Philox key and step counter.  The kernels call
// the one-chain kernels' bodies, so a chain stepped in a batch draws the
// same normals and computes the same values, bit for bit, as when it is
// stepped alone.

// One chain on one level.
struct BatchLevelArg {
    float *x, *f;
    const float *fsplit;  // level 0: the colour-split f (colour k at fsplit + k * fhalf), else null
    i64 fhalf;
    float *xc, *fc;       // the next level's state and right hand side (null on the coarsest level)
    StencilArg<float> s;
};
static_assert(sizeof(StencilArg<float>) == 32 * sizeof(float), "stencil argument: 32 floats");

// One chain: noise key, step counter, coarse Cholesky factors, observables.
struct BatchChainArg {
    u64 seed;
    u64 *d_step;
    const float *Linv, *LinvT;
    float *gv;
    StepEnd end;
};

// Low-rank data of one chain on one level and sweep direction: the B^T x
// arguments, C = M^{-1} B by rows and its CTAs' columns.
struct BatchLowRank {
    LowRankArg lr;
    CorrRows C;  // x += C z rows (FP32 values)
    const int *jobcols;
    int P;       // partial sums per column
};

// B^T x work unit: chain, column j, part p of P.
struct BtJob {
    int chain, j, p, P;
};
// A CTA of one chain's correction.
struct BatchCorrJob {
    int chain;
    CorrJob job;
};
// A CTA of one chain's solve (k_lr_z).
struct BatchZJob {
    int chain, tile;
};
// Up to 256 rows from r0 on of one chain's B_c Sigma^{-1} y.
struct RowJob {
    int chain;
    i64 r0;
};
// B_c Sigma^{-1} y rows of one chain's coarse level (the residual's
// low-rank term), y from its partial sums, destination its coarse f.
struct BatchAddBq {
    i64 nrows;
    const i64 *rows, *ptr;
    const int *col;
    const double *val, *part, *sigma_inv;
    int m, P;
    float *dst;
};

__device__ __forceinline__ void load_stencil_shared(StencilArg<float> &dst, const StencilArg<float> &src) {
    const int t = (threadIdx.z * blockDim.y + threadIdx.y) * blockDim.x + threadIdx.x;
    if (t < 32) reinterpret_cast<float *>(&dst)[t] = reinterpret_cast<const float *>(&src)[t];
    __syncthreads();
}

__device__ __forceinline__ NoiseArgs batch_noise(const BatchChainArg &c, unsigned invocation, unsigned level) {
    NoiseArgs nz;
    nz.buf = nullptr;
    nz.seed = c.seed;
    nz.d_step = c.d_step;
    nz.invocation = invocation;
    nz.level = level;
    return nz;
}

// red-black colour pass of the 7-point level, grid.z = chains x planes
template <int NOISE, bool V8, bool FS>
__global__ void __launch_bounds__(RBP_THREADS) k_sweep_rb_vec_batch(const BatchLevelArg *__restrict__ la,
                                                                    const BatchChainArg *__restrict__ ca, Grid3 g,
                                                                    int colour, int reverse, unsigned invocation,
                                                                    unsigned level) {
    __shared__ StencilArg<float> ss;
    const int chain = blockIdx.z / g.N2, bz = blockIdx.z - chain * g.N2;
    const BatchLevelArg &a = la[chain];
    load_stencil_shared(ss, a.s);
    const NoiseArgs nz = batch_noise(ca[chain], invocation, level);
    const float *fsc = FS ? a.fsplit + colour * a.fhalf : nullptr;
    sweep_rb_vec_body<NOISE, false, V8, FS, true>(a.x, a.f, g, ss, colour, reverse, nz, nullptr, fsc, blockIdx.x, blockIdx.y,
                                            bz);
}

// a pair of colours of an 8-colour level, grid.z = chains x planes of the pair
template <int NOISE>
__global__ void __launch_bounds__(ROW_PAIR_THREADS)
    k_sweep_row_pair_batch(const BatchLevelArg *__restrict__ la, const BatchChainArg *__restrict__ ca, Grid3 g, int pb,
                           int pc, int odd_first, int ncz, unsigned invocation, unsigned level) {
    __shared__ StencilArg<float> ss;
    extern __shared__ __align__(16) unsigned char row_sm[];
    const int chain = blockIdx.z / ncz, bz = blockIdx.z - chain * ncz;
    const BatchLevelArg &a = la[chain];
    load_stencil_shared(ss, a.s);
    const NoiseArgs nz = batch_noise(ca[chain], invocation, level);
    sweep_row_pair_body<float, 27, false, NOISE, 0>(a.x, a.f, g, ss, pb, pc, odd_first, nz, VarField<float>{nullptr, 0},
                                                    blockIdx.y, bz, reinterpret_cast<float *>(row_sm), true, true);
}

// one colour of an 8-colour level with rows too long for a CTA, grid.z =
// chains x colour planes
template <int NOISE>
__global__ void __launch_bounds__(RBP_THREADS) k_sweep_c27_batch(const BatchLevelArg *__restrict__ la,
                                                                 const BatchChainArg *__restrict__ ca, Grid3 g,
                                                                 int colour, int ncz, unsigned invocation,
                                                                 unsigned level) {
    __shared__ StencilArg<float> ss;
    const int chain = blockIdx.z / ncz, bz = blockIdx.z - chain * ncz;
    const BatchLevelArg &a = la[chain];
    load_stencil_shared(ss, a.s);
    const NoiseArgs nz = batch_noise(ca[chain], invocation, level);
    pdl_begin();
    sweep_c27_body<float, false, NOISE, 0>(a.x, a.f, g, ss, colour, nz, VarField<float>{nullptr, 0}, blockIdx.x,
                                           blockIdx.y, bz);
}

// B^T x partial sums and the low-rank noise (NOISE_NONE: the residual's), one
// CTA per job
template <int NOISE>
__global__ void __launch_bounds__(256) k_bt_partial_batch(const BatchLevelArg *__restrict__ la,
                                                          const BatchLowRank *__restrict__ lrs,
                                                          const BatchChainArg *__restrict__ ca,
                                                          const BtJob *__restrict__ jobs, unsigned invocation,
                                                          unsigned level) {
    const BtJob jb = jobs[blockIdx.x];
    LowRankArg lr = lrs[jb.chain].lr;
    if (NOISE == NOISE_NONE) lr.w = nullptr;
    bt_partial_body<float, NOISE>(la[jb.chain].x, lr, batch_noise(ca[jb.chain], invocation, level), jb.j, jb.p, jb.P);
}

// the solve of chains whose corrections do not form z themselves (mode 2)
__global__ void __launch_bounds__(256) k_lr_z_batch(const BatchLowRank *__restrict__ lrs, const BatchZJob *__restrict__ jobs) {
    extern __shared__ double dyn[];
    const BatchZJob jb = jobs[blockIdx.x];
    const BatchLowRank &c = lrs[jb.chain];
    lr_z_body<float>(c.lr, c.P, jb.tile, dyn);
}

// the solve (modes 0 and 1) and x += C z, one CTA per job
template <int MODE>
__global__ void __launch_bounds__(256, MODE == 1 ? 2 : 4)
    k_lr_correct_batch(const BatchLevelArg *__restrict__ la, const BatchLowRank *__restrict__ lrs,
                       const BatchCorrJob *__restrict__ jobs) {
    extern __shared__ double dyn[];
    const BatchCorrJob jb = jobs[blockIdx.x];
    const BatchLowRank &c = lrs[jb.chain];
    lr_correct_body<float, MODE, 1>(la[jb.chain].x, c.lr, c.P, c.C, jb.job, c.jobcols, false, dyn);
}

// f_c -= B_c Sigma^{-1} y, one CTA per job
__global__ void __launch_bounds__(256) k_resid_Bq_batch(const BatchAddBq *__restrict__ bq, const RowJob *__restrict__ jobs) {
    extern __shared__ double qs[];
    const RowJob jb = jobs[blockIdx.x];
    const BatchAddBq &a = bq[jb.chain];
    resid_Bq_body<float>(a.dst, a.nrows, a.rows, a.ptr, a.col, a.val, a.part, a.m, a.P, a.sigma_inv, jb.r0 + threadIdx.x, qs);
}

// residual + restriction, grid.z = chains x coarse tiles in z
template <int NPT>
// Six CTAs per SM: the batched residual-restriction (plain loads, one CTA per
// tile of one chain) gains more from occupancy than it loses to the spills
// this forces (512 chains of 32^3-128^3 cells: 23.1k -> 25.8k samples/s
// against 24.9k with four CTAs per SM, one box).
#ifndef MGMC_RR_BATCH_MINB
#define MGMC_RR_BATCH_MINB 6
#endif
__global__ void __launch_bounds__(RR_THREADS, MGMC_RR_BATCH_MINB) k_resid_restrict_batch(const BatchLevelArg *__restrict__ la, Grid3 gf,
                                                                      Grid3 gc, int tz) {
    __shared__ StencilArg<float> ss;
    extern __shared__ __align__(16) unsigned char rr_smem_b[];
    const int chain = blockIdx.z / tz, bz = blockIdx.z - chain * tz;
    const BatchLevelArg &a = la[chain];
    load_stencil_shared(ss, a.s);
    pdl_begin();
    resid_restrict_tiled_body<float, NPT>(a.x, a.f, a.fc, a.xc, gf, gc, ss, rr_smem_b, blockIdx.x, blockIdx.y, bz);
}

// x += alpha P x_c, grid.z = chains x (coarse planes + 1)
__global__ void __launch_bounds__(128) k_prolong_batch(const BatchLevelArg *__restrict__ la, Grid3 gf, Grid3 gc,
                                                       float alpha, int nzc) {
    const int chain = blockIdx.z / nzc, bz = blockIdx.z - chain * nzc;
    const BatchLevelArg &a = la[chain];
    pdl_begin();
    prolong_add_body<float, 3>(a.x, a.xc, gf, gc, alpha, blockIdx.x, blockIdx.y, nzc - 1 - bz);  // batched chains are 3D
}

// coarse Cholesky sample, grid.y = chains
template <int NOISE>
__global__ void __launch_bounds__(256) k_chol_lower_batch(const BatchLevelArg *__restrict__ la,
                                                          const BatchChainArg *__restrict__ ca, Grid3 g, int ld,
                                                          unsigned invocation, unsigned level) {
    extern __shared__ __align__(16) unsigned char chol_sm_b[];
    const BatchChainArg &c = ca[blockIdx.y];
    const NoiseArgs nz = batch_noise(c, invocation, level);
    chol_gemv_lower_body<float, float, NOISE>(la[blockIdx.y].f, g, c.Linv, ld, c.gv, nz, true, chol_sm_b, blockIdx.x);
}

__global__ void __launch_bounds__(256) k_chol_upper_batch(const BatchLevelArg *__restrict__ la,
                                                          const BatchChainArg *__restrict__ ca, Grid3 g, int ld) {
    extern __shared__ __align__(16) unsigned char chol_sm_b[];
    const BatchChainArg &c = ca[blockIdx.y];
    chol_gemv_upper_body<float, float>(c.gv, g, c.LinvT, ld, la[blockIdx.y].x, true, chol_sm_b, blockIdx.x);
}

// observables and step counters, grid.y = chains
__global__ void __launch_bounds__(256) k_step_end_batch(const BatchLevelArg *__restrict__ la,
                                                        const BatchChainArg *__restrict__ ca) {
    step_end_body<float>(la[blockIdx.y].x, ca[blockIdx.y].end, blockIdx.x, gridDim.x);
}

}  // namespace mgmc
