// Fused diagnostics pass: plaquette windings + pierced list (string finder),
// the 14 screened/unscreened energy sums, and gamma^2 v^2 at pierced corners,
// in one sweep over the valid cells.
//
// Reference: StringFinder.hpp:45-122, PlaquetteWinding.hpp:24-51,
// EnergyKernel.hpp:106-233, Energy.hpp:64-190, Masking.hpp:75-93,
// VelocityKernel.hpp:37-141, Velocity.hpp:62-78.
//
// Windings follow the reference literally: double atan2 of the (double-cast)
// field at each corner, fmod fold into (-pi, pi], lround of the sum / 2 pi.
// Edges whose |dtheta| lies within 1e-12 of pi are counted as "near ties":
// only there could a different correctly-rounded-to-1-ulp atan2 flip a fold.
// Per-cell energy/velocity terms are FP64 whatever the field precision, unless the
// caller asks for FP32 terms on FP32 fields (per_cell_fp32); of FP32 fields the
// gradients are floats, as the reference has them, formed without FP64 where that is
// sure to give the same float. Sums go per thread -> warp shuffle -> block -> per-block partial
// in scratch -> a single-block finalize in a fixed order (deterministic, no
// floating-point atomics).
#include <climits>
#include <cmath>
#include <mutex>

#include <algorithm>
#include <type_traits>

#include "axs_internal.cuh"
#include "fp64_pos.cuh"
#include "sweep.cuh"
#include "winding.cuh"

namespace axs {

struct DiagView {
    const void *data;
    int32_t dtype;
    int nx, ny, nz;
    int ox, oy, oz;          // offset of valid cell (0,0,0) in elements along each axis
    int wx, wy, wz;          // 1: wrap indices periodically on that axis; 0: read ghosts
    int64_t js, ks, cs;
};

struct DiagPartial {
    double e[14];
    double vsum;
    long long cnt[4];  // n_p_plain, n_p_weighted, vel_count, near_tie
    double pad;
};
static_assert(sizeof(DiagPartial) == 160, "partial layout");

constexpr int kDiagThreads = 256;

struct DiagConst {
    double one_over_dx, R, lambda, RpR, m_r, threshold;
    double R2, inv_R, inv_R2, inv_R4;
    double vel_a, vel_b, vel_c;  // gamma^2 v^2 = |phi'|^2 vel_a (1 - vel_b |phi|^2) - vel_c (phi . phi')^2
    int scheme;
    int want_energy, want_plaq, want_vel;
    // single-precision copies for the per_cell_fp32 variant
    float f_one_over_dx, f_R2, f_inv_R, f_inv_R2, f_inv_R4, f_lambda, f_RpR, f_threshold;
    float f_vel_a, f_vel_b, f_vel_c;
    float f_k12h, f_k12l;  // 1/(12 dx) as a float and its remainder (diff1_pairs)
};

template <typename T>
__device__ __forceinline__ int64_t view_off(const DiagView &v, int c, int i, int j, int k)
{
    if (v.wx) i = (i % v.nx + v.nx) % v.nx;
    if (v.wy) j = (j % v.ny + v.ny) % v.ny;
    if (v.wz) k = (k % v.nz + v.nz) % v.nz;
    return c * v.cs + (int64_t)(i + v.ox) + (int64_t)(j + v.oy) * v.js + (int64_t)(k + v.oz) * v.ks;
}

template <typename T>
__device__ __forceinline__ double ld(const DiagView &v, int c, int i, int j, int k)
{
    return (double)__ldg(static_cast<const T *>(v.data) + view_off<T>(v, c, i, j, k));
}

// GRTeclyn diff1 (centred 4th order: weights 1/12, 2/3, times 1/dx) from
// the four neighbours, rounded to the field precision as d1_scalar returns
// amrex::Real. FP32 fields: the reference's expression order with explicit
// round-to-nearest double operations, since a fused multiply-add could move
// the rounded float by one ulp. FP64 fields: contraction allowed.
template <typename T>
__device__ __forceinline__ double diff1_vals(double m2, double m1, double p1, double p2, double inv_dx)
{
    const double wf = 8.33333333333333333333e-2, wn = 6.66666666666666666667e-1;
    if constexpr (sizeof(T) == 4) {
        double r = __dmul_rn(wf, m2);
        r = __dsub_rn(r, __dmul_rn(wn, m1));
        r = __dadd_rn(r, __dmul_rn(wn, p1));
        r = __dsub_rn(r, __dmul_rn(wf, p2));
        return (double)(float)__dmul_rn(r, inv_dx);
    } else {
        // differences first: an FP64 operation less than the sum of four products
        return fma(wn * inv_dx, p1 - m1, -(wf * inv_dx) * (p2 - m2));
    }
}

// float -> double without the conversion unit: GB300 issues FP32 <-> FP64
// conversions at its FP64 rate (1/64 of FP32), and the FP64 per-cell pass
// converts every stencil tap. Normal numbers and zeros by integer operations
// (the same double the conversion gives), the rest by the conversion.
__device__ __forceinline__ double f2d_exact(float x)
{
    const unsigned u = __float_as_uint(x), e = (u >> 23) & 0xffu;
    const unsigned long long sgn = (unsigned long long)(u >> 31) << 63;
    if (e - 1u < 254u)
        return __longlong_as_double(
            (long long)(sgn | ((unsigned long long)(e + 896u) << 52) | ((unsigned long long)(u & 0x7fffffu) << 29)));
    if ((u << 1) == 0u) return __longlong_as_double((long long)sgn);
    return (double)x;
}

// a field value as double: FP32 widened by f2d_exact, FP64 as it is
template <typename T> __device__ __forceinline__ double widen(T x)
{
    if constexpr (sizeof(T) == 4)
        return f2d_exact(x);
    else
        return x;
}

// diff1_vals for FP32 fields from float taps: the same operations; r32 is the
// rounded float the reference squares, the return value its double.
__device__ __forceinline__ double diff1_f32(float m2, float m1, float p1, float p2, double inv_dx, float &r32)
{
    const double wf = 8.33333333333333333333e-2, wn = 6.66666666666666666667e-1;
    double r = __dmul_rn(wf, f2d_exact(m2));
    r = __dsub_rn(r, __dmul_rn(wn, f2d_exact(m1)));
    r = __dadd_rn(r, __dmul_rn(wn, f2d_exact(p1)));
    r = __dsub_rn(r, __dmul_rn(wf, f2d_exact(p2)));
    r32 = __double2float_rn(__dmul_rn(r, inv_dx));
    return f2d_exact(r32);
}

// The float that diff1_f32 rounds to, without FP64 operations (GB300 issues 2
// of them per SM and clock against 128 FP32 ones; the six diff1 values were a
// third of the pass). diff1 = K (8 (p1 - m1) + (m2 - p2)), K = 1/(12 dx), is
// formed as an unevaluated sum p + q of floats with Knuth's and Dekker's exact
// sums and products, to within bound = 2^-41 K (|m2| + |m1| + |p1| + |p2|) of
// what diff1_f32 has before its rounding: 2^-42 for the roundings of the low
// parts, 2^-46 for the double chain's own. Ziv's test: where p + q with the
// bound added and taken away rounds to the same float, that is diff1_f32's;
// otherwise (and near under- or overflow) the answer is false and diff1_f32
// has to be asked.
__device__ __forceinline__ bool diff1_pairs(float m2, float m1, float p1, float p2, float kh, float kl, float &r32)
{
    auto two_diff = [](float x, float y, float &e) {
        const float s = __fsub_rn(x, y), v = __fsub_rn(s, x);
        e = __fsub_rn(__fsub_rn(x, __fsub_rn(s, v)), __fadd_rn(y, v));
        return s;
    };
    float e1, e2;
    const float s1 = two_diff(p1, m1, e1), s2 = two_diff(m2, p2, e2);
    const float u = 8.f * s1, t = __fadd_rn(u, s2), v = __fsub_rn(t, u);
    const float e3 = __fadd_rn(__fsub_rn(u, __fsub_rn(t, v)), __fsub_rn(s2, v));
    const float lo = __fadd_rn(__fmaf_rn(8.f, e1, e2), e3);
    const float p = __fmul_rn(t, kh), pe = __fmaf_rn(t, kh, -p);
    const float q = __fmaf_rn(t, kl, __fmaf_rn(lo, kh, pe));
    const float r = __fadd_rn(p, q), rest = __fsub_rn(q, __fsub_rn(r, p));
    const float size = (fabsf(m2) + fabsf(m1) + fabsf(p1) + fabsf(p2)) * kh, bound = size * 0x1p-41f;
    r32 = r;
    return size > 1e-20f && size < 1e30f && __fadd_rn(r, __fadd_rn(rest, bound)) == r &&
           __fadd_rn(r, __fsub_rn(rest, bound)) == r;
}

// The seven per-cell energy terms (EnergyKernel.hpp:130-190) and the masking
// weight (Masking.hpp:75-93) from psi, Pi and the six diff1 values, in math
// type M: double as the reference computes them, or float for the
// per_cell_fp32 variant.
template <typename M> struct CellConst {
    M R2, inv_R, inv_R2, inv_R4, lambda, RpR, threshold;
};

__device__ __forceinline__ void cell_energy(const CellConst<float> &k, int scheme, float psi1, float psi2, float Pi1,
                                            float Pi2, const float (&g)[2][3], float (&term)[6], float &wgt)
{
    using M = float;
    const M psi_sq = psi1 * psi1 + psi2 * psi2;
    M g1sq = 0, g2sq = 0, cross2 = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        g1sq += g[0][d] * g[0][d];
        g2sq += g[1][d] * g[1][d];
        const M cr = psi1 * g[1][d] - psi2 * g[0][d];
        cross2 += cr * cr;
    }
    const M inv_psq = psi_sq > M(0) ? M(1) / psi_sq : M(0);
    const M gtsq = cross2 * inv_psq * inv_psq;
    const M c1 = Pi1 - k.RpR * psi1, c2 = Pi2 - k.RpR * psi2;
    const M dsq = psi_sq - k.R2;
    const M pot = M(0.25) * k.lambda * dsq * dsq;
    term[0] = (c1 * c1 + c2 * c2 + (g1sq + g2sq) + pot) * k.inv_R4;  // rho
    const M thp = (psi1 * Pi2 - Pi1 * psi2) * inv_psq;
    term[1] = thp * thp * k.inv_R2;                                  // 1/2 (sqrt(2) theta'/R)^2
    term[2] = gtsq * k.inv_R2;                                       // 1/2 sqrt(2)^2 |grad theta|^2 / R^2
    const M rdot = psi1 * c1 + psi2 * c2;
    term[3] = rdot * rdot * inv_psq * k.inv_R4;                      // radial kinetic
    term[4] = (g1sq + g2sq - psi_sq * gtsq) * k.inv_R4;              // radial gradient
    term[5] = pot * k.inv_R4;                                        // radial mass
    wgt = M(1);
    if (scheme != AXS_MASK_NONE) {
        const M mod = sqrt(psi_sq) * k.inv_R;
        if (scheme == AXS_MASK_B) {
            wgt = (mod >= k.threshold) ? M(1) : M(0);
        } else {
            const M f = M(1) + (mod - M(1)) * M(0.70710678118654752440);  // 1 + r / f_a
            wgt = f * f;
        }
    }
}

// The float version for two cells at once, to the same bits: the scalar one's roundings,
// with its sums of products fused as the compiler fuses them.
__device__ __forceinline__ F2 neg(F2 a) { return F2(-a.v.x, -a.v.y); }
__device__ __forceinline__ F2 diff1_pair(F2 m2, F2 p2, F2 p1, F2 m1, float inv_dx)
{
    const float wf = 0.0833333333f, wn = 0.666666667f;
    return fma(F2(wf), m2 - p2, F2(wn) * (p1 - m1)) * F2(inv_dx);
}
__device__ __forceinline__ void cell_energy(const CellConst<float> &k, int scheme, F2 psi1, F2 psi2, F2 Pi1, F2 Pi2,
                                            const F2 (&g)[2][3], F2 (&term)[6], F2 &wgt)
{
    const F2 psi_sq = fma(psi1, psi1, psi2 * psi2);
    F2 g1sq = g[0][0] * g[0][0], g2sq = g[1][0] * g[1][0], cross2;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        if (d) {
            g1sq = fma(g[0][d], g[0][d], g1sq);
            g2sq = fma(g[1][d], g[1][d], g2sq);
        }
        const F2 cr = fma(psi1, g[1][d], neg(psi2 * g[0][d]));
        cross2 = d ? fma(cr, cr, cross2) : cr * cr;
    }
    const F2 inv_psq(psi_sq.v.x > 0.f ? 1.f / psi_sq.v.x : 0.f, psi_sq.v.y > 0.f ? 1.f / psi_sq.v.y : 0.f);
    const F2 gtsq = (cross2 * inv_psq) * inv_psq;
    const F2 c1 = fma(F2(-k.RpR), psi1, Pi1), c2 = fma(F2(-k.RpR), psi2, Pi2);
    const F2 dsq = psi_sq - F2(k.R2);
    const F2 pot = (F2(0.25f * k.lambda) * dsq) * dsq;
    const F2 gsq = g1sq + g2sq;
    term[0] = ((fma(c1, c1, c2 * c2) + gsq) + pot) * F2(k.inv_R4);
    const F2 thp = fma(psi1, Pi2, neg(Pi1 * psi2)) * inv_psq;
    term[1] = (thp * thp) * F2(k.inv_R2);
    term[2] = gtsq * F2(k.inv_R2);
    const F2 rdot = fma(psi1, c1, psi2 * c2);
    term[3] = ((rdot * rdot) * inv_psq) * F2(k.inv_R4);
    term[4] = fma(neg(psi_sq), gtsq, gsq) * F2(k.inv_R4);
    term[5] = pot * F2(k.inv_R4);
    wgt = F2(1.f);
    if (scheme != AXS_MASK_NONE) {
        const F2 mod = F2(sqrtf(psi_sq.v.x), sqrtf(psi_sq.v.y)) * F2(k.inv_R);
        if (scheme == AXS_MASK_B) {
            wgt = F2(mod.v.x >= k.threshold ? 1.f : 0.f, mod.v.y >= k.threshold ? 1.f : 0.f);
        } else {
            const F2 f = fma(mod + F2(-1.f), F2(0.70710678118654752440f), F2(1.f));
            wgt = f * f;
        }
    }
}

// In double, from the diff1 values g and the same in the field precision, gt
// (the reference squares them there). RAW: without the powers of 1/R, which the
// caller puts on the sums (six FP64 operations a cell).
template <typename T, bool RAW>
__device__ __forceinline__ void cell_energy(const CellConst<double> &k, int scheme, double psi1, double psi2,
                                            double Pi1, double Pi2, const double (&g)[2][3], const T (&gt)[2][3],
                                            double (&term)[6], double &wgt)
{
    const double psi_sq = psi1 * psi1 + psi2 * psi2;
    auto square = [&](int c, int d) -> double {
        // the reference squares the float diff1 values in float
        if constexpr (sizeof(T) == 4)
            return f2d_exact(gt[c][d] * gt[c][d]);
        else
            return gt[c][d] * gt[c][d];
    };
    auto cross = [&](int d) { return psi1 * g[1][d] - psi2 * g[0][d]; };
    const double g1sq = square(0, 0) + square(0, 1) + square(0, 2), g2sq = square(1, 0) + square(1, 1) + square(1, 2);
    const double cr0 = cross(0), cr1 = cross(1), cr2 = cross(2);
    const double inv_psq = positive(psi_sq) ? recip_pos(psi_sq) : 0.0;
    const double gtsq_psq = (cr0 * cr0 + cr1 * cr1 + cr2 * cr2) * inv_psq, gtsq = gtsq_psq * inv_psq;
    const double c1 = Pi1 - k.RpR * psi1, c2 = Pi2 - k.RpR * psi2;
    const double dsq = psi_sq - k.R2;
    const double pot = 0.25 * k.lambda * dsq * dsq;
    const double s4 = RAW ? 1.0 : k.inv_R4, s2 = RAW ? 1.0 : k.inv_R2;
    term[0] = (c1 * c1 + c2 * c2 + (g1sq + g2sq) + pot) * s4;  // rho
    const double thp = (psi1 * Pi2 - Pi1 * psi2) * inv_psq;
    term[1] = thp * thp * s2;                                  // 1/2 (sqrt(2) theta'/R)^2
    term[2] = gtsq * s2;                                       // 1/2 sqrt(2)^2 |grad theta|^2 / R^2
    const double rdot = psi1 * c1 + psi2 * c2;
    term[3] = rdot * rdot * inv_psq * s4;                      // radial kinetic
    term[4] = (g1sq + g2sq - gtsq_psq) * s4;                   // radial gradient
    term[5] = pot * s4;                                        // radial mass
    wgt = 1.0;
    if (scheme == AXS_MASK_B) {
        wgt = root_reaches(psi_sq, k.inv_R, k.threshold) ? 1.0 : 0.0;
    } else if (scheme != AXS_MASK_NONE) {
        // 1 + r / f_a, r = |psi| / R - 1
        const double f = (1.0 - 0.70710678118654752440) + sqrt_pos(psi_sq) * (k.inv_R * 0.70710678118654752440);
        wgt = f * f;
    }
}

// Tiled diagnostics pass. A block owns a DTX x DTY tile of cells and marches
// in z over a chunk. Shared memory holds psi1/psi2 of six planes (tile plus a
// 2-cell halo: the five of the gradient stencil and one in flight), Pi1/Pi2 of
// three vertex planes ((DTX+1) x (DTY+1) vertices: z, z+1 and one in flight),
// and for the two vertex planes z and z+1 the single-precision phases (and with
// FP32 per-cell terms gamma^2 v^2), each computed once per vertex. Planes arrive by element-wise
// cp.async one plane ahead of their use, so their latency overlaps the
// current plane's work. Plane loads use element offsets precomputed per work
// item, so the march needs no index division.
constexpr int DTX = 32, DTY = 8, DHX = DTX + 4, DHY = DTY + 4, DVX = DTX + 1, DVY = DTY + 1;
static_assert(DTX * DTY == kDiagThreads, "one cell per thread");
constexpr int kPsiPts = DHX * DHY, kVtxPts = DVX * DVY;
constexpr int kPsiPer = (2 * kPsiPts + kDiagThreads - 1) / kDiagThreads;  // psi loads per thread per plane
constexpr int kPiPer = (2 * kVtxPts + kDiagThreads - 1) / kDiagThreads;   // Pi loads per thread per plane
constexpr int kVtxPer = (kVtxPts + kDiagThreads - 1) / kDiagThreads;      // vertices per thread per plane

// Ring depths for one block barrier per plane: a plane's loads are issued
// before that barrier, so a slot may be refilled only once every thread is
// past the plane that last read it (psi: the 5-plane stencil plus two;
// Pi: read at its vertex plane and again at its cell plane, plus two).
// Vertex planes are computed one plane ahead into a third slot.
// With FP64 per-cell terms the pass is bound by the FP64 pipe (75 % busy with
// about 86 operations a cell; 160 with the diff1 chains, gamma^2 v^2 at every
// vertex, library division and root, and the powers of 1/R in every cell):
// 256^3 on FP32 fields 5.36 -> 2.9 ms.
constexpr int kPsiSlots = 7, kPiSlots = 5, kVtxSlots = 3;
// pierced plaquettes buffered per block; flushed to the global list with one
// atomic once a plane could overflow it (at most 3 entries per cell)
constexpr int kListBuf = 1536, kListFlushAt = kListBuf - 3 * kDiagThreads;
constexpr int kVelQueue = 7 + 3 * 32;  // fewer than 8 left over, and a plane's
template <typename T, bool FAST> struct DiagSmem {
    long long lbuf[kListBuf];
    T ps[kPsiSlots][2][DHY][DHX];
    T pi[kPiSlots][2][DVY][DVX];
    // FAST: gamma^2 v^2 of the vertices; else the pierced plaquettes whose corners'
    // values a warp still has to add up (vel_corners)
    typename std::conditional<FAST, float[kVtxSlots][DVY][DVX], unsigned[kDiagThreads / 32][kVelQueue]>::type gv;
    float th[kVtxSlots][DVY][DVX];
    float tie_value[kDiagThreads / 32][6 * 32];  // of a warp's undecided diff1 values: the float, and which they are
    unsigned char tie[kDiagThreads / 32][6 * 32];
    unsigned char ok[kVtxSlots][DVY][DVX];
};

__device__ __forceinline__ int wrap_or_self(int i, int n, int wrap) { return wrap ? (i % n + n) % n : i; }

template <typename T, bool FAST>
__global__ void __launch_bounds__(kDiagThreads, 2) diag_kernel(const DiagView v, const DiagConst q,
                                                               const uint8_t *__restrict__ mask,
                                                               DiagPartial *__restrict__ partials,
                                                               unsigned long long *__restrict__ list_counter,
                                                               long long *__restrict__ list, long long capacity,
                                                               int tiles_x, int ntiles, int zchunk, long long n_items,
                                                               long long items_per_box, int64_t box_stride,
                                                               uint8_t *__restrict__ tags)
{
    extern __shared__ __align__(16) unsigned char diag_smem_raw[];
    DiagSmem<T, FAST> &sm = *reinterpret_cast<DiagSmem<T, FAST> *>(diag_smem_raw);
    __shared__ int lcount, flush_n;
    __shared__ unsigned long long flush_base;
    const int64_t box_cells = (int64_t)v.nx * v.ny * v.nz;

    double e[14];
#pragma unroll
    for (int s = 0; s < 14; ++s) e[s] = 0.0;
    // per_cell_fp32: one work item's cells are summed in float, then added to e
    // with compensation (Neumaier) for the 13 real-valued sums; the cell count is exact
    float ef[FAST ? 14 : 1], ec[FAST ? 13 : 1];
#pragma unroll
    for (int s = 0; s < (FAST ? 14 : 1); ++s) ef[s] = 0.f;
#pragma unroll
    for (int s = 0; s < (FAST ? 13 : 1); ++s) ec[s] = 0.f;
    auto csum = [](float &sum, float &comp, float x) {
        const float t = sum + x;
        comp += fabsf(sum) >= fabsf(x) ? (sum - t) + x : (x - t) + sum;
        sum = t;
    };
    const CellConst<double> kd{q.R2, q.inv_R, q.inv_R2, q.inv_R4, q.lambda, q.RpR, q.threshold};
    const CellConst<float> kf{q.f_R2, q.f_inv_R, q.f_inv_R2, q.f_inv_R4, q.f_lambda, q.f_RpR, q.f_threshold};
    double vsum = 0.0;
    long long cnt[4] = {0, 0, 0, 0};

    const int tid = threadIdx.x;
    const int lx = tid % DTX, ly = tid / DTX;
    if (tid == 0) lcount = 0;
    int warp_end = 0;  // end of this warp's last append to lbuf (lane-uniform)
    // move the buffered pierced plaquettes to the global list (called by the whole block)
    auto flush = [&]() {
        if (tid == 0) {
            const int nb = lcount;
            flush_n = nb;
            flush_base = nb ? atomicAdd(list_counter, (unsigned long long)nb) : 0ull;
            lcount = 0;
        }
        __syncthreads();
        const int nb = flush_n;
        const unsigned long long b0 = flush_base;
        for (int i = tid; i < nb; i += kDiagThreads)
            if (b0 + i < (unsigned long long)capacity) list[b0 + i] = sm.lbuf[i];
        __syncthreads();
        warp_end = 0;
    };

    int vq_n = 0;  // entries of this warp's plaquette queue (lane-uniform)
    int n_cells = 0;

    for (long long item = blockIdx.x; item < n_items; item += gridDim.x) {
        // boxes of one batch share the view's geometry and sit box_stride apart
        const long long qbox = item / items_per_box, box_item = item % items_per_box;
        const T *__restrict__ base = static_cast<const T *>(v.data) + qbox * box_stride;
        const int tile = (int)(box_item % ntiles);
        const int chunk = (int)(box_item / ntiles);
        const int x0 = (tile % tiles_x) * DTX, y0 = (tile / tiles_x) * DTY;
        const int za = chunk * zchunk, len = min(zchunk, v.nz - za);

        // ---- per-item load plan: in-plane element offsets (wrapped or ghost) ----
        int64_t psi_off[kPsiPer];  // component + in-plane element offset
        bool psi_ok[kPsiPer];
#pragma unroll
        for (int u = 0; u < kPsiPer; ++u) {
            const int idx = tid + u * kDiagThreads;
            const int c = idx / kPsiPts, r = idx % kPsiPts;
            const int xx = x0 - 2 + r % DHX, yy = y0 - 2 + r / DHX;
            psi_ok[u] = idx < 2 * kPsiPts && xx < v.nx + 2 && yy < v.ny + 2 && (v.wx || (xx >= -v.ox && xx < v.nx + v.ox)) &&
                        (v.wy || (yy >= -v.oy && yy < v.ny + v.oy));
            psi_off[u] = c * v.cs + (int64_t)(wrap_or_self(xx, v.nx, v.wx) + v.ox) +
                         (int64_t)(wrap_or_self(yy, v.ny, v.wy) + v.oy) * v.js;
        }
        int64_t pi_off[kPiPer];
        bool pi_ok[kPiPer];
#pragma unroll
        for (int u = 0; u < kPiPer; ++u) {
            const int idx = tid + u * kDiagThreads;
            const int c = idx / kVtxPts, r = idx % kVtxPts;
            const int xx = x0 + r % DVX, yy = y0 + r / DVX;
            pi_ok[u] = idx < 2 * kVtxPts && xx <= v.nx && yy <= v.ny && (v.wx || xx < v.nx + v.ox) &&
                       (v.wy || yy < v.ny + v.oy);
            pi_off[u] = (2 + c) * v.cs + (int64_t)(wrap_or_self(xx, v.nx, v.wx) + v.ox) +
                        (int64_t)(wrap_or_self(yy, v.ny, v.wy) + v.oy) * v.js;
        }
        auto plane_off = [&](int z, bool &zin) -> int64_t {
            zin = v.wz || (z >= -v.oz && z < v.nz + v.oz);
            return (int64_t)(wrap_or_self(z, v.nz, v.wz) + v.oz) * v.ks;
        };
        // psi of plane z (za - 2 <= z <= za + len + 1) sits in slot (z - za + 2) mod
        // kPsiSlots, Pi of vertex plane z (za <= z <= za + len) in slot (z - za) mod kPiSlots
        auto psi_slot = [&](int z) { return (z - za + 2) % kPsiSlots; };
        auto load_psi = [&](int z) {
            bool zin;
            const int64_t po = plane_off(z, zin);
            T *dst = &sm.ps[psi_slot(z)][0][0][0];
#pragma unroll
            for (int u = 0; u < kPsiPer; ++u) {
                const int idx = tid + u * kDiagThreads;
                if (idx < 2 * kPsiPts) cp_async_elem(dst + idx, base + psi_off[u] + po, zin && psi_ok[u], base);
            }
        };
        auto load_pi = [&](int z) {
            if (!q.want_energy && !(FAST && q.want_vel)) return;  // the string finder alone reads psi only
            bool zin;
            const int64_t po = plane_off(z, zin);
            T *pdst = &sm.pi[(z - za) % kPiSlots][0][0][0];
#pragma unroll
            for (int u = 0; u < kPiPer; ++u) {
                const int idx = tid + u * kDiagThreads;
                if (idx < 2 * kVtxPts) cp_async_elem(pdst + idx, base + pi_off[u] + po, zin && pi_ok[u], base);
            }
        };
        // vertex plane z: phases and gamma^2 v^2 from psi and Pi already in shared memory
        auto vertex_plane = [&](int z) {
            const int ts = (z - za) % kVtxSlots;
            const int ps_ = (z - za) % kPiSlots;
            const int slot = psi_slot(z);
#pragma unroll
            for (int u = 0; u < kVtxPer; ++u) {
                const int idx = tid + u * kDiagThreads;
                if (idx >= kVtxPts) break;
                const int vy = idx / DVX, vx = idx % DVX;
                const T a = sm.ps[slot][0][vy + 2][vx + 2], b = sm.ps[slot][1][vy + 2][vx + 2];
                // float conversion keeps the angle to ~1e-7 only away from under/overflow
                if constexpr (sizeof(T) == 4) {
                    const float m = fmaxf(fabsf(a), fabsf(b));
                    sm.ok[ts][vy][vx] = (m > 1e-30f && m < 1e30f) ? 1 : 0;
                } else {
                    const double m = fmax(fabs(a), fabs(b));
                    sm.ok[ts][vy][vx] = (m > 1e-30 && m < 1e30) ? 1 : 0;
                }
                sm.th[ts][vy][vx] = atan2f((float)b, (float)a);
                if constexpr (FAST) {
                    if (!q.want_vel) continue;
                    const float psi1 = a, psi2 = b, Pi1 = sm.pi[ps_][0][vy][vx], Pi2 = sm.pi[ps_][1][vy][vx];
                    const float phi1 = psi1 * q.f_inv_R, phi2 = psi2 * q.f_inv_R;
                    const float pd1 = (Pi1 - q.f_RpR * psi1) * q.f_inv_R2, pd2 = (Pi2 - q.f_RpR * psi2) * q.f_inv_R2;
                    const float phi_sq = phi1 * phi1 + phi2 * phi2;
                    const float pd_sq = pd1 * pd1 + pd2 * pd2;
                    const float re = phi1 * pd1 + phi2 * pd2;
                    sm.gv[ts][vy][vx] = pd_sq * q.f_vel_a * (1.f - q.f_vel_b * phi_sq) - q.f_vel_c * re * re;
                }
            }
        };

        // gamma^2 v^2 (Velocity.hpp:62-78, the constant prefactors folded on the host)
        // of the corners of `take` queued plaquettes of this warp, a corner to a lane,
        // from global memory: 17 FP64 operations for eight plaquettes instead of for
        // every vertex of the grid (an eighth of the pass). Entries: plane in the
        // chunk, orientation, lane of the cell (a warp is a row of cells).
        auto vel_corners = [&](int take) {
            if constexpr (!FAST) {
                __syncwarp();
                vq_n -= take;
                const int k = (tid & 31) >> 2, j = tid & 3;
                if (k < take) {
                    const unsigned en = sm.gv[tid >> 5][vq_n + k];
                    const int pl = (en >> 5) & 3;
                    const int mid = j == 1 || j == 2, far = j >= 2;
                    int x = x0 + (int)(en & 31) + (pl == 0 ? mid : pl == 2 ? far : 0);
                    int y = y0 + ly + (pl == 0 ? far : pl == 1 ? mid : 0);
                    int z = za + (int)(en >> 7) + (pl == 1 ? far : pl == 2 ? mid : 0);
                    const bool on = (v.wx || x < v.nx + v.ox) && (v.wy || y < v.ny + v.oy) && (v.wz || z < v.nz + v.oz);
                    if (v.wx && x == v.nx) x = 0;
                    if (v.wy && y == v.ny) y = 0;
                    if (v.wz && z == v.nz) z = 0;
                    const T *at = base + (x + v.ox) + (int64_t)(y + v.oy) * v.js + (int64_t)(z + v.oz) * v.ks;
                    auto val = [&](int c) { return on ? widen(at[c * v.cs]) : 0.0; };
                    const double psi1 = val(0), psi2 = val(1), Pi1 = val(2), Pi2 = val(3);
                    const double phi1 = psi1 * q.inv_R, phi2 = psi2 * q.inv_R;
                    const double pd1 = (Pi1 - q.RpR * psi1) * q.inv_R2, pd2 = (Pi2 - q.RpR * psi2) * q.inv_R2;
                    const double phi_sq = phi1 * phi1 + phi2 * phi2;
                    const double pd_sq = pd1 * pd1 + pd2 * pd2;
                    const double re = phi1 * pd1 + phi2 * pd2;
                    vsum += pd_sq * q.vel_a * (1.0 - q.vel_b * phi_sq) - q.vel_c * re * re;
                }
                __syncwarp();
            }
        };

        // prologue: psi of za-2 .. za+2 and Pi of za .. za+2 (one group), then the
        // first two vertex planes. Vertex planes run za .. za+len, psi planes
        // za-2 .. za+len+1.
        for (int p = -2; p <= 2; ++p) load_psi(za + p);
        load_pi(za);
        load_pi(za + 1);
        if (len >= 2) load_pi(za + 2);
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        vertex_plane(za);
        vertex_plane(za + 1);

        for (int m = 0; m < len; ++m) {
            const int z = za + m;
            // one plane ahead: psi(z + 3) for the next plane's stencil and vertex
            // plane, Pi(z + 3) for its vertex plane. Their slots were last read
            // two planes back, before the previous plane's barrier.
            if (m + 1 < len) load_psi(z + 3);
            if (m + 3 <= len) load_pi(z + 3);
            cp_async_commit();
            cp_async_wait<1>();  // everything but this plane's group: psi(z + 2), Pi(z + 2)
            // the plane's one barrier: its psi / Pi and vertex planes z, z + 1 are
            // visible, every thread is done with plane z - 1, and the block learns
            // whether the pierced buffer could overflow during this plane
            if (__syncthreads_or(warp_end > kListFlushAt)) flush();
            // vertex plane z + 2 for the next plane, into the slot plane z - 1 read
            if (m + 2 <= len) vertex_plane(z + 2);

            const int x = x0 + lx, y = y0 + ly;
            const int64_t cell = qbox * box_cells + (int64_t)x + (int64_t)v.nx * ((int64_t)y + (int64_t)v.ny * z);
            const bool in = x < v.nx && y < v.ny && (mask == nullptr || mask[cell] != 0);
            int w[3] = {0, 0, 0};
            const int s0 = (m + 2) % kPsiSlots;
            const int sm1 = (m + 1) % kPsiSlots, sp1 = (m + 3) % kPsiSlots, sm2 = m % kPsiSlots,
                      sp2 = (m + 4) % kPsiSlots;
            const int hx = lx + 2, hy = ly + 2;
            // the four taps of diff1 of component c along axis d at the cell of lane l
            auto taps = [&](int c, int d, int l, float (&f)[4]) {
                const T(*pl)[DHX] = sm.ps[s0][c];
                const int x_ = l + 2;
                f[0] = d == 0 ? pl[hy][x_ - 2] : d == 1 ? pl[hy - 2][x_] : sm.ps[sm2][c][hy][x_];
                f[1] = d == 0 ? pl[hy][x_ - 1] : d == 1 ? pl[hy - 1][x_] : sm.ps[sm1][c][hy][x_];
                f[2] = d == 0 ? pl[hy][x_ + 1] : d == 1 ? pl[hy + 1][x_] : sm.ps[sp1][c][hy][x_];
                f[3] = d == 0 ? pl[hy][x_ + 2] : d == 1 ? pl[hy + 2][x_] : sm.ps[sp2][c][hy][x_];
            };
            float gf[2][3] = {};
            if constexpr (sizeof(T) == 4 && !FAST) {
                if (q.want_energy) {
                    // Exact ties are common (at dx = 1/2 the sum of taps is divided by 6, and
                    // the double chain's own roundings decide them): the warp's undecided
                    // values, a few per cent, go through the FP64 chain together, a value to a lane.
                    int n = 0;
                    unsigned undecided = 0;
#pragma unroll
                    for (int cd = 0; cd < 6; ++cd) {
                        float f[4];
                        taps(cd / 3, cd % 3, lx, f);
                        const bool sure = diff1_pairs(f[0], f[1], f[2], f[3], q.f_k12h, q.f_k12l, gf[cd / 3][cd % 3]) || !in;
                        const unsigned who = __ballot_sync(0xffffffffu, !sure);
                        if (!sure) {
                            sm.tie[ly][n + __popc(who & ((1u << lx) - 1u))] = (unsigned char)(cd * 32 + lx);
                            undecided |= 1u << cd;
                        }
                        n += __popc(who);
                    }
                    if (n > 0) {
                        __syncwarp();
                        for (int k = lx; k < n; k += 32) {
                            const int en = sm.tie[ly][k], cd = en >> 5;
                            float f[4], r;
                            taps(cd / 3, cd % 3, en & 31, f);
                            diff1_f32(f[0], f[1], f[2], f[3], q.one_over_dx, r);
                            sm.tie_value[ly][en] = r;
                        }
                        __syncwarp();
#pragma unroll
                        for (int cd = 0; cd < 6; ++cd)
                            if (undecided >> cd & 1u) gf[cd / 3][cd % 3] = sm.tie_value[ly][cd * 32 + lx];
                    }
                }
            }
            if (in) {
                const int t0 = m % kVtxSlots, t1 = (m + 1) % kVtxSlots, tp = m % kPiSlots;
                if (q.want_energy) {
                    const T p1 = sm.ps[s0][0][hy][hx], p2 = sm.ps[s0][1][hy][hx];
                    const T q1 = sm.pi[tp][0][ly][lx], q2 = sm.pi[tp][1][ly][lx];
                    bool done = false;
                    if constexpr (FAST) {
                        const float psq = p1 * p1 + p2 * p2;
                        // float keeps 1/|psi|^4 finite only away from the cores' exact zeros
                        if (psq > 1e-15f && psq < 1e15f) {
                            float g[2][3];
                            const float wf = 0.0833333333f, wn = 0.666666667f;
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                g[c][0] = (wf * (sm.ps[s0][c][hy][hx - 2] - sm.ps[s0][c][hy][hx + 2]) +
                                           wn * (sm.ps[s0][c][hy][hx + 1] - sm.ps[s0][c][hy][hx - 1])) * q.f_one_over_dx;
                                g[c][1] = (wf * (sm.ps[s0][c][hy - 2][hx] - sm.ps[s0][c][hy + 2][hx]) +
                                           wn * (sm.ps[s0][c][hy + 1][hx] - sm.ps[s0][c][hy - 1][hx])) * q.f_one_over_dx;
                                g[c][2] = (wf * (sm.ps[sm2][c][hy][hx] - sm.ps[sp2][c][hy][hx]) +
                                           wn * (sm.ps[sp1][c][hy][hx] - sm.ps[sm1][c][hy][hx])) * q.f_one_over_dx;
                            }
                            float term[6], wgt;
                            cell_energy(kf, q.scheme, p1, p2, q1, q2, g, term, wgt);
#pragma unroll
                            for (int k = 0; k < 6; ++k) {
                                csum(ef[2 * k], ec[2 * k], term[k]);
                                csum(ef[2 * k + 1], ec[2 * k + 1], term[k] * wgt);
                            }
                            csum(ef[12], ec[12], wgt);
                            ef[13] += 1.f;
                            done = true;
                        }
                    }
                    if (!done) {
                        double g[2][3], term[6], wgt;
                        if constexpr (sizeof(T) == 4) {
                            // FP32 fields: taps widened by integer operations (f2d_exact)
                            if constexpr (FAST) {
#pragma unroll
                                for (int c = 0; c < 2; ++c)
#pragma unroll
                                    for (int d = 0; d < 3; ++d) {
                                        float f[4];
                                        taps(c, d, lx, f);
                                        diff1_f32(f[0], f[1], f[2], f[3], q.one_over_dx, gf[c][d]);
                                    }
                            }
#pragma unroll
                            for (int c = 0; c < 2; ++c)
#pragma unroll
                                for (int d = 0; d < 3; ++d) g[c][d] = f2d_exact(gf[c][d]);
                            cell_energy<float, !FAST>(kd, q.scheme, f2d_exact(p1), f2d_exact(p2), f2d_exact(q1),
                                                         f2d_exact(q2), g, gf, term, wgt);
                        } else {
#pragma unroll
                            for (int c = 0; c < 2; ++c) {
                                g[c][0] = diff1_vals<T>(sm.ps[s0][c][hy][hx - 2], sm.ps[s0][c][hy][hx - 1],
                                                        sm.ps[s0][c][hy][hx + 1], sm.ps[s0][c][hy][hx + 2],
                                                        q.one_over_dx);
                                g[c][1] = diff1_vals<T>(sm.ps[s0][c][hy - 2][hx], sm.ps[s0][c][hy - 1][hx],
                                                        sm.ps[s0][c][hy + 1][hx], sm.ps[s0][c][hy + 2][hx],
                                                        q.one_over_dx);
                                g[c][2] = diff1_vals<T>(sm.ps[sm2][c][hy][hx], sm.ps[sm1][c][hy][hx],
                                                        sm.ps[sp1][c][hy][hx], sm.ps[sp2][c][hy][hx], q.one_over_dx);
                            }
                            cell_energy<T, !FAST>(kd, q.scheme, p1, p2, q1, q2, g, g, term, wgt);
                        }
#pragma unroll
                        for (int k = 0; k < 6; ++k) {
                            e[2 * k] += term[k];
                            e[2 * k + 1] += term[k] * wgt;
                        }
                        e[12] += wgt;
                        ++n_cells;
                    }
                }
                if (q.want_plaq || q.want_vel) {
                    // corner phases (x, y, z offsets) in the reference's order
                    const float f000 = sm.th[t0][ly][lx], f100 = sm.th[t0][ly][lx + 1];
                    const float f110 = sm.th[t0][ly + 1][lx + 1], f010 = sm.th[t0][ly + 1][lx];
                    const float f001 = sm.th[t1][ly][lx], f101 = sm.th[t1][ly][lx + 1], f011 = sm.th[t1][ly + 1][lx];
                    const bool ok = sm.ok[t0][ly][lx] & sm.ok[t0][ly][lx + 1] & sm.ok[t0][ly + 1][lx + 1] &
                                    sm.ok[t0][ly + 1][lx] & sm.ok[t1][ly][lx] & sm.ok[t1][ly][lx + 1] &
                                    sm.ok[t1][ly + 1][lx];
                    bool fast = ok;
                    if (fast) fast = winding4_fast(f000, f100, f110, f010, w[0]);
                    if (fast) fast = winding4_fast(f000, f010, f011, f001, w[1]);
                    if (fast) fast = winding4_fast(f000, f001, f101, f100, w[2]);
                    if (!fast) {
                        // near the branch cut or outside the float range: the reference's
                        // double arithmetic for this cell's three plaquettes
                        auto dph = [&](int slot, int ox_, int oy_) {
                            return atan2((double)sm.ps[slot][1][hy + oy_][hx + ox_],
                                         (double)sm.ps[slot][0][hy + oy_][hx + ox_]);
                        };
                        const double d000 = dph(s0, 0, 0), d100 = dph(s0, 1, 0), d110 = dph(s0, 1, 1);
                        const double d010 = dph(s0, 0, 1), d001 = dph(sp1, 0, 0), d101 = dph(sp1, 1, 0);
                        const double d011 = dph(sp1, 0, 1);
                        int ties = 0;
                        w[0] = winding4(d000, d100, d110, d010, ties);
                        w[1] = winding4(d000, d010, d011, d001, ties);
                        w[2] = winding4(d000, d001, d101, d100, ties);
                        cnt[3] += ties;
                    }
                    // StringTagger (StringTagger.hpp:117-151): a cell is tagged when a
                    // plaquette at its low corner is pierced
                    if (tags != nullptr) tags[cell] = (w[0] | w[1] | w[2]) != 0;
                    cnt[0] += (w[0] != 0) + (w[1] != 0) + (w[2] != 0);
                    cnt[1] += abs(w[0]) + abs(w[1]) + abs(w[2]);
                    if constexpr (FAST) {
                        if (q.want_vel && (w[0] | w[1] | w[2])) {
                            const double g000 = sm.gv[t0][ly][lx], g100 = sm.gv[t0][ly][lx + 1];
                            const double g110 = sm.gv[t0][ly + 1][lx + 1], g010 = sm.gv[t0][ly + 1][lx];
                            const double g001 = sm.gv[t1][ly][lx], g101 = sm.gv[t1][ly][lx + 1];
                            const double g011 = sm.gv[t1][ly + 1][lx];
                            double s = 0.0;
                            long long c = 0;
                            if (w[0]) { s += g000 + g100 + g110 + g010; c += 4; }
                            if (w[1]) { s += g000 + g010 + g011 + g001; c += 4; }
                            if (w[2]) { s += g000 + g001 + g101 + g100; c += 4; }
                            vsum += s;
                            cnt[2] += c;
                        }
                    } else {
                        if (q.want_vel) cnt[2] += 4 * ((w[0] != 0) + (w[1] != 0) + (w[2] != 0));
                    }
                }
            }
            if constexpr (!FAST) {
                if (q.want_vel && __any_sync(0xffffffffu, (w[0] | w[1] | w[2]) != 0)) {
#pragma unroll
                    for (int pl = 0; pl < 3; ++pl) {
                        const unsigned hit = __ballot_sync(0xffffffffu, w[pl] != 0);
                        if (w[pl])
                            sm.gv[tid >> 5][vq_n + __popc(hit & ((1u << lx) - 1u))] = (unsigned)m << 7 | pl << 5 | lx;
                        vq_n += __popc(hit);
                    }
                    while (vq_n >= 8) vel_corners(8);
                }
            }
            // ---- pierced plaquettes of this plane into the block's buffer: a warp
            // scan and one shared-memory atomic per warp that has any ----
            if (q.want_plaq && list != nullptr) {
                const int mine = (w[0] != 0) + (w[1] != 0) + (w[2] != 0);
                if (__any_sync(0xffffffffu, mine != 0)) {
                    const int lane = tid & 31;
                    int incl = mine;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int yv = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= o) incl += yv;
                    }
                    const int wtot = __shfl_sync(0xffffffffu, incl, 31);
                    int wbase = 0;
                    if (lane == 31) wbase = atomicAdd(&lcount, wtot);
                    wbase = __shfl_sync(0xffffffffu, wbase, 31);
                    warp_end = wbase + wtot;
                    int pos = wbase + incl - mine;
                    for (int pl = 0; pl < 3; ++pl)
                        if (w[pl]) sm.lbuf[pos++] = 4LL * cell + pl;
                }
            }
        }
        if (vq_n > 0) vel_corners(vq_n);
        __syncthreads();  // the next item's prologue refills the rings
        if constexpr (FAST) {
#pragma unroll
            for (int k = 0; k < 14; ++k) {
                e[k] += (double)ef[k] + (k < 13 ? (double)ec[k < 13 ? k : 0] : 0.0);
                ef[k] = 0.f;
                if (k < 13) ec[k] = 0.f;
            }
        }
    }
    // the rest of the buffer (warp_end > 0: the warp appended since the last flush)
    if (q.want_plaq && list != nullptr && __syncthreads_or(warp_end > 0)) flush();

    if constexpr (!FAST) {  // the terms' powers of 1/R
#pragma unroll
        for (int s = 0; s < 12; ++s) e[s] *= s >= 2 && s < 6 ? kd.inv_R2 : kd.inv_R4;
    }
    e[13] += (double)n_cells;
    // ---- block reduction (fixed order) ----
    __shared__ double red_d[kDiagThreads / 32][15];
    __shared__ long long red_l[kDiagThreads / 32][4];
    const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int s = 0; s < 14; ++s) {
        double xv = e[s];
        for (int o = 16; o > 0; o >>= 1) xv += __shfl_down_sync(0xffffffffu, xv, o);
        if (lane == 0) red_d[warp][s] = xv;
    }
    {
        double xv = vsum;
        for (int o = 16; o > 0; o >>= 1) xv += __shfl_down_sync(0xffffffffu, xv, o);
        if (lane == 0) red_d[warp][14] = xv;
    }
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        long long xv = cnt[s];
        for (int o = 16; o > 0; o >>= 1) xv += __shfl_down_sync(0xffffffffu, xv, o);
        if (lane == 0) red_l[warp][s] = xv;
    }
    __syncthreads();
    if (tid < 15) {
        double xv = 0.0;
        for (int ww = 0; ww < kDiagThreads / 32; ++ww) xv += red_d[ww][tid];
        if (tid < 14)
            partials[blockIdx.x].e[tid] = xv;
        else
            partials[blockIdx.x].vsum = xv;
    } else if (tid >= 32 && tid < 36) {
        long long xv = 0;
        for (int ww = 0; ww < kDiagThreads / 32; ++ww) xv += red_l[ww][tid - 32];
        partials[blockIdx.x].cnt[tid - 32] = xv;
    }
}

// ---------------------------------------------------------------- string finder
// The string finder and the tagger's plaquette criterion (no energy). A warp owns
// a strip of kStripW cells in x by kStripRows in y and marches in z: lane l holds
// the kStripRows + 1 vertices of column x0 + l in registers, the plane before too
// and the plane after in flight, so there is no shared memory and no barrier in
// the march. Only two things are asked of an edge a -> b:
//   - does the short way round cross the negative real axis (the phase difference
//     folds)? With the vertices' imaginary parts of opposite sign (the sign bit: a
//     +-0 belongs to its side, as atan2 has it) it does exactly where cross(a, b) =
//     a1 b2 - a2 b1 has a's sign bit. There the two products have one sign, or a
//     and b lie within the next test's angle, so the sign is exact, underflow included;
//   - is it within 1e-5 of antiparallel, |cross| + 1e-5 dot < 0? Then the lane's
//     cells of that plane take the exact path, as with a vertex outside float range
//     or not a number: per cell the folds of float phases, or, with an edge within
//     1e-5 of +-pi, the reference's double arithmetic.
// The four reduced differences of a plaquette stay below pi each, so its winding is
// -1, 0 or 1, and it is pierced where an odd number of its edges fold: the folds
// are bits, row r of the strip in bit r, and the three plaquettes of eight cells
// come from a few XORs and one shuffle. Columns with pierced cells go to the warp's
// queue; emptying it, with none of the march's registers live, writes the list entries
// (one global atomic for 32 columns) and sums gamma^2 v^2 of the corners. Packed FP32
// pairs are rows r and r + 4.
// A sixth of the instructions of a phase and three edge codes per vertex in shared memory
// (66 against 422 million at 320^3), so the march waits for its loads (16 warps an SM at
// 128 registers; 4 rows a lane with 24 warps took 1.17x as long). 512^3, string finder
// with its list 1.57 -> 0.60 ms, with velocities and no list 1.79 -> 0.63 ms; white
// noise (70 % of the cells pierced), 320^3, list: 0.69 -> 0.60 ms.
constexpr int FTX = 32, FTY = 16;  // energy32_kernel's tile
static_assert(FTX * FTY == 2 * kDiagThreads, "two cells per thread");
constexpr int kStripW = 31, kStripRows = 8, kStripPairs = kStripRows / 2;
constexpr int kStripQueue = 512;  // a warp's queued columns
// Columns with pierced cells from which the columns next to them are queued as well, of the
// strip's 31: from 16 on, fields cut off at 5 cells took 0.93 ms where this takes 0.86, the
// others the same.
constexpr int kStripDense = 24;
constexpr int kFinderBlocks = 2;  // per SM
static_assert(kStripQueue >= 3 * 32 && kStripRows <= 8 && kStripRows % 2 == 0,
              "an empty queue takes three planes' columns; rows are bits of a byte");
// A lane's column of cells in a plane: pierced xy, yz, zx plaquettes, bit per row, in bits
// 0-7, 8-15 and 16-23, the lane in bits 24-28; none pierced: to be taken through the exact
// path, or a column whose vertices the column before it takes.
constexpr unsigned kVerticesOnly = 1u << 29;
struct StripColumn {
    unsigned pierced;
    int z;
};
struct FinderSmem {
    StripColumn queue[kDiagThreads / 32][kStripQueue];
};

// gamma^2 v^2 at a vertex (Velocity.hpp:62-78 with the prefactors folded on the
// host) in single precision, with every operation rounded as written so that the
// plane pass and the after-chunk path agree to the bit
__device__ __forceinline__ float vertex_gv(float psi1, float psi2, float Pi1, float Pi2, const DiagConst &q)
{
    const float phi1 = __fmul_rn(psi1, q.f_inv_R), phi2 = __fmul_rn(psi2, q.f_inv_R);
    const float pd1 = __fmul_rn(__fsub_rn(Pi1, __fmul_rn(q.f_RpR, psi1)), q.f_inv_R2);
    const float pd2 = __fmul_rn(__fsub_rn(Pi2, __fmul_rn(q.f_RpR, psi2)), q.f_inv_R2);
    const float phi_sq = __fadd_rn(__fmul_rn(phi1, phi1), __fmul_rn(phi2, phi2));
    const float pd_sq = __fadd_rn(__fmul_rn(pd1, pd1), __fmul_rn(pd2, pd2));
    const float re = __fadd_rn(__fmul_rn(phi1, pd1), __fmul_rn(phi2, pd2));
    return __fsub_rn(__fmul_rn(__fmul_rn(pd_sq, q.f_vel_a), __fsub_rn(1.f, __fmul_rn(q.f_vel_b, phi_sq))),
                     __fmul_rn(__fmul_rn(q.f_vel_c, re), re));
}

// the same at two vertices, to the same bits
__device__ __forceinline__ F2 vertex_gv(F2 psi1, F2 psi2, F2 Pi1, F2 Pi2, const DiagConst &q)
{
    const F2 phi1 = psi1 * F2(q.f_inv_R), phi2 = psi2 * F2(q.f_inv_R);
    const F2 pd1 = (Pi1 - F2(q.f_RpR) * psi1) * F2(q.f_inv_R2), pd2 = (Pi2 - F2(q.f_RpR) * psi2) * F2(q.f_inv_R2);
    const F2 phi_sq = phi1 * phi1 + phi2 * phi2, pd_sq = pd1 * pd1 + pd2 * pd2, re = phi1 * pd1 + phi2 * pd2;
    return (pd_sq * F2(q.f_vel_a)) * (F2(1.f) - F2(q.f_vel_b) * phi_sq) - (F2(q.f_vel_c) * re) * re;
}

struct CellWindings {
    int w[3], ties;
};

// edge code: fold + 1 in bits 0-1, bit 2 set when the cell must be redone in
// double (winding4_fast's band test on the same float difference)
__device__ __forceinline__ unsigned edge_code(float ta, float tb, bool ok)
{
    const float pi = 3.14159265f, band = 1e-5f;
    const float d = tb - ta;
    const bool bad = !ok || fabsf(fabsf(d) - pi) < band;
    return (unsigned)(1 + (d < -pi) - (d > pi)) | (bad ? 4u : 0u);
}
__device__ __forceinline__ int edge_fold(unsigned c) { return (int)(c & 3u) - 1; }

// A cell's three windings in the reference's double arithmetic, psi read from
// global memory at its seven corners (zero outside the view's ghost region, as
// the plane loads fill it). Out of line: it is rare and needs many registers.
template <typename T>
__device__ __noinline__ CellWindings finder_cell_double(const DiagView v, const T *base, int x, int y, int z)
{
    auto ph = [&](int xx, int yy, int zz) {
        const bool on = (v.wx || xx < v.nx + v.ox) && (v.wy || yy < v.ny + v.oy) && (v.wz || zz < v.nz + v.oz);
        const double a = on ? (double)base[view_off<T>(v, 0, xx, yy, zz)] : 0.0;
        const double b = on ? (double)base[view_off<T>(v, 1, xx, yy, zz)] : 0.0;
        return atan2(b, a);
    };
    const double d000 = ph(x, y, z), d100 = ph(x + 1, y, z), d110 = ph(x + 1, y + 1, z), d010 = ph(x, y + 1, z);
    const double d001 = ph(x, y, z + 1), d101 = ph(x + 1, y, z + 1), d011 = ph(x, y + 1, z + 1);
    CellWindings r;
    r.ties = 0;
    cell_windings_double(d000, d100, d110, d010, d001, d101, d011, r.w, r.ties);
    return r;
}

// A cell whose edges the bits cannot decide: the folds of its float phases or, with an
// edge in the band of edge_code or a vertex outside float range, the double path.
template <typename T>
__device__ __noinline__ CellWindings finder_cell_exact(const DiagView &v, const T *base, int x, int y, int z)
{
    float th[8];
    bool ok[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int xx = x + (c & 1), yy = y + ((c >> 1) & 1), zz = z + (c >> 2);
        const bool on = (v.wx || xx < v.nx + v.ox) && (v.wy || yy < v.ny + v.oy) && (v.wz || zz < v.nz + v.oz);
        const T a = on ? base[view_off<T>(v, 0, xx, yy, zz)] : T(0);
        const T b = on ? base[view_off<T>(v, 1, xx, yy, zz)] : T(0);
        if constexpr (sizeof(T) == 4) {
            const float m = fmaxf(fabsf(a), fabsf(b));
            ok[c] = m > 1e-30f && m < 1e30f;
        } else {
            const double m = fmax(fabs(a), fabs(b));
            ok[c] = m > 1e-30 && m < 1e30;
        }
        th[c] = atan2f((float)b, (float)a);
    }
    // corners c = x + 2 y + 4 z; edges x: 0-1, 2-3, 4-5; y: 0-2, 1-3, 4-6; z: 0-4, 1-5, 2-6
    const int ea[9] = {0, 2, 4, 0, 1, 4, 0, 1, 2}, eb[9] = {1, 3, 5, 2, 3, 6, 4, 5, 6};
    unsigned code[9], bad = 0;
#pragma unroll
    for (int e = 0; e < 9; ++e) bad |= code[e] = edge_code(th[ea[e]], th[eb[e]], ok[ea[e]] && ok[eb[e]]);
    if (bad & 4u) return finder_cell_double<T>(v, base, x, y, z);
    // StringFinder.hpp:45-68 order: xy (000 100 110 010), yz (000 010 011 001), zx (000 001 101 100)
    CellWindings r;
    r.w[0] = edge_fold(code[0]) + edge_fold(code[4]) - edge_fold(code[1]) - edge_fold(code[3]);
    r.w[1] = edge_fold(code[3]) + edge_fold(code[8]) - edge_fold(code[5]) - edge_fold(code[6]);
    r.w[2] = edge_fold(code[6]) + edge_fold(code[2]) - edge_fold(code[7]) - edge_fold(code[0]);
    r.ties = 0;
    return r;
}

// Empty a warp's queue of n columns. Written are the list entries (one global atomic for
// every 32 columns with pierced cells, one for each plaquette of the exact path) and the
// exact path's tags; returned the lane's part of the exact path's counts and (VEL) of the
// sum over the corners of every pierced plaquette.
struct StripCounts {
    double vsum;
    int plain, weighted, ties;
};
template <typename T> struct StripJob {
    const T *base;
    const uint8_t *mask;
    uint8_t *tags;
    unsigned long long *list_counter;
    long long *list;
    long long capacity;
    int64_t cell0;  // number of the strip's first cell in plane 0
    int x0, y0;
};
template <typename T, bool VEL>
__device__ __noinline__ StripCounts strip_drain(const DiagView &v, const DiagConst &q, const StripJob<T> &job,
                                                const StripColumn *queue, int n)
{
    const int lane = threadIdx.x & 31;
    StripCounts r{0.0, 0, 0, 0};
    // corner sums in FP32, compensated (Neumaier; GB300 issues FP64 at 1/64 of the FP32 rate)
    float acc = 0.f, comp = 0.f;
    // VelocityKernel.hpp:37-141: gamma^2 v^2 of the 4 corners of every pierced plaquette of
    // a column (fields are zero outside the view's ghost region). The warp goes through the
    // vertex rows that any lane needs together, so that its loads stay row segments. A lane
    // computes the vertices at its own x, in planes z and z + 1; those at x + 1 come from the
    // next lane where it has that column (a dense network's mostly do), else from memory
    // too. A row's fields are fetched while the one before is computed. 320^3, pass with
    // energies, list and velocities: white noise 1.35 -> 1.22 ms (1.20 with gamma^2 v^2 at every
    // vertex instead), fields cut off at 3 cells 1.21 -> 1.09 (1.12), at 5 cells 0.98 -> 0.86
    // (1.06), at 8 cells 0.78 -> 0.68 (1.04); without the fetch ahead 1.26, 1.16, 1.00, 0.73.
    auto velocity = [&](int x, int y0, int z, unsigned pierced) {
        const int z1 = v.wz && z + 1 == v.nz ? 0 : z + 1;
        const bool onz = v.wz || z + 1 < v.nz + v.oz;
        const T *p0 = job.base + v.ox + (int64_t)v.oy * v.js + (int64_t)(z + v.oz) * v.ks;
        const int64_t up = (int64_t)(z1 - z) * v.ks;
        // the fields at the vertices (xv, y) of planes z and z + 1
        auto fetch = [&](int xv, int y, F2 (&f)[4]) {
            const int xw = v.wx && xv == v.nx ? 0 : xv, yw = v.wy && y == v.ny ? 0 : y;
            const bool on = (v.wx || xv < v.nx + v.ox) && (v.wy || y < v.ny + v.oy);
            const T *c = p0 + xw + (int64_t)yw * v.js;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                f[m].v.x = on ? (float)__ldg(c + m * v.cs) : 0.f;
                f[m].v.y = on && onz ? (float)__ldg(c + m * v.cs + up) : 0.f;
            }
        };
        const unsigned mine = (pierced | pierced >> 8 | pierced >> 16) & 0xffu, vertices = mine | mine << 1;
        // whether the next lane has column x + 1, and the rows that the lane before takes from this one
        const int x_next = __shfl_down_sync(0xffffffffu, x, 1), y_next = __shfl_down_sync(0xffffffffu, y0, 1),
                  z_next = __shfl_down_sync(0xffffffffu, z, 1);
        const bool next = lane < 31 && x_next == x + 1 && y_next == y0 && z_next == z;
        const unsigned asked = __shfl_up_sync(0xffffffffu, next ? vertices : 0u, 1);
        const unsigned own = lane ? vertices | asked : vertices;
        F2 low(0.f), low1(0.f);  // rows k and k + 1 at x and x + 1, planes z and z + 1
        unsigned rows = __reduce_or_sync(0xffffffffu, vertices);
        F2 f[4], f1[4];  // a row ahead
#pragma unroll
        for (int m = 0; m < 4; ++m) f[m] = f1[m] = F2(0.f);
        auto fetch_row = [&]() {
            const int y = __ffs(rows) - 1;
            if (own >> y & 1) fetch(x, y0 + y, f);
            if (!next && (vertices >> y & 1)) fetch(x + 1, y0 + y, f1);
        };
        if (rows) fetch_row();
        while (rows) {
            const int y = __ffs(rows) - 1, k = y - 1;
            const bool here = vertices >> y & 1;
            const F2 c0 = f[0], c1 = f[1], c2 = f[2], c3 = f[3], d0 = f1[0], d1 = f1[1], d2 = f1[2], d3 = f1[3];
            rows &= rows - 1;
            if (rows) fetch_row();
            const F2 g = vertex_gv(c0, c1, c2, c3, q);
            F2 g1;
            g1.v.x = __shfl_down_sync(0xffffffffu, g.v.x, 1);
            g1.v.y = __shfl_down_sync(0xffffffffu, g.v.y, 1);
            if (here && !next) g1 = vertex_gv(d0, d1, d2, d3, q);
            if (here) {
                const F2 high(g.v.x, g1.v.x), high1(g.v.y, g1.v.y);
                if ((mine << 1) >> y & 1) {
                    float s = 0.f;  // corners 000 100 110 010, 000 010 011 001, 000 001 101 100
                    if (pierced >> k & 1) s += low.v.x + low.v.y + high.v.y + high.v.x;
                    if (pierced >> (8 + k) & 1) s += low.v.x + high.v.x + high1.v.x + low1.v.x;
                    if (pierced >> (16 + k) & 1) s += low.v.x + low1.v.x + low1.v.y + low.v.y;
                    const float t = acc + s;
                    comp += fabsf(acc) >= fabsf(s) ? (acc - t) + s : (s - t) + acc;
                    acc = t;
                }
                low = high;
                low1 = high1;
            }
        }
    };
    // Velocities: 31 columns at a time, the last lane with the first of the next 31, which it
    // only computes the vertices of.
    constexpr int kTake = VEL ? 31 : 32;
    for (int i0 = 0; i0 < n; i0 += kTake) {
        const StripColumn e = i0 + lane < n ? queue[i0 + lane] : StripColumn{kVerticesOnly, 0};
        const bool take = lane < kTake && !(e.pierced & kVerticesOnly);
        const unsigned pierced = take ? e.pierced & 0xffffffu : 0u;
        const int dx = e.pierced >> 24 & 31u;
        const int64_t plane = (int64_t)v.nx * v.ny;
        if (job.list != nullptr) {
            int incl = __popc(pierced);
            unsigned long long pos = 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += up;
            }
            if (lane == 31 && incl) pos = atomicAdd(job.list_counter, (unsigned long long)incl);
            pos = __shfl_sync(0xffffffffu, pos, 31) + incl - __popc(pierced);
            const int64_t cell = job.cell0 + dx + plane * e.z;
            for (unsigned p = pierced; p; p &= p - 1) {
                const int b = __ffs(p) - 1;
                if (pos < (unsigned long long)job.capacity) job.list[pos] = 4 * (cell + (int64_t)v.nx * (b & 7)) + (b >> 3);
                ++pos;
            }
        }
        // the pierced cells, then the exact path, four columns at a time, a row a lane
        unsigned exact = __ballot_sync(0xffffffffu, take && !pierced), some = pierced;
        int x = job.x0 + dx, y = job.y0, z = e.z;
        while (true) {
            if constexpr (VEL) velocity(x, y, z, some);
            if (!exact) break;
            unsigned m = exact;
            for (int i = 0; i < lane / 8; ++i) m &= m - 1;
            const int src = m ? __ffs(m) - 1 : 0;
            x = job.x0 + __shfl_sync(0xffffffffu, dx, src);
            y = job.y0 + (lane & 7);
            z = __shfl_sync(0xffffffffu, e.z, src);
            some = 0;
            const int64_t c = job.cell0 + (x - job.x0) + (int64_t)v.nx * (lane & 7) + plane * z;
            if (m && y < min(job.y0 + kStripRows, v.ny) && (job.mask == nullptr || job.mask[c] != 0)) {
                const CellWindings cw = finder_cell_exact<T>(v, job.base, x, y, z);
                r.ties += cw.ties;
                for (int pl = 0; pl < 3; ++pl) {
                    if (cw.w[pl] == 0) continue;
                    some |= 1u << (8 * pl);
                    ++r.plain;
                    r.weighted += abs(cw.w[pl]);
                    if (job.list != nullptr) {
                        const unsigned long long at = atomicAdd(job.list_counter, 1ull);
                        if (at < (unsigned long long)job.capacity) job.list[at] = 4 * c + pl;
                    }
                }
                if (job.tags != nullptr) job.tags[c] = some != 0;
            }
            for (int i = 0; i < 4; ++i) exact &= exact - 1;
        }
    }
    if (VEL) r.vsum = (double)acc + (double)comp;
    return r;
}

// psi at the vertices of a lane's column in one plane
struct StripPlane {
    F2 a1[kStripPairs], a2[kStripPairs];  // rows k, k + kStripPairs
    float b1, b2;                         // row kStripRows
};

// One edge (two, packed): cross and dot products, the antiparallel test into `bad`'s
// sign bit; the value returned has the sign bit of cross.
__device__ __forceinline__ float strip_edge(float a1, float n2, float a2, float b1, float b2, unsigned &bad)
{
    const float cr = fmaf(a1, b2, n2 * b1), dot = fmaf(a1, b1, a2 * b2);
    bad |= __float_as_uint(fmaf(1e-5f, dot, fabsf(cr)));
    return cr;
}
__device__ __forceinline__ F2 strip_edge(F2 a1, F2 n2, F2 a2, F2 b1, F2 b2, unsigned &bad)
{
    const F2 cr = fma(a1, b2, n2 * b1), e = F2(1e-5f) * fma(a1, b1, a2 * b2);
    bad |= __float_as_uint(fabsf(cr.v.x) + e.v.x) | __float_as_uint(fabsf(cr.v.y) + e.v.y);
    return cr;
}
// append to `bits` whether an edge folds: imaginary parts of opposite sign, cross of a2's
__device__ __forceinline__ void strip_fold(unsigned &bits, float a2, float b2, float cr)
{
    const unsigned a = __float_as_uint(a2);
    bits = __funnelshift_l((a ^ __float_as_uint(b2)) & ~(a ^ __float_as_uint(cr)), bits, 1);
}

// VEL (FP32 fields, beside energy32_kernel): also the sum of gamma^2 v^2 over the
// corners of every pierced plaquette. Blocks from e_from on clear their partial
// record's energy sums (energy32_kernel writes those of the blocks below it).
template <typename T, bool VEL>
__global__ void __launch_bounds__(kDiagThreads, kFinderBlocks)
    finder_kernel(const __grid_constant__ DiagView v, const __grid_constant__ DiagConst q,
                  const uint8_t *__restrict__ mask, DiagPartial *__restrict__ partials,
                  unsigned long long *__restrict__ list_counter, long long *__restrict__ list, long long capacity,
                  int strips_x, int strips, int zchunk, long long n_items, long long items_per_box, int64_t box_stride,
                  uint8_t *__restrict__ tags, int e_from)
{
    constexpr int W = kDiagThreads / 32;
    extern __shared__ __align__(16) unsigned char finder_smem_raw[];
    __shared__ StripJob<T> jobs[W];
    __shared__ long long red[W][3];
    __shared__ double redv[W];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    StripColumn *queue = reinterpret_cast<FinderSmem *>(finder_smem_raw)->queue[warp];
    int cnt_p = 0, cnt_w = 0, cnt_tie = 0;  // per-thread counts fit 32 bits
    double vsum = 0.0;

    for (long long item = (long long)blockIdx.x * W + warp; item < n_items; item += (long long)gridDim.x * W) {
        const long long qbox = item / items_per_box, box_item = item % items_per_box;
        const T *__restrict__ base = static_cast<const T *>(v.data) + qbox * box_stride;
        const int strip = (int)(box_item % strips), chunk = (int)(box_item / strips);
        const int x0 = (strip % strips_x) * kStripW, y0 = (strip / strips_x) * kStripRows;
        const int za = chunk * zchunk, zend = min(za + zchunk, v.nz);
        const int64_t cell0 = qbox * v.nx * v.ny * v.nz + x0 + (int64_t)v.nx * y0;
        const int x = x0 + lane;
        if (lane == 0) jobs[warp] = StripJob<T>{base, mask, tags, list_counter, list, capacity, cell0, x0, y0};
        __syncwarp();

        const unsigned valid = lane < kStripW && x < v.nx ? (1u << min(kStripRows, v.ny - y0)) - 1 : 0u;

        // march until the chunk is done or the queue could overflow, then empty the queue with
        // none of the march's registers live, and go on from there
        for (int zs = za; zs < zend;) {
        const int len = zend - zs;
        // in-plane element offsets of the lane's vertices (the host checks that a plane's
        // offsets fit 31 bits). Vertices no cell of the strip has repeat the last one;
        // outside the ghost region psi is zero.
        int off[kStripRows + 1];
        unsigned on = 0;  // bit per row
        const int xv = min(x, v.nx), xw = v.wx && xv == v.nx ? 0 : xv;
#pragma unroll
        for (int r = 0; r <= kStripRows; ++r) {
            const int yv = min(y0 + r, v.ny), yw = v.wy && yv == v.ny ? 0 : yv;
            const bool in = (v.wx || xv < v.nx + v.ox) && (v.wy || yv < v.ny + v.oy);
            on |= (unsigned)in << r;
            off[r] = in ? (xw + v.ox) + (yw + v.oy) * (int)v.js : 0;
        }
        const bool all_on = __all_sync(0xffffffffu, on == (2u << kStripRows) - 1);
        int lz = zs, lzw = zs;  // (zs < nz)
        auto load = [&](StripPlane &p) {
            const bool zin = v.wz || lz < v.nz + v.oz;
            const T *c1 = base + (int64_t)(lzw + v.oz) * v.ks, *c2 = c1 + v.cs;
            if (all_on && zin) {
#pragma unroll
                for (int k = 0; k < kStripPairs; ++k) {
                    p.a1[k] = F2((float)__ldg(c1 + off[k]), (float)__ldg(c1 + off[k + kStripPairs]));
                    p.a2[k] = F2((float)__ldg(c2 + off[k]), (float)__ldg(c2 + off[k + kStripPairs]));
                }
                p.b1 = (float)__ldg(c1 + off[kStripRows]);
                p.b2 = (float)__ldg(c2 + off[kStripRows]);
            } else {
                auto get = [&](const T *c, int r) { return zin && (on >> r & 1) ? (float)__ldg(c + off[r]) : 0.f; };
#pragma unroll
                for (int k = 0; k < kStripPairs; ++k) {
                    p.a1[k] = F2(get(c1, k), get(c1, k + kStripPairs));
                    p.a2[k] = F2(get(c2, k), get(c2, k + kStripPairs));
                }
                p.b1 = get(c1, kStripRows);
                p.b2 = get(c2, kStripRows);
            }
            ++lz;
            lzw = v.wz && lz == v.nz ? 0 : lz;
        };

        int queued = 0;  // warp-uniform
        unsigned X0 = 0, Y0 = 0, bad0 = 0;  // the plane before: x and y edges that fold; bad: sign bit
        // plane zs + j in `cur`, the one before in `prev`; the one after is loaded into `next`
        auto step = [&](int j, const StripPlane &prev, const StripPlane &cur, StripPlane &next) {
            if (j < len) load(next);
            F2 n2[kStripPairs];
            const float nb2 = -cur.b2;
            int least = INT_MAX, most = 0;  // of |psi|^2's bits: NaN lies above, negative below
            unsigned bad1 = 0, bz = 0;
#pragma unroll
            for (int k = 0; k < kStripPairs; ++k) {
                n2[k] = F2(-1.f) * cur.a2[k];
                const F2 s = fma(cur.a1[k], cur.a1[k], cur.a2[k] * cur.a2[k]);
                least = __vimin3_s32(least, __float_as_int(s.v.x), __float_as_int(s.v.y));
                most = __vimax3_s32(most, __float_as_int(s.v.x), __float_as_int(s.v.y));
            }
            {
                const int s = __float_as_int(fmaf(cur.b1, cur.b1, cur.b2 * cur.b2));
                least = min(least, s);
                most = max(most, s);
            }
            const bool outside = least < __float_as_int(1e-36f) || most > __float_as_int(1e36f);
            // x edges (rows 0 .. 8) and y edges (rows 0 .. 7), row 0 appended last
            unsigned xl = 0, xh = 0, yl = 0, yh = 0;
            {
                const float r1 = __shfl_down_sync(0xffffffffu, cur.b1, 1), r2 = __shfl_down_sync(0xffffffffu, cur.b2, 1);
                strip_fold(xh, cur.b2, r2, strip_edge(cur.b1, nb2, cur.b2, r1, r2, bad1));
            }
#pragma unroll
            for (int k = kStripPairs - 1; k >= 0; --k) {
                const F2 a1 = cur.a1[k], a2 = cur.a2[k];
                F2 r1, r2;
                r1.v.x = __shfl_down_sync(0xffffffffu, a1.v.x, 1);
                r1.v.y = __shfl_down_sync(0xffffffffu, a1.v.y, 1);
                r2.v.x = __shfl_down_sync(0xffffffffu, a2.v.x, 1);
                r2.v.y = __shfl_down_sync(0xffffffffu, a2.v.y, 1);
                const F2 cx = strip_edge(a1, n2[k], a2, r1, r2, bad1);
                strip_fold(xl, a2.v.x, r2.v.x, cx.v.x);
                strip_fold(xh, a2.v.y, r2.v.y, cx.v.y);
                const F2 u1 = k + 1 < kStripPairs ? cur.a1[(k + 1) % kStripPairs] : F2(cur.a1[0].v.y, cur.b1);
                const F2 u2 = k + 1 < kStripPairs ? cur.a2[(k + 1) % kStripPairs] : F2(cur.a2[0].v.y, cur.b2);
                const F2 cy = strip_edge(a1, n2[k], a2, u1, u2, bad1);
                strip_fold(yl, a2.v.x, u2.v.x, cy.v.x);
                strip_fold(yh, a2.v.y, u2.v.y, cy.v.y);
            }
            const unsigned X1 = xl | xh << kStripPairs, Y1 = yl | yh << kStripPairs;
            bad1 |= outside ? 0x80000000u : 0u;
            if (j > 0) {
                // z edges to the plane before (rows 0 .. 8)
                unsigned zl = 0, zh = 0;
                strip_fold(zh, cur.b2, prev.b2, strip_edge(cur.b1, nb2, cur.b2, prev.b1, prev.b2, bz));
#pragma unroll
                for (int k = kStripPairs - 1; k >= 0; --k) {
                    const F2 cz = strip_edge(cur.a1[k], n2[k], cur.a2[k], prev.a1[k], prev.a2[k], bz);
                    strip_fold(zl, cur.a2[k].v.x, prev.a2[k].v.x, cz.v.x);
                    strip_fold(zh, cur.a2[k].v.y, prev.a2[k].v.y, cz.v.y);
                }
                const unsigned Z = zl | zh << kStripPairs;
                // the cells of plane zs + j - 1: this column's bits and the next one's
                const unsigned mine = Y0 | Z << 8 | ((bad0 | bz | bad1) >> 31) << 17;
                const unsigned right = __shfl_down_sync(0xffffffffu, mine, 1);
                unsigned pxy = (X0 ^ X0 >> 1 ^ Y0 ^ right) & valid;
                unsigned pyz = (Y0 ^ Y1 ^ Z ^ Z >> 1) & valid;
                unsigned pzx = (Z ^ right >> 8 ^ X0 ^ X1) & valid;
                const bool inexact = valid != 0 && ((mine | right) >> 17 & 1);
                if (inexact) pxy = pyz = pzx = 0;
                unsigned any = pxy | pyz | pzx;
                if (mask != nullptr || tags != nullptr) {
                    const int64_t cell = cell0 + lane + (int64_t)v.nx * v.ny * (zs + j - 1);
                    unsigned keep = 0;
                    for (int k = 0; k < kStripRows; ++k)
                        if (valid >> k & 1) keep |= (unsigned)(mask == nullptr || mask[cell + (int64_t)v.nx * k] != 0) << k;
                    any &= keep;
                    pxy &= keep;
                    pyz &= keep;
                    pzx &= keep;
                    // StringTagger.hpp:117-151: a cell is tagged when a plaquette at its low corner is pierced
                    if (tags != nullptr && !inexact)
                        for (int k = 0; k < kStripRows; ++k)
                            if (keep >> k & 1) tags[cell + (int64_t)v.nx * k] = any >> k & 1;
                }
                cnt_p += __popc(pxy | pyz << 8 | pzx << 16);
                // queue the lane's column if it is inexact, or pierced where anyone asks which cells are
                const bool put = inexact || ((VEL || list != nullptr) && any != 0);
                unsigned with = __ballot_sync(0xffffffffu, put);
                // with velocities, on a plane with many: also the columns next to them, for their vertices
                if (VEL && __popc(with) >= kStripDense) with |= with << 1;
                if (with >> lane & 1)
                    queue[queued + __popc(with & ((1u << lane) - 1))] = StripColumn{
                        pxy | pyz << 8 | pzx << 16 | (unsigned)lane << 24 | (put ? 0u : kVerticesOnly), zs + j - 1};
                queued += __popc(with);
            }
            X0 = X1;
            Y0 = Y1;
            bad0 = bad1;
        };
        StripPlane p0, p1, p2;
        load(p0);
        int j = 0;
        do {
            step(j, p2, p0, p1);
            if (j + 1 <= len) step(j + 1, p0, p1, p2);
            if (j + 2 <= len) step(j + 2, p1, p2, p0);
            j += 3;
        } while (j <= len && queued <= kStripQueue - 3 * 32);
        zs += min(j - 1, len);  // the last vertex plane's cells are still to do
        if (queued) {
            __syncwarp();
            const StripCounts c = strip_drain<T, VEL>(v, q, jobs[warp], queue, queued);
            __syncwarp();
            vsum += c.vsum;
            cnt_p += c.plain;
            cnt_w += c.weighted - c.plain;
            cnt_tie += c.ties;
        }
        }
        __syncwarp();  // the job record is free
    }

    // ---- block reduction (fixed order) into the fused pass's partial record ----
    long long c3[3] = {cnt_p, cnt_w, cnt_tie};
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        for (int o = 16; o > 0; o >>= 1) c3[s] += __shfl_down_sync(0xffffffffu, c3[s], o);
        if (lane == 0) red[warp][s] = c3[s];
    }
    if constexpr (VEL)
        for (int o = 16; o > 0; o >>= 1) vsum += __shfl_down_sync(0xffffffffu, vsum, o);
    if (lane == 0) redv[warp] = VEL ? vsum : 0.0;
    __syncthreads();
    if (tid < 14) {
        if ((int)blockIdx.x >= e_from) partials[blockIdx.x].e[tid] = 0.0;
    } else if (tid == 14) {
        double xv = 0.0;
        for (int ww = 0; ww < W; ++ww) xv += redv[ww];
        partials[blockIdx.x].vsum = xv;
    } else if (tid == 32) {
        long long np = 0, extra = 0, ties = 0;
        for (int ww = 0; ww < W; ++ww) {
            np += red[ww][0];
            extra += red[ww][1];
            ties += red[ww][2];
        }
        DiagPartial &r = partials[blockIdx.x];
        r.cnt[0] = np;                   // n_p_plain
        r.cnt[1] = np + extra;           // n_p_weighted
        r.cnt[2] = VEL ? 4 * np : 0;     // vel_count: the corners of every pierced plaquette
        r.cnt[3] = ties;                 // near_tie
    }
}

// ---------------------------------------------------------------- FP32 per-cell energy sums
// The per_cell_fp32 energy sums on FP32 fields, run beside finder_kernel<float, VEL>
// (windings, the pierced list and the velocity). A block owns a FTX x FTY tile, two
// cells per thread FTY / 2 rows apart, packed, and marches in z. psi of the tile
// plus a 2-cell halo arrives by cp.async in a ring of five planes: the current one, whose
// rows the x and y stencils read, the one two above, whose centre goes to the
// thread's column of five planes in registers, the two on the way, and one that a
// slower warp may still read (one block barrier per plane). Pi comes to registers a plane
// ahead. Per plane the warp's sums of its cells' 13 terms and of their count end on a
// lane each (15 exchanges that halve what a lane holds), which adds them to a
// compensated (Neumaier) FP32 accumulator. After each z-chunk the accumulators go to per-warp FP64 slots. Cells
// where FP32 cannot hold 1/|psi|^4 (|psi|^2 outside (1e-15, 1e15): the cores' exact
// zeros) are queued and take the reference's double arithmetic after the chunk, as the
// fused pass does. VEC: rows, strides and the tile's origin allow 8-byte copies.
// Bound by instruction issue. 512^3: 1.68 -> 0.93 ms (scalar cells, z taps from shared
// memory, 4-byte copies, a full butterfly of each of the 14 sums: 380 instructions a
// cell). Two cells next to each other in x, their sums over five planes first, took
// 0.77 ms, but FP32 partial sums in another order move small boxes' sums by 5e-9.
constexpr int EHX = FTX + 4, EHY = FTY + 4, kEnergySlots = 5, kEnergyBadQ = 1024;
constexpr int kEnergyPts = 2 * EHX * EHY;
struct EnergySmem {
    double ew[kDiagThreads / 32][14];
    float ps[kEnergySlots][2][EHY][EHX];
    int badq[kEnergyBadQ];  // tile-local x | y << 5 | (z - za) << 9
};

struct CellTerms {
    double t[14];
};

// One cell's 14 terms in the reference's double per-cell arithmetic, psi and Pi
// read from global memory (zero outside the view's ghost region).
__device__ __noinline__ CellTerms energy_cell_double(const DiagView v, const DiagConst q, const float *base, int x,
                                                     int y, int z)
{
    auto at = [&](int c, int xx, int yy, int zz) -> double {
        const bool on = (v.wx || (xx >= -v.ox && xx < v.nx + v.ox)) && (v.wy || (yy >= -v.oy && yy < v.ny + v.oy)) &&
                        (v.wz || (zz >= -v.oz && zz < v.nz + v.oz));
        return on ? (double)base[view_off<float>(v, c, xx, yy, zz)] : 0.0;
    };
    double g[2][3];
    for (int c = 0; c < 2; ++c) {
        g[c][0] = diff1_vals<float>(at(c, x - 2, y, z), at(c, x - 1, y, z), at(c, x + 1, y, z), at(c, x + 2, y, z),
                                    q.one_over_dx);
        g[c][1] = diff1_vals<float>(at(c, x, y - 2, z), at(c, x, y - 1, z), at(c, x, y + 1, z), at(c, x, y + 2, z),
                                    q.one_over_dx);
        g[c][2] = diff1_vals<float>(at(c, x, y, z - 2), at(c, x, y, z - 1), at(c, x, y, z + 1), at(c, x, y, z + 2),
                                    q.one_over_dx);
    }
    const CellConst<double> kd{q.R2, q.inv_R, q.inv_R2, q.inv_R4, q.lambda, q.RpR, q.threshold};
    double term[6], wgt;
    float gt[2][3];
    for (int c = 0; c < 2; ++c)
        for (int d = 0; d < 3; ++d) gt[c][d] = (float)g[c][d];
    cell_energy<float, false>(kd, q.scheme, at(0, x, y, z), at(1, x, y, z), at(2, x, y, z), at(3, x, y, z), g, gt, term,
                              wgt);
    CellTerms r;
    for (int k = 0; k < 6; ++k) {
        r.t[2 * k] = term[k];
        r.t[2 * k + 1] = term[k] * wgt;
    }
    r.t[12] = wgt;
    r.t[13] = 1.0;
    return r;
}

// The warp's sums of v[0 .. 13]: lane l returns that of k = 7 b4 + 4 b3 + 2 b2 + b1 of its
// bits (b3 b2 b1 = 7: none), added up in the order of a butterfly from 16 down.
__device__ __forceinline__ float warp_sums14(const float (&v)[14], int lane)
{
    auto fold = [&](float lo, float hi, int o) {
        const bool up = lane & o;
        return (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, o);
    };
    float a[7], b[4];
#pragma unroll
    for (int i = 0; i < 7; ++i) a[i] = fold(v[i], v[i + 7], 16);
#pragma unroll
    for (int i = 0; i < 4; ++i) b[i] = fold(a[i], i < 3 ? a[i + 4] : 0.f, 8);
    const float c0 = fold(b[0], b[2], 4), c1 = fold(b[1], b[3], 4), d = fold(c0, c1, 2);
    return d + __shfl_xor_sync(0xffffffffu, d, 1);
}

constexpr int kEnergyBlocks = 3;  // per SM: 80 registers (64 and 128 took 1.10x as long)
template <bool VEC>
__global__ void __launch_bounds__(kDiagThreads, kEnergyBlocks)
    energy32_kernel(const __grid_constant__ DiagView v, const __grid_constant__ DiagConst q,
                    const uint8_t *__restrict__ mask, DiagPartial *__restrict__ partials, int tiles_x, int ntiles,
                    int zchunk, long long n_items, long long items_per_box, int64_t box_stride, int cnt_from)
{
    __shared__ __align__(16) EnergySmem sm;
    __shared__ int badn, bad_over;
    constexpr int EN = VEC ? 2 : 1;  // elements per copy
    constexpr int PER = (kEnergyPts / EN + kDiagThreads - 1) / kDiagThreads;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int HALF = FTY / 2;
    const int lx = tid % FTX, ly = tid / FTX;                // cells (lx, ly) and (lx, ly + HALF)
    const int sum_of = 7 * (lane >> 4) + ((lane >> 1) & 7);  // the sum the lane keeps
    const bool keeps = (lane & 1) == 0 && (lane & 14) != 14;
    const int64_t box_cells = (int64_t)v.nx * v.ny * v.nz;
    const CellConst<float> kf{q.f_R2, q.f_inv_R, q.f_inv_R2, q.f_inv_R4, q.f_lambda, q.f_RpR, q.f_threshold};
    for (int i = tid; i < (kDiagThreads / 32) * 14; i += kDiagThreads) sm.ew[i / 14][i % 14] = 0.0;
    if (tid == 0) badn = bad_over = 0;
    float acc = 0.f, comp = 0.f;  // running sum of the chunk (13: its cell count, exact)

    for (long long item = blockIdx.x; item < n_items; item += gridDim.x) {
        const long long qbox = item / items_per_box, box_item = item % items_per_box;
        const float *__restrict__ base = static_cast<const float *>(v.data) + qbox * box_stride;
        const int tile = (int)(box_item % ntiles), chunk = (int)(box_item / ntiles);
        const int x0 = (tile % tiles_x) * FTX, y0 = (tile / tiles_x) * FTY;
        const int za = chunk * zchunk, len = min(zchunk, v.nz - za);
        const int x = x0 + lx, y = y0 + ly;

        // load plan: offsets in a plane of both components; elements outside the view's
        // ghost region, and those no cell needs, are zero
        int64_t poff[PER];
        unsigned on = 0;
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int e = (tid + u * kDiagThreads) * EN, r = e % (EHX * EHY);
            const int xx = x0 - 2 + r % EHX, yy = y0 - 2 + r / EHX;
            const bool in = e < kEnergyPts && xx < v.nx + 2 && yy < v.ny + 2 &&
                            (v.wx || (xx >= -v.ox && xx < v.nx + v.ox)) && (v.wy || (yy >= -v.oy && yy < v.ny + v.oy));
            on |= (unsigned)in << u;
            poff[u] = in ? (wrap_or_self(xx, v.nx, v.wx) + v.ox) + (wrap_or_self(yy, v.ny, v.wy) + v.oy) * v.js +
                               (e >= EHX * EHY ? v.cs : 0)
                         : 0;
        }
        // psi planes za - 2, ... in order (plane p in slot (p - za + 2) mod 5)
        int lz = za - 2, lzw = wrap_or_self(za - 2, v.nz, v.wz);
        auto load_psi_next = [&](int slot) {
            const bool zin = v.wz || (lz >= -v.oz && lz < v.nz + v.oz);
            const float *pb = zin ? base + (int64_t)(lzw + v.oz) * v.ks : base;
            float *dst = &sm.ps[slot][0][0][0];
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                const int e = (tid + u * kDiagThreads) * EN;
                const float *src = pb + poff[u];
                const bool in = zin && (on >> u & 1);
                if (e < kEnergyPts) {
                    if constexpr (VEC)
                        cp_async_elem(reinterpret_cast<float2 *>(dst + e), reinterpret_cast<const float2 *>(src), in,
                                      reinterpret_cast<const float2 *>(src));
                    else
                        cp_async_elem(dst + e, src, in, src);
                }
            }
            ++lz;
            lzw = v.wz ? (lzw + 1 == v.nz ? 0 : lzw + 1) : lzw + 1;
        };
        // Pi of the thread's cells, plane za on
        const unsigned valid = x < v.nx ? (unsigned)(y < v.ny) | (unsigned)(y + HALF < v.ny) << 1 : 0u;
        const float *pi_at = base + (valid ? (x + v.ox) + (int64_t)(y + v.oy) * v.js : 0) + (int64_t)(za + v.oz) * v.ks +
                             2 * v.cs;
        F2 pi_next[2];
        auto load_pi_next = [&]() {
#pragma unroll
            for (int c = 0; c < 2; ++c)
                pi_next[c] = F2(valid & 1 ? __ldg(pi_at + c * v.cs) : 0.f,
                                valid & 2 ? __ldg(pi_at + c * v.cs + HALF * v.js) : 0.f);
            pi_at += v.ks;
        };
        auto pair_at = [&](int slot, int c, int yy, int xx) {
            return F2(sm.ps[slot][c][yy][xx], sm.ps[slot][c][yy + HALF][xx]);
        };
        for (int p = 0; p < 5; ++p) load_psi_next(p);  // za - 2 .. za + 2
        cp_async_commit();
        load_pi_next();  // za
        cp_async_wait<0>();
        __syncthreads();
        const int hx = lx + 2, hy = ly + 2;
        F2 col[2][5];  // psi of planes z - 2 .. z + 2, by slot
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int p = 0; p < 4; ++p) col[c][p] = pair_at(p, c, hy, hx);
        __syncthreads();  // slot 0 is loaded again

        // plane za + m, m mod 5 = I
        auto step = [&](auto I, int m) {
            constexpr int i = decltype(I)::value, s0 = (i + 2) % 5, m2 = i, m1 = (i + 1) % 5, p1 = (i + 3) % 5,
                          p2 = (i + 4) % 5;
            const F2 pi1 = pi_next[0], pi2 = pi_next[1];
            // one plane ahead: psi(z + 3), Pi(z + 1)
            if (m + 1 < len) {
                load_psi_next(i);
                load_pi_next();
            }
            cp_async_commit();
            cp_async_wait<1>();  // psi(z + 2)
            __syncthreads();
            F2 g[2][3];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                col[c][p2] = pair_at(p2, c, hy, hx);
                g[c][0] = diff1_pair(pair_at(s0, c, hy, hx - 2), pair_at(s0, c, hy, hx + 2),
                                     pair_at(s0, c, hy, hx + 1), pair_at(s0, c, hy, hx - 1), q.f_one_over_dx);
                g[c][1] = diff1_pair(pair_at(s0, c, hy - 2, hx), pair_at(s0, c, hy + 2, hx),
                                     pair_at(s0, c, hy + 1, hx), pair_at(s0, c, hy - 1, hx), q.f_one_over_dx);
                g[c][2] = diff1_pair(col[c][m2], col[c][p2], col[c][p1], col[c][m1], q.f_one_over_dx);
            }
            const F2 f1 = col[0][s0], f2 = col[1][s0], psq = fma(f1, f1, f2 * f2);
            const bool in0 = psq.v.x > 1e-15f && psq.v.x < 1e15f, in1 = psq.v.y > 1e-15f && psq.v.y < 1e15f;
            F2 term[6], wgt;
            cell_energy(kf, q.scheme, f1, f2, pi1, pi2, g, term, wgt);
            float cells = 2.f;
            if (!__all_sync(0xffffffffu, valid == 3u && in0 && in1 && mask == nullptr)) {
                unsigned take = valid;
                if (mask != nullptr) {
                    const uint8_t *mc = mask + qbox * box_cells + x + (int64_t)v.nx * ((int64_t)y + (int64_t)v.ny * (za + m));
                    if ((take & 1) && mc[0] == 0) take &= ~1u;
                    if ((take & 2) && mc[(int64_t)HALF * v.nx] == 0) take &= ~2u;
                }
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if ((take >> h & 1) && !(h ? in1 : in0)) {
                        // the double path after the chunk
                        take &= ~(1u << h);
                        const int slot = atomicAdd(&badn, 1);
                        if (slot < kEnergyBadQ)
                            sm.badq[slot] = lx | ((ly + h * HALF) << 5) | (m << 9);
                        else
                            bad_over = 1;
                    }
                auto drop = [&](F2 &f) {
                    if (!(take & 1)) f.v.x = 0.f;
                    if (!(take & 2)) f.v.y = 0.f;
                };
#pragma unroll
                for (int k = 0; k < 6; ++k) drop(term[k]);
                drop(wgt);
                cells = (float)__popc(take);
            }
            float ts[14];
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                ts[2 * k] = term[k].v.x + term[k].v.y;
                ts[2 * k + 1] = fmaf(term[k].v.y, wgt.v.y, term[k].v.x * wgt.v.x);
            }
            ts[12] = wgt.v.x + wgt.v.y;
            ts[13] = cells;
            const float mine = warp_sums14(ts, lane), t = acc + mine;
            comp += fabsf(acc) >= fabsf(mine) ? (acc - t) + mine : (mine - t) + acc;
            acc = t;
        };
        for (int m = 0; m < len; m += 5) {
            step(std::integral_constant<int, 0>(), m);
            if (m + 1 < len) step(std::integral_constant<int, 1>(), m + 1);
            if (m + 2 < len) step(std::integral_constant<int, 2>(), m + 2);
            if (m + 3 < len) step(std::integral_constant<int, 3>(), m + 3);
            if (m + 4 < len) step(std::integral_constant<int, 4>(), m + 4);
        }
        __syncthreads();  // the queue is complete; the rings are free for the next chunk
        if (keeps) sm.ew[warp][sum_of] += (double)acc + (double)comp;
        acc = comp = 0.f;
        __syncwarp();  // the double path adds to the same sums
        // the chunk's double-path cells: from the queue or, when it overflowed, by testing
        // every cell again; each warp sums its cells' terms and lane k adds sum k
        const int nbad = badn;
        if (nbad > 0) {
            double d[14];
#pragma unroll
            for (int k = 0; k < 14; ++k) d[k] = 0.0;
            auto add_cell = [&](int x, int y, int z) {
                const CellTerms ct = energy_cell_double(v, q, base, x, y, z);
#pragma unroll
                for (int k = 0; k < 14; ++k) d[k] += ct.t[k];
            };
            if (!bad_over) {
                for (int i = tid; i < nbad; i += kDiagThreads) {
                    const int e = sm.badq[i];
                    add_cell(x0 + (e & 31), y0 + ((e >> 5) & 15), za + (e >> 9));
                }
            } else {
                for (int c = tid; c < FTX * FTY * len; c += kDiagThreads) {
                    const int x = x0 + c % FTX, y = y0 + (c / FTX) % FTY, z = za + c / (FTX * FTY);
                    if (x >= v.nx || y >= v.ny) continue;
                    if (mask != nullptr &&
                        mask[qbox * box_cells + x + (int64_t)v.nx * ((int64_t)y + (int64_t)v.ny * z)] == 0)
                        continue;
                    const float *pc = base + view_off<float>(v, 0, x, y, z);
                    const float p1 = pc[0], p2 = pc[v.cs], psq = p1 * p1 + p2 * p2;
                    if (!(psq > 1e-15f && psq < 1e15f)) add_cell(x, y, z);
                }
            }
#pragma unroll
            for (int k = 0; k < 14; ++k)
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) d[k] += __shfl_xor_sync(0xffffffffu, d[k], o);
            double dm = 0.0;
#pragma unroll
            for (int k = 0; k < 14; ++k)
                if (lane == k) dm = d[k];
            if (lane < 14) sm.ew[warp][lane] += dm;
        }
        __syncthreads();
        if (tid == 0) badn = bad_over = 0;  // published by the next chunk's first barrier
    }
    __syncthreads();
    if (tid < 14) {
        double xv = 0.0;
        for (int ww = 0; ww < kDiagThreads / 32; ++ww) xv += sm.ew[ww][tid];
        partials[blockIdx.x].e[tid] = xv;
    } else if ((int)blockIdx.x >= cnt_from && tid == 14) {
        partials[blockIdx.x].vsum = 0.0;
    } else if ((int)blockIdx.x >= cnt_from && tid >= 32 && tid < 36) {
        partials[blockIdx.x].cnt[tid - 32] = 0;
    }
}

// Sum the per-block partials in a fixed pairwise order and write the result.
__global__ void diag_finalize_kernel(const DiagPartial *__restrict__ partials, int nblocks,
                                     const unsigned long long *__restrict__ list_counter, long long capacity,
                                     int want_list, axs_diag_result *__restrict__ out)
{
    __shared__ double sd[256];
    __shared__ long long sl[256];
    const int t = threadIdx.x;
    for (int f = 0; f < 19; ++f) {
        double xd = 0.0;
        long long xl = 0;
        for (int b = t; b < nblocks; b += 256) {
            if (f < 14)
                xd += partials[b].e[f];
            else if (f == 14)
                xd += partials[b].vsum;
            else
                xl += partials[b].cnt[f - 15];
        }
        sd[t] = xd;
        sl[t] = xl;
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            if (t < o) {
                sd[t] += sd[t + o];
                sl[t] += sl[t + o];
            }
            __syncthreads();
        }
        if (t == 0) {
            if (f < 14)
                out->energy_sums[f] = sd[0];
            else if (f == 14)
                out->vel_sum = sd[0];
            else if (f == 15)
                out->n_p_plain = sl[0];
            else if (f == 16)
                out->n_p_weighted = sl[0];
            else if (f == 17)
                out->vel_count = sl[0];
            else
                out->n_near_tie = sl[0];
        }
        __syncthreads();
    }
    if (t == 0) {
        const long long listed = want_list ? (long long)*list_counter : 0;
        out->n_listed = listed < capacity ? listed : capacity;
        out->status = (want_list && listed > capacity) ? AXS_ERR_CAPACITY : AXS_OK;
    }
}

// Upper bound on the blocks a pass launches (the scratch is sized for it).
static int diag_grid(int64_t ncell)
{
    const int sms = device_sm_count();
    int64_t g = (ncell + kDiagThreads - 1) / kDiagThreads;
    const int64_t cap = (int64_t)(sms > 0 ? sms : 148) * 8;
    if (g > cap) g = cap;
    return (int)(g < 1 ? 1 : g);
}

// Work items (tile, z-chunk), tile fastest; chunks long enough to amortise
// the 4 warm-up planes while giving every resident block several items.
static void diag_plan(const DiagView &v, int nboxes, int max_grid, int tx, int ty, int blocks_per_sm, int &tiles_x,
                      int &ntiles, int &zchunk, long long &items_per_box, long long &items, int &grid)
{
    tiles_x = (v.nx + tx - 1) / tx;
    ntiles = tiles_x * ((v.ny + ty - 1) / ty);
    const int sms = device_sm_count() > 0 ? device_sm_count() : 148;
    const long long resident = (long long)blocks_per_sm * sms;
    const long long tiles_all = (long long)ntiles * nboxes;
    int nch = (int)std::max<long long>(1, (4 * resident + tiles_all - 1) / tiles_all);
    zchunk = std::max(1, (v.nz + nch - 1) / nch);
    if (zchunk < 16 && v.nz >= 16) zchunk = 16;
    if (zchunk > v.nz) zchunk = v.nz;
    items_per_box = (long long)ntiles * ((v.nz + zchunk - 1) / zchunk);
    items = items_per_box * nboxes;
    grid = (int)std::min<long long>(std::min<long long>(items, resident), max_grid);
}

// The string finder's work items (strip, z-chunk), strip fastest, one warp each: as many
// chunks as make the fullest warp's planes fewest (a chunk reads one plane more
// than it has cells, and starts with an empty pipeline).
struct FinderPlan {
    int strips_x, strips, zchunk, grid;
    long long items_per_box, items;
};
static FinderPlan finder_plan(const DiagView &v, int nboxes, int max_grid)
{
    constexpr int W = kDiagThreads / 32;
    FinderPlan f;
    f.strips_x = (v.nx + kStripW - 1) / kStripW;
    f.strips = f.strips_x * ((v.ny + kStripRows - 1) / kStripRows);
    const int sms = device_sm_count() > 0 ? device_sm_count() : 148;
    const long long warps = (long long)std::min(kFinderBlocks * sms, max_grid) * W, all = (long long)f.strips * nboxes;
    long long best = LLONG_MAX;
    f.zchunk = v.nz;
    for (int n = 1; n == 1 || (n <= 64 && v.nz / n >= 4); ++n) {
        const int len = (v.nz + n - 1) / n, chunks = (v.nz + len - 1) / len;
        const long long cost = (all * chunks + warps - 1) / warps * (len + 3);
        if (cost < best) {
            best = cost;
            f.zchunk = len;
        }
    }
    f.items_per_box = (long long)f.strips * ((v.nz + f.zchunk - 1) / f.zchunk);
    f.items = f.items_per_box * nboxes;
    f.grid = (int)std::min<long long>((f.items + W - 1) / W, std::min(kFinderBlocks * sms, max_grid));
    return f;
}

static int64_t diag_scratch_bytes(int64_t ncell) { return 256 + (int64_t)diag_grid(ncell) * sizeof(DiagPartial); }

static int run_diag(const DiagView &v, const axs_diag_params *p, const uint8_t *mask, axs_diag_result *out,
                    int64_t *list, int64_t capacity, void *scratch, int64_t scratch_bytes, cudaStream_t st,
                    int nboxes = 1, int64_t box_stride = 0, uint8_t *tags = nullptr)
{
    AXS_REQUIRE(p != nullptr && out != nullptr, AXS_ERR_INVALID_ARGUMENT, "null params or result");
    AXS_REQUIRE(p->dx > 0.0 && p->R > 0.0 && p->m_r > 0.0, AXS_ERR_INVALID_ARGUMENT,
                "dx, R and m_r must be positive");
    AXS_REQUIRE(p->masking_scheme >= AXS_MASK_NONE && p->masking_scheme <= AXS_MASK_B, AXS_ERR_INVALID_ARGUMENT,
                "bad masking scheme %d", p->masking_scheme);
    AXS_REQUIRE(capacity >= 0, AXS_ERR_INVALID_ARGUMENT, "negative list capacity");
    AXS_REQUIRE(capacity == 0 || list != nullptr, AXS_ERR_INVALID_ARGUMENT, "null list with positive capacity");
    AXS_REQUIRE(nboxes >= 1, AXS_ERR_INVALID_ARGUMENT, "no boxes");
    const int64_t ncell = (int64_t)v.nx * v.ny * v.nz * nboxes;
    const int64_t need = diag_scratch_bytes(ncell);
    AXS_REQUIRE(scratch != nullptr && scratch_bytes >= need, AXS_ERR_WORKSPACE,
                "diagnostics scratch too small (%lld < %lld bytes)", (long long)scratch_bytes, (long long)need);
    AXS_REQUIRE(((uintptr_t)scratch % 16) == 0, AXS_ERR_ALIGNMENT, "scratch must be 16-byte aligned");
    DiagConst q{};
    q.one_over_dx = 1.0 / p->dx;
    q.R = p->R;
    q.R2 = p->R * p->R;
    q.inv_R = 1.0 / p->R;
    q.inv_R2 = 1.0 / q.R2;
    q.inv_R4 = q.inv_R2 * q.inv_R2;
    {
        // Velocity.hpp:62-78: term1 = |phi'|^2/(2 m^2 c1^2) (1 - e1 |phi|^2/c1^3),
        //                     term2 = e1/(4 m^2 c1^5) (phi . phi')^2
        const double c1 = 0.41222, e1 = -0.025763, m2 = p->m_r * p->m_r, c1s = c1 * c1;
        q.vel_a = 1.0 / (2.0 * m2 * c1s);
        q.vel_b = e1 / (c1 * c1s);
        q.vel_c = e1 / (4.0 * m2 * c1s * c1s * c1);
    }
    q.lambda = p->lambda;
    q.RpR = p->R_prime_over_R;
    q.m_r = p->m_r;
    q.threshold = p->masking_threshold;
    q.scheme = p->masking_scheme;
    q.want_energy = p->want_energy != 0;
    q.want_plaq = p->want_plaquettes != 0;
    q.want_vel = p->want_velocity != 0;
    q.f_one_over_dx = (float)q.one_over_dx;
    q.f_k12h = (float)(q.one_over_dx / 12.0);
    q.f_k12l = (float)(q.one_over_dx / 12.0 - (double)q.f_k12h);
    q.f_R2 = (float)q.R2;
    q.f_inv_R = (float)q.inv_R;
    q.f_inv_R2 = (float)q.inv_R2;
    q.f_inv_R4 = (float)q.inv_R4;
    q.f_lambda = (float)q.lambda;
    q.f_RpR = (float)q.RpR;
    q.f_threshold = (float)q.threshold;
    q.f_vel_a = (float)q.vel_a;
    q.f_vel_b = (float)q.vel_b;
    q.f_vel_c = (float)q.vel_c;
    auto *counter = static_cast<unsigned long long *>(scratch);
    auto *partials = reinterpret_cast<DiagPartial *>(static_cast<char *>(scratch) + 256);
    AXS_CUDA_CHECK(cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st));
    int tiles_x, ntiles, zchunk, grid;
    long long items, items_per_box;
    long long *lst = (q.want_plaq && capacity > 0) ? reinterpret_cast<long long *>(list) : nullptr;
    int rc0 = AXS_OK;
    const bool offs31 = (int64_t)(v.ny + 2 * v.oy + 2) * v.js < INT_MAX;  // in-plane offsets in 31 bits
    const FinderPlan f = finder_plan(v, nboxes, diag_grid(ncell));
    auto launch_finder = [&](auto kern, int e_from) -> int {
        AXS_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FinderSmem)));
        kern<<<f.grid, kDiagThreads, sizeof(FinderSmem), st>>>(v, q, mask, partials, counter, lst, capacity, f.strips_x,
                                                               f.strips, f.zchunk, f.items, f.items_per_box, box_stride,
                                                               tags, e_from);
        return launch_status("string finder");
    };
    if (q.want_plaq && !q.want_energy && !q.want_vel && offs31) {
        // windings only
        rc0 = v.dtype != AXS_F64 ? launch_finder(finder_kernel<float, false>, 0)
                                 : launch_finder(finder_kernel<double, false>, 0);
        if (rc0) return rc0;
        diag_finalize_kernel<<<1, 256, 0, st>>>(partials, f.grid, counter, capacity, lst != nullptr, out);
        return launch_status("diagnostics finalize");
    }
    if (q.want_energy && v.dtype == AXS_F32 && p->per_cell_fp32 && offs31) {
        // per-cell FP32 terms: the energy sums (3 blocks per SM) and the windings, the
        // list and the velocity. Each kernel fills its own fields of the partial records
        // and clears the other's in those that the other has no block for.
        const bool strings = q.want_plaq || q.want_vel;
        diag_plan(v, nboxes, diag_grid(ncell), FTX, FTY, kEnergyBlocks, tiles_x, ntiles, zchunk, items_per_box, items, grid);
        const bool vec = (uintptr_t)v.data % 8 == 0 && (v.nx | v.ox | v.js | v.ks | v.cs | box_stride) % 2 == 0;
        (vec ? energy32_kernel<true> : energy32_kernel<false>)<<<grid, kDiagThreads, 0, st>>>(
            v, q, mask, partials, tiles_x, ntiles, zchunk, items, items_per_box, box_stride, strings ? f.grid : 0);
        if ((rc0 = launch_status("energy sums"))) return rc0;
        if (strings) {
            rc0 = q.want_vel ? launch_finder(finder_kernel<float, true>, grid)
                             : launch_finder(finder_kernel<float, false>, grid);
            if (rc0) return rc0;
        }
        diag_finalize_kernel<<<1, 256, 0, st>>>(partials, strings ? std::max(grid, f.grid) : grid, counter, capacity,
                                                lst != nullptr, out);
        return launch_status("diagnostics finalize");
    }
    diag_plan(v, nboxes, diag_grid(ncell), DTX, DTY, 2, tiles_x, ntiles, zchunk, items_per_box, items, grid);
    auto launch = [&](auto kern, size_t smem) -> int {
        AXS_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<grid, kDiagThreads, smem, st>>>(v, q, mask, partials, counter, lst, capacity, tiles_x, ntiles, zchunk,
                                               items, items_per_box, box_stride, tags);
        return AXS_OK;
    };
    if (v.dtype == AXS_F64)
        rc0 = launch(diag_kernel<double, false>, sizeof(DiagSmem<double, false>));
    else if (p->per_cell_fp32)
        rc0 = launch(diag_kernel<float, true>, sizeof(DiagSmem<float, true>));
    else
        rc0 = launch(diag_kernel<float, false>, sizeof(DiagSmem<float, false>));
    if (rc0) return rc0;
    int rc = launch_status("diagnostics");
    if (rc) return rc;
    diag_finalize_kernel<<<1, 256, 0, st>>>(partials, grid, counter, capacity, lst != nullptr, out);
    return launch_status("diagnostics finalize");
}

// One periodic box in level layout (an ensemble member), without the pierced list.
int diag_level_box(const void *data, int32_t dtype, int nx, int ny, int nz, const LevelGeom &g,
                   const axs_diag_params *p, axs_diag_result *out, void *scratch, int64_t scratch_bytes,
                   cudaStream_t st)
{
    DiagView v{data, dtype, nx, ny, nz, g.ox, g.oy, 0, 1, 1, 1, g.js, g.ks, g.cs};
    return run_diag(v, p, nullptr, out, nullptr, 0, scratch, scratch_bytes, st);
}

int64_t diag_scratch_bytes_for(int64_t ncell) { return diag_scratch_bytes(ncell); }

// The refinement tagger's plaquette criterion on a periodic level: the string
// finder's pass (same windings, bit for bit) writing one tag byte per cell
// (x fastest) instead of a pierced list. `out` is a device result record.
int diag_level_plaquette_tags(const void *state, int32_t dtype, int nx, int ny, int nz, const LevelGeom &g, double dx,
                              uint8_t *tags, axs_diag_result *out, void *scratch, int64_t scratch_bytes,
                              cudaStream_t st)
{
    DiagView v{state, dtype, nx, ny, nz, g.ox, g.oy, 0, 1, 1, 1, g.js, g.ks, g.cs};
    axs_diag_params p{};
    p.dx = dx;
    p.R = 1.0;
    p.m_r = 1.0;
    p.masking_scheme = AXS_MASK_NONE;
    p.boundary = AXS_BOUNDARY_PERIODIC;
    p.want_plaquettes = 1;
    return run_diag(v, &p, nullptr, out, nullptr, 0, scratch, scratch_bytes, st, 1, 0, tags);
}

// nboxes boxes of one geometry, box_stride elements apart, with explicit ghost
// layers (refined patches), summed into one result. A pierced-list entry is
// 4 * (q * nx * ny * nz + cell) + plane for box q.
int diag_ghost_boxes(const void *data, int32_t dtype, int nx, int ny, int nz, int ox, int oy, int oz, int64_t js,
                     int64_t ks, int64_t cs, int nboxes, int64_t box_stride, const axs_diag_params *p,
                     axs_diag_result *out, int64_t *list, int64_t capacity, void *scratch, int64_t scratch_bytes,
                     cudaStream_t st)
{
    DiagView v{data, dtype, nx, ny, nz, ox, oy, oz, 0, 0, 0, js, ks, cs};
    return run_diag(v, p, nullptr, out, list, capacity, scratch, scratch_bytes, st, nboxes, box_stride);
}

}  // namespace axs

using namespace axs;

extern "C" {

int axs_diagnostics_scratch_bytes(int32_t nx, int32_t ny, int32_t nz, int64_t *bytes)
{
    AXS_REQUIRE(bytes != nullptr, AXS_ERR_INVALID_ARGUMENT, "null output");
    AXS_REQUIRE(nx > 0 && ny > 0 && nz > 0, AXS_ERR_INVALID_ARGUMENT, "empty box");
    *bytes = diag_scratch_bytes((int64_t)nx * ny * nz);
    return AXS_OK;
}

int axs_diagnostics(const axs_fab *state, const axs_diag_params *p, const uint8_t *mask, axs_diag_result *out,
                    int64_t *list, int64_t capacity, void *scratch, int64_t scratch_bytes, void *stream)
{
    AXS_REQUIRE(p != nullptr, AXS_ERR_INVALID_ARGUMENT, "null params");
    const int periodic = p->boundary == AXS_BOUNDARY_PERIODIC;
    AXS_REQUIRE(p->boundary == AXS_BOUNDARY_GHOSTS || periodic, AXS_ERR_INVALID_ARGUMENT, "bad boundary mode");
    const int need_ng = periodic ? 0 : (p->want_energy ? 2 : 1);
    int rc = validate_fab(state, "state", 4, need_ng);
    if (rc) return rc;
    DiagView v{state->data, state->dtype, state->nx, state->ny, state->nz, state->ng, state->ng, state->ng,
               periodic, periodic, periodic, state->jstride, state->kstride, state->cstride};
    return run_diag(v, p, mask, out, list, capacity, scratch, scratch_bytes, (cudaStream_t)stream);
}

int axs_level_diagnostics(const axs_level *lv, const axs_diag_params *p, const uint8_t *mask, axs_diag_result *out,
                          int64_t *list, int64_t capacity, void *scratch, int64_t scratch_bytes, void *stream)
{
    LevelGeom g;
    AXS_REQUIRE(lv != nullptr && lv->state != nullptr, AXS_ERR_INVALID_ARGUMENT, "null level");
    int rc = level_geom(lv->dtype, lv->nx, lv->ny, lv->nz, g);
    if (rc) return rc;
    // indices wrap on every axis: the sweeps keep the x/y padding current but
    // not its corners, which the xy plaquette at (nx-1, ny-1) would read
    DiagView v{lv->state, lv->dtype, lv->nx, lv->ny, lv->nz, g.ox, g.oy, 0, 1, 1, 1, g.js, g.ks, g.cs};
    return run_diag(v, p, mask, out, list, capacity, scratch, scratch_bytes, (cudaStream_t)stream);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Diagnostics without caller-provided scratch.
//
// Some host codes cannot hand this library any extra device memory: an AMReX
// application, for instance, gives most of the GPU to its own arena at start-up
// and expects plugins to work inside the buffers they are passed, and other
// callers run under a fixed device-memory budget where a cudaMalloc from a
// plugin is not allowed. For them the diagnostics pass can use the scratch
// array below, a file-scope device array that every GPU loading this library
// holds until the process exits. Its size caps the per-block partials the pass
// needs (256 bytes of header + 160 bytes per block); on a 152-SM GB300 a pass
// uses at most 1216 blocks, i.e. about 195 KB of the 256 KiB.
namespace axs {
constexpr size_t kStaticDiagScratchBytes = 256 * 1024;
static __device__ __align__(256) unsigned char g_static_diag_scratch[kStaticDiagScratchBytes];

// Device address of g_static_diag_scratch, looked up once per device with that
// device current (host code must not use the symbol itself as an address).
static int static_scratch_address(void **out)
{
    constexpr int kMaxDevices = 64;
    static void *addr[kMaxDevices] = {};
    static std::mutex mu;
    int dev = 0;
    AXS_CUDA_CHECK(cudaGetDevice(&dev));
    AXS_REQUIRE(dev >= 0 && dev < kMaxDevices, AXS_ERR_UNSUPPORTED, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lock(mu);
    if (addr[dev] == nullptr) {
        void *p = nullptr;
        AXS_CUDA_CHECK(cudaGetSymbolAddress(&p, g_static_diag_scratch));
        addr[dev] = p;
    }
    *out = addr[dev];
    return AXS_OK;
}
}  // namespace axs

extern "C" {

int axs_diagnostics_static_scratch(const axs_fab *state, const axs_diag_params *p, const uint8_t *mask,
                                   axs_diag_result *result_dev, int64_t *pierced_dev, int64_t pierced_capacity,
                                   void *stream)
{
    AXS_REQUIRE(state != nullptr, AXS_ERR_INVALID_ARGUMENT, "null state");
    const int64_t ncell = (int64_t)state->nx * state->ny * state->nz;
    AXS_REQUIRE(ncell > 0, AXS_ERR_INVALID_ARGUMENT, "empty box");
    const int64_t need = diag_scratch_bytes(ncell);
    AXS_REQUIRE(need <= (int64_t)kStaticDiagScratchBytes, AXS_ERR_WORKSPACE,
                "diagnostics needs %lld scratch bytes on this device, more than the %lld-byte static array; "
                "use axs_diagnostics with caller-provided scratch",
                (long long)need, (long long)kStaticDiagScratchBytes);
    void *scratch = nullptr;
    int rc = static_scratch_address(&scratch);
    if (rc) return rc;
    // run_diag clears the list counter in the array before the pass; the
    // per-block partials are overwritten in full.
    return axs_diagnostics(state, p, mask, result_dev, pierced_dev, pierced_capacity, scratch,
                           (int64_t)kStaticDiagScratchBytes, stream);
}

}  // extern "C"
