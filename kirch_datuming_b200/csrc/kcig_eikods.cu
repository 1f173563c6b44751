// First-arrival traveltime tables on the GPU, the role of eikods2d
// (src/eikods2d.cpp:149-765, SERECKIRCH/src/eikods.cpp:66-211,
// SERECKIRCH/src/neighbors.cpp): for each source, the time T, its first
// derivatives with respect to the source position (tdl1 in the relative
// coordinate, tds1 in the source coordinate) and the branch-aware spatial
// gradients (gradz, gradx).
//
// eikods2d marches the front with a binary heap (fast marching).  Here every
// source's grid is solved by Gauss-Seidel sweeps in the four diagonal
// orderings, repeated until four consecutive sweeps change nothing, with the
// same local problem: the same constant-slowness box around the source
// (neighbors.cpp:418-484), the same first/second-order upwind quadratic in
// double precision (neighbors.cpp:106-188, 271-302) and the same rounding of
// every operation (explicit round-to-nearest intrinsics, no contraction).  For
// order 1 the update is monotone and the converged sweeps reach exactly the
// marching result; for order 2 the marching result also depends on the order
// in which the heap accepts points, and the two differ by up to ~2.5e-4 s at a
// fraction of the points.  The derivative recursion of eikods.cpp:119-211
// (each point from its upwind neighbours, in order of increasing time) is
// solved the same way: sweeps until nothing changes give exactly the ordered
// result.
//
// Execution: a CTA solves one source at a time, one anti-diagonal per step (the
// points of a diagonal depend on others' only), thread t taking rows t,
// t + blockDim, ...  Two sweep orderings run along the diagonals iz + ix =
// const, two along iz - ix = const, so every source's working values are kept
// in both diagonal-major layouts: the rows a step needs are contiguous and
// come by 16-byte cp.async into a shared-memory ring (diagonals p - 2 .. p + D
// around the current one), fetched D steps ahead.  A value that changes is
// written to the ring and to both layouts.  In the plain layout every row of
// a diagonal is a cache line of its own, and a sweep ran at one L1 wavefront
// per row and step: 400 sources of 601 x 1601 in 83 ms, 169 ms with
// tdl1/tds1, now 28 and 66 ms.
//
// Points whose inputs did not change since their previous evaluation are
// skipped (a stamp of the sweep of its last change beside every value), and
// so are whole blocks of diagonals without a change in reach: both change no
// result.  The quiet sweeps that end a pass cost only that test.  There is no
// wait other than the barriers and every loop has a fixed bound.
#include <float.h>
#include <math.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

#include "kcig_common.h"
#include "kcig_div.h"

namespace kcig {
namespace {

constexpr float kFar = FLT_MAX;  // not yet reached (neighbors.cpp:423-426)

struct EikSource {
    int st0, en0, st1, en1;  // constant-slowness box, inclusive and clamped to the grid
    int ic;                  // box centre (its slowness is the box's)
    float xs0, xs1, xs2;     // source minus origin: depth, lateral, third axis
};

// Reciprocals of the divisors of the local problem; [second order on axis 0]
// [on axis 1] of the two-axis sum, [axis][second order] of one axis
struct EikRecip {
    double two[2][2], one[2][2];
};

struct EikArgs {
    const float *vv;   // [2][nd + 2 kEikBorder][np] slowness squared, both layouts (skew_index)
    const double *dw;  // [2][nd + 2 kEikBorder][np] derivative of vv along axis l
    const float *vplain;  // [nx][nz]
    const EikSource *src;
    float *T, *dl1;    // [nsrc][nx][nz]
    unsigned char *work;  // per CTA: slot_bytes
    size_t slot_bytes;
    int *next;         // sources handed out so far
    int *status;       // set to 1 when a source has no fixed point within max_iter
    int *iters;        // [nsrc] sweeps the traveltime pass took (0: no fixed point)
    int nsrc, nz, nx, np, nd, order, max_iter;
    int blk_shift, nblk;  // diagonals per skipping block (a power of two), blocks
    float d0, d1, d2;  // sampling: depth, lateral, third axis
    float rdx0, rdx1;  // 1 / d^2 rounded to float (neighbors.cpp:19-30)
    DivF dd0, dd1;     // d^2 of both axes
    EikRecip rc;
};

// Diagonal-major layouts: family 0 holds diagonal p = iz + ix, family 1 p = iz
// - ix + nx - 1, each as a row of np >= nz + 2 entries (np a multiple of 16)
// indexed by iz; kEikBorder border rows before and after, and every entry
// outside the grid, keep the border value for good.
constexpr int kEikBorder = 8;
__host__ __device__ __forceinline__ size_t skew_row(int p, int np) { return (size_t)(p + kEikBorder) * np; }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint2 lds64(uint32_t addr)
{
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float lds32(uint32_t addr)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// neighbors.cpp:106-160 for one axis, with stencil() (:271-276): the
// smaller neighbour, or the second-order one-sided value when the sample two
// steps further is not larger.  a2 / b2 are kFar where that sample is outside
// the grid or not reached, which fails the comparisons exactly as the marching
// code's bounds and status checks do.
__device__ __forceinline__ bool upd_axis(float a, float b, float a2, float b2, int order, double &stencil, float &value)
{
    value = fminf(a, b);  // never NaN
    const double v = (double)value;
    const float t2 = (a < b) ? a2 : b2;
    const bool second = order > 1 && a != b && value >= t2;
    const double s2 = div_by(__fma_rn(4.0, v, -(double)t2), 3.0, 1.0 / 3.0);  // 4 v is exact
    stencil = second ? s2 : v;
    return second;
}

// neighbors.cpp:278-302 updaten() past its sums: root of A t^2 - 2 B t + C =
// v1, `false` if it is not above `value` (not causal)
__device__ __forceinline__ bool upd_root(double A, double B, double C, double y, double v1, float value, float &res)
{
    B = div_by(B, A, y);
    const double discr = __dadd_rn(__dmul_rn(B, B), div_by(__dsub_rn(v1, C), A, y));
    const double t = __dadd_rn(B, __dsqrt_rn(discr));
    res = __double2float_rn(t);
    return !(discr < 0.0) && !(t <= (double)value);
}

// neighbors.cpp:106-188 qsolve() on a 2-D grid (the third axis never
// contributes): the two-axis root, else the one of the smaller axis alone.
// (The sums over the axes do not depend on their order.)
__device__ __forceinline__ float qsolve2d(float zm, float zp, float zm2, float zp2, float xm, float xp, float xm2,
                                          float xp2, float vv, float rdx0, float rdx1, int order, const EikRecip &rc)
{
    double s0, s1;
    float v0, v1;
    const bool o0 = upd_axis(zm, zp, zm2, zp2, order, s0, v0), o1 = upd_axis(xm, xp, xm2, xp2, order, s1, v1);
    const double d0 = o0 ? __dmul_rn((double)rdx0, 2.25) : (double)rdx0;
    const double d1 = o1 ? __dmul_rn((double)rdx1, 2.25) : (double)rdx1;
    const double b0 = __dmul_rn(s0, d0), b1 = __dmul_rn(s1, d1);
    const double c0 = __dmul_rn(__dmul_rn(s0, s0), d0), c1 = __dmul_rn(__dmul_rn(s1, s1), d1);
    // the marching code sorts the axes by value: the first keeps its place
    // unless the second is smaller
    const bool swap = !(v0 <= v1);
    const float lo = swap ? v1 : v0, hi = swap ? v0 : v1;
    const double w = (double)vv;
    float t;
    if (upd_root(__dadd_rn(d0, d1), __dadd_rn(b0, b1), __dadd_rn(c0, c1),
                 o0 ? (o1 ? rc.two[1][1] : rc.two[1][0]) : (o1 ? rc.two[0][1] : rc.two[0][0]), w, hi, t) &&
        hi < kFar)
        return t;
    if (upd_root(swap ? d1 : d0, swap ? b1 : b0, swap ? c1 : c0,
                 swap ? (o1 ? rc.one[1][1] : rc.one[1][0]) : (o0 ? rc.one[0][1] : rc.one[0][0]), w, lo, t) &&
        lo < kFar)
        return t;
    return kFar;
}

// ------------------------------------------------------------- kernels --

__global__ void k_slowness2(const float *__restrict__ vel, float *__restrict__ vv, size_t n, int is_slowness2)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float v = vel[i];
    // eikods2d.cpp:325-335: v = 1 / (v * v) with the product in float
    vv[i] = is_slowness2 ? v : __double2float_rn(__ddiv_rn(1.0, (double)__fmul_rn(v, v)));
}

// derivative of slowness squared along axis l (eikods.cpp:197-204)
__global__ void k_dw(const float *__restrict__ vv, double *__restrict__ dw, int nz, int nx, int l, float dl)
{
    const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i0 >= (size_t)nz * nx) return;
    const int ii = l == 0 ? (int)(i0 % nz) : (int)(i0 / nz), n = l == 0 ? nz : nx;
    const size_t s = l == 0 ? 1 : (size_t)nz;
    const double den = __dmul_rn(2.0, (double)dl);
    double w;
    if (0 < ii && ii < n - 1) {
        w = __ddiv_rn((double)__fsub_rn(vv[i0 + s], vv[i0 - s]), den);
    } else if (ii == 0) {
        const double u = __dadd_rn(-(double)vv[i0 + 2 * s], __dmul_rn(4.0, (double)vv[i0 + s]));
        w = __ddiv_rn(__dsub_rn(u, __dmul_rn(3.0, (double)vv[i0])), den);
    } else {
        const double u = __dsub_rn(__dmul_rn(3.0, (double)vv[i0]), __dmul_rn(4.0, (double)vv[i0 - s]));
        w = __ddiv_rn(__dadd_rn(u, (double)vv[i0 - 2 * s]), den);
    }
    dw[i0] = w;
}

// a plain [nx][nz] array into both layouts, `border` outside the grid
template <class V>
__global__ void k_skew(const V *__restrict__ in, V *__restrict__ out, int nz, int nx, int np, int nd, V border)
{
    const int iz = blockIdx.y * blockDim.x + threadIdx.x, p = (int)blockIdx.x - kEikBorder, fam = blockIdx.z;
    if (iz >= np) return;
    const int ix = fam == 0 ? p - iz : iz + nx - 1 - p;
    out[((size_t)fam * (nd + 2 * kEikBorder)) * np + skew_row(p, np) + iz] =
        iz < nz && ix >= 0 && ix < nx ? in[(size_t)ix * nz + iz] : border;
}

constexpr int kEikS = 8, kEikD = 5;  // ring slots (a power of two), prefetch distance: kEikS >= kEikD + 3
static_assert((kEikS & (kEikS - 1)) == 0 && kEikS >= kEikD + 3 && kEikD >= 3, "ring too small");
static_assert(kEikBorder >= kEikD + 1, "the last steps fetch border rows");
constexpr int kEikPad = 2;           // rows -2, -1 in front of a ring row (16 bytes of pairs)

// bytes of one CTA's working values: {value, stamp} pairs in both layouts,
// and with derivatives the final time in both
inline size_t eik_slot_bytes(int nd, int np, bool deriv)
{
    return 2 * (size_t)(nd + 2 * kEikBorder) * np * (deriv ? 12 : 8);
}
// shared memory: the pair ring, the time ring (derivative pass; its border
// pads four floats), the blocks' last changes
inline size_t eik_smem(int np, int nblk, bool deriv)
{
    const size_t rings = (size_t)kEikS * ((np + kEikPad) * 8 + (deriv ? (np + 4) * 4 : 0)) + 2 * (size_t)nblk * 4;
    return std::max(rings, (size_t)32 * 33 * 4);  // at least one window of eik_unskew
}

// What a sweep works on: one source's pairs ({value, stamp}: the time or tdl1,
// and 1 + the sweep of its last change, 0: none) and final times in both
// layouts, the rings, the blocks' last changes.
struct EikMem {
    uint2 *W;
    const float *TT;
    uint2 *RP;
    float *RT;
    unsigned *last;
};

// One sweep along the diagonals of family FAM, ST = +1 or -1 its direction.
// MODE 0: traveltime; MODE 1: the source derivative recursion on the final
// traveltime.  Every address advances by a constant per step and the ring
// slots rotate through registers: the loop is bound by instructions (a point
// takes 2.9 evaluations a pass on the salt model, 30 of 32 lanes busy) and by
// the serial chain of one step.  One CTA of 19 warps without spills per SM is
// as fast for 400 sources as two at 48 registers (66 ms against 78) and faster
// for 148 (28 against 38), with half the working memory.
template <int MODE, int ROWS, int FAM, int ST>
__device__ __forceinline__ bool eik_sweep(const EikArgs &a, const EikSource &sc, const EikMem &m, int sweep)
{
    const int nz = a.nz, nx = a.nx, np = a.np, nd = a.nd, nthr = blockDim.x, tid = threadIdx.x;
    const int NR = np + kEikPad, NT = np + 4;
    const size_t fam_len = (size_t)(nd + 2 * kEikBorder) * np;
    uint2 *Wf = m.W + FAM * fam_len, *Wo = m.W + (1 - FAM) * fam_len;
    const unsigned *lastf = m.last + FAM * a.nblk;
    const uint32_t rp = (uint32_t)__cvta_generic_to_shared(m.RP + kEikPad), rt = (uint32_t)__cvta_generic_to_shared(m.RT + 4);
    const bool f_on = tid < np / 2, g_on = MODE == 1 && tid < np / 4;  // blockDim >= np / 2 (the launcher)
    bool changed = false, piped = false;
    for (int bi = 0; bi < a.nblk; bi++) {
        const int blk = ST > 0 ? bi : a.nblk - 1 - bi;
        // a change of this sweep or the one before, here or next door
        // (blocks are at least as long as the stencil's reach)
        bool need = sweep == 0 || lastf[blk] >= (unsigned)sweep;
        if (!need && blk > 0) need = lastf[blk - 1] >= (unsigned)sweep;
        if (!need && blk + 1 < a.nblk) need = lastf[blk + 1] >= (unsigned)sweep;
        if (!need) {
            piped = false;
            continue;
        }
        const int b0 = blk << a.blk_shift, b1 = min(nd, b0 + (1 << a.blk_shift));
        const int p0 = ST > 0 ? b0 : b1 - 1, n = b1 - b0;
        // diagonal p sits in ring slot p mod kEikS; its rows are fetched kEikD steps ahead
        const uint2 *src = Wf + skew_row(p0 + ST * kEikD, np) + 2 * tid;
        const float *srcT = MODE == 1 ? m.TT + FAM * fam_len + skew_row(p0 + ST * kEikD, np) + 4 * tid : nullptr;
        if (!piped) {  // fill the ring
            cp_wait<0>();
            __syncthreads();
            for (int q = -2; q < kEikD; q++) {
                const int p = p0 + ST * q, slot = p & (kEikS - 1);
                if (f_on) cp_async16(rp + (slot * NR + 2 * tid) * 8, Wf + skew_row(p, np) + 2 * tid);
                if (g_on) cp_async16(rt + (slot * NT + 4 * tid) * 4, m.TT + FAM * fam_len + skew_row(p, np) + 4 * tid);
            }
            cp_commit();
            cp_wait<0>();
            __syncthreads();
            piped = true;
        }
        // slots of p + ST d, d = -2 .. 2, as byte offsets of a row's first pair
        uint32_t o[5];
#pragma unroll
        for (int d = 0; d < 5; d++) o[d] = (uint32_t)((p0 + ST * (d - 2)) & (kEikS - 1)) * (uint32_t)NR * 8u;
        uint32_t oD = (uint32_t)((p0 + ST * kEikD) & (kEikS - 1));  // slot being fetched
        const float *vp = a.vv + FAM * fam_len + skew_row(p0, np) + tid;
        const double *wp = MODE == 1 ? a.dw + FAM * fam_len + skew_row(p0, np) + tid : nullptr;
        float v_nxt[ROWS];  // the model's values one step ahead
        double w_nxt[ROWS];
#pragma unroll
        for (int qr = 0; qr < ROWS; qr++) {
            const bool in = tid + qr * nthr < np;
            if (MODE == 0) v_nxt[qr] = in ? __ldg(vp + qr * nthr) : 0.0f;
            else w_nxt[qr] = in ? __ldg(wp + qr * nthr) : 0.0;
        }
        int p = p0;
        for (int k = 0; k < n; k++, p += ST) {
            if (f_on) cp_async16(rp + oD * (uint32_t)NR * 8u + tid * 16, src);
            src += ST * np;
            if (MODE == 1) {
                if (g_on) cp_async16(rt + oD * (uint32_t)NT * 4u + tid * 16, srcT);
                srcT += ST * np;
            }
            oD = (oD + (uint32_t)ST) & (kEikS - 1);
            cp_commit();
            float v_cur[ROWS];
            double w_cur[ROWS];
            if (MODE == 0) vp += ST * np;
            else wp += ST * np;
#pragma unroll
            for (int qr = 0; qr < ROWS; qr++) {
                const bool in = tid + qr * nthr < np;
                if (MODE == 0) {
                    v_cur[qr] = v_nxt[qr];
                    if (in) v_nxt[qr] = __ldg(vp + qr * nthr);
                } else {
                    w_cur[qr] = w_nxt[qr];
                    if (in) w_nxt[qr] = __ldg(wp + qr * nthr);
                }
            }
            // physical diagonals p - 2 .. p + 2, and the two an x step leads to
            const uint32_t m2 = ST > 0 ? o[0] : o[4], m1 = ST > 0 ? o[1] : o[3];
            const uint32_t p1 = ST > 0 ? o[3] : o[1], p2 = ST > 0 ? o[4] : o[0];
#pragma unroll
            for (int qr = 0; qr < ROWS; qr++) {
                const int iz = tid + qr * nthr, ix = FAM ? iz + nx - 1 - p : p - iz;
                if (iz >= nz || (unsigned)ix >= (unsigned)nx) continue;
                const uint32_t r = rp + iz * 8;
                const uint2 zm = lds64(r + m1 - 8), zp = lds64(r + p1 + 8);
                const uint2 xm = lds64(r + (FAM ? p1 : m1)), xp = lds64(r + (FAM ? m1 : p1));
                unsigned snew = max(max(zm.y, zp.y), max(xm.y, xp.y));
                float nv;
                if (MODE == 0) {
                    const uint2 zm2 = lds64(r + m2 - 16), zp2 = lds64(r + p2 + 16);
                    const uint2 xm2 = lds64(r + (FAM ? p2 : m2)), xp2 = lds64(r + (FAM ? m2 : p2));
                    snew = max(snew, max(max(zm2.y, zp2.y), max(xm2.y, xp2.y)));
                    // inputs as at its previous evaluation: it would come out the same
                    if (sweep > 0 && snew < (unsigned)sweep) continue;
                    const bool in_box = iz >= sc.st0 && iz <= sc.en0 && ix >= sc.st1 && ix <= sc.en1;
                    if (in_box) continue;
                    nv = qsolve2d(__uint_as_float(zm.x), __uint_as_float(zp.x), __uint_as_float(zm2.x),
                                  __uint_as_float(zp2.x), __uint_as_float(xm.x), __uint_as_float(xp.x),
                                  __uint_as_float(xm2.x), __uint_as_float(xp2.x), v_cur[qr], a.rdx0, a.rdx1, a.order, a.rc);
                    if (!(nv < __uint_as_float(lds64(r + o[2]).x))) continue;
                } else {
                    if (sweep > 0 && snew < (unsigned)sweep) continue;
                    // eikods.cpp:149-211 (eikods_dt1) for one point, branch-free; tds1 follows from the
                    // final tdl1 (k_tds1)
                    const uint32_t q = (uint32_t)NT * 4u, t = rt + iz * 4;
                    const uint32_t tm = ((p - 1) & (kEikS - 1)) * q, tp = ((p + 1) & (kEikS - 1)) * q;
                    const float t0 = lds32(t + (p & (kEikS - 1)) * q);
                    double rhs = 0.0, den = 0.0;
                    float e[2], el[2];  // of an axis without an upwind neighbour: not used
                    bool up[2], quick = true;
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        const int ii = j == 0 ? iz : ix, len = j == 0 ? nz : nx;
                        const float ta = lds32(j == 0 ? t + tm - 4 : t + (FAM ? tp : tm));
                        const float tb = lds32(j == 0 ? t + tp + 4 : t + (FAM ? tm : tp));
                        const float la = __uint_as_float(j == 0 ? zm.x : xm.x);
                        const float lb = __uint_as_float(j == 0 ? zp.x : xp.x);
                        const bool use_b = ii == 0 || (ii != len - 1 && ta > tb);
                        const float t1 = use_b ? tb : ta, l1 = use_b ? lb : la;
                        const DivF &dd = j == 0 ? a.dd0 : a.dd1;
                        up[j] = t1 < t0;
                        e[j] = up[j] ? __fsub_rn(t0, t1) : 1.0f;
                        el[j] = __fmul_rn(e[j], l1);
                        quick = quick && div_quick(e[j], dd) && (div_quick(el[j], dd) || el[j] == 0.0f);
                    }
                    // one test for the point's four divisions (never-reached times, infinite slopes)
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        const DivF &dd = j == 0 ? a.dd0 : a.dd1;
                        const double term = (double)(quick ? div_known(el[j], dd) : __fdiv_rn(el[j], dd.div));
                        const double dterm = (double)(quick ? div_known(e[j], dd) : __fdiv_rn(e[j], dd.div));
                        rhs = up[j] ? __dadd_rn(rhs, term) : rhs;
                        den = up[j] ? __dadd_rn(den, dterm) : den;
                    }
                    nv = den != 0.0 ? __double2float_rn(__ddiv_rn(__dadd_rn(__dmul_rn(0.5, w_cur[qr]), rhs), den)) : 0.0f;
                    if (!(nv != __uint_as_float(lds64(r + o[2]).x))) continue;
                }
                const uint2 e = make_uint2(__float_as_uint(nv), (unsigned)sweep + 1u);
                const int op = FAM ? iz + ix : iz - ix + nx - 1;
                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(r + o[2]), "r"(e.x), "r"(e.y) : "memory");
                Wf[skew_row(p, np) + iz] = e;
                Wo[skew_row(op, np) + iz] = e;
                m.last[FAM * a.nblk + blk] = e.y;
                m.last[(1 - FAM) * a.nblk + (op >> a.blk_shift)] = e.y;
                changed = true;
            }
            const uint32_t nxt = (uint32_t)((p + 3 * ST) & (kEikS - 1)) * (uint32_t)NR * 8u;
            o[0] = o[1];
            o[1] = o[2];
            o[2] = o[3];
            o[3] = o[4];
            o[4] = nxt;
            cp_wait<kEikD - 3>();
            __syncthreads();
        }
    }
    cp_wait<0>();
    return __syncthreads_or(changed) != 0;
}

// One pass over one source: sweeps in the four orderings (z+ x+), (z- x+),
// (z+ x-), (z- x-) until each has changed nothing.  Returns the sweeps it
// took, 0 without a fixed point.
template <int MODE, int ROWS>
__device__ __forceinline__ int eik_pass(const EikArgs &a, const EikSource &sc, const EikMem &m)
{
    const int nthr = blockDim.x, tid = threadIdx.x;
    const unsigned border = MODE == 0 ? __float_as_uint(kFar) : 0u;
    for (int q = tid; q < kEikS * kEikPad; q += nthr)
        m.RP[(q / kEikPad) * (a.np + kEikPad) + q % kEikPad] = make_uint2(border, 0u);
    if (MODE == 1)
        for (int q = tid; q < kEikS * 4; q += nthr) m.RT[(q >> 2) * (a.np + 4) + (q & 3)] = kFar;
    for (int q = tid; q < 2 * a.nblk; q += nthr) m.last[q] = 0u;
    __syncthreads();
    int quiet = 0;
    for (int sweep = 0; sweep < 4 * a.max_iter; sweep++) {
        bool any;
        switch (sweep & 3) {
        case 0: any = eik_sweep<MODE, ROWS, 0, 1>(a, sc, m, sweep); break;
        case 1: any = eik_sweep<MODE, ROWS, 1, -1>(a, sc, m, sweep); break;
        case 2: any = eik_sweep<MODE, ROWS, 1, 1>(a, sc, m, sweep); break;
        default: any = eik_sweep<MODE, ROWS, 0, -1>(a, sc, m, sweep); break;
        }
        quiet = any ? 0 : quiet + 1;
        // four quiet sweeps in a row (one of each ordering): a fixed point
        if (quiet >= 4) return sweep + 1;
    }
    return 0;
}

// The values of a layout-0 pair array into the plain [nx][nz] order: a warp
// takes 32 rows and walks the diagonals, a window of 32 of them in shared
// memory (33 floats a row); column ix of the rows is complete once diagonal
// ix + r0 + 31 has been read.  Reads and writes are whole 32-row segments.
__device__ __forceinline__ void eik_unskew(const uint2 *W, float *out, int nz, int nx, int np, int nd, float *sh,
                                           int warps)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp >= warps) return;
    float *win = sh + warp * 32 * 33;
    for (int r0 = warp * 32; r0 < nz; r0 += warps * 32) {
        const int row = min(r0 + lane, np - 1);
        const int d1 = r0 + 31 + nx;  // one past the last diagonal read
        constexpr int U = 16;  // diagonals in flight
        for (int d = r0; d < d1; d += U) {
            float v[U];
#pragma unroll
            for (int q = 0; q < U; q++)
                v[q] = __uint_as_float(__ldcg(&W[skew_row(min(d + q, nd + kEikBorder - 1), np) + row].x));
#pragma unroll
            for (int q = 0; q < U; q++) {
                if (d + q >= d1) break;
                win[((d + q) & 31) * 33 + lane] = v[q];
                __syncwarp();
                const int ix = d + q - r0 - 31;
                if (ix >= 0 && r0 + lane < nz) out[(size_t)ix * nz + r0 + lane] = win[((ix + r0 + lane) & 31) * 33 + lane];
                __syncwarp();
            }
        }
    }
}

// Sources one after another per CTA: the time pass, its result to the plain
// layout, then (DERIV) the derivative pass in the same working memory.  RPT:
// rows per thread; MAXT: the block sizes it is compiled for.
template <int RPT, int MAXT, bool DERIV>
__global__ void __launch_bounds__(MAXT) k_eik_solve(const EikArgs a)
{
    extern __shared__ __align__(16) unsigned char eik_smem_raw[];
    __shared__ int cur;
    const int nz = a.nz, nx = a.nx, np = a.np, nd = a.nd, nthr = blockDim.x, tid = threadIdx.x;
    uint2 *RP = reinterpret_cast<uint2 *>(eik_smem_raw);                       // [kEikS][np + kEikPad]
    float *RT = reinterpret_cast<float *>(RP + kEikS * (np + kEikPad));        // [kEikS][np + 4] (DERIV)
    unsigned *last = reinterpret_cast<unsigned *>(RT + (DERIV ? kEikS * (np + 4) : 0));
    const size_t fam_len = (size_t)(nd + 2 * kEikBorder) * np;
    uint2 *W = reinterpret_cast<uint2 *>(a.work + (size_t)blockIdx.x * a.slot_bytes);
    float *TT = reinterpret_cast<float *>(W + 2 * fam_len);
    const int uwarps = max(1, min(nthr / 32, (int)((unsigned)(kEikS * (np + kEikPad) * 8) / (32 * 33 * 4))));
    for (;;) {
        if (tid == 0) cur = atomicAdd(a.next, 1);
        __syncthreads();
        const int js = cur;
        __syncthreads();
        if (js >= a.nsrc) return;
        const EikSource sc = a.src[js];
        const size_t nzx = (size_t)nz * nx;
        // initial state: nothing reached, the box at straight-ray times
        // (neighbors.cpp:418-484)
        const unsigned far = __float_as_uint(kFar);
        for (size_t i = tid; i < fam_len; i += nthr) reinterpret_cast<uint4 *>(W)[i] = make_uint4(far, 0u, far, 0u);
        __syncthreads();
        {
            const double v1 = (double)a.vplain[sc.ic];
            const int bz = sc.en0 - sc.st0 + 1, nb = bz * (sc.en1 - sc.st1 + 1);
            for (int q = tid; q < nb; q += nthr) {
                const int iz = sc.st0 + q % bz, iy = sc.st1 + q / bz;
                const double e0 = (double)__fsub_rn(sc.xs0, __fmul_rn((float)iz, a.d0));
                const double e1 = (double)__fsub_rn(sc.xs1, __fmul_rn((float)iy, a.d1));
                const double e2 = (double)__fsub_rn(sc.xs2, __fmul_rn(0.0f, a.d2));
                double d2 = __dadd_rn(0.0, __dmul_rn(e0, e0));
                d2 = __dadd_rn(d2, __dmul_rn(e1, e1));
                d2 = __dadd_rn(d2, __dmul_rn(e2, e2));
                const uint2 e = make_uint2(__float_as_uint(__fsqrt_rn(__double2float_rn(__dmul_rn(v1, d2)))), 0u);
                W[skew_row(iz + iy, np) + iz] = e;
                W[fam_len + skew_row(iz - iy + nx - 1, np) + iz] = e;
            }
        }
        __syncthreads();
        const EikMem mem = {W, TT, RP, RT, last};
        const int n = eik_pass<0, RPT>(a, sc, mem);
        if (tid == 0) {
            a.iters[js] = n;
            if (n == 0) atomicExch(a.status, 1);
        }
        __syncthreads();
        eik_unskew(W, a.T + (size_t)js * nzx, nz, nx, np, nd, reinterpret_cast<float *>(RP), uwarps);
        __syncthreads();
        if (DERIV) {
            // two pairs a thread, eight loads in flight (fam_len is a multiple of 16)
            uint4 *W4 = reinterpret_cast<uint4 *>(W);
            uint2 *T2 = reinterpret_cast<uint2 *>(TT);
            for (size_t i = tid; i < fam_len; i += 8 * (size_t)nthr) {
                uint4 v[8];
#pragma unroll
                for (int q = 0; q < 8; q++)
                    if (i + q * (size_t)nthr < fam_len) v[q] = W4[i + q * (size_t)nthr];
#pragma unroll
                for (int q = 0; q < 8; q++)
                    if (i + q * (size_t)nthr < fam_len) {
                        T2[i + q * (size_t)nthr] = make_uint2(v[q].x, v[q].z);
                        W4[i + q * (size_t)nthr] = make_uint4(0u, 0u, 0u, 0u);
                    }
            }
            __syncthreads();
            if (eik_pass<1, RPT>(a, sc, mem) == 0 && tid == 0) atomicExch(a.status, 1);
            __syncthreads();
            eik_unskew(W, a.dl1 + (size_t)js * nzx, nz, nx, np, nd, reinterpret_cast<float *>(RP), uwarps);
            __syncthreads();
        }
    }
}

// tds1 from the final time and tdl1 (eikods.cpp:149-211): tdl1 minus the
// time's derivative along axis l where the point has an upwind neighbour
__global__ void k_tds1(const float *__restrict__ T, const float *__restrict__ dl1, float *__restrict__ ds1, int nz,
                       int nx, int l, float d0, float d1)
{
    const size_t nzx = (size_t)nz * nx;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nzx) return;
    const float *t = T + (size_t)blockIdx.y * nzx;
    const size_t o = (size_t)blockIdx.y * nzx + i;
    const int iz = (int)(i % nz), ix = (int)(i / nz);
    const float t0 = t[i];
    double den = 0.0, dt = 0.0;
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const int ii = j == 0 ? iz : ix, n = j == 0 ? nz : nx;
        const size_t s = j == 0 ? 1 : (size_t)nz;
        const float dj = j == 0 ? d0 : d1;
        const float ta = ii > 0 ? t[i - s] : kFar, tb = ii < n - 1 ? t[i + s] : kFar;
        const bool use_b = ii == 0 || (ii != n - 1 && ta > tb);
        const float t1 = use_b ? tb : ta;
        const bool up = t1 < t0;
        const double dterm = (double)__fdiv_rn(__fsub_rn(t0, t1), __fmul_rn(dj, dj));
        den = up ? __dadd_rn(den, dterm) : den;
        if (l == j) {
            const float ta2 = ii > 1 ? t[i - 2 * s] : kFar, tb2 = ii < n - 2 ? t[i + 2 * s] : kFar;
            const float t2 = use_b ? tb2 : ta2;
            const bool three = use_b ? (ii < n - 2 && t1 > tb2) : (ii > 1 && t1 > ta2);
            const double num3 = use_b ? __dsub_rn(__dadd_rn(-(double)t2, __dmul_rn(4.0, (double)t1)),
                                                  __dmul_rn(3.0, (double)t0))
                                      : __dadd_rn(__dsub_rn(__dmul_rn(3.0, (double)t0), __dmul_rn(4.0, (double)t1)),
                                                  (double)t2);
            const double d3 = __ddiv_rn(num3, __dmul_rn(2.0, (double)dj));
            const double d2p = (double)__fdiv_rn(use_b ? __fsub_rn(t1, t0) : __fsub_rn(t0, t1), dj);
            dt = up ? (three ? d3 : d2p) : dt;
        }
    }
    ds1[o] = den != 0.0 ? __double2float_rn(__dsub_rn((double)dl1[o], dt)) : 0.0f;
}

// branch-aware spatial gradient along one axis (eikods2d.cpp:30-68)
__device__ __forceinline__ float upwind_grad(const float *t, size_t i0, int ii, int n, size_t s, float dd)
{
    const size_t a = i0 - s, b = i0 + s;
    size_t i1;
    if (ii == 0) i1 = b;
    else if (ii != n - 1 && t[b] < t[a]) i1 = b;
    else i1 = a;
    if (!(t[i1] < t[i0])) return 0.0f;
    const float two_d = __fmul_rn(2.0f, dd);
    if (i1 == b) {
        if (ii < n - 2 && t[i1 + s] < t[i1]) {
            const float u = __fadd_rn(-t[i1 + s], __fmul_rn(4.0f, t[i1]));
            return __fdiv_rn(__fsub_rn(u, __fmul_rn(3.0f, t[i0])), two_d);
        }
        return __fdiv_rn(__fsub_rn(t[i1], t[i0]), dd);
    }
    if (ii > 1 && t[i1 - s] < t[i1]) {
        const float u = __fsub_rn(__fmul_rn(3.0f, t[i0]), __fmul_rn(4.0f, t[i1]));
        return __fdiv_rn(__fadd_rn(u, t[i1 - s]), two_d);
    }
    return __fdiv_rn(__fsub_rn(t[i0], t[i1]), dd);
}

__global__ void k_upwind_grads(const float *__restrict__ T, float *__restrict__ gz, float *__restrict__ gx, int nz,
                               int nx, float dz, float dx)
{
    const size_t nzx = (size_t)nz * nx;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nzx) return;
    const float *t = T + (size_t)blockIdx.y * nzx;
    const size_t o = (size_t)blockIdx.y * nzx + i;
    const int iz = (int)(i % nz), ix = (int)(i / nz);
    if (gz) gz[o] = upwind_grad(t, i, iz, nz, 1, dz);
    if (gx) gx[o] = upwind_grad(t, i, ix, nx, (size_t)nz, dx);
}

// host side of neighbors.cpp:428-445: the box around the source, in the
// reference's own float arithmetic
EikSource source_box(float s0, float s1, float s2, float o0, float o1, float o2, float d0, float d1, int nz, int nx,
                     int b0, int b1)
{
    const float xs[3] = {s0 - o0, s1 - o1, s2 - o2};
    const float d[2] = {d0, d1};
    const int n[2] = {nz, nx}, b[2] = {b0, b1};
    int st[3], en[3];
    for (int j = 0; j < 2; j++) {
        const int is = (int)(xs[j] / d[j] + 0.5);
        st[j] = is - b[j];
        en[j] = is + b[j];
        st[j] = st[j] < 0 ? 0 : (st[j] >= n[j] ? n[j] - 1 : st[j]);
        en[j] = en[j] < 0 ? 0 : (en[j] >= n[j] ? n[j] - 1 : en[j]);
    }
    st[2] = en[2] = 0;  // a 2-D grid: the third axis clamps to its one sample
    EikSource e;
    e.st0 = st[0];
    e.en0 = en[0];
    e.st1 = st[1];
    e.en1 = en[1];
    e.ic = (st[0] + en[0]) / 2 + n[0] * ((st[1] + en[1]) / 2 + n[1] * (st[2] + en[2]) / 2);
    e.xs0 = xs[0];
    e.xs1 = xs[1];
    e.xs2 = xs[2];
    return e;
}

struct DevBuf {
    void *p = nullptr;
    cudaStream_t st = nullptr;
    ~DevBuf()
    {
        if (p) cudaFreeAsync(p, st);
    }
};

// The calls' device memory comes from a stream-ordered pool of the library,
// one per device, that keeps up to a sixteenth of the device between calls
// (mapping and unmapping memory anew cost more than the solve on small
// grids: ~16 ms per GB).  On a device with less than a 32nd free (5.7 GB) a call
// gives back what it used (kEikKeep at most stays); the library's other
// allocations take it back when they fail, and eik_release_pool at any time.
constexpr uint64_t kEikKeep = 256ull << 20;
std::mutex g_pool_mu;
std::map<int, cudaMemPool_t> g_pools;

int eik_pool(cudaMemPool_t *out)
{
    int dev = 0;
    KCIG_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(g_pool_mu);
    auto it = g_pools.find(dev);
    if (it == g_pools.end()) {
        cudaMemPoolProps pr = {};
        pr.allocType = cudaMemAllocationTypePinned;
        pr.location.type = cudaMemLocationTypeDevice;
        pr.location.id = dev;
        cudaMemPool_t pool;
        KCIG_CUDA(cudaMemPoolCreate(&pool, &pr));
        cudaDeviceProp dp;
        KCIG_CUDA(cudaGetDeviceProperties(&dp, dev));
        uint64_t keep = (uint64_t)dp.totalGlobalMem / 16;
        KCIG_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
        it = g_pools.emplace(dev, pool).first;
    }
    *out = it->second;
    return KCIG_OK;
}

// memory the pool holds and no call uses
size_t eik_pool_idle(cudaMemPool_t pool)
{
    uint64_t held = 0, used = 0;
    cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &held);
    cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used);
    return held > used ? held - used : 0;
}

// Gives back what a call leaves in the pool where the device is `full`.
// Declared before the call's buffers, so that they have been freed by then.
struct PoolSettle {
    cudaMemPool_t pool;
    cudaStream_t st;
    bool full = false;
    ~PoolSettle()
    {
        if (!full || cudaStreamSynchronize(st) != cudaSuccess) return;
        cudaMemPoolTrimTo(pool, kEikKeep);
        cudaGetLastError();
    }
};

// Whether the device is nearly full without what the pool holds idle; fr: what
// is free with it.  (A query takes ~0.15 ms: calls below kEikKeep go without.)
int eik_device_full(cudaMemPool_t pool, size_t *fr, bool *full)
{
    size_t tot = 0;
    KCIG_CUDA(cudaMemGetInfo(fr, &tot));
    *full = *fr < tot / 32;
    *fr += eik_pool_idle(pool);
    return KCIG_OK;
}

}  // namespace

int eik_release_pool()
{
    int dev = 0;
    KCIG_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(g_pool_mu);
    auto it = g_pools.find(dev);
    if (it != g_pools.end()) KCIG_CUDA(cudaMemPoolTrimTo(it->second, 0));
    return KCIG_OK;
}
}  // namespace kcig

using namespace kcig;

extern "C" int kcig_eikods(const float *vel, int nz, int nx, float o1, float o2, float d1, float d2, float o3,
                           float d3, const float *shots, int nshot, const kcig_eikods_opts *opt, float *time,
                           float *tdl1, float *tds1, float *gradz, float *gradx, int *iters, void *stream)
{
    if (!vel || !time || !shots || !opt || nz < 3 || nx < 3 || nshot < 1 || !(d1 > 0.0f) || !(d2 > 0.0f))
        return set_error(KCIG_ERR_ARG, "kcig_eikods: bad arguments");
    if (opt->order != 1 && opt->order != 2) return set_error(KCIG_ERR_ARG, "kcig_eikods: order must be 1 or 2");
    if (opt->l != 0 && opt->l != 1) return set_error(KCIG_ERR_ARG, "kcig_eikods: l must be 0 or 1");
    if ((tdl1 == nullptr) != (tds1 == nullptr))
        return set_error(KCIG_ERR_ARG, "kcig_eikods: tdl1 and tds1 go together");
    // the rings hold kEikS diagonals of nz rows, 12 bytes a row
    if (nz > 1400) return set_error(KCIG_ERR_ARG, "kcig_eikods: nz=%d above 1400", nz);
    const int max_iter = opt->max_iter > 0 ? opt->max_iter : 256;
    const int b0 = opt->b1 < 1 ? 1 : opt->b1, b1 = opt->b2 < 1 ? 1 : opt->b2;
    cudaStream_t st = (cudaStream_t)stream;
    const size_t nzx = (size_t)nz * nx;

    std::vector<EikSource> hs(nshot);
    for (int j = 0; j < nshot; j++)
        hs[j] = source_box(shots[3 * j], shots[3 * j + 1], shots[3 * j + 2], o1, o2, o3, d1, d2, nz, nx, b0, b1);

    const bool deriv = tdl1 != nullptr;
    const int np = (nz + 2 + 15) / 16 * 16, nd = nz + nx - 1;
    const size_t fam_len = (size_t)(nd + 2 * kEikBorder) * np;
    // skipping blocks of 16 diagonals (more on grids that would need over 1024)
    int blk_shift = 4;
    while (((nd - 1) >> blk_shift) + 1 > 1024) blk_shift++;
    const int nblk = ((nd - 1) >> blk_shift) + 1;
    const int rows = nz <= 1024 ? 1 : 2;
    const int threads = ((std::max((nz + rows - 1) / rows, np / 2) + 31) / 32) * 32;
    const size_t smem = eik_smem(np, nblk, deriv), slot = (eik_slot_bytes(nd, np, deriv) + 255) / 256 * 256;
    const void *kern =
        threads <= 640 && rows == 1
            ? (deriv ? (const void *)k_eik_solve<1, 640, true> : (const void *)k_eik_solve<1, 640, false>)
            : rows == 1 ? (deriv ? (const void *)k_eik_solve<1, 1024, true> : (const void *)k_eik_solve<1, 1024, false>)
                        : (deriv ? (const void *)k_eik_solve<2, 704, true> : (const void *)k_eik_solve<2, 704, false>);
    KCIG_TRY(set_dyn_smem(kern, (int)smem));
    // one CTA per source up to the resident ones, and to half of the free
    // memory (32 MB of working values a source on 601 x 1601)
    int per_sm = 0, sms = 0, dev = 0;
    KCIG_CUDA(cudaGetDevice(&dev));
    KCIG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    KCIG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
    int slots = std::min(nshot, std::max(1, per_sm) * sms);
    cudaMemPool_t pool;
    KCIG_TRY(eik_pool(&pool));
    PoolSettle settle{pool, st};
    if (slots * slot > kEikKeep) {
        size_t fr = 0;
        KCIG_TRY(eik_device_full(pool, &fr, &settle.full));
        slots = (int)std::max<size_t>(1, std::min<size_t>(slots, fr / 2 / slot));
    }

    DevBuf bvv, bsk, bdw, bdp, bsrc, bstat, bit, bwork;
    bvv.st = bsk.st = bdw.st = bdp.st = bsrc.st = bstat.st = bit.st = bwork.st = st;
    KCIG_CUDA(cudaMallocFromPoolAsync(&bvv.p, nzx * sizeof(float), pool, st));
    KCIG_CUDA(cudaMallocFromPoolAsync(&bsk.p, 2 * fam_len * sizeof(float), pool, st));
    KCIG_CUDA(cudaMallocFromPoolAsync(&bsrc.p, nshot * sizeof(EikSource), pool, st));
    KCIG_CUDA(cudaMallocFromPoolAsync(&bstat.p, 2 * sizeof(int), pool, st));
    KCIG_CUDA(cudaMallocFromPoolAsync(&bit.p, nshot * sizeof(int), pool, st));
    for (;; slots /= 2) {  // fewer sources at a time where memory is short
        const cudaError_t e = cudaMallocFromPoolAsync(&bwork.p, slots * slot, pool, st);
        if (e == cudaSuccess) break;
        if (e != cudaErrorMemoryAllocation || slots == 1) return cuda_error(e, "cudaMallocFromPoolAsync(work)");
        cudaGetLastError();
        bwork.p = nullptr;
    }
    if (deriv) {
        KCIG_CUDA(cudaMallocFromPoolAsync(&bdp.p, nzx * sizeof(double), pool, st));
        KCIG_CUDA(cudaMallocFromPoolAsync(&bdw.p, 2 * fam_len * sizeof(double), pool, st));
    }
    KCIG_CUDA(cudaMemcpyAsync(bsrc.p, hs.data(), nshot * sizeof(EikSource), cudaMemcpyHostToDevice, st));
    KCIG_CUDA(cudaMemsetAsync(bstat.p, 0, 2 * sizeof(int), st));

    EikArgs a;
    a.vv = (const float *)bsk.p;
    a.dw = (const double *)bdw.p;
    a.vplain = (const float *)bvv.p;
    a.src = (const EikSource *)bsrc.p;
    a.T = time;
    a.dl1 = tdl1;
    a.work = (unsigned char *)bwork.p;
    a.slot_bytes = slot;
    a.status = (int *)bstat.p;
    a.next = a.status + 1;
    a.iters = (int *)bit.p;
    a.nsrc = nshot;
    a.nz = nz;
    a.nx = nx;
    a.np = np;
    a.nd = nd;
    a.order = opt->order;
    a.max_iter = max_iter;
    a.blk_shift = blk_shift;
    a.nblk = nblk;
    a.d0 = d1;
    a.d1 = d2;
    a.d2 = d3;
    a.rdx0 = (float)(1. / (d1 * d1));
    a.rdx1 = (float)(1. / (d2 * d2));
    a.dd0 = div_prepare(d1 * d1);
    a.dd1 = div_prepare(d2 * d2);
    for (int i = 0; i < 2; i++) {
        const double w0 = (double)a.rdx0 * (i ? 2.25 : 1.0);
        a.rc.one[0][i] = 1.0 / w0;
        a.rc.one[1][i] = 1.0 / ((double)a.rdx1 * (i ? 2.25 : 1.0));
        for (int j = 0; j < 2; j++) a.rc.two[i][j] = 1.0 / (w0 + (double)a.rdx1 * (j ? 2.25 : 1.0));
    }

    const unsigned g1 = (unsigned)((nzx + 255) / 256);
    const dim3 gs(nd + 2 * kEikBorder, (np + 127) / 128, 2);
    k_slowness2<<<g1, 256, 0, st>>>(vel, (float *)bvv.p, nzx, opt->vel_is_slowness2);
    k_skew<float><<<gs, 128, 0, st>>>((const float *)bvv.p, (float *)bsk.p, nz, nx, np, nd, 0.0f);
    if (deriv) {
        k_dw<<<g1, 256, 0, st>>>((const float *)bvv.p, (double *)bdp.p, nz, nx, opt->l, opt->l == 0 ? d1 : d2);
        k_skew<double><<<gs, 128, 0, st>>>((const double *)bdp.p, (double *)bdw.p, nz, nx, np, nd, 0.0);
    }
    KCIG_CUDA(cudaGetLastError());
    void *args[] = {&a};
    KCIG_CUDA(cudaLaunchKernel(kern, dim3(slots), dim3(threads), args, smem, st));
    if (deriv) {
        for (int j = 0; j < nshot; j += 65535) {
            const size_t o = (size_t)j * nzx;
            k_tds1<<<dim3(g1, std::min(65535, nshot - j)), 256, 0, st>>>(time + o, tdl1 + o, tds1 + o, nz, nx, opt->l, d1,
                                                                       d2);
            KCIG_CUDA(cudaGetLastError());
        }
    }
    if (gradz || gradx) {
        k_upwind_grads<<<dim3(g1, nshot), 256, 0, st>>>(time, gradz, gradx, nz, nx, d1, d2);
        KCIG_CUDA(cudaGetLastError());
    }
    int status = 0;
    std::vector<int> hit(nshot);
    KCIG_CUDA(cudaMemcpyAsync(&status, bstat.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    KCIG_CUDA(cudaMemcpyAsync(hit.data(), bit.p, nshot * sizeof(int), cudaMemcpyDeviceToHost, st));
    KCIG_CUDA(cudaStreamSynchronize(st));
    if (iters)
        for (int j = 0; j < nshot; j++) iters[j] = hit[j];
    if (status)
        return set_error(KCIG_ERR_DEVICE, "kcig_eikods: sweeps found no fixed point within max_iter=%d", max_iter);
    return KCIG_OK;
}

// fixed-geometry entry point: sources at depth zsrc and lateral positions
// p0 + k*dp (shotgen's float arithmetic), order 2, derivative = tds1
extern "C" int kcig_eikonal_tables(const float *vel, int nz, int nx, float dz, float dx, float z0, float x0, int npos,
                                   float p0, float dp, float zsrc, int b1, int b2, int iterations, float *time,
                                   float *deriv, void *stream)
{
    if (npos < 1) return set_error(KCIG_ERR_ARG, "kcig_eikonal_tables: npos < 1");
    std::vector<float> shots(3 * (size_t)npos);
    for (int j = 0; j < npos; j++) {
        shots[3 * j] = zsrc;
        shots[3 * j + 1] = p0 + (float)j * dp;
        shots[3 * j + 2] = 0.0f;
    }
    kcig_eikods_opts o;
    o.order = 2;
    o.b1 = b1;
    o.b2 = b2;
    o.l = 1;
    o.vel_is_slowness2 = 0;
    o.max_iter = iterations;
    cudaMemPool_t pool;
    KCIG_TRY(eik_pool(&pool));
    PoolSettle settle{pool, (cudaStream_t)stream};
    DevBuf dl1;
    dl1.st = (cudaStream_t)stream;
    size_t fr = 0;
    if (deriv && (size_t)npos * nz * nx * sizeof(float) > kEikKeep) KCIG_TRY(eik_device_full(pool, &fr, &settle.full));
    if (deriv)
        KCIG_CUDA(cudaMallocFromPoolAsync(&dl1.p, (size_t)npos * nz * nx * sizeof(float), pool, (cudaStream_t)stream));
    return kcig_eikods(vel, nz, nx, z0, x0, dz, dx, 0.0f, 1.0f, shots.data(), npos, &o, time, (float *)dl1.p, deriv,
                       nullptr, nullptr, nullptr, stream);
}
