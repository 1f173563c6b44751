// Datuming between depth levels on the device: the frequency-domain
// Kirchhoff extrapolation of the reference's kirchdat2d_freq
// (src/kirchdat2d_frequency_cs.cpp) and the datum-depth slice of greensol_auto
// (src/greensol_auto.cpp).
//
// Layout in HBM.  After the forward transforms the spectra are kept
// frequency-major, U[iw][is][ih] (complex FP32): one ns x nh matrix per
// frequency.  For cmp = 0 the receiver operator is the same for every shot
// and the source operator the same for every receiver, so each side is one
// complex matrix product per frequency:
//     receiver side  Utmp[iw] = U[iw] . Kr[iw],   Kr[ic][ih]  (nh x nh)
//     source side    Uout[iw] = Ks[iw] . Utmp[iw], Ks[is][ic]  (ns x ns)
// (k_cgemm, batched over a chunk of frequencies, skipping the K tiles outside
// the aperture band).  The operators of a chunk are built on the device
// (k_dat_op_fft; k_dat_op for filters beyond 63 samples): per term the weight of :508-523 (aperture taper, distance,
// tau) precomputed on the host in the reference's arithmetic, times the
// anti-aliasing weight (:197-226) and the filter H(tau, w) (:98-182), which is
// evaluated in FP64 with exact phase reduction (the reference's FP32 phase
// omega * m loses ~1e-3 rad at high frequencies).  For cmp = 1 the receiver
// operator moves with the shot and the source side walks common-receiver
// gathers (:556-619), so the sums run term by term (k_dat_rcv_cmp1,
// k_dat_src_cmp1) over per-chunk tables of aH for the table pairs they use.
// Transforms: cuFFT R2C / C2R of length nfft on batches of traces
// (k_dat_prep reverses, tapers and pads; k_dat_finish scales, reverses and
// trims), with tiled transposes between trace-major and frequency-major.
#include <cuda_runtime.h>
#include <cufft.h>
#include <math.h>

#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <map>
#include <mutex>
#include <vector>

#include "kcig_common.h"
#include "kcig_tc.h"

namespace kcig {
namespace {

constexpr int kFilterMax = 64;  // filter samples kept in shared memory (longer filters recompute them)

struct DatEntry {
    float w;     // term weight before the anti-alias weight (0: no term)
    float tau;   // table traveltime of the term
    float dtau;  // |slope| x coordinate step, the anti-alias phase increment
};

struct DatOpArgs {
    const DatEntry *ent;
    int ne;
    float2 *out;  // [nf][ne]
    int f0, nf, nfft, K;
    float dt, antialias;
};

// antialias_weight_iw (:197-226), in the reference's float arithmetic, its
// per-term part (fnyq, fmax, fpass) taken once per term and the frequency
// iw / (nfft dt) once per chunk: the same float operations, the same weights.
// mode 1: the weight is 1 at every frequency; 0: 0 at iw > 0; 2: the taper
// between fpass and fmax
struct DatAa {
    int mode;
    float fpass, fmax, den;
};

__device__ __forceinline__ DatAa dat_aa_term(float antialias, float dtau, float dt)
{
    DatAa t{1, 0.0f, 0.0f, 0.0f};
    if (antialias <= 0.0f) return t;
    dtau = __fmul_rn(fabsf(dtau), antialias);
    if (dtau <= 1e-12f || !isfinite(dtau)) return t;
    const float fnyq = __fdiv_rn(0.5f, dt);
    const float fmax = __fdiv_rn(0.5f, dtau);
    if (fmax >= fnyq) return t;
    if (fmax <= 0.0f) {
        t.mode = 0;
        return t;
    }
    t.mode = 2;
    t.fmax = fmax;
    t.fpass = __fmul_rn(0.8f, fmax);
    t.den = __fsub_rn(fmax, t.fpass);
    return t;
}

// freq = iw / (nfft dt) as dat_aa forms it
__device__ __forceinline__ float dat_aa_at(const DatAa &t, int iw, float freq)
{
    if (t.mode == 1 || iw <= 0) return 1.0f;
    if (t.mode == 0) return 0.0f;
    if (freq <= t.fpass) return 1.0f;
    if (freq >= t.fmax) return 0.0f;
    const float x = __fdiv_rn(__fsub_rn(freq, t.fpass), t.den);
    return __fmul_rn(0.5f, __fadd_rn(1.0f, cospif(x)));
}

// sqrt(t^2 - 1) for t = 1 + u, written without the cancellation of t^2 - 1
__device__ __forceinline__ double dat_root(int j, double dt_over_tau)
{
    if (j < 0) return 0.0;
    const double u = (double)(j + 1) * dt_over_tau;
    return sqrt(u * (2.0 + u));
}

// One thread per operator term, looping over the chunk's frequencies:
// out[c][e] = w aa(iw) H(tau, iw), H = lin . sum_k F[k]/dt exp(-i w k) with
// F the second differences of sqrt(t^2 - 1) (build_filter_F, :98-116), lin =
// (1-delta) exp(-i w m) + delta exp(-i w (m-1)), m = ceil(tau/dt) (:128-181).
__global__ void __launch_bounds__(128) k_dat_op(const DatOpArgs a)
{
    extern __shared__ double zs[];  // [nf][2]: cos w, sin w of the chunk's frequencies; [nf] frequencies; filters
    float *fq = reinterpret_cast<float *>(zs + 2 * a.nf);
    const float fden = __fmul_rn((float)a.nfft, a.dt);
    for (int c = threadIdx.x; c < a.nf; c += blockDim.x) {
        double s, co;
        sincospi(2.0 * (double)(a.f0 + c) / (double)a.nfft, &s, &co);
        zs[2 * c] = co;
        zs[2 * c + 1] = s;
        fq[c] = __fdiv_rn((float)(a.f0 + c), fden);
    }
    __syncthreads();
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.ne) return;
    const DatEntry d = a.ent[e];
    float2 *o = a.out + e;
    if (d.w == 0.0f || !(d.tau > 0.0f) || !isfinite(d.tau) || a.K <= 0) {
        for (int c = 0; c < a.nf; c++) o[(size_t)c * a.ne] = make_float2(0.0f, 0.0f);
        return;
    }
    const double r = (double)a.dt / (double)d.tau, inv_dt = 1.0 / (double)a.dt;
    const int K = a.K;
    // the filter samples in shared memory, F[128 k] of this thread (in a
    // local array they spilled past L1; 21 -> 17 ms at the benchmark size)
    const bool cached = K <= kFilterMax;
    double *F = reinterpret_cast<double *>(zs + 2 * a.nf + (a.nf + 1) / 2) + threadIdx.x;
    if (cached) {
        double p2 = 0.0, p1 = 0.0;
        for (int k = 0; k < K; k++) {
            const double ck = dat_root(k, r);
            F[128 * k] = (ck - 2.0 * p1 + p2) * inv_dt;
            p2 = p1;
            p1 = ck;
        }
    }
    const double q = (double)d.tau * inv_dt, mceil = ceil(q), delta = mceil - q;
    const long long m = (long long)mceil;
    const DatAa aa = dat_aa_term(a.antialias, d.dtau, a.dt);
    for (int c = 0; c < a.nf; c++) {
        const int iw = a.f0 + c;
        const float wa = __fmul_rn(d.w, dat_aa_at(aa, iw, fq[c]));
        if (fabsf(wa) < 1e-20f) {  // the reference skips these terms (:525)
            o[(size_t)c * a.ne] = make_float2(0.0f, 0.0f);
            continue;
        }
        const double zr = zs[2 * c], zi = zs[2 * c + 1];  // exp(-i w) = zr - i zi
        // Horner from the last filter sample down: S = ((F[K-1] z + F[K-2]) z + ...) z + F[0]
        double sr, si = 0.0;
        if (cached) {
            sr = F[128 * (K - 1)];
            for (int k = K - 2; k >= 0; k--) {
                const double tr = sr * zr + si * zi, ti = si * zr - sr * zi;
                sr = tr + F[128 * k];
                si = ti;
            }
        } else {  // long filters: the samples from three running roots
            double c0 = dat_root(K - 1, r), c1 = dat_root(K - 2, r), c2 = dat_root(K - 3, r);
            sr = (c0 - 2.0 * c1 + c2) * inv_dt;
            for (int k = K - 2; k >= 0; k--) {
                c0 = c1;
                c1 = c2;
                c2 = dat_root(k - 2, r);
                const double tr = sr * zr + si * zi, ti = si * zr - sr * zi;
                sr = tr + (c0 - 2.0 * c1 + c2) * inv_dt;
                si = ti;
            }
        }
        // exp(-i w m) with the phase reduced exactly: (iw m) mod nfft, nfft a
        // power of two and iw m >= 0
        const long long red = ((long long)iw * m) & (long long)(a.nfft - 1);
        float es, ec;
        sincospif(__fdiv_rn(2.0f * (float)red, (float)a.nfft), &es, &ec);
        const double lr = (1.0 - delta) + delta * zr, li = delta * zi;  // (1-delta) + delta exp(+i w)
        const double mr = (double)ec * lr + (double)es * li, mi = (double)ec * li - (double)es * lr;
        const double hr = mr * sr - mi * si, hi = mr * si + mi * sr;
        o[(size_t)c * a.ne] = make_float2((float)(wa * hr), (float)(wa * hi));
    }
}

// ---- the same operators by short FFTs ---------------------------------------
// A term's factor is a real FIR filter of K + 1 samples placed at n = m - 1 ..
// m - 1 + K (the K filter samples, and the split of tau between samples m - 1
// and m as a two-sample filter over them):
//     H(iw) = sum_n G[n] W_N^(iw n),  W_N = exp(-2 pi i / nfft).
// For the frequencies iw = a + M b (M = nfft / Q, b = 0 .. Q - 1) of one
// residue a, W_N^(iw n) = W_N^(a n) W_Q^(b n): a Q-point FFT over n mod Q of
// G[n] W_N^(a n) gives all of them, and since G is real the half above
// nfft / 2 is the conjugate of residue M - a.  Residues a = 0 .. M / 2 give
// every frequency; the spectra's rows are kept in that order (dat_row), so a
// chunk of rows is a group of residues.  About 30 FP64 operations per (term,
// frequency) for Q = 64 in place of Horner's five per filter sample and the
// phase's own sine and cosine: 17.1 -> 6.7 ms for 400 x 400 terms, 8193
// frequencies and 51 filter samples (10.5 GB of operators written).
//
// A block of 256 threads takes 256 / T entries, T = Q / 8 sub-threads per
// entry with eight points each: an 8-point DFT in registers, the twiddles, an
// exchange through shared memory, a T-point DFT.
// Lanes are entries, so every table read is a broadcast, the exchange has no
// bank conflicts and a row is stored as 256 consecutive bytes per warp.
struct C64 {
    double x, y;
};
__device__ __forceinline__ C64 operator+(C64 a, C64 b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ C64 operator-(C64 a, C64 b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ C64 operator*(C64 a, C64 b) { return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
__device__ __forceinline__ C64 mul_mi(C64 a) { return {a.y, -a.x}; }  // -i a

__device__ __forceinline__ void dft2(C64 *v)
{
    const C64 t = v[0];
    v[0] = t + v[1];
    v[1] = t - v[1];
}
__device__ __forceinline__ void dft4(C64 *v)
{
    const C64 a = v[0] + v[2], b = v[0] - v[2], c = v[1] + v[3], d = mul_mi(v[1] - v[3]);
    v[0] = a + c;
    v[1] = b + d;
    v[2] = a - c;
    v[3] = b - d;
}
__device__ __forceinline__ void dft8(C64 *v)
{
    constexpr double r = 0.70710678118654752440;
    C64 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    dft4(e);
    dft4(o);
    const C64 o1 = {(o[1].x + o[1].y) * r, (o[1].y - o[1].x) * r};   // W_8 o1
    const C64 o2 = mul_mi(o[2]);
    const C64 o3 = {(o[3].y - o[3].x) * r, -(o[3].x + o[3].y) * r};  // W_8^3 o3
    v[0] = e[0] + o[0];
    v[4] = e[0] - o[0];
    v[1] = e[1] + o1;
    v[5] = e[1] - o1;
    v[2] = e[2] + o2;
    v[6] = e[2] - o2;
    v[3] = e[3] + o3;
    v[7] = e[3] - o3;
}

// row of frequency w in the residue order (Q = 0: the natural order)
__device__ __forceinline__ int dat_row(int w, int Q, int M)
{
    if (Q == 0) return w;
    int a = w & (M - 1), b = w >> (__ffs(M) - 1);  // M is a power of two
    if (a == 0) return b;
    if (2 * a > M) {
        a = M - a;
        b += Q / 2;
    }
    return Q / 2 + 1 + (a - 1) * Q + b;
}

// W_N^(a q) for the residues a = 0 .. M / 2 and q = 0 .. 2 Q - 1
__global__ void k_dat_twiddles(C64 *tw, int Q, int M)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (M / 2 + 1) * 2 * Q) return;
    const long long n = (long long)(i / (2 * Q)) * (i % (2 * Q)) % ((long long)M * Q);
    double s, c;
    sincospi(2.0 * (double)n / (double)((long long)M * Q), &s, &c);
    tw[i] = {c, -s};
}

struct DatFftArgs {
    const DatEntry *ent;
    const C64 *tw;   // [M / 2 + 1][2 Q]
    float2 *out;     // [rows of residues a0 .. a0 + na - 1][ne]
    int ne, a0, na, M, K, nfft;
    float dt, antialias;
};
constexpr int kOpGroup = 4;  // residues of one block: the filters are formed once for them

template <int Q>
__host__ __device__ constexpr int dat_op_smem()
{
    // exchange (or the filter roots), twiddles of the group, W_Q, entry phases, row frequencies
    return 8 * 256 * 16 + kOpGroup * 2 * Q * 16 + Q * 16 + kOpGroup * (2048 / Q) * 16 + (kOpGroup * Q + 4) * 4;
}

template <int Q>
__global__ void __launch_bounds__(256, 2) k_dat_op_fft(const DatFftArgs a)
{
    constexpr int T = Q / 8, EB = 256 / T, G = kOpGroup;
    extern __shared__ __align__(16) unsigned char osm[];
    C64 *xch = reinterpret_cast<C64 *>(osm);              // [Q][EB]
    double *root = reinterpret_cast<double *>(osm);       // [Q][EB], before the exchange is used
    C64 *tw = xch + 8 * 256;                              // [G][2 Q]
    C64 *wq = tw + G * 2 * Q;                             // [Q]
    C64 *ph = wq + Q;                                     // [G][EB]
    float *fq = reinterpret_cast<float *>(ph + G * EB);   // rows of the group
    const int en = threadIdx.x % EB, j = threadIdx.x / EB, e = blockIdx.x * EB + en;
    const int M = a.M, K = a.K;
    const int g0 = a.a0 + blockIdx.y * G, g1 = min(a.a0 + a.na, g0 + G);
    // rows of residue r start at r ? Q / 2 + 1 + (r - 1) Q : 0
    auto row_of = [](int r) { return r ? Q / 2 + 1 + (r - 1) * Q : 0; };
    const int row0 = row_of(g0), nrow = (g1 == M / 2 + 1 ? M / 2 * Q + 1 : row_of(g1)) - row0;
    float2 *o = a.out + (size_t)(row0 - row_of(a.a0)) * a.ne + e;
    DatEntry d{0.0f, 0.0f, 0.0f};
    if (e < a.ne) d = a.ent[e];
    const bool on = d.w != 0.0f && d.tau > 0.0f && isfinite(d.tau);
    if (!__syncthreads_or(on)) {  // terms outside the aperture
        if (e < a.ne)
            for (int r = j; r < nrow; r += T) o[(size_t)r * a.ne] = make_float2(0.0f, 0.0f);
        return;
    }
    for (int i = threadIdx.x; i < (g1 - g0) * 2 * Q; i += 256) tw[i] = a.tw[(size_t)g0 * 2 * Q + i];
    for (int i = threadIdx.x; i < Q; i += 256) {
        double s, c;
        sincospi(2.0 * i / Q, &s, &c);
        wq[i] = {c, -s};
    }
    const float fden = __fmul_rn((float)a.nfft, a.dt);
    for (int i = threadIdx.x; i < nrow; i += 256) {
        const int r = row0 + i;  // the inverse of dat_row
        int iw = r * M;
        if (r > Q / 2) {
            const int res = (r - Q / 2 - 1) / Q + 1, b = (r - Q / 2 - 1) % Q;
            iw = 2 * res == M || b < Q / 2 ? res + M * b : M - res + M * (b - Q / 2);
        }
        fq[i] = __fdiv_rn((float)iw, fden);
    }
    // roots sqrt(t^2 - 1) of the filter, shared by the entry's sub-threads
    const double rr = on ? (double)a.dt / (double)d.tau : 0.0, inv_dt = 1.0 / (double)a.dt;
    for (int k = j; k < K; k += T) root[k * EB + en] = dat_root(k, rr);
    const double q = on ? (double)d.tau * inv_dt : 1.0, mceil = ceil(q), delta = mceil - q;
    const long long n0 = (long long)mceil - 1;  // first sample of the filter, >= 0
    // phases W_M^(residue t0) of the samples' whole turns t0 = n0 / Q
    for (int g = j; g < g1 - g0; g += T) {
        const long long t = ((n0 / Q) % M) * (g0 + g) % M;
        double s, c;
        sincospi(2.0 * (double)t / (double)M, &s, &c);
        ph[g * EB + en] = {c, -s};
    }
    __syncthreads();
    // sample at place p = j + T i of the circle: G[k] = delta F[k] + (1 - delta) F[k - 1], k = p - n0 mod Q
    const int p0 = (int)(n0 & (Q - 1));
    double g[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int k = (j + T * i - p0) & (Q - 1);
        auto R = [&](int n) { return n >= 0 && n < K ? root[n * EB + en] : 0.0; };
        const double c0 = R(k), c1 = R(k - 1), c2 = R(k - 2), c3 = R(k - 3);
        const double f0 = k < K ? c0 - 2.0 * c1 + c2 : 0.0;                // F[k] dt
        const double f1 = k >= 1 && k <= K ? c1 - 2.0 * c2 + c3 : 0.0;     // F[k - 1] dt
        g[i] = on && k <= K ? (delta * f0 + (1.0 - delta) * f1) * inv_dt : 0.0;
    }
    const DatAa aa = dat_aa_term(a.antialias, d.dtau, a.dt);
    for (int r = g0; r < g1; r++) {
        __syncthreads();  // the roots, or the last residue's exchange, are read
        const C64 *tr = tw + (r - g0) * 2 * Q;
        C64 v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int p = j + T * i;
            const C64 z = tr[p < p0 ? p + Q : p];
            v[i] = {g[i] * z.x, g[i] * z.y};
        }
        dft8(v);
        if (T > 1) {
#pragma unroll
            for (int m = 0; m < 8; m++) xch[(m * T + j) * EB + en] = m ? v[m] * wq[j * m] : v[m];
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = xch[(j * 8 + i) * EB + en];  // m = j (8 / T) + i / T, its T sub-threads
#pragma unroll
            for (int i = 0; i < 8; i += T) {
                if (T == 8) dft8(v + i);
                else if (T == 4) dft4(v + i);
                else dft2(v + i);
            }
        }
        const C64 c = ph[(r - g0) * EB + en];
        const int base = row_of(r) - row0;
        if (e < a.ne) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                // output b = m + 8 l
                const int b = T > 1 ? j * (8 / T) + i / T + 8 * (i % T) : i;
                int slot = b;
                bool conj = false;
                if (b >= Q / 2 && !(r == 0 && b == Q / 2)) {
                    if (r == 0 || 2 * r == M) continue;  // its own mirror image
                    slot = Q / 2 + Q - 1 - b;
                    conj = true;
                }
                // (r = 0, b = 0 is frequency 0: fq = 0, below every fpass)
                const C64 h = v[i] * c;
                const float wa = __fmul_rn(d.w, aa.mode == 1 ? 1.0f : dat_aa_at(aa, r + slot, fq[base + slot]));
                o[(size_t)(base + slot) * a.ne] =
                    !on || fabsf(wa) < 1e-20f  // the reference skips these terms (:525)
                        ? make_float2(0.0f, 0.0f)
                        : make_float2((float)(wa * h.x), (float)(conj ? -(wa * h.y) : wa * h.y));
            }
        }
    }
}

// Batched complex GEMM, FP32: C[z] = A[z] . B[z] (row-major, complex
// interleaved), 64x64 tiles of C per CTA, 4x4 per thread, K in steps of 8.
// band >= 0: the nonzero terms satisfy |k - m| <= band (band_rows) or
// |k - n| <= band, so a tile reads only the K range that can touch it.
struct CGemmArgs {
    const float2 *A;
    const float2 *B;
    float2 *C;
    long long sA, sB, sC;  // batch strides (elements)
    int lda, ldb, ldc;
    int M, N, K;
    int band, band_rows;
    int a_trans;           // tensor-core kernel only: A(m, k) at A[k * lda + m]
    int a_vec;             // tensor-core kernel only: row-major A rows start on 16 bytes (lda, sA even)
};

__global__ void __launch_bounds__(256) k_cgemm(const CGemmArgs a)
{
    constexpr int BM = 64, BN = 64, BK = 8;
    __shared__ __align__(16) float2 As[BK][BM + 2];
    __shared__ __align__(16) float2 Bs[BK][BN + 2];
    const int z = blockIdx.z;
    const float2 *A = a.A + (size_t)z * a.sA;
    const float2 *B = a.B + (size_t)z * a.sB;
    float2 *C = a.C + (size_t)z * a.sC;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    int k_lo = 0, k_hi = a.K;
    if (a.band >= 0) {
        const int c0 = a.band_rows ? m0 : n0, c1 = (a.band_rows ? min(a.M, m0 + BM) : min(a.N, n0 + BN)) - 1;
        k_lo = max(0, c0 - a.band);
        k_hi = min(a.K, c1 + a.band + 1);
    }
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    float ar[4][4], ai[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) ar[i][j] = ai[i][j] = 0.0f;
    for (int k0 = k_lo; k0 < k_hi; k0 += BK) {
#pragma unroll
        for (int rr = 0; rr < 2; rr++) {
            const int e = tid + 256 * rr;
            const int mm = e >> 3, kk = e & 7, gm = m0 + mm, gk = k0 + kk;
            As[kk][mm] = (gm < a.M && gk < k_hi) ? A[(size_t)gm * a.lda + gk] : make_float2(0.0f, 0.0f);
            const int kb = e >> 6, nn = e & 63, gkb = k0 + kb, gn = n0 + nn;
            Bs[kb][nn] = (gkb < k_hi && gn < a.N) ? B[(size_t)gkb * a.ldb + gn] : make_float2(0.0f, 0.0f);
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            const float4 a01 = *reinterpret_cast<const float4 *>(&As[kk][ty * 4]);
            const float4 a23 = *reinterpret_cast<const float4 *>(&As[kk][ty * 4 + 2]);
            const float4 b01 = *reinterpret_cast<const float4 *>(&Bs[kk][tx * 4]);
            const float4 b23 = *reinterpret_cast<const float4 *>(&Bs[kk][tx * 4 + 2]);
            const float xr[4] = {a01.x, a01.z, a23.x, a23.z}, xi[4] = {a01.y, a01.w, a23.y, a23.w};
            const float yr[4] = {b01.x, b01.z, b23.x, b23.z}, yi[4] = {b01.y, b01.w, b23.y, b23.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    ar[i][j] = fmaf(xr[i], yr[j], ar[i][j]);
                    ar[i][j] = fmaf(-xi[i], yi[j], ar[i][j]);
                    ai[i][j] = fmaf(xr[i], yi[j], ai[i][j]);
                    ai[i][j] = fmaf(xi[i], yr[j], ai[i][j]);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= a.M) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int gn = n0 + tx * 4 + j;
            if (gn < a.N) C[(size_t)gm * a.ldc + gn] = make_float2(ar[i][j], ai[i][j]);
        }
    }
}

// The same batched complex GEMM on the tensor cores (tcgen05, kind::tf32,
// accumulators in TMEM) with FP32 accuracy from three TF32 products:
// x = hi + lo (hi = TF32(x), lo = TF32(x - hi), both rounded to nearest),
// a.b ~ ah.bh + ah.bl + al.bh,
// the dropped al.bl and the TF32 rounding of lo being ~2^-22 relative.
// The complex product runs as four real products on separate real and
// imaginary planes of both operands: Cr = Ar.Br - Ai.Bi and Ci = Ar.Bi +
// Ai.Br, the minus by the instruction's negate-A bit, so no operand value is
// stored twice.  CTA tile: 128 rows x TNC complex columns (Cr and Ci each a
// 128 x TNC FP32 accumulator in TMEM); K in chunks of 8 complex through S
// pipeline stages, each holding the hi and lo of Ar, Ai (128 x 8) and Br, Bi
// (TNC x 8) in the canonical K-major layout.  Two groups of 8 producer warps
// take alternate chunks: each loads its next chunk while it splits and
// stores the current one; after the main loop all 16 warps read the
// accumulators out.  Warp 16 allocates TMEM and one of its lanes issues the
// MMAs (12 per chunk).  One CTA per SM.  Every mbarrier wait is bounded; a
// wait that gives up sets *status, and the CTA stops issuing work, waits
// (bounded) for its own MMAs and frees its TMEM.
#ifndef KCIG_CGEMM_TNC
#define KCIG_CGEMM_TNC 208  // complex columns of a CTA tile: 400 columns in two tiles (4% padding)
#endif
#ifndef KCIG_CGEMM_STAGES
#define KCIG_CGEMM_STAGES 4
#endif
namespace tcg {
constexpr int TM = 128, TNC = KCIG_CGEMM_TNC, KC = 8, S = KCIG_CGEMM_STAGES;
static_assert(TNC % 16 == 0 && TNC >= 16 && TNC <= 256, "an M = 128 MMA takes N = 16 .. 256 in steps of 16");
constexpr int TMEM_COLS = TNC <= 64 ? 128 : TNC <= 128 ? 256 : 512;  // Cr at column 0, Ci at TMEM_COLS / 2
constexpr int AK = TM * 16 + 32;                    // byte stride of an A plane's two k-groups (padded)
constexpr int BK = TNC * 16;                        // byte stride of a B plane's two k-groups
constexpr int A_PLANE = 2 * AK, B_PLANE = 2 * BK;   // one plane: 8 real k = two 16-byte k-groups
constexpr int STAGE = 4 * A_PLANE + 4 * B_PLANE;    // Ar, Ai, Br, Bi, each hi and lo
constexpr int SMEM = S * STAGE + 128;               // + barriers and slots
constexpr int PRODUCERS = 16;                       // warps
constexpr int THREADS = 32 * (PRODUCERS + 1);
constexpr int RB = (2 * TNC + 255) / 256;           // B items (column, k-group) per producer thread
static_assert(SMEM <= 227 * 1024, "shared memory of one CTA");
}  // namespace tcg

// a bounded mbarrier wait: at most 2^22 polls, each suspending the thread for
// up to 1 us (a few seconds in all; a tile's whole main loop takes ~20 us)
__device__ __forceinline__ bool dat_wait(uint64_t *bar, uint32_t parity)
{
    const uint32_t addr = tc::smem_u32(bar);
    for (uint32_t i = 0; i < (1u << 22); i++) {
        uint32_t ready;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ready)
            : "r"(addr), "r"(parity), "r"(1000u)
            : "memory");
        if (ready) return true;
    }
    return false;
}

// x rounded to 10 mantissa bits (half an ulp added to the magnitude's bits,
// the low 13 bits cleared): the TF32 value nearest x, on the integer pipes
__device__ __forceinline__ float tf32_round(float x)
{
    return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xFFFFE000u);
}

__device__ __forceinline__ void tc_store_split(uint8_t *hi, uint8_t *lo, uint32_t off, float4 v)
{
    float4 h, l;
    h.x = tf32_round(v.x);
    h.y = tf32_round(v.y);
    h.z = tf32_round(v.z);
    h.w = tf32_round(v.w);
    l.x = tf32_round(v.x - h.x);
    l.y = tf32_round(v.y - h.y);
    l.z = tf32_round(v.z - h.z);
    l.w = tf32_round(v.w - h.w);
    *reinterpret_cast<float4 *>(hi + off) = h;
    *reinterpret_cast<float4 *>(lo + off) = l;
}

// the real parts and the imaginary parts of four complex values, split into
// TF32 hi / lo, into one 16-byte row segment of the four planes re_hi, re_lo,
// im_hi, im_lo (`plane` bytes apart, in that order)
__device__ __forceinline__ void tc_store_planes(uint8_t *base, int plane, uint32_t off, const float2 *v)
{
    tc_store_split(base, base + plane, off, make_float4(v[0].x, v[1].x, v[2].x, v[3].x));
    tc_store_split(base + 2 * plane, base + 3 * plane, off, make_float4(v[0].y, v[1].y, v[2].y, v[3].y));
}

__global__ void __launch_bounds__(tcg::THREADS, 1) k_cgemm_tc(const CGemmArgs a, int *status)
{
    using namespace tcg;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + S * STAGE);
    uint64_t *empty = full + S;
    uint64_t *done = empty + S;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(done + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tslot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int z = blockIdx.z;
    const float2 *A = a.A + (size_t)z * a.sA;
    const float2 *B = a.B + (size_t)z * a.sB;
    float2 *C = a.C + (size_t)z * a.sC;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TNC;
    int k_lo = 0, k_hi = a.K;
    if (a.band >= 0) {
        const int c0 = a.band_rows ? m0 : n0, c1 = (a.band_rows ? min(a.M, m0 + TM) : min(a.N, n0 + TNC)) - 1;
        // even start (16-byte loads of A cover k, k+1); the terms added below
        // the band have zero operator entries
        k_lo = max(0, c0 - a.band) & ~1;
        k_hi = min(a.K, c1 + a.band + 1);
    }
    const int nchunks = k_hi > k_lo ? (k_hi - k_lo + KC - 1) / KC : 0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; s++) {
            tc::mbar_init(&full[s], 8);
            tc::mbar_init(&empty[s], 1);
        }
        tc::mbar_init(done, 1);
        *abort_flag = 0;
    }
    if (warp == PRODUCERS) tc::tmem_alloc(tslot, TMEM_COLS);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tslot;

    if (warp < PRODUCERS) {
        // ---- producers: group g (warps 8g .. 8g+7) stores chunks g, g+2, ...
        // into stage i % S.  A item: (row t % 128, k-group t / 128), four
        // complex k; B item e: (column e % TNC, k-group e / TNC), four complex k
        const int g = warp >> 3, t = threadIdx.x & 255;
        struct Chunk {
            float2 a[4], b[RB][4];
        };
        const int arow = t & 127, aj = t >> 7;
        auto load = [&](int i, Chunk &c) {
            const int k0 = k_lo + i * KC + 4 * aj;  // even
            const int gm = m0 + arow;
#pragma unroll
            for (int q = 0; q < 4; q++) c.a[q] = make_float2(0.0f, 0.0f);
            if (gm < a.M) {
                if (a.a_trans) {
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (k0 + q < k_hi) c.a[q] = A[(size_t)(k0 + q) * a.lda + gm];
                } else {
                    const float2 *src = A + (size_t)gm * a.lda + k0;
                    if (a.a_vec && k0 + 3 < k_hi) {  // two 16-byte loads
                        const float4 p = *reinterpret_cast<const float4 *>(src);
                        const float4 r = *reinterpret_cast<const float4 *>(src + 2);
                        c.a[0] = make_float2(p.x, p.y);
                        c.a[1] = make_float2(p.z, p.w);
                        c.a[2] = make_float2(r.x, r.y);
                        c.a[3] = make_float2(r.z, r.w);
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (k0 + q < k_hi) c.a[q] = src[q];
                    }
                }
            }
#pragma unroll
            for (int rr = 0; rr < RB; rr++) {
                const int e = t + 256 * rr, j = e / TNC, n = e - j * TNC, gn = n0 + n;
                const int kb = k_lo + i * KC + 4 * j;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    c.b[rr][q] = make_float2(0.0f, 0.0f);
                    if (e < 2 * TNC && gn < a.N && kb + q < k_hi) c.b[rr][q] = B[(size_t)(kb + q) * a.ldb + gn];
                }
            }
        };
        // group g takes chunks g, g+2, g+4, ...: the loads of its next chunk
        // are issued before the current one is split and stored
        Chunk nxt;
        if (g < nchunks) load(g, nxt);
        for (int i = g; i < nchunks; i += 2) {
            const int slot = i % S;
            const Chunk c = nxt;
            if (i + 2 < nchunks) load(i + 2, nxt);
            if (i >= S && !dat_wait(&empty[slot], ((i / S) - 1) & 1)) {
                atomicExch(status, 1);
                *abort_flag = 1;
            }
            if (__any_sync(0xffffffffu, *abort_flag)) break;  // warp-uniform, as the arrival below is per warp
            uint8_t *st = smem + slot * STAGE;
            // row r of a plane, k-group j: j * stride + (r / 8) * 128 + (r % 8) * 16
            tc_store_planes(st, A_PLANE, (uint32_t)(aj * AK + (arow >> 3) * 128 + (arow & 7) * 16), c.a);
#pragma unroll
            for (int rr = 0; rr < RB; rr++) {
                const int e = t + 256 * rr, j = e / TNC, n = e - j * TNC;
                if (e < 2 * TNC)
                    tc_store_planes(st + 4 * A_PLANE, B_PLANE, (uint32_t)(j * BK + (n >> 3) * 128 + (n & 7) * 16),
                                    c.b[rr]);
            }
            tc::fence_async_smem();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&full[slot]);
        }
    } else if (lane == 0) {
        // ---- MMA issuer: Cr += Ar.Br - Ai.Bi, Ci += Ar.Bi + Ai.Br, three
        // TF32 products each
        const uint32_t id = tc::idesc_tf32(TM, TNC), id_neg = id | (1u << 13);  // bit 13: negate A
        const uint32_t Dr = tmem, Di = tmem + TMEM_COLS / 2;
        for (int i = 0; i < nchunks; i++) {
            const int slot = i % S;
            if (!dat_wait(&full[slot], (i / S) & 1)) {
                atomicExch(status, 2);
                *abort_flag = 1;
            }
            if (*abort_flag) break;
            tc::fence_after();
            const uint32_t st = tc::smem_u32(smem + slot * STAGE), sb = st + 4 * A_PLANE;
            const uint64_t arh = tc::sdesc(st, AK, 128), arl = tc::sdesc(st + A_PLANE, AK, 128);
            const uint64_t aih = tc::sdesc(st + 2 * A_PLANE, AK, 128), ail = tc::sdesc(st + 3 * A_PLANE, AK, 128);
            const uint64_t brh = tc::sdesc(sb, BK, 128), brl = tc::sdesc(sb + B_PLANE, BK, 128);
            const uint64_t bih = tc::sdesc(sb + 2 * B_PLANE, BK, 128), bil = tc::sdesc(sb + 3 * B_PLANE, BK, 128);
            const uint32_t acc = i > 0 ? 1u : 0u;
            tc::mma_tf32(Dr, arh, brh, id, acc);
            tc::mma_tf32(Dr, arh, brl, id, 1u);
            tc::mma_tf32(Dr, arl, brh, id, 1u);
            tc::mma_tf32(Dr, aih, bih, id_neg, 1u);
            tc::mma_tf32(Dr, aih, bil, id_neg, 1u);
            tc::mma_tf32(Dr, ail, bih, id_neg, 1u);
            tc::mma_tf32(Di, arh, bih, id, acc);
            tc::mma_tf32(Di, arh, bil, id, 1u);
            tc::mma_tf32(Di, arl, bih, id, 1u);
            tc::mma_tf32(Di, aih, brh, id, 1u);
            tc::mma_tf32(Di, aih, brl, id, 1u);
            tc::mma_tf32(Di, ail, brh, id, 1u);
            tc::commit(&empty[slot]);
        }
        tc::commit(done);  // tracks every MMA issued, also after an abort
    }
    __syncwarp();
    // ---- epilogue: warps 0-15 read the accumulators; warp w owns TMEM lanes
    // 32 (w % 4) .. +31 and a quarter of the columns, 32 at a time
    bool ok = true;
    if (warp < PRODUCERS || lane == 0) ok = dat_wait(done, 0);
    if (!ok) atomicExch(status, 3);
    if (warp < PRODUCERS) {
        tc::fence_after();
        constexpr int QC = (TNC / 4 + 31) / 32 * 32;  // columns per quarter, whole 32-column loads
        const int q = warp & 3, quarter = warp >> 2;
        const int gm = m0 + 32 * q + lane;
        const uint32_t lanes = (uint32_t)(32 * q) << 16;
        const bool live = __all_sync(0xffffffffu, ok && !*abort_flag);  // warp-uniform: TMEM loads are collective
        for (int cb = 0; cb < QC; cb += 32) {
            const int c0 = quarter * QC + cb;
            if (c0 >= TNC) break;  // the accumulators' unused columns
            float vr[32], vi[32];
            if (nchunks > 0 && live) {
                tc::tmem_ld32(tmem + lanes + c0, vr);
                tc::tmem_ld32(tmem + lanes + TMEM_COLS / 2 + c0, vi);
            } else {
#pragma unroll
                for (int c = 0; c < 32; c++) vr[c] = vi[c] = 0.0f;
            }
            if (gm < a.M && live) {
                float2 *dst = C + (size_t)gm * a.ldc + n0 + c0;
#pragma unroll
                for (int c = 0; c < 32; c++)
                    if (c0 + c < TNC && n0 + c0 + c < a.N) dst[c] = make_float2(vr[c], vi[c]);
            }
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == PRODUCERS) tc::tmem_free(tmem, TMEM_COLS);
}

// Frequencies a thread of the cmp = 1 sums carries in registers: the term's
// indices and weight (table lookups, a double product on the source side) are
// formed once for all of them, and as many independent loads are in flight.
constexpr int kCmp1F = 4;

// cmp = 1 receiver side (:493-546 with s_abs = s0 + is ds): one thread per
// (shot, trace) and kCmp1F frequencies, the sum over the aperture of
// geom[ic][ih] tau (aH)[pair], pair = (table row cc = cabs[is][ic], column
// c = cabs[is][ih]) looked up in the chunk's band table P[c][row][j],
// j = c - cc + band.  Lanes along ih: the pair table, geom and tau are read
// coalesced, the input spectrum is one value per warp.
struct RcvCmp1Args {
    const float2 *U;   // [nf][ns][nh] (the chunk's input spectra)
    float2 *Utmp;      // [nf][ns][nh]
    const float2 *P;   // [nf][nrow * (2 band + 1)]
    const float *Ptau; // [nrow * (2 band + 1)]
    const int *cabs;   // [ns][nh]
    const float *geom; // [nh][nh], the input trace first
    int ns, nh, aper, band, row0, nrow, nf;
    long long sU;      // U batch stride
};

__global__ void __launch_bounds__(128) k_dat_rcv_cmp1(const RcvCmp1Args a)
{
    const int tr = blockIdx.x * blockDim.x + threadIdx.x, f0 = blockIdx.y * kCmp1F;
    const int ntr = a.ns * a.nh;
    if (tr >= ntr) return;
    const int is = tr / a.nh, ih = tr - is * a.nh;
    const int wid = 2 * a.band + 1;
    const size_t sP = (size_t)a.nrow * wid;
    const float2 *U[kCmp1F], *P[kCmp1F];
    float sr[kCmp1F], si[kCmp1F];
#pragma unroll
    for (int j = 0; j < kCmp1F; j++) {
        const size_t f = min(f0 + j, a.nf - 1);  // past the chunk: the last frequency again, not stored
        U[j] = a.U + f * a.sU + (size_t)is * a.nh;
        P[j] = a.P + f * sP;
        sr[j] = si[j] = 0.0f;
    }
    const int cih = a.cabs[tr];
    const int left = max(0, ih - a.aper), right = min(a.nh - 1, ih + a.aper);
    // no branch on a zero weight (its term is dropped by selection, so a NaN
    // trace outside the taper stays outside): the loads of several terms overlap
#pragma unroll 4
    for (int ic = left; ic <= right; ic++) {
        const float g = __ldg(a.geom + (size_t)ic * a.nh + ih);
        const int cc = __ldg(a.cabs + (size_t)is * a.nh + ic);
        const size_t pi = (size_t)(cc - a.row0) * wid + (cih - cc + a.band);
        const float w = __fmul_rn(g, __ldg(a.Ptau + pi));
#pragma unroll
        for (int j = 0; j < kCmp1F; j++) {
            const float2 h = __ldg(P[j] + pi), u = __ldg(U[j] + ic);
            const float xr = fmaf(w, u.x * h.x - u.y * h.y, sr[j]), xi = fmaf(w, u.x * h.y + u.y * h.x, si[j]);
            sr[j] = g != 0.0f ? xr : sr[j];
            si[j] = g != 0.0f ? xi : si[j];
        }
    }
#pragma unroll
    for (int j = 0; j < kCmp1F; j++)
        if (f0 + j < a.nf) a.Utmp[(size_t)(f0 + j) * ntr + tr] = make_float2(sr[j], si[j]);
}

// cmp = 1 source side (:556-619): one thread per output trace (shot is, trace
// ih) and kCmp1F frequencies.  The common-receiver gathers r that send the
// shot to this trace are listed per trace (cnt in gath, in order of r; one
// gather when |ds| >= |dh|): each gather's neighbouring shots are summed, and
// the gathers' sums added in that order.  Lanes along ih take neighbouring
// gathers, so ihmap[ic][r] and the input spectra are read coalesced.
// It was one thread per (frequency, shot) walking every gather that holds
// the shot, a few hundred threads a chunk: 19.4 ms of a 64 x 96 trace call
// with 513 frequencies, now 0.55 ms (receiver side 2.0 -> 0.82 ms).
struct SrcCmp1Args {
    const float2 *Utmp;  // [nf][ns][nh]
    float2 *Uout;        // [nf][ns][nh]
    const float2 *P;     // [nf][ns][ns]: aH of pair (c_s[ic], c_s[is]) at [is][ic]
    const double *gw;    // [ns][ns]: ds sdatum tau / (pi dist) at [is][ic]
    const int *sleft, *sright;  // [nr] the gather's shot range
    const int *ihmap;    // [ns][nr]: trace of shot is in gather r, -1 outside
    const int *goff;     // [ns * nh + 1] first entry of each output trace in gath
    const int *gath;     // gathers, in order
    const float *ramp;   // [nramp] edge taper by the distance from the window's end; past it 1
    int ns, nh, nr, aper, jump, nramp, nf;
    long long sUout;
};

__global__ void __launch_bounds__(128) k_dat_src_cmp1(const SrcCmp1Args a)
{
    const int tr = blockIdx.x * blockDim.x + threadIdx.x, f0 = blockIdx.y * kCmp1F;
    const int ntr = a.ns * a.nh;
    if (tr >= ntr) return;
    const int is = tr / a.nh;
    const float2 *Ut[kCmp1F], *P[kCmp1F];
    float2 o[kCmp1F];
#pragma unroll
    for (int j = 0; j < kCmp1F; j++) {
        const size_t f = min(f0 + j, a.nf - 1);
        Ut[j] = a.Utmp + f * ntr;
        P[j] = a.P + f * a.ns * a.ns + (size_t)is * a.ns;
        o[j] = make_float2(0.0f, 0.0f);
    }
    const double *gw = a.gw + (size_t)is * a.ns;
    for (int q = a.goff[tr]; q < a.goff[tr + 1]; q++) {
        const int ir = a.gath[q];
        const int il = max(a.sleft[ir], is - a.jump * a.aper), iu = min(a.sright[ir], is + a.jump * a.aper);
        float accr[kCmp1F], acci[kCmp1F];
#pragma unroll
        for (int j = 0; j < kCmp1F; j++) accr[j] = acci[j] = 0.0f;
#pragma unroll 4
        for (int ic = il; ic <= iu; ic += a.jump) {
            const int hh = __ldg(a.ihmap + (size_t)ic * a.nr + ir);
            const float cl = ic - il < a.nramp ? __ldg(a.ramp + (ic - il)) : 1.0f;
            const float cu = iu - ic < a.nramp ? __ldg(a.ramp + (iu - ic)) : 1.0f;
            const float w = (float)((double)__fmul_rn(cl, cu) * __ldg(gw + ic));
            const size_t at = (size_t)ic * a.nh + max(hh, 0);
#pragma unroll
            for (int j = 0; j < kCmp1F; j++) {
                const float2 h = __ldg(P[j] + ic), u = __ldg(Ut[j] + at);
                const float xr = fmaf(w, u.x * h.x - u.y * h.y, accr[j]), xi = fmaf(w, u.x * h.y + u.y * h.x, acci[j]);
                accr[j] = hh >= 0 ? xr : accr[j];  // a shot the gather does not hold
                acci[j] = hh >= 0 ? xi : acci[j];
            }
        }
#pragma unroll
        for (int j = 0; j < kCmp1F; j++) {
            o[j].x += accr[j];
            o[j].y += acci[j];
        }
    }
#pragma unroll
    for (int j = 0; j < kCmp1F; j++)
        if (f0 + j < a.nf) a.Uout[(size_t)(f0 + j) * a.sUout + tr] = o[j];
}

// reverse in time, edge taper and zero-pad one batch of traces (:287-306):
// a thread writes four consecutive samples of a padded trace (one 16-byte
// store; nfft is a power of two >= 4), up to 1024 block rows walk the
// batch's traces (several traces per block: ~10 waves at full size)
__global__ void k_dat_prep(const float *in, const float *wtr, float *pad, int tr0, int nb, int nt, int nfft)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= (nfft >> 2)) return;
    for (int b = blockIdx.y; b < nb; b += gridDim.y) {
        const float w = wtr[tr0 + b];
        const float *src = in + (size_t)(tr0 + b) * nt + (nt - 1);  // src[-t]: sample nt - 1 - t
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int t = 4 * q + j;
            float x = 0.0f;
            if (t < nt) {
                const float y = src[-t];
                x = w == 1.0f ? y : __fmul_rn(w, y);
            }
            v[j] = x;
        }
        reinterpret_cast<float4 *>(pad + (size_t)b * nfft)[q] = make_float4(v[0], v[1], v[2], v[3]);
    }
}

// scale by 1/nfft, optionally reverse, trim to nt (:476-487): threads along
// the output samples, up to 1024 block rows walk the batch's traces
__global__ void k_dat_finish(const float *pad, float *out, int tr0, int nb, int nt, int nfft, float scale, int reverse)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt) return;
    const int ts = reverse ? nt - 1 - t : t;
    for (int b = blockIdx.y; b < nb; b += gridDim.y)
        out[(size_t)(tr0 + b) * nt + t] = __fmul_rn(pad[(size_t)b * nfft + ts], scale);
}

// tiled transposes between spec[b][nw] (a batch of traces) and U[row][ntr],
// the rows in dat_row's order
__global__ void k_dat_to_fmajor(const float2 *spec, float2 *U, int tr0, int nb, int nw, int ntr, int Q, int M)
{
    __shared__ float2 tile[32][33];
    const int w0 = blockIdx.x * 32, b0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int b = b0 + r, w = w0 + threadIdx.x;
        if (b < nb && w < nw) tile[r][threadIdx.x] = spec[(size_t)b * nw + w];
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int w = w0 + r, b = b0 + threadIdx.x;
        if (b < nb && w < nw) U[(size_t)dat_row(w, Q, M) * ntr + tr0 + b] = tile[threadIdx.x][r];
    }
}

__global__ void k_dat_to_tmajor(const float2 *U, float2 *spec, int tr0, int nb, int nw, int ntr, int Q, int M)
{
    __shared__ float2 tile[32][33];
    const int w0 = blockIdx.y * 32, b0 = blockIdx.x * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int w = w0 + r, b = b0 + threadIdx.x;
        if (b < nb && w < nw) tile[r][threadIdx.x] = U[(size_t)dat_row(w, Q, M) * ntr + tr0 + b];
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int b = b0 + r, w = w0 + threadIdx.x;
        if (b < nb && w < nw) spec[(size_t)b * nw + w] = tile[threadIdx.x][r];
    }
}

__global__ void k_green_gather(const float *table, const int *ix, float *out, int ngx, int nx, int nz, int idatum)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ngx * ngx) return;
    const int i1 = i / ngx, i2 = i - i1 * ngx;
    out[i] = table[((size_t)i1 * nx + ix[i2]) * nz + idatum];
}

// ------------------------------------------------------------ host side --

// the reference's float arithmetic for indices and weights (x86-64 SSE, no
// contraction): every operation below rounds to float as it does there
inline int f2i(float x) { return (int)x; }

float taper_host(int left, int center, int right, int tap, int stride)  // taper_weight (:229-240)
{
    if (center < left || center > right) return 0.0f;
    if (tap <= 0) return 1.0f;
    if (stride < 1) stride = 1;
    const float width = (float)tap * (float)stride;
    const float ul = fminf(1.0f, fmaxf(0.0f, (float)(center - left) / width));
    const float ur = fminf(1.0f, fmaxf(0.0f, (float)(right - center) / width));
    return 0.5f * (1.0f - cosf((float)M_PI * ul)) * 0.5f * (1.0f - cosf((float)M_PI * ur));
}

float edge_host(int i, int n, int tap)  // data_edge_taper_weight (:255-279)
{
    if (tap <= 0 || n <= 1) return 1.0f;
    int ntap = tap;
    const int max_tap = (n - 1) / 2;
    if (ntap > max_tap) ntap = max_tap;
    if (ntap <= 0) return 1.0f;
    if (i < ntap) return 0.5f * (1.0f - cosf((float)M_PI * ((float)i / (float)ntap)));
    if (i > n - 1 - ntap) return 0.5f * (1.0f - cosf((float)M_PI * ((float)(n - 1 - i) / (float)ntap)));
    return 1.0f;
}

float slope_host(const float *t, int n, int row, int col, float dcoord)  // :184-194, t[row][col] row-major n x n
{
    if (n <= 1 || dcoord == 0.0f) return 0.0f;
    if (row <= 0) return (t[(size_t)1 * n + col] - t[col]) / dcoord;
    if (row >= n - 1) return (t[(size_t)(n - 1) * n + col] - t[(size_t)(n - 2) * n + col]) / dcoord;
    return 0.5f * (t[(size_t)(row + 1) * n + col] - t[(size_t)(row - 1) * n + col]) / dcoord;
}

int rcv_index(const kcig_datum_params &p, int is, int ih)  // :502, :507
{
    const float s = p.cmp ? p.s0 + (float)is * p.ds : 0.0f;
    return f2i((s + p.h0 + (float)ih * p.dh - p.rg0) / p.drg + 0.5f);
}

int src_index(const kcig_datum_params &p, int is)  // :583, :638
{
    return f2i((p.s0 + (float)is * p.ds - p.sg0) / p.dsg + 0.5f);
}

// w = coef / M_PI * d * datum * tau / dist, in double as written, then float
float term_weight(float coef, float d, float datum, float tau, float dist)
{
    return (float)(coef / M_PI * d * datum * tau / dist);
}

struct Stage {
    cudaEvent_t ev[6] = {};
};

thread_local float g_last_ms[5] = {0, 0, 0, 0, 0};
thread_local int g_last_launches = 0;

struct DBuf {
    void *p = nullptr;
    ~DBuf()
    {
        if (p) cudaFree(p);
    }
    template <class T>
    T *as() const
    {
        return (T *)p;
    }
};

int dalloc(DBuf &b, size_t bytes, const char *what)
{
    if (bytes == 0) bytes = 16;
    const cudaError_t e = cudaMalloc(&b.p, bytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        b.p = nullptr;
        return set_error(KCIG_ERR_NOMEM, "kcig_green_slice: cannot allocate %.3f GB for %s on the device",
                         bytes / 1e9, what);
    }
    return KCIG_OK;
}

template <class T>
int upload(DBuf &b, const std::vector<T> &v, cudaStream_t st, const char *what)
{
    KCIG_TRY(dalloc(b, v.size() * sizeof(T), what));
    if (!v.empty()) KCIG_CUDA(cudaMemcpyAsync(b.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st));
    return KCIG_OK;
}

int cufft_error(cufftResult r, const char *what)
{
    return set_error(KCIG_ERR_CUDA, "%s failed: cufftResult %d", what, (int)r);
}

// ---- device buffers and transform plans kept between calls
// The spectra alone take nw x traces x 8 bytes (10.5 GB for 400 x 400
// traces and 8193 frequencies); allocating them, planning the transforms and
// freeing it all again cost a fifth of a call.  One cache per device, held
// by a call for its whole run (kcig_datum_freq is synchronous on its
// stream), so calls on one device from several threads run one after the
// other.  Buffers only grow.  A call that cannot allocate frees every cached
// buffer and tries once more; kcig_datum_release frees a device's cache.
enum CacheSlot {
    CB_U,       // spectra, frequency-major [nw][ntr]
    CB_UFULL,   // receiver-side spectra kept for interm
    CB_UT,      // receiver-side spectra of one chunk of frequencies
    CB_KR,      // receiver operator of one chunk
    CB_KS,      // source operator of one chunk
    CB_PAD,     // one batch of padded traces
    CB_SPEC,    // one batch of trace-major spectra
    CB_WORK,    // cuFFT work area, shared by the four plans
    CB_IN,      // host-memory calls: the input, output and interm cubes
    CB_OUT,
    CB_INTERM,
    CB_STATUS,  // tensor-core GEMM status word
    CB_WTR,     // uploads: trace weights, operator entries, cmp = 1 walk tables
    CB_RCV,
    CB_SRC,
    CB_CABS,
    CB_GEOM,
    CB_RTAU,
    CB_SGW,
    CB_SL,
    CB_SR,
    CB_IHM,
    CB_GOFF,
    CB_GATH,
    CB_RAMP,
    CB_TW,      // twiddles of the operators' FFTs
    CB_COUNT
};

const char *const kSlotName[CB_COUNT] = {
    "the spectra", "the receiver-side spectra", "the receiver-side chunk", "the receiver operator",
    "the source operator", "the transform buffer", "the transform buffer", "the transform work area",
    "the input traces", "the output traces", "the intermediate traces", "a status word", "trace weights",
    "receiver terms", "source terms", "receiver indices", "receiver weights", "receiver pair times",
    "source pair weights", "gather ranges", "gather ranges", "gather traces", "gather lists", "gather lists",
    "the edge taper", "twiddles"};

struct CBuf {
    void *p = nullptr;
    size_t n = 0;
    template <class T>
    T *as() const
    {
        return (T *)p;
    }
};

// an R2C / C2R plan pair of one transform length and batch
struct FftPair {
    cufftHandle f = 0, b = 0;
    bool ok = false;
    int nfft = 0, batch = 0;
    size_t work = 0;
};

struct DatumCache {
    std::mutex mu;
    CBuf buf[CB_COUNT];
    FftPair full, tail;
    std::vector<cudaEvent_t> ev;
    cudaStream_t copy = nullptr;  // host-memory calls: the cubes' copies, batch by batch
};

std::mutex g_caches_mu;
std::map<int, DatumCache *> g_caches;  // never destroyed: the process exit or kcig_datum_release frees them

DatumCache &cache_of(int dev)
{
    std::lock_guard<std::mutex> g(g_caches_mu);
    DatumCache *&c = g_caches[dev];
    if (!c) c = new DatumCache;
    return *c;
}

void free_buffers(DatumCache &c)
{
    for (CBuf &b : c.buf) {
        if (b.p) cudaFree(b.p);
        b = CBuf{};
    }
}

void free_pair(FftPair &q)
{
    if (q.ok) {
        cufftDestroy(q.f);
        cufftDestroy(q.b);
    }
    q = FftPair{};
}

// the plan pair for (nfft, batch), work area left to the caller
int make_pair(FftPair &q, int nfft, int nw, int batch)
{
    if (q.ok && q.nfft == nfft && q.batch == batch) return KCIG_OK;
    free_pair(q);
    cufftResult cr;
    if ((cr = cufftCreate(&q.f)) != CUFFT_SUCCESS) return cufft_error(cr, "cufftCreate");
    if ((cr = cufftCreate(&q.b)) != CUFFT_SUCCESS) {
        cufftDestroy(q.f);
        q = FftPair{};
        return cufft_error(cr, "cufftCreate");
    }
    q.ok = true;
    int n = nfft;
    size_t wf = 0, wb = 0;
    if ((cr = cufftSetAutoAllocation(q.f, 0)) != CUFFT_SUCCESS || (cr = cufftSetAutoAllocation(q.b, 0)) != CUFFT_SUCCESS) {
        free_pair(q);
        return cufft_error(cr, "cufftSetAutoAllocation");
    }
    if ((cr = cufftMakePlanMany(q.f, 1, &n, nullptr, 1, nfft, nullptr, 1, nw, CUFFT_R2C, batch, &wf)) != CUFFT_SUCCESS) {
        free_pair(q);
        return cufft_error(cr, "cufftPlanMany (R2C)");
    }
    if ((cr = cufftMakePlanMany(q.b, 1, &n, nullptr, 1, nw, nullptr, 1, nfft, CUFFT_C2R, batch, &wb)) != CUFFT_SUCCESS) {
        free_pair(q);
        return cufft_error(cr, "cufftPlanMany (C2R)");
    }
    q.nfft = nfft;
    q.batch = batch;
    q.work = std::max(wf, wb);
    return KCIG_OK;
}

// every slot at least need[slot] bytes (0: not used by this call)
int ensure_buffers(DatumCache &c, const size_t *need)
{
    for (int attempt = 0; attempt < 2; attempt++) {
        int bad = -1;
        for (int i = 0; i < CB_COUNT && bad < 0; i++) {
            CBuf &b = c.buf[i];
            if (need[i] == 0 || b.n >= need[i]) continue;
            if (b.p) cudaFree(b.p);
            b = CBuf{};
            if (cudaMalloc(&b.p, need[i]) != cudaSuccess) {
                cudaGetLastError();
                b.p = nullptr;
                bad = i;
            } else {
                b.n = need[i];
            }
        }
        if (bad < 0) return KCIG_OK;
        free_buffers(c);
        KCIG_TRY(eik_release_pool());  // what the table calls keep
        if (attempt == 1)
            return set_error(KCIG_ERR_NOMEM, "kcig_datum_freq: cannot allocate %.3f GB for %s on the device",
                             need[bad] / 1e9, kSlotName[bad]);
    }
    return KCIG_OK;
}

template <class T>
size_t upload_bytes(const std::vector<T> &v)
{
    return std::max<size_t>(16, v.size() * sizeof(T));
}

template <class T>
int upload_to(const CBuf &b, const std::vector<T> &v, cudaStream_t st)
{
    if (!v.empty()) KCIG_CUDA(cudaMemcpyAsync(b.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st));
    return KCIG_OK;
}

int validate(const kcig_datum_params &p)
{
    if (p.cmp != 0 && p.cmp != 1) return set_error(KCIG_ERR_ARG, "cmp must be 0 or 1.");
    if (p.bf_p <= 0 || p.bf_n_leaf <= 1) return set_error(KCIG_ERR_ARG, "Need bf_p > 0 and bf_n_leaf > 1.");
    if (p.bf_p >= p.bf_n_leaf)
        return set_error(KCIG_ERR_ARG,
                         "Need bf_p < bf_n_leaf for meaningful butterfly interpolation / exact leaf-stage settings.");
    if (p.data_taper < 0) return set_error(KCIG_ERR_ARG, "data_taper must be >= 0.");
    if (!(p.antialias >= 0.0f)) return set_error(KCIG_ERR_ARG, "antialias must be >= 0.");
    if (p.nt <= 0 || p.nh <= 0 || p.ns <= 0 || p.nsg <= 0 || p.nrg <= 0)
        return set_error(KCIG_ERR_ARG, "kcig_datum_freq: sizes must be positive");
    if (!(p.dt > 0.0f)) return set_error(KCIG_ERR_ARG, "kcig_datum_freq: dt must be positive");
    if ((long long)p.ns * p.nh > 0x7fffffffLL) return set_error(KCIG_ERR_ARG, "kcig_datum_freq: too many traces");
    return KCIG_OK;
}

int sizes(const kcig_datum_params &p, const float *st, const float *rt, int *nsam_out, int *nfft_out)
{
    const float ratio = p.length / p.dt;
    if (!(fabsf(ratio) < 1e8f)) return set_error(KCIG_ERR_ARG, "kcig_datum_freq: length / dt out of range");
    const int nsam = f2i(ratio) + 2;
    float max_tau = 0.0f;  // choose_nfft (:82-96)
    for (size_t i = 0; i < (size_t)p.nrg * p.nrg; i++)
        if (rt[i] > max_tau) max_tau = rt[i];
    for (size_t i = 0; i < (size_t)p.nsg * p.nsg; i++)
        if (st[i] > max_tau) max_tau = st[i];
    const float steps = ceilf(max_tau / p.dt);
    if (!(steps < 5e8f)) return set_error(KCIG_ERR_ARG, "kcig_datum_freq: table traveltimes too long for an FFT");
    const long long need = (long long)p.nt + (long long)steps + (nsam - 2) + 2;
    long long n = 1;
    while (n < need) n <<= 1;
    if (n > (1LL << 30)) return set_error(KCIG_ERR_ARG, "kcig_datum_freq: nfft %lld too large", n);
    *nsam_out = nsam;
    *nfft_out = (int)n;
    return KCIG_OK;
}

// Operator terms of one side in the reference's arithmetic.  Dense matrices
// of DatEntry: receiver (cmp 0) at [ic][ih] (the K x N operand), source
// (cmp 0) at [is][ic]; for cmp = 1, the band table of receiver pairs and the
// source pair matrix, whose entries carry w = 1 (the geometric factor is
// applied by the sums).
struct Host {
    std::vector<DatEntry> rcv, src;
    // cmp = 1 receiver side
    std::vector<int> cabs;        // [ns][nh]
    std::vector<float> geom, rtau;  // [nh][nh] (input trace first), [nrow][2 band + 1]
    int band = 0, row0 = 0, nrow = 0;
    // cmp = 1 source side
    std::vector<double> sgw;   // [ns][ns] geometric weight times tau
    std::vector<float> ramp;   // edge taper by the distance from a window's end
    std::vector<int> sleft, sright, ihmap;  // [nr], [nr], [ns][nr]
    std::vector<int> goff, gath;            // the gathers of each output trace, in order
    int nr = 0, jump = 1;
};

int build_receiver(const kcig_datum_params &p, const float *rt, Host &h)
{
    const int nh = p.nh, ns = p.ns, aper = p.aperture, nrg = p.nrg;
    if (p.cmp == 0) {
        h.rcv.assign((size_t)nh * nh, DatEntry{0.0f, 0.0f, 0.0f});
        for (int ih = 0; ih < nh; ih++) {
            const int c = rcv_index(p, 0, ih);
            const int left = std::max(0, ih - aper), right = std::min(nh - 1, ih + aper);
            for (int ic = left; ic <= right; ic++) {
                const int cc = rcv_index(p, 0, ic);
                if (c < 0 || c >= nrg || cc < 0 || cc >= nrg) return set_error(KCIG_ERR_ARG, "Receiver table too small.");
                const float coef = taper_host(left, ic, right, p.taper, 1);
                const float tau = rt[(size_t)cc * nrg + c];
                const float dist = p.rdatum * p.rdatum + (float)((ic - ih) * (ic - ih)) * p.dh * p.dh;
                DatEntry &e = h.rcv[(size_t)ic * nh + ih];
                e.w = term_weight(coef, p.dh, p.rdatum, tau, dist);
                e.tau = tau;
                e.dtau = slope_host(rt, nrg, cc, c, p.drg) * fabsf(p.dh);
            }
        }
        return KCIG_OK;
    }
    h.cabs.resize((size_t)ns * nh);
    int lo = 0x7fffffff, hi = -0x7fffffff - 1;
    for (int is = 0; is < ns; is++)
        for (int ih = 0; ih < nh; ih++) {
            const int c = rcv_index(p, is, ih);
            h.cabs[(size_t)is * nh + ih] = c;
            if (aper >= 0 && (c < 0 || c >= nrg)) return set_error(KCIG_ERR_ARG, "Receiver table too small.");
            lo = std::min(lo, c);
            hi = std::max(hi, c);
        }
    h.geom.assign((size_t)nh * nh, 0.0f);
    int band = 0;
    for (int ih = 0; ih < nh; ih++) {
        const int left = std::max(0, ih - aper), right = std::min(nh - 1, ih + aper);
        for (int ic = left; ic <= right; ic++) {
            const float coef = taper_host(left, ic, right, p.taper, 1);
            const float dist = p.rdatum * p.rdatum + (float)((ic - ih) * (ic - ih)) * p.dh * p.dh;
            h.geom[(size_t)ic * nh + ih] = (float)(coef / M_PI * p.dh * p.rdatum / dist);
        }
        for (int is = 0; is < ns && left <= right; is++) {
            const int c = h.cabs[(size_t)is * nh + ih];
            band = std::max(band, std::abs(c - h.cabs[(size_t)is * nh + left]));
            band = std::max(band, std::abs(c - h.cabs[(size_t)is * nh + right]));
        }
    }
    if (aper < 0 || lo > hi) {
        lo = hi = 0;
    }
    h.band = band;
    h.row0 = lo;
    h.nrow = hi - lo + 1;
    const int wid = 2 * band + 1;
    h.rcv.assign((size_t)h.nrow * wid, DatEntry{0.0f, 0.0f, 0.0f});
    h.rtau.assign((size_t)h.nrow * wid, 0.0f);
    for (int r = 0; r < h.nrow; r++)
        for (int j = 0; j < wid; j++) {
            const int cc = h.row0 + r, c = cc + j - band;
            if (cc < 0 || cc >= nrg || c < 0 || c >= nrg) continue;
            DatEntry &e = h.rcv[(size_t)r * wid + j];
            e.w = 1.0f;
            e.tau = rt[(size_t)cc * nrg + c];
            e.dtau = slope_host(rt, nrg, cc, c, p.drg) * fabsf(p.dh);
            h.rtau[(size_t)r * wid + j] = e.tau;
        }
    return KCIG_OK;
}

int build_source(const kcig_datum_params &p, const float *st, Host &h)
{
    const int ns = p.ns, nh = p.nh, aper = p.aperture, nsg = p.nsg;
    std::vector<int> cs(ns);
    for (int is = 0; is < ns; is++) cs[is] = src_index(p, is);
    if (p.cmp == 0) {
        h.src.assign((size_t)ns * ns, DatEntry{0.0f, 0.0f, 0.0f});
        for (int is = 0; is < ns; is++) {
            const int c = cs[is];
            if (c < 0 || c >= nsg) return set_error(KCIG_ERR_ARG, "Source table too small.");
            const int left = std::max(0, is - aper), right = std::min(ns - 1, is + aper);
            for (int ic = left; ic <= right; ic++) {
                const int cc = cs[ic];
                if (cc < 0 || cc >= nsg) return set_error(KCIG_ERR_ARG, "Source table too small.");
                const float coef = taper_host(left, ic, right, p.taper, 1);
                const float tau = st[(size_t)cc * nsg + c];
                const float dist = p.sdatum * p.sdatum + (float)((ic - is) * (ic - is)) * p.ds * p.ds;
                DatEntry &e = h.src[(size_t)is * ns + ic];
                e.w = term_weight(coef, p.ds, p.sdatum, tau, dist);
                e.tau = tau;
                e.dtau = slope_host(st, nsg, cc, c, p.dsg) * fabsf(p.ds);
            }
        }
        return KCIG_OK;
    }
    // the common-receiver walk (:556-579), in float as the reference
    const float ds = p.ds, dh = p.dh;
    const float s = fabsf((float)(ns - 1) * ds), hl = fabsf((float)(nh - 1) * dh);
    const bool wide = fabsf(ds) >= fabsf(dh);
    const int jump = wide ? 1 : f2i(dh / ds + 0.5f);
    const float dr = wide ? fabsf(dh) : fabsf(ds);
    const int nr = f2i((s + hl) / dr + 1.5f);
    if (jump < 1) return set_error(KCIG_ERR_ARG, "kcig_datum_freq: cmp=1 needs dh / ds >= 1 when |ds| < |dh|");
    if (nr < 0 || (long long)nr * ns > 0x7fffffffLL) return set_error(KCIG_ERR_ARG, "kcig_datum_freq: cmp=1 gather count");
    h.nr = nr;
    h.jump = jump;
    h.sleft.resize(nr);
    h.sright.resize(nr);
    h.ihmap.assign((size_t)nr * ns, -1);
    h.goff.assign((size_t)ns * nh + 1, 0);
    const float as = ds <= 0.f ? -1.f : 0.f, ah = dh <= 0.f ? -1.f : 0.f, bl = ds <= 0.f ? 0.f : -1.f;
    for (int ir = 0; ir < nr; ir++) {
        const float r = (float)ir * dr + as * s + ah * hl;
        int sl = f2i(((float)ir * dr + as * s + bl * hl) / ds + 0.5f);
        int sr = f2i(((float)ir * dr + as * s + as * hl) / ds + 0.5f);
        if (sl < 0) sl = 0;
        if (sr > ns - 1) sr = ns - 1;
        const int left = f2i((r - (float)sl * ds) / dh + 0.5f);
        if (left < 0 || left > nh - 1) sl++;
        const int right = f2i((r - (float)sr * ds) / dh + 0.5f);
        if (right < 0 || right > nh - 1) sr--;
        h.sleft[ir] = sl;
        h.sright[ir] = sr;
        for (int is = sl; is <= sr; is += jump) {
            if (is < 0 || is >= ns) continue;
            const int c = cs[is];
            if (c < 0 || c >= nsg) return set_error(KCIG_ERR_ARG, "Source table too small.");
            const int ih = f2i((r - (float)is * ds) / dh + 0.5f);
            if (ih < 0 || ih >= nh) continue;
            h.ihmap[(size_t)is * nr + ir] = ih;
            h.goff[(size_t)is * nh + ih + 1]++;
        }
    }
    // the gathers that hold each output trace, in order of r
    for (size_t t = 0; t < (size_t)ns * nh; t++) h.goff[t + 1] += h.goff[t];
    h.gath.resize(h.goff.back());
    std::vector<int> at(h.goff.begin(), h.goff.end() - 1);
    for (int ir = 0; ir < nr; ir++)
        for (int is = std::max(0, h.sleft[ir]); is <= std::min(ns - 1, h.sright[ir]); is++) {
            const int ih = h.ihmap[(size_t)is * nr + ir];
            if (ih >= 0) h.gath[at[(size_t)is * nh + ih]++] = ir;
        }
    // half of taper_weight (:229-240), by the distance from a window's end
    if (p.taper > 0) {
        const float width = (float)p.taper * (float)jump;
        for (int k = 0; k < ns && (float)k < width; k++)
            h.ramp.push_back((float)(0.5 * (1.0 - cos(M_PI * (double)((float)k / width)))));
    }
    const double kw = (double)ds * (double)p.sdatum / M_PI;
    h.src.assign((size_t)ns * ns, DatEntry{0.0f, 0.0f, 0.0f});
    h.sgw.assign((size_t)ns * ns, 0.0);
    const float jds = fabsf((float)jump * ds);
    for (int is = 0; is < ns; is++)
        for (int ic = std::max(0, is - jump * aper); ic <= std::min(ns - 1, is + jump * aper); ic++) {
            const int c = cs[is], cc = cs[ic];
            if (c < 0 || c >= nsg || cc < 0 || cc >= nsg) continue;
            DatEntry &e = h.src[(size_t)is * ns + ic];
            e.w = 1.0f;
            e.tau = st[(size_t)cc * nsg + c];
            e.dtau = slope_host(st, nsg, cc, c, p.dsg) * jds;
            const float dist = p.sdatum * p.sdatum + (float)((ic - is) * (ic - is)) * ds * ds;
            h.sgw[(size_t)is * ns + ic] = kw * (double)e.tau / (double)dist;
        }
    return KCIG_OK;
}

int launch_op(const DatEntry *ent, int ne, float2 *out, int f0, int nf, int nfft, int K, const kcig_datum_params &p,
              cudaStream_t st, int &launches)
{
    if (ne <= 0) return KCIG_OK;
    DatOpArgs a;
    a.ent = ent;
    a.ne = ne;
    a.out = out;
    a.f0 = f0;
    a.nf = nf;
    a.nfft = nfft;
    a.K = K;
    a.dt = p.dt;
    a.antialias = p.antialias;
    // shared memory: cos, sin and frequency of the chunk's frequencies, then
    // each thread's filter samples (128 threads)
    const size_t sm = (size_t)nf * 2 * sizeof(double) + (size_t)(nf + 1) / 2 * sizeof(double) +
                      (size_t)std::min(K, kFilterMax) * 128 * sizeof(double);
    KCIG_TRY(set_dyn_smem((const void *)k_dat_op, (int)sm));
    k_dat_op<<<(ne + 127) / 128, 128, sm, st>>>(a);
    launches++;
    KCIG_CUDA(cudaGetLastError());
    return KCIG_OK;
}

// Q of the FFT form: the smallest of 8 .. 64 that holds the filter's K + 1
// samples, with at least two residues; 0 (longer filters): Horner's rule
int op_points(int K, int nfft)
{
    if (K < 1) return 0;
    for (int Q = 8; Q <= 64; Q *= 2)
        if (K + 1 <= Q) return nfft >= 2 * Q ? Q : 0;
    return 0;
}

template <int Q>
int launch_op_q(const DatFftArgs &a, cudaStream_t st)
{
    KCIG_TRY(set_dyn_smem((const void *)k_dat_op_fft<Q>, dat_op_smem<Q>()));
    constexpr int EB = 2048 / Q;
    k_dat_op_fft<Q><<<dim3((a.ne + EB - 1) / EB, (a.na + kOpGroup - 1) / kOpGroup), 256, dat_op_smem<Q>(), st>>>(a);
    KCIG_CUDA(cudaGetLastError());
    return KCIG_OK;
}

int launch_op_fft(const DatEntry *ent, int ne, float2 *out, const C64 *tw, int Q, int M, int a0, int na, int nfft, int K,
                  const kcig_datum_params &p, cudaStream_t st, int &launches)
{
    if (ne <= 0) return KCIG_OK;
    DatFftArgs a;
    a.ent = ent;
    a.tw = tw;
    a.out = out;
    a.ne = ne;
    a.a0 = a0;
    a.na = na;
    a.M = M;
    a.K = K;
    a.nfft = nfft;
    a.dt = p.dt;
    a.antialias = p.antialias;
    launches++;
    switch (Q) {
    case 8: return launch_op_q<8>(a, st);
    case 16: return launch_op_q<16>(a, st);
    case 32: return launch_op_q<32>(a, st);
    default: return launch_op_q<64>(a, st);
    }
}

int launch_gemm(const float2 *A, long long sA, int lda, const float2 *B, long long sB, int ldb, float2 *C,
                long long sC, int ldc, int M, int N, int K, int band, int band_rows, int batch, cudaStream_t st,
                int &launches)
{
    CGemmArgs g;
    g.a_trans = 0;
    g.a_vec = 0;
    g.A = A;
    g.B = B;
    g.C = C;
    g.sA = sA;
    g.sB = sB;
    g.sC = sC;
    g.lda = lda;
    g.ldb = ldb;
    g.ldc = ldc;
    g.M = M;
    g.N = N;
    g.K = K;
    g.band = band;
    g.band_rows = band_rows;
    for (int z0 = 0; z0 < batch; z0 += 65535) {
        const int nz = std::min(65535, batch - z0);
        CGemmArgs gz = g;
        gz.A += (size_t)z0 * sA;
        gz.B += (size_t)z0 * sB;
        gz.C += (size_t)z0 * sC;
        k_cgemm<<<dim3((N + 63) / 64, (M + 63) / 64, nz), 256, 0, st>>>(gz);
        launches++;
        KCIG_CUDA(cudaGetLastError());
    }
    return KCIG_OK;
}

int launch_gemm_tc(const float2 *A, long long sA, int lda, const float2 *B, long long sB, int ldb, float2 *C,
                   long long sC, int ldc, int M, int N, int K, int band, int band_rows, int batch, int *status,
                   cudaStream_t st, int &launches, int a_trans = 0)
{
    CGemmArgs g;
    g.a_trans = a_trans;
    g.a_vec = !a_trans && lda % 2 == 0 && sA % 2 == 0 && ((uintptr_t)A & 15) == 0;
    g.A = A;
    g.B = B;
    g.C = C;
    g.sA = sA;
    g.sB = sB;
    g.sC = sC;
    g.lda = lda;
    g.ldb = ldb;
    g.ldc = ldc;
    g.M = M;
    g.N = N;
    g.K = K;
    g.band = band;
    g.band_rows = band_rows;
    KCIG_TRY(set_dyn_smem((const void *)k_cgemm_tc, tcg::SMEM));
    for (int z0 = 0; z0 < batch; z0 += 65535) {
        const int nz = std::min(65535, batch - z0);
        CGemmArgs gz = g;
        gz.A += (size_t)z0 * sA;
        gz.B += (size_t)z0 * sB;
        gz.C += (size_t)z0 * sC;
        k_cgemm_tc<<<dim3((N + tcg::TNC - 1) / tcg::TNC, (M + tcg::TM - 1) / tcg::TM, nz), tcg::THREADS, tcg::SMEM, st>>>(
            gz, status);
        launches++;
        KCIG_CUDA(cudaGetLastError());
    }
    return KCIG_OK;
}

// the GEMMs of cmp = 0 run on the tensor cores; KCIG_DATUM_GEMM=simt selects
// the FP32 CUDA-core kernel instead (a diagnostic comparison)
bool gemm_on_tensor_cores()
{
    const char *e = getenv("KCIG_DATUM_GEMM");
    return !(e && strcmp(e, "simt") == 0);
}

// traces per transform batch: as many as keep a batch's padded traces at
// 1 GB, or KCIG_DATUM_BATCH (smaller batches and a tail batch on small cases)
long long transform_batch(long long ntr, int nfft)
{
    long long b = ((long long)1 << 28) / nfft;
    const char *e = getenv("KCIG_DATUM_BATCH");
    if (e && atoll(e) > 0) b = std::min(b, atoll(e));
    return std::max<long long>(1, std::min<long long>(ntr, b));
}

}  // namespace
}  // namespace kcig

using namespace kcig;

extern "C" int kcig_datum_params_init(kcig_datum_params *p)
{
    if (!p) return set_error(KCIG_ERR_ARG, "kcig_datum_params_init: null");
    *p = kcig_datum_params{};
    p->aperture = 50;
    p->taper = 10;
    p->data_taper = 0;
    p->cmp = 1;
    p->antialias = 1.0f;
    p->length = 0.025f;
    p->use_bf = 1;
    p->bf_p = 12;
    p->bf_n_leaf = 16;
    p->bf_panel_levels = 1;
    p->bf_amp_eps = 1e-20f;
    p->bf_phase_tol = 2.0f;
    return KCIG_OK;
}

extern "C" int kcig_datum_sizes(const kcig_datum_params *p, const float *stable, const float *rtable, int *nsam,
                                int *nfft)
{
    if (!p || !stable || !rtable || !nsam || !nfft) return set_error(KCIG_ERR_ARG, "kcig_datum_sizes: null argument");
    KCIG_TRY(validate(*p));
    return sizes(*p, stable, rtable, nsam, nfft);
}

extern "C" int kcig_datum_release(void)
{
    int dev = 0;
    KCIG_CUDA(cudaGetDevice(&dev));
    DatumCache &c = cache_of(dev);
    std::lock_guard<std::mutex> hold(c.mu);
    free_buffers(c);
    free_pair(c.full);
    free_pair(c.tail);
    for (cudaEvent_t e : c.ev) cudaEventDestroy(e);
    c.ev.clear();
    if (c.copy) cudaStreamDestroy(c.copy);
    c.copy = nullptr;
    return eik_release_pool();
}

extern "C" int kcig_datum_last_timing(float *ms5, int *launches)
{
    if (ms5)
        for (int i = 0; i < 5; i++) ms5[i] = g_last_ms[i];
    if (launches) *launches = g_last_launches;
    return KCIG_OK;
}

extern "C" int kcig_green_slice(const float *table, int nz, int nx, int ngx, float oz, float ox, float dz, float dx,
                                float ogx, float dgx, float datum, float *tgreen, int memory, void *stream)
{
    if (!table || !tgreen || nz <= 0 || nx <= 0 || ngx <= 0) return set_error(KCIG_ERR_ARG, "kcig_green_slice: bad arguments");
    if (memory != KCIG_MEM_HOST && memory != KCIG_MEM_DEVICE) return set_error(KCIG_ERR_ARG, "kcig_green_slice: bad memory kind");
    // src/greensol_auto.cpp:68-69 and :75-82: float operands, double 0.5
    const int idatum = (int)((datum - oz) / dz + 0.5);
    if (idatum < 0 || idatum >= nz) return set_error(KCIG_ERR_ARG, "Datum out of range.");
    std::vector<int> ix(ngx);
    for (int i = 0; i < ngx; i++) {
        const float gx = ogx + (float)i * dgx;
        ix[i] = (int)((gx - ox) / dx + 0.5);
        if (ix[i] < 0 || ix[i] >= nx) return set_error(KCIG_ERR_ARG, "Receiver table too small.");
    }
    if (memory == KCIG_MEM_HOST) {
        for (int i1 = 0; i1 < ngx; i1++)
            for (int i2 = 0; i2 < ngx; i2++)
                tgreen[(size_t)i1 * ngx + i2] = table[((size_t)i1 * nx + ix[i2]) * nz + idatum];
        return KCIG_OK;
    }
    cudaStream_t st = (cudaStream_t)stream;
    DBuf dix;
    KCIG_TRY(upload(dix, ix, st, "table indices"));
    const int n = ngx * ngx;
    k_green_gather<<<(n + 255) / 256, 256, 0, st>>>(table, dix.as<int>(), tgreen, ngx, nx, nz, idatum);
    KCIG_CUDA(cudaGetLastError());
    KCIG_CUDA(cudaStreamSynchronize(st));
    return KCIG_OK;
}

extern "C" int kcig_datum_freq(const kcig_datum_params *pp, const float *stable, const float *rtable, const float *in,
                               float *out, float *interm, int memory, void *stream)
{
    if (!pp || !stable || !rtable || !in || !out) return set_error(KCIG_ERR_ARG, "kcig_datum_freq: null argument");
    if (memory != KCIG_MEM_HOST && memory != KCIG_MEM_DEVICE) return set_error(KCIG_ERR_ARG, "kcig_datum_freq: bad memory kind");
    const kcig_datum_params p = *pp;
    KCIG_TRY(validate(p));
    cudaStream_t st = (cudaStream_t)stream;
    // host copies of the tables (indices, weights and nfft are decided there)
    std::vector<float> sth, rth;
    const float *stp = stable, *rtp = rtable;
    if (memory == KCIG_MEM_DEVICE) {
        sth.resize((size_t)p.nsg * p.nsg);
        rth.resize((size_t)p.nrg * p.nrg);
        KCIG_CUDA(cudaMemcpyAsync(sth.data(), stable, sth.size() * 4, cudaMemcpyDeviceToHost, st));
        KCIG_CUDA(cudaMemcpyAsync(rth.data(), rtable, rth.size() * 4, cudaMemcpyDeviceToHost, st));
        KCIG_CUDA(cudaStreamSynchronize(st));
        stp = sth.data();
        rtp = rth.data();
    }
    int nsam = 0, nfft = 0;
    KCIG_TRY(sizes(p, stp, rtp, &nsam, &nfft));
    if (nfft < 4) return set_error(KCIG_ERR_ARG, "kcig_datum_freq: transform length %d below 4", nfft);
    const int nw = nfft / 2 + 1, K = nsam - 1;
    const int ns = p.ns, nh = p.nh, nt = p.nt;
    const long long ntr = (long long)ns * nh;
    Host h;
    KCIG_TRY(build_receiver(p, rtp, h));  // the receiver side's checks come first, as in the reference
    KCIG_TRY(build_source(p, stp, h));
    // cmp = 0 with shots and receivers on the same positions, tables and
    // datums: Ks[a][b] == Kr[b][a] term for term, so one operator serves both
    // sides (the source side reads it transposed) and is built once
    bool shared_op = p.cmp == 0 && ns == nh && gemm_on_tensor_cores();
    for (size_t a0 = 0; shared_op && a0 < (size_t)ns; a0++)
        for (size_t b0 = 0; b0 < (size_t)ns; b0++) {
            const DatEntry &x = h.src[a0 * ns + b0], &y = h.rcv[b0 * nh + a0];
            if (memcmp(&x, &y, sizeof(DatEntry)) != 0) {
                shared_op = false;
                break;
            }
        }
    std::vector<float> wtr((size_t)ntr);
    for (int is = 0; is < ns; is++) {
        const float ws = edge_host(is, ns, p.data_taper);
        for (int ih = 0; ih < nh; ih++) wtr[(size_t)is * nh + ih] = ws * edge_host(ih, nh, p.data_taper);
    }

    // ---- device buffers and transform plans, kept between calls on this device
    int dev = 0;
    KCIG_CUDA(cudaGetDevice(&dev));
    DatumCache &c = cache_of(dev);
    std::lock_guard<std::mutex> hold(c.mu);
    // declared after the lock: on every return the stream is idle before
    // the next call may reuse the buffers
    struct StreamIdle {
        cudaStream_t s, s2;
        ~StreamIdle()
        {
            cudaStreamSynchronize(s);
            if (s2) cudaStreamSynchronize(s2);
        }
    } idle{st, nullptr};
    int launches = 0;
    const size_t spec_bytes = (size_t)nw * ntr * sizeof(float2);
    const bool tcore = gemm_on_tensor_cores();
    // per-frequency bytes of a chunk: Utmp + both operators
    const size_t op_r = h.rcv.size(), op_s = shared_op ? 0 : h.src.size();
    const size_t per_f = (interm ? 0 : (size_t)ntr * sizeof(float2)) + (op_r + op_s) * sizeof(float2);
    int chunk = (int)std::max<size_t>(1, std::min<size_t>(256, ((size_t)1536 << 20) / std::max<size_t>(per_f, 1)));
    // rows of the spectra in residue order when the operators come from FFTs:
    // a chunk is then a group of residues (Q rows each; the first Q / 2 + 1,
    // the last Q / 2).  Spreads so wide that a residue's Q rows pass the
    // chunk's memory keep Horner's rule, which takes any number of rows: FFTs
    // halve the operators' time, but their GEMMs take ten times that.
    const int Q0 = op_points(K, nfft), Q = chunk >= Q0 ? Q0 : 0, M = Q ? nfft / Q : 0;
    chunk = std::min(chunk, nw);
    const int chunk_res = Q ? std::max(1, chunk / Q) : 0;
    struct Chunk {
        int f0, nf, a0, na;
    };
    std::vector<Chunk> chunks;
    if (Q) {
        auto row_of = [&](int r) { return r == 0 ? 0 : r > M / 2 ? nw : Q / 2 + 1 + (r - 1) * Q; };
        for (int a0 = 0; a0 <= M / 2; a0 += chunk_res) {
            const int a1 = std::min(M / 2 + 1, a0 + chunk_res);
            chunks.push_back({row_of(a0), row_of(a1) - row_of(a0), a0, a1 - a0});
        }
        chunk = 0;
        for (const Chunk &k : chunks) chunk = std::max(chunk, k.nf);
    } else {
        for (int f0 = 0; f0 < nw; f0 += chunk) chunks.push_back({f0, std::min(chunk, nw - f0), 0, 0});
    }
    // transform batches
    const int B = (int)transform_batch(ntr, nfft);
    const int tail = (int)(ntr % B);
    // plans first (their work area is sized with the buffers); a plan that
    // does not fit beside the cached buffers gets a second try without them
    for (int attempt = 0;; attempt++) {
        int rc = make_pair(c.full, nfft, nw, B);
        if (rc == KCIG_OK && tail) rc = make_pair(c.tail, nfft, nw, tail);
        if (rc == KCIG_OK) break;
        if (attempt == 1) return rc;
        free_buffers(c);
    }
    size_t need[CB_COUNT] = {};
    need[CB_U] = spec_bytes;
    if (interm)
        need[CB_UFULL] = spec_bytes;
    else
        need[CB_UT] = (size_t)chunk * ntr * sizeof(float2);
    need[CB_KR] = (size_t)chunk * std::max<size_t>(op_r, 1) * sizeof(float2);
    need[CB_KS] = (size_t)chunk * std::max<size_t>(op_s, 1) * sizeof(float2);
    need[CB_PAD] = (size_t)B * nfft * 4;
    need[CB_SPEC] = (size_t)B * nw * sizeof(float2);
    need[CB_WORK] = std::max<size_t>(16, std::max(c.full.work, tail ? c.tail.work : 0));
    if (memory == KCIG_MEM_HOST) {
        need[CB_IN] = need[CB_OUT] = (size_t)ntr * nt * 4;
        if (interm) need[CB_INTERM] = (size_t)ntr * nt * 4;
    }
    need[CB_STATUS] = sizeof(int);
    need[CB_TW] = Q ? (size_t)(M / 2 + 1) * 2 * Q * sizeof(C64) : 16;
    need[CB_WTR] = upload_bytes(wtr);
    need[CB_RCV] = upload_bytes(h.rcv);
    need[CB_SRC] = upload_bytes(h.src);
    if (p.cmp == 1) {
        need[CB_CABS] = upload_bytes(h.cabs);
        need[CB_GEOM] = upload_bytes(h.geom);
        need[CB_RTAU] = upload_bytes(h.rtau);
        need[CB_SGW] = upload_bytes(h.sgw);
        need[CB_SL] = upload_bytes(h.sleft);
        need[CB_SR] = upload_bytes(h.sright);
        need[CB_IHM] = upload_bytes(h.ihmap);
        need[CB_GOFF] = upload_bytes(h.goff);
        need[CB_GATH] = upload_bytes(h.gath);
        need[CB_RAMP] = upload_bytes(h.ramp);
    }
    KCIG_TRY(ensure_buffers(c, need));
    const CBuf *bf = c.buf;
    cufftResult cr;
    for (FftPair *q : {&c.full, &c.tail}) {
        if (q == &c.tail && !tail) continue;
        for (cufftHandle hq : {q->f, q->b}) {
            if ((cr = cufftSetWorkArea(hq, bf[CB_WORK].p)) != CUFFT_SUCCESS) return cufft_error(cr, "cufftSetWorkArea");
            if ((cr = cufftSetStream(hq, st)) != CUFFT_SUCCESS) return cufft_error(cr, "cufftSetStream");
        }
    }
    const float *d_in = in;
    float *d_out = out, *d_interm = interm;
    cudaStream_t cs = nullptr;
    if (memory == KCIG_MEM_HOST) {
        if (!c.copy) KCIG_CUDA(cudaStreamCreateWithFlags(&c.copy, cudaStreamNonBlocking));
        cs = idle.s2 = c.copy;
        d_in = bf[CB_IN].as<float>();
        d_out = bf[CB_OUT].as<float>();
        if (interm) d_interm = bf[CB_INTERM].as<float>();
    }
    KCIG_CUDA(cudaMemsetAsync(bf[CB_STATUS].p, 0, sizeof(int), st));
    KCIG_TRY(upload_to(bf[CB_WTR], wtr, st));
    KCIG_TRY(upload_to(bf[CB_RCV], h.rcv, st));
    KCIG_TRY(upload_to(bf[CB_SRC], h.src, st));
    if (p.cmp == 1) {
        KCIG_TRY(upload_to(bf[CB_CABS], h.cabs, st));
        KCIG_TRY(upload_to(bf[CB_GEOM], h.geom, st));
        KCIG_TRY(upload_to(bf[CB_RTAU], h.rtau, st));
        KCIG_TRY(upload_to(bf[CB_SGW], h.sgw, st));
        KCIG_TRY(upload_to(bf[CB_SL], h.sleft, st));
        KCIG_TRY(upload_to(bf[CB_SR], h.sright, st));
        KCIG_TRY(upload_to(bf[CB_IHM], h.ihmap, st));
        KCIG_TRY(upload_to(bf[CB_GOFF], h.goff, st));
        KCIG_TRY(upload_to(bf[CB_GATH], h.gath, st));
        KCIG_TRY(upload_to(bf[CB_RAMP], h.ramp, st));
    }
    float2 *const U = bf[CB_U].as<float2>();
    float2 *const Kr = bf[CB_KR].as<float2>(), *const Ks = bf[CB_KS].as<float2>();
    float *const pad = bf[CB_PAD].as<float>();
    float2 *const spec = bf[CB_SPEC].as<float2>();
    int *const dstatus = bf[CB_STATUS].as<int>();
    // events: four stage bounds, four per chunk of frequencies (read once
    // the call has finished, so the chunks are queued back to back), and for
    // host-memory calls per batch of traces: its input copied, its interm
    // and output traces finished
    const int nchunk = (int)chunks.size();
    const int nbatch = (int)((ntr + B - 1) / B);
    while (c.ev.size() < 4 + 4 * (size_t)nchunk + 3 * (size_t)nbatch) {
        cudaEvent_t e;
        KCIG_CUDA(cudaEventCreate(&e));
        c.ev.push_back(e);
    }
    cudaEvent_t *const ev = c.ev.data();
    cudaEvent_t *const bev = ev + 4 + 4 * nchunk;
    // host-memory calls: a batch's input goes over on the copy stream while
    // the batch before it is transformed; its output comes back once its
    // inverse transform is done, while later batches are transformed
    auto copy_in = [&](int ib) -> int {
        const long long t0 = (long long)ib * B;
        const size_t n = (size_t)std::min<long long>(B, ntr - t0) * nt;
        KCIG_CUDA(cudaMemcpyAsync(bf[CB_IN].as<float>() + t0 * nt, in + t0 * nt, n * 4, cudaMemcpyHostToDevice, cs));
        KCIG_CUDA(cudaEventRecord(bev[ib], cs));
        return KCIG_OK;
    };
    if (cs) KCIG_TRY(copy_in(0));
    KCIG_CUDA(cudaEventRecord(ev[0], st));
    // ---- forward: reverse, taper, pad, R2C, to frequency-major
    for (long long t0 = 0, ib = 0; t0 < ntr; t0 += B, ib++) {
        const int nb = (int)std::min<long long>(B, ntr - t0);
        if (cs) KCIG_CUDA(cudaStreamWaitEvent(st, bev[ib], 0));
        k_dat_prep<<<dim3((nfft / 4 + 255) / 256, std::min(nb, 1024)), 256, 0, st>>>(d_in, bf[CB_WTR].as<float>(), pad,
                                                                                    (int)t0, nb, nt, nfft);
        launches++;
        KCIG_CUDA(cudaGetLastError());
        if ((cr = cufftExecR2C(nb == B ? c.full.f : c.tail.f, (cufftReal *)pad, (cufftComplex *)spec)) != CUFFT_SUCCESS)
            return cufft_error(cr, "cufftExecR2C");
        launches++;
        k_dat_to_fmajor<<<dim3((nw + 31) / 32, (nb + 31) / 32), dim3(32, 8), 0, st>>>(spec, U, (int)t0, nb, nw,
                                                                                     (int)ntr, Q, M);
        launches++;
        KCIG_CUDA(cudaGetLastError());
        if (cs && ib + 1 < nbatch) KCIG_TRY(copy_in((int)ib + 1));
    }
    KCIG_CUDA(cudaEventRecord(ev[1], st));
    // ---- per chunk of frequencies: operators, receiver side, source side
    if (Q) {
        const int n = (M / 2 + 1) * 2 * Q;
        k_dat_twiddles<<<(n + 255) / 256, 256, 0, st>>>(bf[CB_TW].as<C64>(), Q, M);
        launches++;
        KCIG_CUDA(cudaGetLastError());
    }
    auto build_op = [&](const DatEntry *ent, size_t ne, float2 *K_out, const Chunk &k) -> int {
        if (Q)
            return launch_op_fft(ent, (int)ne, K_out, bf[CB_TW].as<C64>(), Q, M, k.a0, k.na, nfft, K, p, st, launches);
        return launch_op(ent, (int)ne, K_out, k.f0, k.nf, nfft, K, p, st, launches);
    };
    for (int ic = 0; ic < nchunk; ic++) {
        const int f0 = chunks[ic].f0, nf = chunks[ic].nf;
        cudaEvent_t *const ce = ev + 4 + 4 * ic;
        float2 *Uc = U + (size_t)f0 * ntr;
        float2 *Utc = interm ? bf[CB_UFULL].as<float2>() + (size_t)f0 * ntr : bf[CB_UT].as<float2>();
        KCIG_CUDA(cudaEventRecord(ce[0], st));
        KCIG_TRY(build_op(bf[CB_RCV].as<DatEntry>(), op_r, Kr, chunks[ic]));
        if (op_s) KCIG_TRY(build_op(bf[CB_SRC].as<DatEntry>(), op_s, Ks, chunks[ic]));
        KCIG_CUDA(cudaEventRecord(ce[1], st));
        if (p.cmp == 0) {
            if (tcore)
                KCIG_TRY(launch_gemm_tc(Uc, ntr, nh, Kr, (long long)nh * nh, nh, Utc, ntr, nh, ns, nh, nh,
                                        p.aperture >= 0 ? p.aperture : 0, 0, nf, dstatus, st, launches));
            else
                KCIG_TRY(launch_gemm(Uc, ntr, nh, Kr, (long long)nh * nh, nh, Utc, ntr, nh, ns, nh, nh,
                                     p.aperture >= 0 ? p.aperture : 0, 0, nf, st, launches));
        } else {
            RcvCmp1Args a;
            a.U = Uc;
            a.Utmp = Utc;
            a.P = Kr;
            a.Ptau = bf[CB_RTAU].as<float>();
            a.cabs = bf[CB_CABS].as<int>();
            a.geom = bf[CB_GEOM].as<float>();
            a.ns = ns;
            a.nh = nh;
            a.aper = p.aperture;
            a.band = h.band;
            a.row0 = h.row0;
            a.nrow = h.nrow;
            a.nf = nf;
            a.sU = ntr;
            k_dat_rcv_cmp1<<<dim3((unsigned)((ntr + 127) / 128), (nf + kCmp1F - 1) / kCmp1F), 128, 0, st>>>(a);
            launches++;
            KCIG_CUDA(cudaGetLastError());
        }
        KCIG_CUDA(cudaEventRecord(ce[2], st));
        if (p.cmp == 0) {
            if (tcore && shared_op)
                KCIG_TRY(launch_gemm_tc(Kr, (long long)nh * nh, nh, Utc, ntr, nh, Uc, ntr, nh, ns, nh, ns,
                                        p.aperture >= 0 ? p.aperture : 0, 1, nf, dstatus, st, launches, 1));
            else if (tcore)
                KCIG_TRY(launch_gemm_tc(Ks, (long long)ns * ns, ns, Utc, ntr, nh, Uc, ntr, nh, ns, nh, ns,
                                        p.aperture >= 0 ? p.aperture : 0, 1, nf, dstatus, st, launches));
            else
                KCIG_TRY(launch_gemm(Ks, (long long)ns * ns, ns, Utc, ntr, nh, Uc, ntr, nh, ns, nh, ns,
                                     p.aperture >= 0 ? p.aperture : 0, 1, nf, st, launches));
        } else {
            SrcCmp1Args a;
            a.Utmp = Utc;
            a.Uout = Uc;
            a.P = Ks;
            a.gw = bf[CB_SGW].as<double>();
            a.sleft = bf[CB_SL].as<int>();
            a.sright = bf[CB_SR].as<int>();
            a.ihmap = bf[CB_IHM].as<int>();
            a.goff = bf[CB_GOFF].as<int>();
            a.gath = bf[CB_GATH].as<int>();
            a.ramp = bf[CB_RAMP].as<float>();
            a.ns = ns;
            a.nh = nh;
            a.nr = h.nr;
            a.aper = p.aperture;
            a.jump = h.jump;
            a.nramp = (int)h.ramp.size();
            a.nf = nf;
            a.sUout = ntr;
            k_dat_src_cmp1<<<dim3((unsigned)((ntr + 127) / 128), (nf + kCmp1F - 1) / kCmp1F), 128, 0, st>>>(a);
            launches++;
            KCIG_CUDA(cudaGetLastError());
        }
        KCIG_CUDA(cudaEventRecord(ce[3], st));
    }
    KCIG_CUDA(cudaEventRecord(ev[2], st));
    // ---- inverse: to trace-major, C2R, scale, reverse, trim
    auto inverse = [&](const float2 *Usrc, float *dst, int reverse, cudaEvent_t *done) -> int {
        for (long long t0 = 0, ib = 0; t0 < ntr; t0 += B, ib++) {
            const int nb = (int)std::min<long long>(B, ntr - t0);
            k_dat_to_tmajor<<<dim3((nb + 31) / 32, (nw + 31) / 32), dim3(32, 8), 0, st>>>(Usrc, spec, (int)t0, nb, nw,
                                                                                         (int)ntr, Q, M);
            launches++;
            KCIG_CUDA(cudaGetLastError());
            if ((cr = cufftExecC2R(nb == B ? c.full.b : c.tail.b, (cufftComplex *)spec, (cufftReal *)pad)) != CUFFT_SUCCESS)
                return cufft_error(cr, "cufftExecC2R");
            launches++;
            k_dat_finish<<<dim3((nt + 255) / 256, std::min(nb, 1024)), 256, 0, st>>>(pad, dst, (int)t0, nb, nt, nfft,
                                                                                  1.0f / (float)nfft, reverse);
            launches++;
            KCIG_CUDA(cudaGetLastError());
            if (cs) KCIG_CUDA(cudaEventRecord(done[ib], st));
        }
        return KCIG_OK;
    };
    cudaEvent_t *const done_im = bev + nbatch, *const done_out = bev + 2 * nbatch;
    if (interm) KCIG_TRY(inverse(bf[CB_UFULL].as<float2>(), d_interm, 0, done_im));
    KCIG_TRY(inverse(U, d_out, 1, done_out));
    KCIG_CUDA(cudaEventRecord(ev[3], st));
    if (cs) {
        // queued after every inverse launch, so a copy to pageable memory
        // (which holds the host until it is done) leaves the device busy
        auto copy_out = [&](float *host, const float *dev_src, const cudaEvent_t *done) -> int {
            for (long long t0 = 0, ib = 0; t0 < ntr; t0 += B, ib++) {
                const size_t n = (size_t)std::min<long long>(B, ntr - t0) * nt;
                KCIG_CUDA(cudaStreamWaitEvent(cs, done[ib], 0));
                KCIG_CUDA(cudaMemcpyAsync(host + t0 * nt, dev_src + t0 * nt, n * 4, cudaMemcpyDeviceToHost, cs));
            }
            return KCIG_OK;
        };
        if (interm) KCIG_TRY(copy_out(interm, d_interm, done_im));
        KCIG_TRY(copy_out(out, d_out, done_out));
        KCIG_CUDA(cudaStreamSynchronize(cs));
    }
    int dev_status = 0;
    KCIG_CUDA(cudaMemcpyAsync(&dev_status, dstatus, sizeof(int), cudaMemcpyDeviceToHost, st));
    KCIG_CUDA(cudaStreamSynchronize(st));
    if (dev_status)
        return set_error(KCIG_ERR_DEVICE, "kcig_datum_freq: a tensor-core GEMM gave up waiting (stage %d)", dev_status);
    float t, ms_op = 0.0f, ms_r = 0.0f, ms_s = 0.0f;
    for (int ic = 0; ic < nchunk; ic++) {
        const cudaEvent_t *ce = ev + 4 + 4 * ic;
        cudaEventElapsedTime(&t, ce[0], ce[1]);
        ms_op += t;
        cudaEventElapsedTime(&t, ce[1], ce[2]);
        ms_r += t;
        cudaEventElapsedTime(&t, ce[2], ce[3]);
        ms_s += t;
    }
    cudaEventElapsedTime(&t, ev[0], ev[1]);
    g_last_ms[0] = t;
    g_last_ms[1] = ms_op;
    g_last_ms[2] = ms_r;
    g_last_ms[3] = ms_s;
    cudaEventElapsedTime(&t, ev[2], ev[3]);
    g_last_ms[4] = t;
    g_last_launches = launches;
    return KCIG_OK;
}
