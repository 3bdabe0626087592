// ps_fit.cuh -- fit kernels of the GB300 period-search engine (sm_103a),
// shared by the single-object launchers (ps_engine.cu) and the multi-object
// packed launch (ps_pack.cu).
//
// One CTA is one fit slot.  A slot pulls fits (period index, initial pole)
// from a device work counter and runs the whole Levenberg-Marquardt fit on
// the device: model evaluation (the reference's mrqcof with curv, blmatrix,
// bright and conv), the damped normal-equation solve (gauss_errc), the
// accept/reject and lambda update (mrqmin) and the stop rule of the driver
// loop (period_search_BOINC.cpp:868-893).  Nothing returns to the host until
// every fit of the launch is done.
//
// Evaluation of one parameter vector, per tile of P observations:
//   1. point set-up (one thread per point, FP64): solar phase angle, phase
//      function, body rotation f = fmod(omega*t + phi0, 2*pi) and the rotated
//      Earth/Sun directions with their beta/lambda/omega derivatives;
//   2. facet stage (one warp per point, lanes over facets): mu, mu0, the
//      Lommel-Seeliger + Lambert law, brightness, rotation and scattering
//      derivatives; lit facets write W[p][i] = Darea_i * s_pi * g_i;
//   3. shape contraction J[p][k] = Scale_p * sum_i W[p][i] * Dsph[i][k]
//      (the reference's sum over lit facets of dbr * Dg);
//   4. relative lightcurves: per-lightcurve sums, then the renormalisation of
//      mrqcof.c:90-104 from a per-slot scratch copy of the lightcurve's rows;
//   5. normal-matrix accumulation alpha = J^T W J, beta, chi^2 over the free
//      parameters, each alpha element summed over points in data order.
// The three convexity rows (conv.c) are three more rows of the same
// contraction with W[c][i] = Darea_i * g_i * n_i[c].
//
// The mixed form runs the contraction on the tensor cores when the shape
// tables allow it (tensor_basis_ok): tcgen05 FP16 MMAs with the basis split
// into high and low FP16 parts (scaled by a power of two) resident in Tensor
// Memory for the CTA's lifetime (A = [Dsph_hi^T; Dsph_lo^T], 128 lanes, two
// facets per column) and W split the same way in shared memory (B), so that
// the four partial products give the contraction to FP32 accuracy; the
// normal-matrix accumulation runs as TF32 high/low MMAs.  Otherwise both run
// on the SIMT pipes.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <mutex>
#include <type_traits>

#include "ps_engine.h"
#include "ps_tc.cuh"

namespace psg {

namespace {

constexpr double kPi = 3.14159265358979323846;
constexpr double kTwoPi = 2 * kPi;
constexpr double kRad2Deg = 180 / kPi;
constexpr double kDeg2Rad = kPi / 180;
constexpr double kTinyMu = 1e-8;
// 2*pi split for the mixed form's phase reduction: hi = 2*pi rounded to
// double, lo = 2*pi - hi.
constexpr double kTwoPiHi = 6.283185307179586;
constexpr double kTwoPiLo = 2.4492935982947064e-16;
constexpr double kInvTwoPi = 0.15915494309189535;

__constant__ double c_beta_pole[PS_N_POLES] = {0, 0, 0, 0, 60, 60, 60, -60, -60, -60};
// blmatrix.c:9-46 entry by entry: factor a (0 zero, 1 cos beta, 2 sin beta,
// 3 one) | factor b << 2 (0 one, 1 cos lambda, 2 sin lambda) | 16 negated;
// rows of B, then dB/dbeta, then dB/dlambda
__constant__ unsigned char c_bl_code[27] = {5,  9,  18, 27, 7, 0, 6,  10, 1,  22, 26, 17, 0, 0,
                                            0,  5,  9,  18, 25, 5, 0, 23, 27, 0,  26, 6,  0};
__constant__ double c_lambda_pole[PS_N_POLES] = {0, 90, 180, 270, 60, 180, 300, 60, 180, 300};

// Arithmetic type of the facet stage, the contraction and the model rows.
template <int FORM> struct RealOf { using T = double; };
template <> struct RealOf<PS_FORM_MIXED> { using T = float; };

template <int FORM>
struct Smem {
    using R = typename RealOf<FORM>::T;
    double *cg, *atry, *beta, *da, *alpha, *covar, *area, *gv, *ym, *red, *dave, *col, *misc;
    R *areaR, *gvR, *W, *J, *pt;
    R *pt2;       // the other point set-up buffer (== pt unless set-up runs one tile ahead)
    float *accs;  // mixed form: per-point FP32 weights and residuals of a tile
    float *davef; // mixed form: FP32 copy of a relative lightcurve's derivative sums
    R *bmat;      // [27] rotation matrix and its beta/lambda derivatives, [27..29] phase
                  // function a, d, k, [30] Lommel-Seeliger and [31] Lambert weight
    float *dsph;  // FP32 basis in shared memory (mixed form), or nullptr
    // tensor-core contraction: operand tiles, MMA-completion barrier, Tensor
    // Memory address slot and the abort flag set when a wait gives up
    unsigned char *bhi, *blo;
    uint64_t *mbar, *mbar2;   // completion of the contraction MMAs / of the alpha MMAs
    float4 *fac;              // per facet pair (2j, 2j + 1): {nx, nx', ny, ny'}, {nz, nz', Area, Area'} (fac_at)
    float *fpart;             // [4][P][9] facet-sum partials of the four facet quarters
    unsigned char *aop;       // alpha/beta MMA operands
    unsigned char *pref;      // per-point data prefetched for the contraction window
    int *flist;               // the free parameters' columns (tensor-core path)
    // FP64 form: lit-facet count of each point of the tile, and its lit
    // facets in increasing order ([P][wcols], the W row holds their values)
    int *nlit;
    uint16_t *lidx;
    double *phase;          // FP64 form: [4][phase_tiles * P] first set-up part of the CTA's next tiles
    uint32_t *tslot;
    int *abort;
};

template <int FORM>
__device__ inline Smem<FORM> carve(char *base, const SlotLayout &L)
{
    using R = typename RealOf<FORM>::T;
    Smem<FORM> s;
    s.cg = reinterpret_cast<double *>(base + L.cg);
    s.atry = reinterpret_cast<double *>(base + L.atry);
    s.beta = reinterpret_cast<double *>(base + L.beta);
    s.da = reinterpret_cast<double *>(base + L.da);
    s.alpha = reinterpret_cast<double *>(base + L.alpha);
    s.covar = reinterpret_cast<double *>(base + L.covar);
    s.area = reinterpret_cast<double *>(base + L.area);
    s.gv = reinterpret_cast<double *>(base + L.gv);
    s.areaR = reinterpret_cast<R *>(base + L.areaR);
    s.gvR = reinterpret_cast<R *>(base + L.gvR);
    s.W = reinterpret_cast<R *>(base + L.W);
    s.J = reinterpret_cast<R *>(base + L.J);
    s.pt = reinterpret_cast<R *>(base + L.pt);
    s.pt2 = reinterpret_cast<R *>(base + L.pt2);
    s.accs = reinterpret_cast<float *>(base + L.accs);
    s.davef = reinterpret_cast<float *>(base + L.davef);
    s.bmat = reinterpret_cast<R *>(base + L.bmat);
    s.ym = reinterpret_cast<double *>(base + L.ym);
    s.red = reinterpret_cast<double *>(base + L.red);
    s.dave = reinterpret_cast<double *>(base + L.dave);
    s.col = reinterpret_cast<double *>(base + L.col);
    s.misc = reinterpret_cast<double *>(base + L.misc);
    s.nlit = L.form == PS_FORM_FP64 ? reinterpret_cast<int *>(base + L.lit) : nullptr;
    s.lidx = L.form == PS_FORM_FP64 ? reinterpret_cast<uint16_t *>(base + L.lit + 4 * static_cast<size_t>(L.P))
                                     : nullptr;
    s.phase = L.form == PS_FORM_FP64 ? reinterpret_cast<double *>(base + L.phase) : nullptr;
    s.dsph = L.dsph_smem == kBasisSmem ? reinterpret_cast<float *>(base + L.dsph) : nullptr;
    if (basis_on_tensor(L.dsph_smem)) {
        s.bhi = reinterpret_cast<unsigned char *>(base + L.bhi);
        s.blo = reinterpret_cast<unsigned char *>(base + L.blo);
        s.mbar = reinterpret_cast<uint64_t *>(base + L.tcm);
        s.tslot = reinterpret_cast<uint32_t *>(base + L.tcm + 8);
        s.abort = reinterpret_cast<int *>(base + L.tcm + 12);
        s.mbar2 = reinterpret_cast<uint64_t *>(base + L.tcm + 16);
        s.fac = reinterpret_cast<float4 *>(base + L.fac);
        s.fpart = reinterpret_cast<float *>(base + L.fpart);
        s.aop = reinterpret_cast<unsigned char *>(base + L.aop);
        s.pref = reinterpret_cast<unsigned char *>(base + L.pref);
        s.flist = reinterpret_cast<int *>(base + L.flist);
        // wide path: the SIMT accumulation's weighted rows are staged in the
        // operand region (free between a tile's readback and the next
        // tile's facet stage)
        if (L.dsph_smem == kBasisTensorWide) s.W = reinterpret_cast<R *>(base + L.bhi);
    } else {
        s.bhi = s.blo = nullptr;
        s.mbar = s.mbar2 = nullptr;
        s.tslot = nullptr;
        s.fac = nullptr;
        s.fpart = nullptr;
        s.aop = nullptr;
        s.pref = nullptr;
        s.flist = nullptr;
        s.abort = nullptr;
    }
    return s;
}

// misc slots
enum : int {
    M_CHISQ = 0,   // chi^2 accumulator of the current evaluation
    M_AVE = 1,     // relative-lightcurve model sum
    M_AREA = 2,    // sum of facet areas of the current evaluation
    M_CHK = 3,     // 3 convexity residuals (sum Area*n) of the current evaluation
    M_INVAVE = 6,  // mixed form: 1 / sum of the current relative lightcurve's model
    M_CL = 7,      // exp(log cl)
    M_TRIG = 8,    // cos/sin of the pole angles beta, lambda (4 doubles)
    M_PIV = 12,    // pivot broadcast of the solvers (2 doubles + status)
    M_RED = 16,    // 16 doubles of block-reduction scratch
    M_LM = 32,     // 4 doubles: lambda, ochisq, dev, iter_diff of the fit, broadcast from thread 0
    M_WEXP = 36,   // tensor-core path: exponent of the evaluation's W scale
    M_LIT = 37     // FP64 form: the CTA's count of lit facet-point pairs (an unsigned 64-bit integer)
};

// FP64 form: the CTA's lit facet-point counter in misc.
__device__ inline unsigned long long *lit_counter(double *misc)
{
    return reinterpret_cast<unsigned long long *>(misc + M_LIT);
}

// Facet table of the tensor-core path, interleaved by facet pairs so that
// the facet stage loads each pair's components as FP32x2 register pairs:
// float4 2j = {nx_2j, nx_2j+1, ny_2j, ny_2j+1}, float4 2j + 1 = {nz_2j,
// nz_2j+1, Area_2j, Area_2j+1}.  Component c (0 nx, 1 ny, 2 nz, 3 Area) of
// facet i:
__device__ inline float &fac_at(float4 *fac, int i, int c)
{
    return reinterpret_cast<float *>(fac)[(i >> 1) * 8 + 2 * c + (i & 1)];
}

// Row j of packed lower-triangle element e (j*(j+1)/2 <= e < (j+1)*(j+2)/2),
// from an FP32 square root corrected in integers.
__device__ inline int tri_row(int e)
{
    int j = static_cast<int>((sqrtf(8.0f * static_cast<float>(e) + 1.0f) - 1.0f) * 0.5f);
    while (j * (j + 1) / 2 > e) j--;
    while ((j + 1) * (j + 2) / 2 <= e) j++;
    return j;
}

constexpr int kSlotThreads = threads_of<PS_FORM_MIXED>();   // of a whole CTA of the mixed form

// The threads of one fit.  A fit slot is a CTA, or (NT = kTeamThreads) one of
// the two teams of a CTA that runs two fits side by side (fit_kernel_pair):
// the thread's number in its team, and the team's barrier (named barriers 2
// and 3; 1, 4 and 5 serve the Cholesky solve's helper warp).
template <int NT>
__device__ inline int team_thread()
{
    return NT == kTeamThreads ? static_cast<int>(threadIdx.x) % kTeamThreads : static_cast<int>(threadIdx.x);
}
template <int NT>
__device__ inline void team_sync()
{
    if constexpr (NT == kTeamThreads) __barrier_sync_count(2 + threadIdx.x / kTeamThreads, NT);
    else __syncthreads();
}

template <class T>
__device__ inline T warp_sum(T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Asynchronous global -> shared copies (cp.async, 8 or 16 bytes, both
// addresses aligned to the size), completed by cp_async_wait_all of the
// issuing thread.
__device__ inline void cp_async8(void *dst_smem, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst_smem))),
                 "l"(src)
                 : "memory");
}
__device__ inline void cp_async16(void *dst_smem, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst_smem))),
                 "l"(src)
                 : "memory");
}
__device__ inline void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ inline void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Rotation phase omega*t + phi0 reduced to [0, 2*pi).  The FP64 form rounds
// the product and the sum separately and reduces with fmod, as the
// reference does (matrix.c:21-22).  The mixed form reduces in FP64 with a
// two-part 2*pi (the product rounded once), exact to ~1e-16 rad, and hands
// the phase on in FP32 (its only use is the FP32 cos/sin), so the final
// wrap into [0, 2*pi) runs in FP32.
__device__ inline double rotation_phase_fp64(double omg, double t, double phi0)
{
    return fmod(__dadd_rn(__dmul_rn(omg, t), phi0), kTwoPi);
}

__device__ inline float rotation_phase_mixed(double omg, double t, double phi0)
{
    constexpr float kTwoPiF = 6.28318548f;   // 2*pi rounded to FP32
    const double x = fma(omg, t, phi0);
    const double q = floor(x * kInvTwoPi);
    double f = fma(-q, kTwoPiHi, x);
    f = fma(-q, kTwoPiLo, f);
    float ff = static_cast<float>(f);
    if (ff < 0.f) ff += kTwoPiF;
    if (ff >= kTwoPiF) ff -= kTwoPiF;
    return ff;
}

// FP64 form: sum_i W[p][i] Dsph[i][k] (ds = Dsph + k) for point p of the
// tile.  Model rows sum over the point's lit facets, in increasing order as
// bright.c:79-86 does (a dense sum over all facets adds only exact zeros,
// so the two agree bit for bit); convexity rows sum over every facet.
template <class S>
__device__ inline double contract_fp64(const S &s, const double *ds, int p, int C, int F, int wcols, bool conv)
{
    const double *Wp = s.W + static_cast<size_t>(p) * wcols;
    double acc = 0;
    if (conv) {
        for (int i = 0; i < F; i++) acc = acc + Wp[i] * ds[static_cast<size_t>(i) * C];
    } else {
        const uint16_t *idx = s.lidx + static_cast<size_t>(p) * wcols;
        const int n = s.nlit[p];
        for (int j = 0; j < n; j++) acc = acc + Wp[j] * ds[static_cast<size_t>(idx[j]) * C];
    }
    return acc;
}

// Lit-facet terms of the Lommel-Seeliger + Lambert law (bright.c:65-74,
// 116-117).  The reference divides four times by mu + mu0; both forms
// multiply by one reciprocal instead (the FP64 form's correctly rounded, so
// each quotient is within an ulp of the reference's; the mixed form's
// approximate).
template <class R, int FORM>
struct LitTerms {
    R sv, dsmu, dsmu0, dcls_w;  // s, ds/dmu, ds/dmu0, mu*mu0/(mu+mu0)
    __device__ inline LitTerms(R mu, R mu0, R cl, R cls)
    {
        const R dnom = mu + mu0;
        if constexpr (FORM == PS_FORM_FP64) {
            const R r = 1.0 / dnom;
            sv = mu * mu0 * (cl + cls * r);
            const R q0 = mu0 * r, q1 = mu * r;
            dsmu = cls * (q0 * q0) + cl * mu0;
            dsmu0 = cls * (q1 * q1) + cl * mu;
            dcls_w = mu * mu0 * r;
        } else {
            R r;
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(dnom));   // ~1 ulp: the mixed form's budget
            sv = mu * mu0 * (cl + cls * r);
            const R q0 = mu0 * r, q1 = mu * r;
            dsmu = cls * (q0 * q0) + cl * mu0;
            dsmu0 = cls * (q1 * q1) + cl * mu;
            dcls_w = mu * mu0 * r;
        }
    }
};

// One butterfly level over lane bit m: of the pair (a, c) a lane keeps a
// (bit clear) or c (bit set), adding the partner lane's copy of it; one
// shuffle carries the half each lane gives away.  ia, ic: the values' ids.
__device__ inline double fold_pair(double a, double c, int ia, int ic, int m, int lane, int &id)
{
    const bool hi = (lane & m) != 0;
    const double give = hi ? a : c, keep = hi ? c : a;
    id = hi ? ic : ia;
    return keep + __shfl_xor_sync(0xffffffffu, give, m);
}

// Sums nine FP64 values over the warp and stores sum k at out[k] (the last at
// out8): every level pairs the same lanes as warp_sum, so each sum is
// warp_sum's bit for bit, in 12 shuffles and 12 additions instead of 45.  Each
// sum ends in the lanes that kept it; they store it (the same value).
__device__ inline void warp_sum9(const double (&v)[9], double *out, double *out8, int lane)
{
    double w[5];
    int iw[5];
#pragma unroll
    for (int j = 0; j < 4; j++) w[j] = fold_pair(v[2 * j], v[2 * j + 1], 2 * j, 2 * j + 1, 16, lane, iw[j]);
    w[4] = v[8] + __shfl_xor_sync(0xffffffffu, v[8], 16);
    iw[4] = 8;
    double x[3];
    int ix[3];
    x[0] = fold_pair(w[0], w[1], iw[0], iw[1], 8, lane, ix[0]);
    x[1] = fold_pair(w[2], w[3], iw[2], iw[3], 8, lane, ix[1]);
    x[2] = w[4] + __shfl_xor_sync(0xffffffffu, w[4], 8);
    ix[2] = iw[4];
    double y[2];
    int iy[2];
    y[0] = fold_pair(x[0], x[1], ix[0], ix[1], 4, lane, iy[0]);
    y[1] = x[2] + __shfl_xor_sync(0xffffffffu, x[2], 4);
    iy[1] = ix[2];
    int iz;
    const double z = fold_pair(y[0], y[1], iy[0], iy[1], 2, lane, iz);
    *(iz < 8 ? out + iz : out8) = z + __shfl_xor_sync(0xffffffffu, z, 1);
}

// Lists the lit facets of a point with Earth and Sun directions e, f in
// increasing order into idx (one warp); returns their count.
__device__ inline int list_lit_fp64(const DevObject &ob, double e1, double e2, double e3, double f1, double f2,
                                    double f3, uint16_t *idx)
{
    const int lane = threadIdx.x & 31, F = ob.nfac;
    // The lit test in FP32 where it is decided beyond its rounding: the FP32
    // dot products of the FP32-rounded unit vectors are within ~4e-7 of the
    // FP64 ones, so outside a 1e-4 band (scaled by the direction's 1-norm)
    // around kTinyMu the FP64 test gives the same answer; inside it the FP64
    // test runs (on the FP64 unit, which the first pass then leaves alone).
    // Each value converted once, on a lane of its own (a conversion is an FP64
    // instruction for the whole warp), and handed round.
    const double own = lane == 0 ? e1 : lane == 1 ? e2 : lane == 2 ? e3 : lane == 3 ? f1 : lane == 4 ? f2 : f3;
    const float ownf = static_cast<float>(own);
    const float e1f = __shfl_sync(0xffffffffu, ownf, 0), e2f = __shfl_sync(0xffffffffu, ownf, 1),
                e3f = __shfl_sync(0xffffffffu, ownf, 2), f1f = __shfl_sync(0xffffffffu, ownf, 3),
                f2f = __shfl_sync(0xffffffffu, ownf, 4), f3f = __shfl_sync(0xffffffffu, ownf, 5);
    const float band_e = 1e-4f * fmaxf(1.f, fabsf(e1f) + fabsf(e2f) + fabsf(e3f));
    const float band_f = 1e-4f * fmaxf(1.f, fabsf(f1f) + fabsf(f2f) + fabsf(f3f));
    const float tiny = static_cast<float>(kTinyMu);
    int n = 0;
    // Three rounds of 32 facets at a time, their loads ahead of the ballots
    // (one by one, the loads' latency made the list 5.6 of a point's 22 kcycles
    // in the chi^2 pass; one period's ten FP64 fits 38.8 -> 37.5 ms, 400 fits 515
    // -> 475 ms).
    constexpr int kRounds = 3;
    for (int i0 = 0; i0 < F; i0 += 32 * kRounds) {
        float nxf[kRounds], nyf[kRounds], nzf[kRounds];
#pragma unroll
        for (int r = 0; r < kRounds; r++) {
            const int i = min(i0 + 32 * r + lane, F - 1);
            nxf[r] = ob.nx_f[i];
            nyf[r] = ob.ny_f[i];
            nzf[r] = ob.nz_f[i];
        }
#pragma unroll
        for (int r = 0; r < kRounds; r++) {
            const int i = i0 + 32 * r + lane;
            const float muf = e1f * nxf[r] + e2f * nyf[r] + e3f * nzf[r];
            const float mu0f = f1f * nxf[r] + f2f * nyf[r] + f3f * nzf[r];
            bool lit = i < F && muf > tiny + band_e && mu0f > tiny + band_f;
            if (i < F && !lit && !(muf < tiny - band_e || mu0f < tiny - band_f)) {
                const double mu = e1 * ob.nx[i] + e2 * ob.ny[i] + e3 * ob.nz[i];
                const double mu0 = f1 * ob.nx[i] + f2 * ob.ny[i] + f3 * ob.nz[i];
                lit = mu > kTinyMu && mu0 > kTinyMu;
            }
            const unsigned m = __ballot_sync(0xffffffffu, lit);
            if (lit) idx[n + __popc(m & ((1u << lane) - 1u))] = static_cast<uint16_t>(i);
            n += __popc(m);
        }
    }
    __syncwarp();
    return n;
}

// FP64 facet stage of point p of the tile (bright.c:59-120), one warp.  A
// first pass lists the point's lit facets in increasing order (s.lidx,
// s.nlit); the law and the facet sums then run over that list with every
// lane busy (an FP64 instruction holds its sub-partition's FP64 unit for
// the whole warp, however few lanes are active), lane l taking the list's
// entries l, l + 32, ...  W is left in the W row at the list positions.
// The facet sums go to s.red[p * kRedStride + 0..7], brightness, U, V and the
// Lambert derivative, and the scattering-weight derivative to the point's
// record.
// count: add the point's lit facets to the CTA's counter.
__device__ inline void facet_point_fp64(const DevObject &ob, Smem<PS_FORM_FP64> &s, int p, int wcols, double cl,
                                        double cls, bool count)
{
    const int lane = threadIdx.x & 31;
    double *pt = s.pt + p * kPointStride;
    const double e1 = pt[0], e2 = pt[1], e3 = pt[2];
    const double f1 = pt[3], f2 = pt[4], f3 = pt[5];
    uint16_t *idx = s.lidx + static_cast<size_t>(p) * wcols;
    const int n = list_lit_fp64(ob, e1, e2, e3, f1, f2, f3, idx);
    // The rotation derivatives sum_i Area_i (dsmu_i (n_i . D_k) + dsmu0_i
    // (n_i . E_k)) (bright.c:87-104; D_k, E_k: the derivative directions of
    // the Earth and Sun vectors) are D_k . U + E_k . V with U = sum Area
    // dsmu n and V = sum Area dsmu0 n: the law accumulates U and V, the six
    // dot products run once per point (tile_rows_fp64).
    double br = 0, ux = 0, uy = 0, uz = 0, vx = 0, vy = 0, vz = 0, dcl = 0, dcls = 0;
    double *Wp = s.W + static_cast<size_t>(p) * wcols;
    for (int j = lane; j < n; j += 32) {
        const int i = idx[j];
        const double nx = ob.nx[i], ny = ob.ny[i], nz = ob.nz[i];
        const double mu = e1 * nx + e2 * ny + e3 * nz;
        const double mu0 = f1 * nx + f2 * ny + f3 * nz;
        const double ar = s.area[i];
        const LitTerms<double, PS_FORM_FP64> lt(mu, mu0, cl, cls);
        br = br + ar * lt.sv;
        Wp[j] = ob.darea[i] * lt.sv * s.gv[i];
        const double cu = ar * lt.dsmu, cv = ar * lt.dsmu0;
        ux = ux + cu * nx;
        uy = uy + cu * ny;
        uz = uz + cu * nz;
        vx = vx + cv * nx;
        vy = vy + cv * ny;
        vz = vz + cv * nz;
        dcl = dcl + mu * mu0 * ar;
        dcls = dcls + ar * lt.dcls_w;
    }
    const double v9[9] = {br, ux, uy, uz, vx, vy, vz, dcl, dcls};
    warp_sum9(v9, s.red + p * kRedStride, pt + kPtSum, lane);
    if (lane == 0) {
        s.nlit[p] = n;
        if (count) atomicAdd(lit_counter(s.misc), static_cast<unsigned long long>(n));
    }
}

// Accumulates the rows J[0..np) (model values in ym) of one tile into the
// normal matrix M (lower triangle), bv and chi^2 (mrqcof.c:106-136) on the
// SIMT pipes of the mixed form: FP32 partial sums, every element over the
// points in data order, added to the FP64 totals every few tiles.  A warp
// takes units of 4 rows by 32 columns of the matrix (a lane one column, four
// rows from one 16-byte broadcast of the weighted rows): two loads for four
// products, where an element per thread takes two each and waits for shared
// memory.  Unit u is unit u of the list of row groups' column panels
// (alpha_unit); warp w takes w, w + 16, ...
// Measured (87 free parameters): an evaluation's accumulation of 33 tiles 566
// -> 280 kcycles, 1010 fits 165 -> 148 ms.
constexpr int kTilesPerFlush = 8;
// The tensor-core path's FP32 alpha accumulator in Tensor Memory (products
// of TF32 high/low parts) is added to the FP64 normal matrix every 16 tiles.
constexpr int kTcTilesPerFlush = 16;

// Units of a warp by kernel variant: at most 45 units (90 free parameters), or
// 80 with up to 128 coefficients (KU 2).
template <int KU>
constexpr int kAlphaUnits = KU == 2 ? 5 : 3;
// The SIMT contraction of one coefficient per lane (KU 1) needs the registers
// of the partial sums for its loads in flight: there the loops over the units
// are not unrolled, which puts the sums in local memory (48 bytes a thread,
// read and written once a tile; 304 fits of 20 steps with 16 coefficients 22.0
// -> 21.0 ms).  With two per lane the contraction is a call, which saves them anyhow, and the
// packed kernel is slower without the unrolling (28.2 against 21.9 ms).
template <int KU>
constexpr int kAlphaUnroll = KU == 1 ? 1 : kAlphaUnits<KU>;

// Unit u: its first row (a group of four rows has the panels of 32 columns
// that reach its last row's diagonal) and, in the upper half, its first
// column; -1 past the end.
__device__ inline int alpha_unit(int u, int mf)
{
    for (int r = 0; r < mf; r += 4) {
        const int panels = (min(r + 4, mf) + 31) / 32;
        if (u < panels) return r | (32 * u) << 16;
        u -= panels;
    }
    return -1;
}

// Pitch of the weighted rows (16-byte groups of four).
PSG_HD inline int alpha_pitch(int mf) { return (mf + 3) & ~3; }

template <int KU>
__device__ inline void flush_partials(double *M, double *bv, int mf, const int (&unit)[kAlphaUnits<KU>],
                                      float4 (&accA)[kAlphaUnits<KU>], float &accB)
{
    const int tid = threadIdx.x, lane = tid & 31;
#pragma unroll kAlphaUnroll<KU>
    for (int q = 0; q < kAlphaUnits<KU>; q++) {
        if (unit[q] >= 0) {
            const int r0 = unit[q] & 0xffff, k = (unit[q] >> 16) + lane;
            const float v[4] = {accA[q].x, accA[q].y, accA[q].z, accA[q].w};
#pragma unroll
            for (int r = 0; r < 4; r++)
                if (r0 + r < mf && k <= r0 + r) M[(r0 + r) * mf + k] += static_cast<double>(v[r]);
        }
        accA[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (tid < mf) bv[tid] += static_cast<double>(accB);
    accB = 0.f;
}

template <int KU>
__device__ void accumulate_tile(const DevObject &ob, Smem<PS_FORM_MIXED> &s, int np, int q0pt, bool conv,
                                double conv_sig, bool chi2, const int (&unit)[kAlphaUnits<KU>],
                                float4 (&accA)[kAlphaUnits<KU>], float &accB)
{
    constexpr int NT = threads_of<PS_FORM_MIXED>();
    const int tid = threadIdx.x, lane = tid & 31;
    const int ma = ob.ma, mf = ob.mfit, mp = alpha_pitch(mf);
    float *wt = s.W;  // [np][mp], reuses the facet-weight tile
    // per point: FP32 weight sig2i*w and residual; chi^2 of the tile
    // summed over one warp in FP64
    float *dyv = s.accs;
    float *wtp = dyv + 32;
    if (tid < 32) {
        double c2 = 0;
        if (tid < np) {
            const int q = q0pt + tid;
            const double sig2i = conv ? 1 / (conv_sig * conv_sig) : ob.sig2i[q];
            const double wg = ob.weight[q];
            const double dy = (conv ? 0.0 : ob.bright[q]) - s.ym[tid];
            dyv[tid] = static_cast<float>(dy);
            wtp[tid] = static_cast<float>(sig2i * wg);
            if (chi2) c2 = dy * dy * sig2i * wg;
        }
        if (chi2) {
            c2 = warp_sum(c2);
            if (tid == 0) s.misc[M_CHISQ] += c2;
        }
    }
    __syncthreads();
    for (int e = tid; e < np * mp; e += NT) {
        const int p = e / mp, j = e - p * mp;
        wt[e] = j < mf ? s.J[p * ma + ob.free_list[j]] * wtp[p] : 0.f;
    }
    __syncthreads();
#pragma unroll kAlphaUnroll<KU>
    for (int q = 0; q < kAlphaUnits<KU>; q++) {
        if (unit[q] < 0) continue;
        const float *jc = s.J + ob.free_list[min((unit[q] >> 16) + lane, mf - 1)];
        const float4 *wr = reinterpret_cast<const float4 *>(wt + (unit[q] & 0xffff));
        float4 acc = accA[q];
#pragma unroll 8
        for (int p = 0; p < np; p++) {
            const float x = jc[p * ma];
            const float4 w = wr[p * (mp / 4)];
            acc.x = fmaf(w.x, x, acc.x);
            acc.y = fmaf(w.y, x, acc.y);
            acc.z = fmaf(w.z, x, acc.z);
            acc.w = fmaf(w.w, x, acc.w);
        }
        accA[q] = acc;
    }
    if (tid < mf) {
        float acc = accB;
        for (int p = 0; p < np; p++) acc = fmaf(dyv[p], wt[p * mp + tid], acc);
        accB = acc;
    }
    __syncthreads();
}

// Basis element Dsph[i][k] of the mixed form: from shared memory with an
// explicit shared-space load, or from global memory through the read-only
// path.
template <bool SMEM_D>
__device__ inline float load_basis(const float *d, int idx)
{
    if constexpr (SMEM_D) {
        float v;
        const unsigned addr = static_cast<unsigned>(__cvta_generic_to_shared(d + idx));
        asm("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
        return v;
    } else {
        return __ldg(d + idx);
    }
}

// Mixed-form shape contraction J[p][k] = Scale_p * sum_i W[p][i] Dsph[i][k]
// of one tile, FP32 on the SIMT pipes.  Register tile: warp w owns points
// (w % 8) + 8 r (r < 4) and coefficients lane + 32 ((w / 8) + 2 u) (u < KU);
// W is read four facets at a time (float4 broadcast), Dsph one coalesced row
// per facet.  Bound by the latency of those loads, so by what the compiler
// keeps in flight: a function of its own (contract_mixed_call) has all
// registers for it, also those of the partial sums of the normal matrix, which
// inlined it shares them with.  304 fits of 20 steps with 81 coefficients and
// 512 facets 168.3 -> 90.4 ms, with 49 coefficients and 288 facets 36.4 -> 29.9;
// one coefficient per lane with the basis in L2 is better inlined (49
// coefficients, 648 facets: 72.0 ms, 119 as a call).  Unrolled by four facet
// groups with the basis in shared memory, by two else (81 coefficients: four
// 91.5 ms, none 95.3, two 86.6).
template <int NT, int KU, bool SMEM_D>
__device__ __forceinline__ void contract_mixed(const float *Wf, const float *pt, float *J, const float *dsph, int np,
                                               int F, int C, int ma, int wcols, bool conv)
{
    static_assert(NT == 512, "the register tile assumes 16 warps");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = warp & 7, half = warp >> 3;
    constexpr int kPW = 4;
    float acc[kPW][KU];
#pragma unroll
    for (int r = 0; r < kPW; r++)
#pragma unroll
        for (int u = 0; u < KU; u++) acc[r][u] = 0.f;
    int kk[KU];
    bool kv[KU];
#pragma unroll
    for (int u = 0; u < KU; u++) {
        kk[u] = lane + 32 * (half + 2 * u);
        kv[u] = kk[u] < C;
    }
    bool any = false;
#pragma unroll
    for (int u = 0; u < KU; u++) any |= kv[u];
    if (any) {
#pragma unroll (SMEM_D ? 4 : 2)
        for (int i = 0; i < F; i += 4) {
            float4 w4[kPW];
#pragma unroll
            for (int r = 0; r < kPW; r++) {
                const int p = g + 8 * r;
                w4[r] = (p < np) ? *reinterpret_cast<const float4 *>(Wf + static_cast<size_t>(p) * wcols + i)
                                 : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int ii = 0; ii < 4; ii++) {
                float d[KU];
#pragma unroll
                for (int u = 0; u < KU; u++) d[u] = kv[u] ? load_basis<SMEM_D>(dsph, (i + ii) * C + kk[u]) : 0.f;
#pragma unroll
                for (int r = 0; r < kPW; r++) {
                    const float wv = ii == 0 ? w4[r].x : ii == 1 ? w4[r].y : ii == 2 ? w4[r].z : w4[r].w;
#pragma unroll
                    for (int u = 0; u < KU; u++) acc[r][u] = fmaf(wv, d[u], acc[r][u]);
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < kPW; r++) {
        const int p = g + 8 * r;
        if (p < np) {
            const float sc = conv ? 1.f : pt[p * kPointStride + 24];
#pragma unroll
            for (int u = 0; u < KU; u++)
                if (kv[u]) J[p * ma + kk[u]] = sc * acc[r][u];
        }
    }
}

template <int NT, int KU, bool SMEM_D>
__device__ __noinline__ void contract_mixed_call(const float *Wf, const float *pt, float *J, const float *dsph, int np,
                                                 int F, int C, int ma, int wcols, bool conv)
{
    contract_mixed<NT, KU, SMEM_D>(Wf, pt, J, dsph, np, F, C, ma, wcols, conv);
}

// Mixed-form point set-up in three parts (bright.c:27-57, phasec.c,
// matrix.c): setup_mixed_phase (the rotation phase and its cos and sin into
// pt[28], pt[29]), setup_mixed_geo (the phase function into pt[24..27], the
// products of the pole matrix and its beta/lambda derivatives with the Earth
// and Sun vectors into pt[0..17], the time into pt[30]) and
// setup_mixed_rotate (the rotation about the spin axis into pt[0..23]).  The
// rotation fm commutes out of the products (matrix.c): with u = B ee,
// e = fm u, de/dbeta = fm (dB/dbeta ee), de/dlambda = fm (dB/dlambda ee) and
// de/domega = (dfm/domega) u = t (e_y, -e_x, 0); the same for the Sun vector.
// The tensor-core path runs the first two on different warps (the FP64
// rotation phase holds its sub-partition's FP64 unit for the whole warp)
// and applies the rotation where it reads the records; the SIMT variants
// run all three (setup_point).
__device__ inline void setup_mixed_phase(double td, double omg, double phi0, float *pt)
{
    const float f = rotation_phase_mixed(omg, td, phi0);
    float sf, cf;
    sincosf(f, &sf, &cf);
    pt[28] = cf;
    pt[29] = sf;
}

// part < 0: all of it; part 0: the phase function and the pole matrix's
// products; part 1: its derivatives' products and the time (two warps of
// the tensor-core path share the work).
__device__ inline void setup_mixed_geo(float4 g0, float4 g1, const float *bm, float *pt, int part = -1)
{
    const float ee[3] = {g0.x, g0.y, g0.z}, e0v[3] = {g1.x, g1.y, g1.z};
    if (part <= 0) {
        const float alpha = g0.w;
        const float php0 = bm[27], php1 = bm[28], php2 = bm[29];
        const float inv_w = 1.f / php1;
        const float ex = expf(-alpha * inv_w);
        const float pe = __fmul_rn(php0, ex);
        pt[24] = fmaf(php2, alpha, __fadd_rn(1.f, pe));   // one rounding wherever it is formed
        pt[25] = ex;
        pt[26] = pe * alpha * (inv_w * inv_w);
        pt[27] = alpha;
    }
    if (part != 0) pt[30] = g1.w;
#pragma unroll
    for (int m = 0; m < 3; m++) {
        if ((part == 0 && m != 0) || (part == 1 && m == 0)) continue;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const float *row = bm + 9 * m + 3 * k;
            pt[6 * m + k] = row[0] * ee[0] + row[1] * ee[1] + row[2] * ee[2];
            pt[6 * m + 3 + k] = row[0] * e0v[0] + row[1] * e0v[1] + row[2] * e0v[2];
        }
    }
}

__device__ inline void setup_mixed_rotate(float *pt)
{
    const float cf = pt[28], sf = pt[29], t = pt[30];
    float u[18];
#pragma unroll
    for (int i = 0; i < 18; i++) u[i] = pt[i];
#pragma unroll
    for (int m = 0; m < 3; m++) {
        const float *ue = u + 6 * m, *us = u + 6 * m + 3;
        const float r0 = cf * ue[0] + sf * ue[1], r1 = cf * ue[1] - sf * ue[0];
        const float s0 = cf * us[0] + sf * us[1], s1 = cf * us[1] - sf * us[0];
        if (m == 0) {
            pt[0] = r0;
            pt[1] = r1;
            pt[2] = ue[2];
            pt[3] = s0;
            pt[4] = s1;
            pt[5] = us[2];
            // d/domega (column 2 of de and de0)
            pt[6 + 2] = t * r1;
            pt[6 + 3 + 2] = -t * r0;
            pt[6 + 6 + 2] = 0.f;
            pt[15 + 2] = t * s1;
            pt[15 + 3 + 2] = -t * s0;
            pt[15 + 6 + 2] = 0.f;
        } else {
            const int j = m - 1;   // column 0: d/dbeta, 1: d/dlambda
            pt[6 + j] = r0;
            pt[6 + 3 + j] = r1;
            pt[6 + 6 + j] = ue[2];
            pt[15 + j] = s0;
            pt[15 + 3 + j] = s1;
            pt[15 + 6 + j] = us[2];
        }
    }
}

// 1 + a exp(-alpha / d) + k alpha (phasec.c), one rounding wherever it is formed.
__device__ inline double phase_scale_fp64(double a, double k, double ex, double alpha)
{
    return fma(k, alpha, __dadd_rn(1.0, __dmul_rn(a, ex)));
}

// Point set-up of observation q (bright.c:27-57, phasec.c, matrix.c): the
// rotated Earth and Sun directions with their beta/lambda/omega derivatives,
// the phase function and its derivatives, into pt[0..27].
__device__ inline void setup_point(const DevObject &ob, const FitConfig &cfg, int q, double omg, const float *bm,
                                   float *pt)
{
    setup_mixed_phase(ob.tim[q], omg, cfg.phi0, pt);
    setup_mixed_geo(ob.geo_f[2 * q], ob.geo_f[2 * q + 1], bm, pt);
    setup_mixed_rotate(pt);
}

// FP64 form: the point set-up in two parts.  The first is what every point
// needs once, a point per lane: the cos and sin of the rotation phase, the
// phase function's exponential and its derivative by d, into ph[0..3][stride].
__device__ inline void setup_phase_fp64(const DevObject &ob, const FitConfig &cfg, int q, double omg,
                                        const double *bm, double *ph, int stride)
{
    const double alpha = ob.alpha_pt[q], php0 = bm[27], php1 = bm[28];
    const double ex = exp(-alpha / php1);
    const double f = rotation_phase_fp64(omg, ob.tim[q], cfg.phi0);
    ph[0] = cos(f);
    ph[stride] = sin(f);
    ph[2 * stride] = ex;
    ph[3 * stride] = php0 * ex * alpha / (php1 * php1);
}

// The second, of the point's directions the row i of e = fm B ee (part 0) or
// of its derivative by beta (1), lambda (2) or omega (3), and the same of the
// Sun vector: twelve parts of at most 14 FP64 instructions, a warp each with
// a point per lane.  The zeros and ones of the rotation fm are left out of
// the reference's products (matrix.c), which changes no value.
__device__ inline void setup_row_fp64(const DevObject &ob, int q, int part, int i, const double *bm,
                                      const double *ph, int stride, double *pt)
{
    const double ee[3] = {ob.eex[q], ob.eey[q], ob.eez[q]}, es[3] = {ob.e0x[q], ob.e0y[q], ob.e0z[q]};
    const double *B = bm + (part == 3 ? 0 : 9 * part);
    double x = 0, y = 0;
    if (i == 2) {
        if (part < 3) {
#pragma unroll
            for (int j = 0; j < 3; j++) {
                x = fma(B[6 + j], ee[j], x);
                y = fma(B[6 + j], es[j], y);
            }
        }
    } else {
        const double cf = ph[0], sf = ph[stride];
        double f0 = i == 0 ? cf : -sf, f1 = i == 0 ? sf : cf;
        if (part == 3) {
            const double t = ob.tim[q];
            f0 = __dmul_rn(-t, i == 0 ? sf : cf);
            f1 = i == 0 ? __dmul_rn(t, cf) : __dmul_rn(-t, sf);
        }
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const double m = fma(f1, B[3 + j], __dmul_rn(f0, B[j]));
            x = fma(m, ee[j], x);
            y = fma(m, es[j], y);
        }
    }
    // directions at pt[0..5], derivative column part - 1 at pt[6..14] and pt[15..23]
    pt[part == 0 ? i : 6 + i * 3 + part - 1] = x;
    pt[part == 0 ? 3 + i : 15 + i * 3 + part - 1] = y;
}

// The part of the FP64 form's set-up that the model value needs: the rotated
// Earth and Sun directions into e[0..5] and the phase function (returned),
// by the operations of setup_phase_fp64 and setup_row_fp64.
__device__ inline double setup_point_light(const DevObject &ob, const FitConfig &cfg, int q, double omg,
                                           const double *bm, double (&e)[6])
{
    const double ee[3] = {ob.eex[q], ob.eey[q], ob.eez[q]}, e0v[3] = {ob.e0x[q], ob.e0y[q], ob.e0z[q]};
    const double alpha = ob.alpha_pt[q];
    const double f = rotation_phase_fp64(omg, ob.tim[q], cfg.phi0);
    const double cf = cos(f), sf = sin(f);
    const double fm[9] = {cf, sf, 0.0, -sf, cf, 0.0, 0.0, 0.0, 1.0};
#pragma unroll
    for (int i = 0; i < 3; i++) {
        double x = 0, y = 0;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            double m = 0;
#pragma unroll
            for (int k = 0; k < 3; k++) m = m + fm[i * 3 + k] * bm[k * 3 + j];
            x = x + m * ee[j];
            y = y + m * e0v[j];
        }
        e[i] = x;
        e[3 + i] = y;
    }
    return phase_scale_fp64(bm[27], bm[29], exp(-alpha / bm[28]), alpha);
}

// ---------------------------------------------------------------------------
// Tensor-core contraction of the mixed form (kBasisTensor).
// ---------------------------------------------------------------------------
constexpr uint32_t kTcWaitTries = 1u << 22;   // mbarrier polls before a wait gives up
constexpr int kErrTcTimeout = 16;             // ps_fit.err_code of a fit cut short by a failed wait

// Tensor Memory columns: the basis [0, Fp/2) (FP16 pairs of facets, Fp =
// tc_kpad(F)), from tc_dcol on a contraction accumulator of 64 columns for
// each team (column p: A W_hi^T for point p, 32 + p: A W_lo^T), then an alpha
// accumulator of 2 tc_arows(mfit) columns for each team.  The wide path
// (kBasisTensorWide) has the second basis region R2 at [Fp/2, 3 Fp/4), the
// accumulator at tc_dcol and R2's accumulator at tc_dcol + 64 (columns
// 0..31: products with the first half of the facets, 32..63: with the second
// half), and no alpha accumulator.
__device__ inline uint32_t tc_r2col(int F) { return static_cast<uint32_t>(tc_kpad(F) >> 1); }

__device__ inline uint32_t tc_cols(int F, int mf, bool wide, int teams)
{
    uint32_t n = 32;
    while (n < (wide ? tc_dcol(F, true) + 128u : tc_dcol(F) + static_cast<uint32_t>(teams * (64 + 2 * tc_arows(mf)))))
        n <<= 1;
    return n;
}

// Per-thread view of the CTA's tensor-core state (every thread keeps the
// same values).
struct TcState {
    uint32_t tbase = 0;     // Tensor Memory base address
    int basis_exp = 0;      // the basis is held scaled by 2^basis_exp
    uint32_t phase = 0;     // parity of the contraction barrier's next phase
    uint32_t aphase = 0;    // parity of the alpha barrier's next phase
    bool apending = false;  // alpha MMAs committed and not waited for
    bool afresh = true;     // the alpha accumulator holds nothing since the last flush
    bool wide = false;      // kBasisTensorWide layout
    uint32_t dcol = 0, acol = 0;   // Tensor Memory columns of the contraction and the alpha accumulator
};

// Every thread of the team waits for the barrier's phase; true when all saw
// it, else the abort flag is set.
template <int NT>
__device__ inline bool team_wait(Smem<PS_FORM_MIXED> &s, uint64_t *mbar, uint32_t phase)
{
    const bool ok = tc::mbar_wait(mbar, phase, kTcWaitTries);
    if constexpr (NT == kTeamThreads) {
        if (!ok) *s.abort = 1;
        team_sync<NT>();
        return !*s.abort;
    } else {
        if (__syncthreads_and(ok)) return true;
        if (threadIdx.x == 0) *s.abort = 1;
        __syncthreads();
        return false;
    }
}

// Waits for the committed alpha MMAs (their operands' shared memory is then
// free); a wait that gives up sets the abort flag.
template <int NT>
__device__ inline void tc_alpha_wait(Smem<PS_FORM_MIXED> &s, TcState &t)
{
    if (!t.apending || *s.abort) return;
    t.apending = false;
    if (!team_wait<NT>(s, s.mbar2, t.aphase)) {
        t.apending = true;   // tc_teardown waits once more
        return;
    }
    t.aphase ^= 1u;
    tc::fence_after_sync();
}

// Allocates the CTA's Tensor Memory (s0: the shared memory of its first
// team), initialises the team's barriers, stages the team's facet constants
// (zero for the padding facets) and loads the basis operand into Tensor
// Memory.  The operand is formed once per object (basis_words): formed here
// from the FP64 basis, its conversions took about 45 us of every launch.
template <int NT, bool WIDE = false>
__device__ void tc_setup(const DevObject &ob, Smem<PS_FORM_MIXED> &s0, Smem<PS_FORM_MIXED> &s, TcState &t)
{
    constexpr int kTeams = kSlotThreads / NT;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int ttid = team_thread<NT>(), team = tid / NT;
    const int F = ob.nfac, Fp = tc_kpad(F);
    if (warp == 0) tc::tmem_alloc(s0.tslot, tc_cols(F, ob.mfit, WIDE, kTeams));
    if (ttid == 0) {
        tc::mbar_init(s.mbar, 1);
        tc::mbar_init(s.mbar2, 1);
        *s.abort = 0;
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tbase = *s0.tslot;
    for (int i = ttid; i < Fp; i += NT) {
        fac_at(s.fac, i, 0) = i < F ? ob.nx_f[i] : 0.f;
        fac_at(s.fac, i, 1) = i < F ? ob.ny_f[i] : 0.f;
        fac_at(s.fac, i, 2) = i < F ? ob.nz_f[i] : 0.f;
        fac_at(s.fac, i, 3) = 0.f;
    }
    for (int j = ttid; j < ob.mfit; j += NT) s.flist[j] = ob.free_list[j];
    // lanes 32 (warp % 4) .. + 31, eight columns at a time, the warps of a
    // lane quarter in turn
    const uint32_t row = tbase + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    const uint32_t *src = ob.basis_tc + (tid & 127);
    const int cols = WIDE ? 3 * (Fp / 4) : Fp / 2;
    for (int j0 = 8 * (warp >> 2); j0 < cols; j0 += kSlotThreads / 16) {
        uint32_t v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = src[static_cast<size_t>(j0 + j) * 128];
        tc::tmem_st8(row + static_cast<uint32_t>(j0), v);
    }
    tc::tmem_wait_st();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    t.tbase = tbase;
    t.basis_exp = ob.basis_exp;
    t.wide = WIDE;
    t.dcol = tc_dcol(F, WIDE) + 64u * team;
    t.acol = tc_dcol(F) + 64u * kTeams + static_cast<uint32_t>(2 * tc_arows(ob.mfit) * team);
}

// Releases the Tensor Memory.  After an abandoned wait the MMAs in flight
// get one more bounded wait first.
template <int NT>
__device__ void tc_teardown(Smem<PS_FORM_MIXED> &s, const TcState &t, int F, int mf)
{
    if (*s.abort && team_thread<NT>() == 0) {
        tc::mbar_wait(s.mbar, t.phase, kTcWaitTries);
        if (t.apending) tc::mbar_wait(s.mbar2, t.aphase, kTcWaitTries);
    }
    tc::fence_before_sync();
    __syncthreads();   // both teams
    if ((threadIdx.x >> 5) == 0)
        tc::tmem_dealloc(t.tbase, tc_cols(F, mf, t.wide, threads_of<PS_FORM_MIXED>() / NT));
}

// Issues the alpha/beta MMAs of the operands in s.aop (built and fenced,
// behind a CTA barrier) and commits them to the alpha barrier.  Called by
// every thread; the elected thread of warp 0 issues.
template <int NT>
__device__ inline void tc_alpha_issue(Smem<PS_FORM_MIXED> &s, TcState &t, int mf)
{
    if (__shfl_sync(0xffffffffu, team_thread<NT>() >> 5, 0) == 0 && !*s.abort && tc::elect_one()) {
        tc::fence_after_sync();
        const uint32_t idesc = tc::idesc_tf32(128, 2 * tc_arows(mf));
        const uint32_t a0 = tc::smem_u32(s.aop), b0 = tc::smem_u32(s.aop + 16384), d = t.tbase + t.acol;
        for (int kk = 0; kk < 4; kk++) {
            const uint32_t off = static_cast<uint32_t>(kk) * 256;
            tc::mma_tf32_ss(d, tc::smem_desc(a0 + off, 128, 1024), tc::smem_desc(b0 + off, 128, 1024), idesc,
                            (t.afresh && kk == 0) ? 0u : 1u);
        }
        tc::mma_commit(s.mbar2);
    }
    t.apending = true;
    t.afresh = false;
}

// Issues D = A [W_hi; W_lo]^T for the tile as Fp/16 FP16 MMAs of 128 x 64 x
// 16 and a commit to the barrier.  The issuing thread is elected
// (elect.sync in a warp-uniform branch): picked by its number, it took about
// 70 cycles per MMA whatever the shape, more than the MMAs themselves (18 MMAs
// of 288 facets: issue 1.8 -> 1.1 kcycles a tile; the wide path's 64: 4.9 ->
// 2.4; 1010 wide fits 174 -> 165 ms).  The facet stage has written the operand: FP16 high parts of W
// in rows 0..31, low parts in rows 32..63, canonical K-major layout (8-row x
// 8-facet core matrices, K-adjacent ones 128 bytes apart).
template <int NT, bool WIDE = false>
__device__ void contract_tc_issue(Smem<PS_FORM_MIXED> &s, int F, TcState &t)
{
    const int tid = team_thread<NT>(), warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int Fp = tc_kpad(F), kcs = Fp >> 3;
    const uint32_t tbase = t.tbase;
    tc::fence_proxy_async();
    tc::fence_before_sync();
    team_sync<NT>();
    if (warp == 0 && !*s.abort && tc::elect_one()) {
        tc::fence_after_sync();
        const uint32_t idesc = tc::idesc_f16(128, 64);
        const uint32_t sbo = static_cast<uint32_t>(kcs) * 128;
        const uint32_t d = tbase + t.dcol;
        const uint64_t b0 = tc::smem_desc(tc::smem_u32(s.bhi), 128, sbo);
        // one K step: 8 columns of A, 256 bytes (16 in the descriptor) of B
        const int steps = Fp / 16;
        tc::mma_f16_ts(d, tbase, b0, idesc, 0);
#pragma unroll 4
        for (int ks = 1; ks < steps; ks++) tc::mma_f16_ts(d, tbase + 8u * ks, b0 + 16u * ks, idesc, 1);
        if constexpr (WIDE) {
            // R2 against the W_hi rows (N = 32) of each facet half: the
            // products of lanes 0.. with the first half land in columns
            // 0..31, those of lanes 64.. with the second half in 32..63
            const uint32_t idesc32 = tc::idesc_f16(128, 32), d2 = d + 64, a2 = tbase + tc_r2col(F);
            const int half_steps = Fp / 32;
            for (int h = 0; h < 2; h++) {
                const uint64_t bh = b0 + static_cast<uint64_t>(16 * h * half_steps);
                tc::mma_f16_ts(d2 + 32u * h, a2, bh, idesc32, 0);
#pragma unroll 4
                for (int ks = 1; ks < half_steps; ks++)
                    tc::mma_f16_ts(d2 + 32u * h, a2 + 8u * ks, bh + 16u * ks, idesc32, 1);
            }
        }
        tc::mma_commit(s.mbar);
    }
}

// Earth and Sun directions of a point record (setup_mixed_phase,
// setup_mixed_geo) rotated about the spin axis.
__device__ inline void rotate_directions(const float *pt, float (&e)[6])
{
    const float cf = pt[28], sf = pt[29];
    e[0] = cf * pt[0] + sf * pt[1];
    e[1] = cf * pt[1] - sf * pt[0];
    e[2] = pt[2];
    e[3] = cf * pt[3] + sf * pt[4];
    e[4] = cf * pt[4] - sf * pt[3];
    e[5] = pt[5];
}

// The Lommel-Seeliger + Lambert law on a pair of facets (fac_at's two float4
// of the pair) as FP32x2 operations, one paired instruction each.
// Branch-free: the 8 points of a warp see different lit facets, so a branch
// would diverge on almost every step (and a warp-uniform skip of groups
// unlit for all 8 points measured slower, twice); unlit and padding facets
// get zero area (every term vanishes) and a safe denominator.
struct LitPair {
    float2 ax, m, m0, r, mm;   // area (0 when unlit), mu, mu0, 1 / (mu + mu0), mu mu0
    __device__ inline LitPair(const float4 &fa, const float4 &fb, const float2 &E1, const float2 &E2, const float2 &E3,
                              const float2 &F1, const float2 &F2, const float2 &F3)
    {
        const float2 nx = make_float2(fa.x, fa.y), ny = make_float2(fa.z, fa.w), nz = make_float2(fb.x, fb.y);
        float2 mu = __fmul2_rn(E1, nx), mu0 = __fmul2_rn(F1, nx);
        mu = __ffma2_rn(E2, ny, mu);
        mu0 = __ffma2_rn(F2, ny, mu0);
        mu = __ffma2_rn(E3, nz, mu);
        mu0 = __ffma2_rn(F3, nz, mu0);
        const bool lit0 = mu.x > float(kTinyMu) && mu0.x > float(kTinyMu);
        const bool lit1 = mu.y > float(kTinyMu) && mu0.y > float(kTinyMu);
        // Area (= Darea g, also the weight of W: the Lambert and
        // Lommel-Seeliger terms share it)
        ax = make_float2(lit0 ? fb.z : 0.f, lit1 ? fb.w : 0.f);
        m = make_float2(lit0 ? mu.x : 1.f, lit1 ? mu.y : 1.f);
        m0 = make_float2(lit0 ? mu0.x : 1.f, lit1 ? mu0.y : 1.f);
        const float2 dnom = __fadd2_rn(m, m0);
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(dnom.x));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(dnom.y));
        mm = __fmul2_rn(m, m0);
    }
    // s = mu mu0 (cl + cls / (mu + mu0))
    __device__ inline float2 law(const float2 &CL, const float2 &CLS) const
    {
        return __fmul2_rn(mm, __ffma2_rn(CLS, r, CL));
    }
};

// Facet stage of the tensor-core path (bright.c:59-120).  Warp w takes
// points 8 (w % 4) .. +7 (lane / 4) and the facet quarter w / 4, each lane
// of a point taking two adjacent facets of every 8 (lane % 4), so that one
// warp store covers a whole 8-point x 8-facet core matrix of the MMA
// operand [W_hi; W_lo] (FP16 pairs, W scaled by wscale = 2^k so that the
// evaluation's largest W is just below 2^14).  The per-point
// sums (brightness, Lambert and scattering derivatives, U, V) are reduced over
// the four lanes into s.fpart[(quarter * 32 + p) * 9 + 0..8], for
// point_sums_tc.  The tile's operand region must be free (previous MMAs waited
// for).
template <int NT>
__device__ void facet_stage_tc(const DevObject &ob, Smem<PS_FORM_MIXED> &s, int np, float cl, float cls,
                               float wscale)
{
    static_assert(NT % 128 == 0, "warps: 4 point groups x facet quarters");
    const int tid = team_thread<NT>(), lane = tid & 31, warp = tid >> 5;
    const int kcs = tc_kpad(ob.nfac) >> 3;   // 8-facet core matrices per row group
    const int cq = kcs >> 2;                 // per facet quarter
    const int g = warp & 3, p = g * 8 + (lane >> 2), fl = lane & 3;
    // The point records of this path hold the pole products before the
    // rotation about the spin axis (setup_mixed_geo) and its cos/sin
    // (setup_mixed_phase): Earth and Sun directions rotated here.
    float e1 = 0, e2 = 0, e3 = 0, f1 = 0, f2 = 0, f3 = 0;
    if (p < np) {
        float e[6];
        rotate_directions(s.pt + p * kPointStride, e);
        e1 = e[0];
        e2 = e[1];
        e3 = e[2];
        f1 = e[3];
        f2 = e[4];
        f3 = e[5];
    }
    // The rotation derivatives sum_i Area_i (dsmu (n_i . D_k) + dsmu0 (n_i .
    // E_k)) over the lit facets are D_k . U + E_k . V with U = sum Area dsmu
    // n and V = sum Area dsmu0 n (D_k, E_k: the derivative directions of the
    // Earth and Sun vectors), so the facet loop accumulates U and V.
    // A lane's two facets of each 8 run as the halves of FP32x2 operations
    // (one paired instruction each, on the facet table's interleaved pairs),
    // each half summing its own facets; the halves are added at the end.
    const float2 E1 = make_float2(e1, e1), E2 = make_float2(e2, e2), E3 = make_float2(e3, e3);
    const float2 F1 = make_float2(f1, f1), F2 = make_float2(f2, f2), F3 = make_float2(f3, f3);
    const float2 CL = make_float2(cl, cl), CLS = make_float2(cls, cls), WS = make_float2(wscale, wscale);
    const float2 z2 = make_float2(0.f, 0.f);
    uint32_t *bh = reinterpret_cast<uint32_t *>(s.bhi), *bl = reinterpret_cast<uint32_t *>(s.blo);
    // (a team of 8 warps takes two quarters per warp, one after the other)
#pragma unroll 1
    for (int part = 0; part < kSlotThreads / NT; part++) {
        const int quarter = (warp >> 2) + part * (NT / 128);
        float2 br = z2, dcl = z2, dcls = z2, ux = z2, uy = z2, uz = z2, vx = z2, vy = z2, vz = z2;
        for (int kc = quarter * cq; kc < (quarter + 1) * cq; kc++) {
            const int i = kc * 8 + 2 * fl;
            const int cm = g * kcs + kc;    // core matrix (8-point group, 8-facet group)
            const float4 fa = s.fac[i], fb = s.fac[i + 1];
            const float2 nx = make_float2(fa.x, fa.y), ny = make_float2(fa.z, fa.w), nz = make_float2(fb.x, fb.y);
            // (unlit facets carry zero area: no branch, see LitPair)
            const LitPair lp(fa, fb, E1, E2, E3, F1, F2, F3);
            const float2 ax = lp.ax, m = lp.m, m0 = lp.m0, r = lp.r, mm = lp.mm;
            const float2 sv = lp.law(CL, CLS);
            const float2 q0 = __fmul2_rn(m0, r), q1 = __fmul2_rn(m, r);
            const float2 dsmu = __ffma2_rn(CLS, __fmul2_rn(q0, q0), __fmul2_rn(CL, m0));
            const float2 dsmu0 = __ffma2_rn(CLS, __fmul2_rn(q1, q1), __fmul2_rn(CL, m));
            const float2 axs = __fmul2_rn(ax, sv);
            br = __fadd2_rn(br, axs);
            const float2 wv = __fmul2_rn(axs, WS);
            const float2 cu = __fmul2_rn(ax, dsmu), cv = __fmul2_rn(ax, dsmu0);
            ux = __ffma2_rn(cu, nx, ux);
            uy = __ffma2_rn(cu, ny, uy);
            uz = __ffma2_rn(cu, nz, uz);
            vx = __ffma2_rn(cv, nx, vx);
            vy = __ffma2_rn(cv, ny, vy);
            vz = __ffma2_rn(cv, nz, vz);
            dcl = __ffma2_rn(mm, ax, dcl);
            dcls = __ffma2_rn(ax, __fmul2_rn(mm, r), dcls);
            const uint32_t hp = tc::pack_f16x2(wv.x, wv.y);
            bh[cm * 32 + lane] = hp;
            bl[cm * 32 + lane] = tc::pack_f16x2(wv.x - tc::f16_lo(hp), wv.y - tc::f16_hi(hp));
        }
        float v[9] = {br.x + br.y, dcl.x + dcl.y, dcls.x + dcls.y, ux.x + ux.y, uy.x + uy.y,
                      uz.x + uz.y, vx.x + vx.y, vy.x + vy.y, vz.x + vz.y};
#pragma unroll
        for (int k = 0; k < 9; k++) {
            v[k] += __shfl_xor_sync(0xffffffffu, v[k], 1);
            v[k] += __shfl_xor_sync(0xffffffffu, v[k], 2);
        }
        if (fl == 0) {
            float *fp = s.fpart + (quarter * 32 + p) * 9;
#pragma unroll
            for (int k = 0; k < 9; k++) fp[k] = v[k];
        }
    }
}

// The sums of point p of the tile from its four quarters' partials (FP32: the
// J columns they feed are): brightness, the three rotation derivatives, the
// Lambert and the scattering-weight derivatives.  Formed in the contraction
// window by the warp that writes the J columns: at the end of the facet stage
// they held all warps for a barrier and some 700 cycles a tile.
__device__ inline void point_sums_tc(const Smem<PS_FORM_MIXED> &s, int p, float (&v)[6])
{
    float t[9];
#pragma unroll
    for (int k = 0; k < 9; k++) {
        float a = 0.f;
#pragma unroll
        for (int q = 0; q < 4; q++) a += s.fpart[(q * 32 + p) * 9 + k];
        t[k] = a;
    }
    // D_k . U with D_k = fm u_k (k: beta, lambda) is u_k . fm^T U; the
    // omega derivative is D_2 = t (e_y, -e_x, 0), e = fm u_0
    const float *pt = s.pt + p * kPointStride;
    const float cf = pt[28], sf = pt[29], tt = pt[30];
    const float Ux = cf * t[3] - sf * t[4], Uy = sf * t[3] + cf * t[4], Uz = t[5];
    const float Vx = cf * t[6] - sf * t[7], Vy = sf * t[6] + cf * t[7], Vz = t[8];
    v[0] = t[0];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float *ue = pt + 6 * (k + 1), *us = ue + 3;
        v[1 + k] = ue[0] * Ux + ue[1] * Uy + ue[2] * Uz + us[0] * Vx + us[1] * Vy + us[2] * Vz;
    }
    v[3] = tt * (pt[1] * Ux - pt[0] * Uy + pt[4] * Vx - pt[3] * Vy);
    v[4] = t[1];
    v[5] = t[2];
}

// Convexity rows (conv.c:12-29) on the tensor-core path: rows 0..2 of the
// MMA operand hold Darea g n_c (scaled by wscale) split into FP16 high and
// low parts; the residuals sum Area n_c in FP64.
template <int NT>
__device__ void conv_rows_tc(const DevObject &ob, Smem<PS_FORM_MIXED> &s, float wscale)
{
    const int tid = team_thread<NT>(), lane = tid & 31, warp = tid >> 5;
    const int F = ob.nfac, half = tc_kpad(F) >> 1;
    uint32_t *bh = reinterpret_cast<uint32_t *>(s.bhi), *bl = reinterpret_cast<uint32_t *>(s.blo);
    for (int e = tid; e < 3 * half; e += NT) {
        const int c = e / half, i = 2 * (e - c * half);
        const double *nc = (c == 0) ? ob.nx : (c == 1) ? ob.ny : ob.nz;
        float w[2], h[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            w[u] = i + u < F ? static_cast<float>(ob.darea[i + u] * s.gv[i + u] * nc[i + u]) * wscale : 0.f;
            h[u] = tc::round_f16(w[u]);
        }
        // row c of the first 8-row group, facets i, i + 1 of core matrix i / 8
        const int off = (i >> 3) * 32 + c * 4 + ((i & 7) >> 1);
        bh[off] = tc::pack_f16x2(h[0], h[1]);
        bl[off] = tc::pack_f16x2(w[0] - h[0], w[1] - h[1]);
    }
    if (warp < 3) {
        const double *nc = (warp == 0) ? ob.nx : (warp == 1) ? ob.ny : ob.nz;
        double res = 0;
        for (int i = lane; i < F; i += 32) res = res + s.area[i] * nc[i];
        res = warp_sum(res);
        if (lane == 0) s.red[warp * kRedStride] = res;
    }
}

// Waits for the tile's MMAs, stages the accumulator (lane m = row m) in
// shared memory and writes J[p][k] = Scale_p jscale (D[k][p] + D[k][32 + p]
// + D[64 + k][p] + D[64 + k][32 + p]): basis high and low parts times W high
// and low parts, jscale undoing the operands' power-of-two scales.  A wait
// that gives up sets the abort flag; the caller ends the fit.
template <int NT, bool WIDE = false>
__device__ void contract_tc_finish(Smem<PS_FORM_MIXED> &s, int np, int F, int C, int ma, bool conv, TcState &t,
                                   float jscale)
{
    const int tid = team_thread<NT>(), lane = tid & 31, warp = tid >> 5;
    const uint32_t tbase = t.tbase;
    if (*s.abort) return;
    if (!team_wait<NT>(s, s.mbar, t.phase)) return;
    t.phase ^= 1u;
    tc::fence_after_sync();
    // every warp reads, for 8 points of its lane quadrant's rows (warp w may
    // access Tensor Memory lanes 32 (w % 4) .. + 31), the products with W_hi
    // (column p) and W_lo (column 32 + p) and stages their sum Y[m][p]
    float *Y = reinterpret_cast<float *>(s.bhi);   // [128][33]
    float *Y2 = Y + 128 * 33;                      // wide path: [128][33] from R2's accumulator
#pragma unroll
    for (int part = 0; part < kSlotThreads / NT; part++) {
        const int quad = warp & 3, pg = (warp >> 2) + part * (NT / 128);
        const uint32_t taddr = tbase + (static_cast<uint32_t>(quad * 32) << 16) + t.dcol + 8 * pg;
        float *yr = Y + (quad * 32 + lane) * 33 + 8 * pg;
        uint32_t vh[8], vl[8];
        tc::tmem_ld8(taddr, vh);
        tc::tmem_ld8(taddr + 32, vl);
        tc::tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; j++) yr[j] = __uint_as_float(vh[j]) + __uint_as_float(vl[j]);
        if constexpr (WIDE) {
            // lanes 0..63 hold the first facet half's products (columns
            // 0..31), lanes 64..127 the second half's (columns 32..63)
            uint32_t v2[8];
            tc::tmem_ld8(taddr + 64 + (quad >= 2 ? 32 : 0), v2);
            tc::tmem_wait_ld();
            float *y2 = Y2 + (quad * 32 + lane) * 33 + 8 * pg;
#pragma unroll
            for (int j = 0; j < 8; j++) y2[j] = __uint_as_float(v2[j]);
        }
    }
    team_sync<NT>();
    if constexpr (WIDE) {
        // J[p][k] = Scale_p jscale (high part of k times W_hi and W_lo + low
        // part of k times W: from R1's lanes C + k for k < 128 - C, else
        // from R2's two facet halves); thread: k = tid % 128, points
        // tid / 128 + 4 i
        const int k = tid & 127, L1 = 128 - C;
        if (k < C) {
            for (int p = tid >> 7; p < np; p += NT / 128) {
                const float sc = (conv ? 1.f : s.pt[p * kPointStride + 24]) * jscale;
                const float lo = k < L1 ? Y[(C + k) * 33 + p] : Y2[(k - L1) * 33 + p] + Y2[(64 + k - L1) * 33 + p];
                s.J[p * ma + k] = sc * (Y[k * 33 + p] + lo);
            }
        }
        return;
    }
    // J[p][k] = Scale_p jscale (Y[k][p] + Y[64 + k][p]); thread: k = tid % 64,
    // points tid / 64 + 8 i (C <= 64 on this path)
    {
        const int k = tid & 63;
        if (k < C) {
            const float *yh = Y + k * 33, *yl = Y + (64 + k) * 33;
            for (int p = tid >> 6; p < np; p += NT / 64) {
                const float sc = (conv ? 1.f : s.pt[p * kPointStride + 24]) * jscale;
                s.J[p * ma + k] = sc * (yh[p] + yl[p]);
            }
        }
    }
}

// alpha/beta accumulation of one tile on the tensor cores (mrqcof.c:106-136):
// D += A B^T over the tile's points with A = [Wt_hi; Wt_lo] (row j: the
// weighted column J[.][l_j] sig^-2 w of free parameter j, 128 x 32) and B =
// [Jt_hi; Jt_lo] (row k < mfit: column J[.][l_k]; row mfit: the residuals
// dy; the low parts from row tc_arows(mfit) on), both split into TF32 high
// and low parts, so that the four quadrants of the FP32 accumulator (128
// lanes x 2 tc_arows(mfit) columns) sum to alpha (and beta in column mfit)
// at FP32 accuracy.  The accumulator stays in Tensor Memory across tiles
// until tc_alpha_flush.  chi^2 is summed in FP64 by warp 0, unless the
// caller has prepared the weights, residuals and chi^2 (prepared).  With
// rows (a relative lightcurve's second pass) the operands are built straight
// from the parked rows (stride rw: renormalisation factor in column 0, y/ave
// in ma, residual in ma + 1, weight in ma + 2), renormalising on the way
// (mrqcof.c:90-104).
template <int NT>
__device__ void accumulate_tile_tc(const DevObject &ob, Smem<PS_FORM_MIXED> &s, int np, int q0pt, bool conv,
                                   double conv_sig, TcState &t, bool prepared, const float *rows = nullptr,
                                   int rw = 0)
{
    const int tid = team_thread<NT>(), lane = tid & 31, warp = tid >> 5;
    const int ma = ob.ma, mf = ob.mfit;
    float *dyv = s.accs;
    float *wtp = dyv + 32;
    if (tid < 32 && !prepared) {
        double c2 = 0;
        if (tid < np) {
            const int q = q0pt + tid;
            const double sig2i = conv ? 1 / (conv_sig * conv_sig) : ob.sig2i[q];
            const double wg = ob.weight[q];
            const double dy = (conv ? 0.0 : ob.bright[q]) - s.ym[tid];
            dyv[tid] = static_cast<float>(dy);
            wtp[tid] = static_cast<float>(sig2i * wg);
            c2 = dy * dy * sig2i * wg;
        }
        c2 = warp_sum(c2);
        if (tid == 0) s.misc[M_CHISQ] += c2;
    }
    tc_alpha_wait<NT>(s, t);
    team_sync<NT>();
    // operands in the canonical K-major layout, K = the tile's 32 points
    // (zero beyond np): 8-row x 4-point core matrices, K-adjacent ones 128
    // bytes apart, 8-row groups 1024 bytes apart; high parts in rows 0..63,
    // low parts in rows 64..127
    unsigned char *Ab = s.aop, *Bb = s.aop + 16384;
    // (row groups of A past rg_end hold what was there: their lanes of the
    // accumulator are not read; B has none)
    const int rg_end = tc_arows(mf) >> 3;
    // warp w: core matrices c = w + (warps) i of both operands (row group c / 8,
    // points 4 (c % 8) .. + 3), the same J element feeding A and B
    constexpr int NW = NT / 32;
#pragma unroll
    for (int i = 0; i < 64 / NW; i++) {
        const int c = warp + NW * i, rg = c >> 3, kc = c & 7;
        if (rg < rg_end) {
            const int row = rg * 8 + (lane >> 2), p = kc * 4 + (lane & 3);
            float va = 0.f, vb = 0.f;
            if (p < np) {
                if (rows) {
                    const float *r = rows + static_cast<size_t>(p) * rw;
                    if (row < mf) {
                        const int l = s.flist[row];
                        vb = l == 0 ? 0.f : r[0] * (r[l] - r[ma] * s.davef[l]);
                        va = vb * r[ma + 2];
                    } else if (row == mf) {
                        vb = r[ma + 1];
                    }
                } else if (row < mf) {
                    vb = s.J[p * ma + s.flist[row]];
                    va = vb * wtp[p];
                } else if (row == mf) {
                    vb = dyv[p];
                }
            }
            const uint32_t ah = tc::to_tf32(va), bh = tc::to_tf32(vb);
            const uint32_t al = tc::to_tf32(va - __uint_as_float(ah)), bl = tc::to_tf32(vb - __uint_as_float(bh));
            reinterpret_cast<uint32_t *>(Ab + (rg * 8 + kc) * 128)[lane] = ah;
            reinterpret_cast<uint32_t *>(Ab + ((rg + 8) * 8 + kc) * 128)[lane] = al;
            reinterpret_cast<uint32_t *>(Bb + (rg * 8 + kc) * 128)[lane] = bh;
            reinterpret_cast<uint32_t *>(Bb + ((rg + rg_end) * 8 + kc) * 128)[lane] = bl;
        }
    }
    tc::fence_proxy_async();
    tc::fence_before_sync();
    team_sync<NT>();
    tc_alpha_issue<NT>(s, t, mf);
}

// Adds the alpha accumulator to the FP64 normal matrix M (lower triangle)
// and bv, and marks it empty: each quadrant pair is summed on the way out of
// Tensor Memory (rows m and 64 + m, columns k and 64 + k).
template <int NT>
__device__ void tc_alpha_flush(const DevObject &ob, Smem<PS_FORM_MIXED> &s, double *M, double *bv, TcState &t)
{
    const int tid = team_thread<NT>(), lane = tid & 31, warp = tid >> 5;
    const int mf = ob.mfit;
    if (t.afresh) return;
    tc_alpha_wait<NT>(s, t);
    if (*s.abort) return;
    float *S = reinterpret_cast<float *>(s.bhi);   // [128][65], after the tile's contraction
    // 8 of the column pairs (k, nb + k) of the warp's lane quadrant at a time
    const int quad = warp & 3, nb = tc_arows(mf);
    for (int c0 = 8 * (warp >> 2); c0 < nb; c0 += NT / 16) {
        const uint32_t taddr = t.tbase + (static_cast<uint32_t>(quad * 32) << 16) + t.acol + c0;
        float *sr = S + (quad * 32 + lane) * 65 + c0;
        uint32_t vh[8], vl[8];
        tc::tmem_ld8(taddr, vh);
        tc::tmem_ld8(taddr + nb, vl);
        tc::tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; j++) sr[j] = __uint_as_float(vh[j]) + __uint_as_float(vl[j]);
    }
    team_sync<NT>();
    const int ntri = mf * (mf + 1) / 2;
    for (int e = tid; e < ntri; e += NT) {
        const int j = tri_row(e);
        const int k = e - j * (j + 1) / 2;
        M[j * mf + k] += static_cast<double>(S[j * 65 + k] + S[(64 + j) * 65 + k]);
    }
    for (int j = tid; j < mf; j += NT) bv[j] += static_cast<double>(S[j * 65 + mf] + S[(64 + j) * 65 + mf]);
    t.afresh = true;
    tc::fence_before_sync();
    team_sync<NT>();
}

// The parts of an evaluation at parameters a[] that do not depend on the
// points: facet areas (s.area, s.gv), their sum, the rotation matrices and
// the phase and scattering parameters (s.bmat), the scale of the tensor-core
// operand; clears chi^2.  Ends with a barrier.
template <int FORM, int KU, int NT>
__device__ void shape_prologue(const DevObject &ob, Smem<FORM> &s, const double *a)
{
    using R = typename RealOf<FORM>::T;
    constexpr bool kFP64 = FORM == PS_FORM_FP64;
    constexpr bool kPipe = !kFP64 && (KU == 0 || KU == 3);
    const int tid = team_thread<NT>(), lane = tid & 31, warp = tid >> 5;
    const int F = ob.nfac, C = ob.ncoef, ma = ob.ma;
    // The scalars' exp, cos and sin on the last warp (the pole angles on two
    // lanes at once), which has no facets on the usual grids, while the
    // other warps compute the curvature.
    if (warp == NT / 32 - 1) {
        if (lane < 2) {
            const double x = a[C + lane];
            s.misc[M_TRIG + 2 * lane] = cos(x);
            s.misc[M_TRIG + 2 * lane + 1] = sin(x);
        } else if (lane == 2) {
            s.misc[M_CL] = exp(a[ma - 2]);
            s.misc[M_CHISQ] = 0;
        }
    }
    // curv.c:10-39 -- g_i = exp(sum over (m,l) of P_l^m (c cos + c' sin)), FP64.
    // (a team of fewer threads takes the places of several: the area sum's
    // order is that of the form's full slot)
    constexpr int NV = threads_of<FORM>();
#pragma unroll
    for (int part = 0; part < NV / NT; part++) {
        const int vt = tid + part * NT;
        double asum = 0;
        for (int i = vt; i < F; i += NV) {
            double g = 0;
            if constexpr (kFP64) {
                for (int q = 0; q < ob.npairs; q++) {
                    int m = ob.pair_m[q], n = ob.pair_n[q];
                    double fsum = a[n] * ob.fc[m * F + i];
                    if (m != 0) fsum = fsum + a[n + 1] * ob.fs[m * F + i];
                    g = g + ob.pleg[q * F + i] * fsum;
                }
            } else {
                // the same sum as the dot product of the facet's FP64 basis row
                // (Dsph[i][n] = P_l^m cos(m phi_i), Dsph[i][n + 1] = P_l^m
                // sin(m phi_i)) with the shape coefficients: independent loads
                // instead of a pair-index chain per term; it rounds differently
                // from curv.c's order by about 1e-16
                const double *drow = ob.dsph + static_cast<size_t>(i) * ob.ncoef;
#pragma unroll 7
                for (int k = 0; k < ob.ncoef; k++) g = fma(drow[k], a[k], g);
            }
            g = exp(g);
            double ar = ob.darea[i] * g;
            s.area[i] = ar;
            s.gv[i] = g;
            if constexpr (!kFP64) {
                if constexpr (kPipe) {
                    fac_at(s.fac, i, 3) = static_cast<float>(ar);
                } else {
                    s.areaR[i] = static_cast<R>(ar);
                    s.gvR[i] = static_cast<R>(g);
                }
            }
            asum += ar;
        }
        asum = warp_sum(asum);
        if (lane == 0) s.misc[M_RED + (vt >> 5)] = asum;
    }
    team_sync<NT>();
    // Every scalar once, on a warp of its own (an FP64 instruction holds the
    // FP64 unit for the whole warp): the area sum, blmatrix.c:9-46 in FP64
    // from the angles' cos/sin, one entry per lane, stored in the
    // facet-stage type with the phase and scattering parameters.
    if (tid == 0) {
        double t = 0;
#pragma unroll
        for (int i = 0; i < NV / 32; i++) t += s.misc[M_RED + i];
        s.misc[M_AREA] = t;
    } else if (warp == 2) {
        R v;
        if (lane < 27) {
            const int code = c_bl_code[lane];
            const int fa = code & 3, fb = (code >> 2) & 3;
            const double va = fa == 1 ? s.misc[M_TRIG] : fa == 2 ? s.misc[M_TRIG + 1] : fa == 3 ? 1.0 : 0.0;
            const double vb = fb == 1 ? s.misc[M_TRIG + 2] : fb == 2 ? s.misc[M_TRIG + 3] : 1.0;
            const double p = va * vb;
            v = R((code & 16) ? -p : p);
        } else {
            v = R(lane == 31 ? s.misc[M_CL] : a[lane == 30 ? C + 7 : C + 3 + (lane - 27)]);
        }
        s.bmat[lane] = v;
    } else if (kPipe && warp == 1) {
        // Scale of the contraction operand W = Darea g s: s <= |cl| +
        // |cls| / 2 (mu mu0 <= 1, mu mu0 / (mu + mu0) <= 1/2), and the
        // convexity rows' W <= Darea g, so 2^k puts the evaluation's largest
        // W just below 2^14.
        float mx = 0.f;
        for (int i = lane; i < F; i += 32) mx = fmaxf(mx, fac_at(s.fac, i, 3));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float wmax =
            mx * fmaxf(1.f, fabsf(static_cast<float>(s.misc[M_CL])) + 0.5f * fabsf(static_cast<float>(a[C + 7])));
        if (lane == 0) s.misc[M_WEXP] = (wmax > 0.f && wmax < 1e30f) ? static_cast<double>(13 - ilogbf(wmax)) : 0.0;
    }
    team_sync<NT>();
}

// ---------------------------------------------------------------------------
// Mixed form's model evaluation (mrqcof) at parameters a[] into M (mfit x mfit,
// lower triangle accumulated then mirrored) and vector bv.  Leaves chi^2,
// the facet-area sum and the convexity residuals in misc.  fresh = false:
// chi2_mixed has just run at the same parameters (an accepted step): neither
// the shape's terms nor chi^2 are formed again.
// ---------------------------------------------------------------------------
template <int KU, int NT>
__device__ void evaluate_mixed(const DevObject &ob, const FitConfig &cfg, const SlotLayout &L,
                               Smem<PS_FORM_MIXED> &s, const double *a, double *M, double *bv, float *scratch,
                               TcState &tcs, bool fresh = true)
{
    using R = float;
    // tensor-core path: the point set-up of the next tile runs on warps 1..15
    // while thread 0 issues the current tile's MMAs
    constexpr bool kPipe = KU == 0 || KU == 3;
    // alpha/beta on the tensor cores (KU 0), or on the SIMT pipes behind the
    // wide tensor-core contraction (KU 3: 65..96 coefficients)
    constexpr bool kTcAlpha = KU == 0;
    constexpr bool kWide = KU == 3;
    constexpr bool kAlias = NT == kTeamThreads;   // alpha's operands lie over the contraction's (make_layout)
    static_assert(NT == threads_of<PS_FORM_MIXED>() || KU == 0, "teams: the tensor-core path only");
    const int tid = team_thread<NT>(), lane = tid & 31, warp = tid >> 5;
    const int F = ob.nfac, C = ob.ncoef, ma = ob.ma, mf = ob.mfit, P = L.P;
    const int wcols = L.wcols;
    const int RW = rel_row_stride(ma);   // parked row of a relative lightcurve
    const R *nxR = ob.nx_f, *nyR = ob.ny_f, *nzR = ob.nz_f, *dareaR = ob.darea_f;

    if (fresh) shape_prologue<PS_FORM_MIXED, KU, NT>(ob, s, a);
    else if (tid == 0) s.misc[M_CHISQ] = 0;
    for (int e = tid; e < mf * mf; e += NT) M[e] = 0;
    for (int j = tid; j < mf; j += NT) bv[j] = 0;
    const double omg = a[C + 2];
    team_sync<NT>();
    const R cls = s.bmat[30], cl = s.bmat[31];
    // power-of-two scales of the tensor-core contraction's operands
    const int wexp = kPipe ? static_cast<int>(s.misc[M_WEXP]) : 0;
    const float wscale = ldexpf(1.f, wexp);
    const float jscale = ldexpf(1.f, -(wexp + tcs.basis_exp));

    const double conv_sig = cfg.conv_sig;
    float4 accA[kAlphaUnits<KU>];
    float accB = 0.f;
#pragma unroll
    for (int u = 0; u < kAlphaUnits<KU>; u++) accA[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    int unit[kAlphaUnits<KU>];
    if constexpr (!kTcAlpha) {
#pragma unroll
        for (int u = 0; u < kAlphaUnits<KU>; u++) unit[u] = alpha_unit(warp + u * (NT / 32), mf);
    }
    int tiles_since_flush = 0;
    const float *dsphF = s.dsph ? s.dsph : ob.dsph_f;
    // Point set-up threads.  An FP64 instruction holds its sub-partition's
    // FP64 unit for the whole warp however few lanes are active, so the
    // set-up keeps its points on one warp, lane = point (FP64 only for the
    // rotation phase).  On the tensor-core path warp 1 sets up the evaluation's first tile here; later tiles are set
    // up in the contraction window of the tile before (warps 1..3).
    const int pipe_sp = warp == 1 ? lane : -1;
    if constexpr (kPipe) {
        if (ob.n_lc > 1 && pipe_sp >= 0 && pipe_sp < min(P, ob.lc_npts[0])) {
            const int q = ob.lc_start[0] + pipe_sp;
            float *pt0 = s.pt + pipe_sp * kPointStride;
            setup_mixed_phase(ob.tim[q], omg, cfg.phi0, pt0);
            setup_mixed_geo(ob.geo_f[2 * q], ob.geo_f[2 * q + 1], s.bmat, pt0);
        }
        team_sync<NT>();   // the first tile's facet stage reads it
    }

    for (int lc = 0; lc < ob.n_lc; lc++) {
        const int start = ob.lc_start[lc], npts = ob.lc_npts[lc];
        const bool rel = ob.lc_rel[lc] != 0;
        const bool conv = (lc == ob.n_lc - 1);
        if (rel) {
            for (int l = tid; l < ma; l += NT) s.dave[l] = 0;
            if (tid == 0) s.misc[M_AVE] = 0;
        }
        // ---- pass 1: model rows of this lightcurve, tile by tile ----
        for (int t0 = 0; t0 < npts; t0 += P) {
            const int np = min(P, npts - t0);
            if (!conv) {
                // 1. point set-up (bright.c:27-57, phasec.c, matrix.c), one
                // thread per point on as few warps as possible; with the
                // tensor cores it was done during the previous tile's MMAs
                if constexpr (!kPipe) {
                    if (warp == 0 && lane < np)
                        setup_point(ob, cfg, start + t0 + lane, omg, s.bmat, s.pt + lane * kPointStride);
                }
                // (with the tensor cores the set-up is a tile old: the
                // barrier after the previous tile's contraction ordered it)
                if constexpr (!kPipe) team_sync<NT>();
                // 2. facet stage (bright.c:59-120), one warp per point
                if constexpr (kPipe) {
                    // prefetch for the contraction window: the next tile's
                    // times (warp 1) and geometry (warps 2 and 3, a copy
                    // each), this tile's accumulation data (warp 14)
                    if (kTcAlpha && warp == NT / 32 - 2) {
                        if (!rel && lane < np) {
                            const int q = start + t0 + lane;
                            double *d = reinterpret_cast<double *>(s.pref + kPrefAcc) + 3 * lane;
                            cp_async8(d, ob.sig2i + q);
                            cp_async8(d + 1, ob.weight + q);
                            cp_async8(d + 2, ob.bright + q);
                        }
                        cp_async_commit();
                    } else if (warp >= 1 && warp <= 3) {
                        const int nlc = t0 + P < npts ? lc : lc + 1, nt0 = t0 + P < npts ? t0 + P : 0;
                        if (nlc < ob.n_lc - 1 && lane < min(P, ob.lc_npts[nlc] - nt0)) {
                            const int q = ob.lc_start[nlc] + nt0 + lane;
                            if (warp == 1) {
                                cp_async8(reinterpret_cast<double *>(s.pref + kPrefTim) + lane, ob.tim + q);
                            } else {
                                float4 *g = reinterpret_cast<float4 *>(s.pref + (warp == 2 ? kPrefGeo : kPrefGeo2)) +
                                            2 * lane;
                                cp_async16(g, ob.geo_f + 2 * q);
                                cp_async16(g + 1, ob.geo_f + 2 * q + 1);
                            }
                        }
                        cp_async_commit();
                    }
                    if constexpr (kAlias) tc_alpha_wait<NT>(s, tcs);   // the operands share their memory
                    facet_stage_tc<NT>(ob, s, np, cl, cls, wscale);
                }
                else
                for (int p = warp; p < np; p += NT / 32) {
                    const R *pt = s.pt + p * kPointStride;
                    const R e1 = pt[0], e2 = pt[1], e3 = pt[2];
                    const R f1 = pt[3], f2 = pt[4], f3 = pt[5];
                    R de[9], de0[9];
#pragma unroll
                    for (int k = 0; k < 9; k++) {
                        de[k] = pt[6 + k];
                        de0[k] = pt[15 + k];
                    }
                    R br = 0, r0 = 0, r1 = 0, r2 = 0, dcl = 0, dcls = 0;
                    R *Wp = s.W + static_cast<size_t>(p) * wcols;
                    for (int i = lane; i < F; i += 32) {
                        const R nx = nxR[i], ny = nyR[i], nz = nzR[i];
                        const R mu = e1 * nx + e2 * ny + e3 * nz;
                        const R mu0 = f1 * nx + f2 * ny + f3 * nz;
                        R w = 0;
                        if (mu > R(kTinyMu) && mu0 > R(kTinyMu)) {
                            const R ar = s.areaR[i];
                            const LitTerms<R, PS_FORM_MIXED> lt(mu, mu0, cl, cls);
                            br = br + ar * lt.sv;
                            w = dareaR[i] * lt.sv * s.gvR[i];
                            const R s0 = nx * de[0] + ny * de[3] + nz * de[6];
                            const R s1 = nx * de[1] + ny * de[4] + nz * de[7];
                            const R s2 = nx * de[2] + ny * de[5] + nz * de[8];
                            const R t0v = nx * de0[0] + ny * de0[3] + nz * de0[6];
                            const R t1v = nx * de0[1] + ny * de0[4] + nz * de0[7];
                            const R t2v = nx * de0[2] + ny * de0[5] + nz * de0[8];
                            r0 = r0 + ar * (lt.dsmu * s0 + lt.dsmu0 * t0v);
                            r1 = r1 + ar * (lt.dsmu * s1 + lt.dsmu0 * t1v);
                            r2 = r2 + ar * (lt.dsmu * s2 + lt.dsmu0 * t2v);
                            dcl = dcl + mu * mu0 * ar;
                            dcls = dcls + ar * lt.dcls_w;
                        }
                        Wp[i] = w;
                    }
                    br = warp_sum(br);
                    r0 = warp_sum(r0);
                    r1 = warp_sum(r1);
                    r2 = warp_sum(r2);
                    dcl = warp_sum(dcl);
                    dcls = warp_sum(dcls);
                    if (lane == 0) {
                        double *rd = s.red + p * kRedStride;
                        rd[0] = br;
                        rd[1] = r0;
                        rd[2] = r1;
                        rd[3] = r2;
                        rd[4] = dcl;
                        rd[5] = dcls;
                    }
                }
            } else if constexpr (kPipe) {
                if constexpr (kAlias) tc_alpha_wait<NT>(s, tcs);
                conv_rows_tc<NT>(ob, s, wscale);
            } else {
                // convexity rows (conv.c:12-29): W = Darea g n_c, residual =
                // sum Area n_c (the residual in FP64 in both forms)
                for (int p = warp; p < np; p += NT / 32) {
                    const double *nc = (p == 0) ? ob.nx : (p == 1) ? ob.ny : ob.nz;
                    double res = 0;
                    R *Wp = s.W + static_cast<size_t>(p) * wcols;
                    for (int i = lane; i < F; i += 32) {
                        res = res + s.area[i] * nc[i];
                        Wp[i] = R(ob.darea[i] * s.gv[i] * nc[i]);
                    }
                    res = warp_sum(res);
                    if (lane == 0) s.red[p * kRedStride] = res;
                }
            }
            // (the tensor-core issue below begins with a barrier of its own)
            if constexpr (!kPipe) team_sync<NT>();
            // 3. shape contraction and the remaining columns of J
            if constexpr (kPipe) {
                contract_tc_issue<NT, kWide>(s, F, tcs);   // the work below overlaps the MMAs
            } else {
                if (s.dsph)
                    contract_mixed_call<NT, KU, true>(s.W, s.pt, s.J, dsphF, np, F, C, ma, wcols, conv);
                else if constexpr (KU == 2)
                    contract_mixed_call<NT, KU, false>(s.W, s.pt, s.J, dsphF, np, F, C, ma, wcols, conv);
                else
                    contract_mixed<NT, KU, false>(s.W, s.pt, s.J, dsphF, np, F, C, ma, wcols, conv);
            }
            // remaining columns of J: one thread per point (not thread 0 on the
            // tensor-core path: it issues the MMAs)
            const int jp = kPipe ? (tid + 32) % NT : tid;
            if (jp < np) {
                const int p = jp;
                R *Jp = s.J + p * ma;
                const double *rd = s.red + p * kRedStride;
                if (!conv) {
                    R v[6];
                    if constexpr (kPipe) {
                        point_sums_tc(s, p, v);
                    } else {
#pragma unroll
                        for (int k = 0; k < 6; k++) v[k] = R(rd[k]);
                    }
                    const R *pt = s.pt + p * kPointStride;
                    const R scale = pt[24];
                    const R br = v[0];
                    Jp[C] = scale * v[1];
                    Jp[C + 1] = scale * v[2];
                    Jp[C + 2] = scale * v[3];
                    Jp[C + 3] = br * pt[25];
                    Jp[C + 4] = br * pt[26];
                    Jp[C + 5] = br * pt[27];
                    Jp[C + 6] = scale * v[4] * cl;
                    Jp[C + 7] = scale * v[5];
                    s.ym[p] = static_cast<double>(br * scale);
                } else {
                    for (int k = C; k < ma; k++) Jp[k] = 0;
                    s.ym[p] = rd[0];
                    s.misc[M_CHK + p] = rd[0];
                }
            }
            if constexpr (kPipe) {
                // the accumulation's per-point FP64 work (weights, residuals,
                // chi^2) of an absolute lightcurve or of the convexity rows,
                // here on the last warp but one (its own copy of the model value) while
                // thread 0 issues the contraction and the last writes the J
                // columns (same per-point values and reduction as in the
                // accumulation itself)
                if (rel && warp == NT / 32 - 1) {
                    // relative lightcurve: park the model value with the
                    // row and add the tile to the lightcurve sum
                    double y = 0;
                    if (jp < np) {
                        y = s.ym[jp];
                        scratch[static_cast<size_t>(t0 + jp) * RW + ma] = R(y);
                    }
                    y = warp_sum(y);
                    if (lane == 0) s.misc[M_AVE] += y;
                }
                if (kTcAlpha && !rel && warp == NT / 32 - 2) {
                    double c2 = 0;
                    cp_async_wait_all();
                    if (lane < np) {
                        const int q = start + t0 + lane;
                        const double *pa = reinterpret_cast<const double *>(s.pref + kPrefAcc) + 3 * lane;
                        float br = 0.f;
                        if (!conv) {
#pragma unroll
                            for (int h = 0; h < 4; h++) br += s.fpart[(h * 32 + lane) * 9];
                        }
                        const double ymv = conv ? s.red[lane * kRedStride]
                                                : static_cast<double>(br * s.pt[lane * kPointStride + 24]);
                        const double sig2i = conv ? 1 / (conv_sig * conv_sig) : pa[0];
                        const double wg = conv ? ob.weight[q] : pa[1];
                        const double dy = (conv ? 0.0 : pa[2]) - ymv;
                        s.accs[lane] = static_cast<float>(dy);
                        s.accs[32 + lane] = static_cast<float>(sig2i * wg);
                        if (fresh) c2 = dy * dy * sig2i * wg;
                    }
                    if (fresh) {
                        c2 = warp_sum(c2);
                        if (lane == 0) s.misc[M_CHISQ] += c2;
                    }
                }
            }
            bool next_setup = false;
            if constexpr (kPipe) {
                // point set-up of the next tile into the other buffer, one
                // point per lane: the rotation phase on warp 1, the phase
                // function and pole products on warps 2 and 3 (the facet
                // stage applies the rotation)
                const int nlc = t0 + P < npts ? lc : lc + 1, nt0 = t0 + P < npts ? t0 + P : 0;
                next_setup = nlc < ob.n_lc - 1;   // the last lightcurve is the convexity rows
                if (next_setup && warp >= 1 && warp <= 3) {
                    const bool have = lane < min(P, ob.lc_npts[nlc] - nt0);
                    float *ptn = s.pt2 + lane * kPointStride;
                    cp_async_wait_all();
                    if (warp == 1) {
                        if (have) setup_mixed_phase(reinterpret_cast<const double *>(s.pref + kPrefTim)[lane], omg,
                                                    cfg.phi0, ptn);
                    } else {
                        const float4 *g =
                            reinterpret_cast<const float4 *>(s.pref + (warp == 2 ? kPrefGeo : kPrefGeo2)) + 2 * lane;
                        if (have) setup_mixed_geo(g[0], g[1], s.bmat, ptn, warp - 2);
                    }
                }
                contract_tc_finish<NT, kWide>(s, np, F, C, ma, conv, tcs, jscale);
            }
            team_sync<NT>();
            if (next_setup) {
                R *t = s.pt;
                s.pt = s.pt2;
                s.pt2 = t;
            }
            if (rel) {
                // 4a. lightcurve sums and a copy of the rows (mrqcof.c:51-88)
                // (on the tensor-core path the last warp has parked the model
                // values and summed them during the contraction; the FP64
                // column sums run on sub-partitions 2 and 3)
                R *dst = scratch + static_cast<size_t>(t0) * RW;
                for (int e = tid; e < np * ma; e += NT) {
                    int p = e / ma, l = e - p * ma;
                    dst[static_cast<size_t>(p) * RW + l] = s.J[e];
                }
                if (!kPipe && tid < np) dst[static_cast<size_t>(tid) * RW + ma] = R(s.ym[tid]);
                for (int l = kPipe ? tid - 64 : tid; l < ma; l += NT) {
                    if (l < 0) break;
                    float d = 0.f;
                    for (int p = 0; p < np; p++) d += s.J[p * ma + l];
                    s.dave[l] += static_cast<double>(d);
                }
                if (!kPipe && warp == 0) {
                    const double v = warp_sum(lane < np ? s.ym[lane] : 0.0);
                    if (lane == 0) s.misc[M_AVE] += v;
                }
                team_sync<NT>();
                continue;
            }
            // 5. accumulate (mrqcof.c:106-136)
            if constexpr (kTcAlpha) {
                accumulate_tile_tc<NT>(ob, s, np, start + t0, conv, conv_sig, tcs, true);
                if (++tiles_since_flush == kTcTilesPerFlush) {
                    tc_alpha_flush<NT>(ob, s, M, bv, tcs);
                    tiles_since_flush = 0;
                }
            } else {
                accumulate_tile<KU>(ob, s, np, start + t0, conv, conv_sig, fresh, unit, accA, accB);
                if (++tiles_since_flush == kTilesPerFlush) {
                    flush_partials<KU>(M, bv, mf, unit, accA, accB);
                    tiles_since_flush = 0;
                }
            }
        }
        if (!rel) continue;
        // ---- pass 2: renormalise and accumulate (mrqcof.c:90-136) ----
        const double ave = s.misc[M_AVE];
        // the renormalisation runs in FP32 on FP32 copies, with one
        // reciprocal of the lightcurve sum (computed once, not per warp; the
        // FP64 form divides as the reference does)
        for (int l = tid; l < ma; l += NT) s.davef[l] = static_cast<float>(s.dave[l]);
        if (tid == 0) s.misc[M_INVAVE] = 1.0 / ave;
        team_sync<NT>();
        const double inv_ave = s.misc[M_INVAVE];
        if constexpr (kTcAlpha) {
            // The per-point FP64 work of the whole lightcurve at once, one
            // tile per warp (the tiles' FP64 chains on different
            // sub-partitions): renormalisation factor coef and y/ave into
            // the row's columns 0 (unused by the renormalised row) and ma,
            // residual and weight into ma + 1 and ma + 2; the tiles' chi^2
            // sums are added in tile order (16 tiles a round).
            for (int r0 = 0; r0 * P < npts; r0 += NT / 32) {
                const int tt = r0 + warp;
                const int p = tt * P + lane;
                double c2 = 0;
                if (lane < P && p < npts) {
                    const int q = start + p;
                    R *row = scratch + static_cast<size_t>(p) * RW;
                    const double yt = static_cast<double>(row[ma]);
                    const double coef = ob.sig[q] * npts * inv_ave;
                    const double ym = coef * yt;
                    const double sig2i = ob.sig2i[q];
                    const double wg = ob.weight[q];
                    const double dy = ob.bright[q] - ym;
                    row[0] = static_cast<float>(coef);
                    row[ma] = static_cast<float>(yt * inv_ave);
                    row[ma + 1] = static_cast<float>(dy);
                    row[ma + 2] = static_cast<float>(sig2i * wg);
                    if (fresh) c2 = dy * dy * sig2i * wg;
                }
                if (!fresh) continue;   // chi^2 is known
                c2 = warp_sum(c2);
                if (lane == 0) s.red[warp] = c2;
                team_sync<NT>();
                if (tid == 0)
                    for (int w = 0; w < NT / 32 && (r0 + w) * P < npts; w++) s.misc[M_CHISQ] += s.red[w];
                if ((r0 + NT / 32) * P < npts) team_sync<NT>();
            }
        }
        for (int t0 = 0; t0 < npts; t0 += P) {
            const int np = min(P, npts - t0);
            const R *src = scratch + static_cast<size_t>(t0) * RW;
            // model values of the tile in FP64 (parked as FP32); on the
            // tensor-core path they were prepared above, and the tile's residuals and
            // weights go where the accumulation reads them
            if constexpr (kTcAlpha) {
                // operands built from the parked rows (renormalised on the way)
                accumulate_tile_tc<NT>(ob, s, np, start + t0, false, conv_sig, tcs, true, src, RW);
                if (++tiles_since_flush == kTcTilesPerFlush) {
                    tc_alpha_flush<NT>(ob, s, M, bv, tcs);
                    tiles_since_flush = 0;
                }
                continue;
            }
            if (tid < np) {
                const int q = start + t0 + tid;
                const double yt = static_cast<double>(src[static_cast<size_t>(tid) * RW + ma]);
                const double coef = ob.sig[q] * npts * inv_ave, ytr = yt * inv_ave;
                s.ym[tid] = coef * yt;
                s.accs[tid] = static_cast<float>(coef);        // consumed before the
                s.accs[32 + tid] = static_cast<float>(ytr);    // accumulation reuses it
            }
            team_sync<NT>();
            for (int e = tid; e < np * ma; e += NT) {
                const int p = e / ma, l = e - p * ma;
                const R v = src[static_cast<size_t>(p) * RW + l];
                const R out = s.accs[p] * (v - s.accs[32 + p] * s.davef[l]);
                s.J[e] = (l == 0) ? R(0) : out;
            }
            team_sync<NT>();
            accumulate_tile<KU>(ob, s, np, start + t0, false, conv_sig, fresh, unit, accA, accB);
            if (++tiles_since_flush == kTilesPerFlush) {
                flush_partials<KU>(M, bv, mf, unit, accA, accB);
                tiles_since_flush = 0;
            }
        }
    }
    if constexpr (kTcAlpha) tc_alpha_flush<NT>(ob, s, M, bv, tcs);
    else flush_partials<KU>(M, bv, mf, unit, accA, accB);
    team_sync<NT>();
    // mirror the lower triangle (mrqcof.c:139-141)
    for (int e = tid; e < mf * mf; e += NT) {
        const int j = e / mf, k = e - j * mf;
        if (k > j) M[e] = M[k * mf + j];
    }
    team_sync<NT>();
}

// ---------------------------------------------------------------------------
// FP64 form's model evaluation (mrqcof), by one CTA or (SPLIT) by the CTAs of
// a thread-block cluster.  Bound by the FP64 units: a warp's FP64 instruction
// holds its sub-partition's unit for 64 cycles however few lanes are active,
// so every stage keeps its lanes full and its warps spread evenly over the
// four sub-partitions, and what is the same for a point is computed once.
//
// SPLIT: one fit's point tiles are dealt round-robin to the cluster's CTAs,
// which compute their tiles' model rows (tile_rows_fp64) at the same time;
// after each round every CTA takes the round's tiles in data order -- its own
// from its shared memory, the others' through distributed shared memory --
// and runs what sums over points: the relative lightcurves' sums, parked rows
// and second pass, and chi^2 in full, the normal matrix and beta for its
// share of the elements only.  Every sum therefore runs in the same order as
// with one CTA, and the split fit is bit-identical to it.  Every CTA computes
// the convexity rows; then each copies its share of the matrix into the
// others, so that all of them take the same LM decisions and keep the same
// control flow (and the same sequence of cluster barriers).
//
// Measured (980 points, 288 facets): one evaluation 4.97 -> 4.33 ms, 400 fits
// 577 -> 548 ms with the set-up in twelve parts, the dot products, residuals
// and renormalisation factors once per point, the contraction's points in
// order of their lit counts and beta's elements among alpha's units.  Of an
// evaluation's 8.8 Mcycles the FP64 instructions take 7.7 on full units
// (contraction 3.3, facet law 3.0, alpha 0.8).
// ---------------------------------------------------------------------------
constexpr int kMaxSplit = 16;
constexpr int kWarpsFp64 = threads_of<PS_FORM_FP64>() / 32;

// Where the first set-up part of point `lane` of the group's tile `slot` lies:
// the four values' distance in stride.
__device__ inline double *phase_at(const SlotLayout &L, const Smem<PS_FORM_FP64> &s, int slot, int lane, int &stride)
{
    const bool own = L.phase_tiles > 1;
    stride = own ? L.phase_tiles * L.P : 1;
    return own ? s.phase + slot * L.P + lane : s.pt + lane * kPointStride + kPtPhase;
}

// First part of the set-up (setup_phase_fp64) of the CTA's next
// L.phase_tiles tiles, warp w the w-th, a point per lane: with one tile at a
// time the set-up ran on 8 lanes of 4 warps (28 of a tile's 320 kcycles; 7 now,
// with the second part).  (lc, t0): the first of these tiles; step: tiles from one
// of the CTA's tiles to its next.
__device__ inline void setup_group_fp64(const DevObject &ob, const FitConfig &cfg, const SlotLayout &L,
                                        Smem<PS_FORM_FP64> &s, int lc, int t0, int step, double omg)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < L.phase_tiles) {
        int skip = warp * step;
        while (lc < ob.n_lc - 1) {
            const int nt = (ob.lc_npts[lc] - t0 + L.P - 1) / L.P;
            if (skip < nt) break;
            skip -= nt;
            lc++;
            t0 = 0;
        }
        if (lc < ob.n_lc - 1) {
            t0 += skip * L.P;
            if (lane < min(L.P, ob.lc_npts[lc] - t0)) {
                int stride;
                double *ph = phase_at(L, s, warp, lane, stride);
                setup_phase_fp64(ob, cfg, ob.lc_start[lc] + t0 + lane, omg, s.bmat, ph, stride);
            }
        }
    }
    __syncthreads();
}

// Model rows of one tile of np points from q0 on into s.J / s.ym
// (bright.c:14-126), its first set-up part in the group's slot `slot`; conv:
// the convexity rows (conv.c:12-29).  Leaves with a barrier.
__device__ void tile_rows_fp64(const DevObject &ob, const SlotLayout &L, Smem<PS_FORM_FP64> &s, int q0, int np,
                               bool conv, int slot, bool count)
{
    constexpr int NW = kWarpsFp64;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int F = ob.nfac, C = ob.ncoef, ma = ob.ma, wcols = L.wcols;
    const double cls = s.bmat[30], cl = s.bmat[31];
    if (!conv) {
        // second part of the set-up: twelve parts, a warp each
        static_assert(NW == 12, "twelve set-up parts");
        const int part = warp & 3, i = warp >> 2;
        if (lane < np) {
            int stride;
            const double *ph = phase_at(L, s, slot, lane, stride);
            double *pt = s.pt + lane * kPointStride;
            setup_row_fp64(ob, q0 + lane, part, i, s.bmat, ph, stride, pt);
            if (part == 3 && i == 2) {
                const double alpha = ob.alpha_pt[q0 + lane], ex = ph[2 * stride];
                pt[24] = phase_scale_fp64(s.bmat[27], s.bmat[29], ex, alpha);
                pt[25] = ex;
                pt[26] = ph[3 * stride];
                pt[27] = alpha;
            }
        }
        __syncthreads();
        for (int p = warp; p < np; p += NW) facet_point_fp64(ob, s, p, wcols, cl, cls, count);
    } else {
        for (int p = warp; p < np; p += NW) {
            const double *nc = (p == 0) ? ob.nx : (p == 1) ? ob.ny : ob.nz;
            double res = 0;
            double *Wp = s.W + static_cast<size_t>(p) * wcols;
            for (int i = lane; i < F; i += 32) {
                res = res + s.area[i] * nc[i];
                Wp[i] = ob.darea[i] * s.gv[i] * nc[i];
            }
            res = warp_sum(res);
            if (lane == 0) s.red[p * kRedStride] = res;
        }
    }
    __syncthreads();
    // Contraction: outputs (point, coefficient) in units of 32 lanes.  A lane
    // runs as long as its point's lit list, a unit as long as its longest, so
    // the points are taken in order of their counts (each warp orders them
    // itself, into its byte of the points' records): a unit's points then have
    // nearly the same count.
    auto ord = [&](int r) -> unsigned char & {
        return reinterpret_cast<unsigned char *>(s.pt + r * kPointStride + kPtOrder)[warp];
    };
    {
        const int n = lane < np ? (conv ? F : s.nlit[lane]) : -1;
        int r = 0;
#pragma unroll
        for (int o = 0; o < 32; o++) {
            const int m = __shfl_sync(0xffffffffu, n, o);
            r += (m > n || (m == n && o < lane)) ? 1 : 0;
        }
        if (lane < np) ord(r) = static_cast<unsigned char>(lane);
        __syncwarp();
    }
    for (int o = tid; o < np * C; o += NW * 32) {
        const int r = o / C, k = o - r * C, p = ord(r);
        const double acc = contract_fp64(s, ob.dsph + k, p, C, F, wcols, conv);
        s.J[p * ma + k] = conv ? acc : s.pt[p * kPointStride + 24] * acc;
    }
    // the remaining columns, a point per lane of the last warp (which has the
    // fewest units): D_k . U + E_k . V with D_k = (de[k], de[3 + k], de[6 + k])
    // and E_k likewise from de0
    if (warp == NW - 1 && lane < np) {
        const int p = lane;
        double *Jp = s.J + p * ma;
        const double *rd = s.red + p * kRedStride;
        if (!conv) {
            const double *pt = s.pt + p * kPointStride, *de = pt + 6, *de0 = pt + 15;
            const double scale = pt[24];
            const double br = rd[0];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                double v = fma(de[k], rd[1], __dmul_rn(de[3 + k], rd[2]));
                v = fma(de[6 + k], rd[3], v);
                v = fma(de0[k], rd[4], v);
                v = fma(de0[3 + k], rd[5], v);
                v = fma(de0[6 + k], rd[6], v);
                Jp[C + k] = scale * v;
            }
            Jp[C + 3] = br * pt[25];
            Jp[C + 4] = br * pt[26];
            Jp[C + 5] = br * pt[27];
            Jp[C + 6] = scale * rd[7] * cl;
            Jp[C + 7] = scale * pt[kPtSum];
            s.ym[p] = br * scale;
        } else {
            for (int k = C; k < ma; k++) Jp[k] = 0;
            s.ym[p] = rd[0];
            s.misc[M_CHK + p] = rd[0];
        }
    }
    __syncthreads();
}

// Elements of the normal matrix's lower triangle, then of beta, in units of
// 32 lanes dealt to the cluster's CTAs and then to a CTA's warps: calls
// fn(e) for the calling thread's elements e.
template <class Fn>
__device__ inline void for_share(int n, int rank, int cs, Fn fn)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int u = warp * cs + rank; u * 32 < n; u += kWarpsFp64 * cs) {
        const int e = u * 32 + lane;
        if (e < n) fn(e);
    }
}

// Accumulates the rows Jrows[0..np) (model values ymv) of one tile into the
// normal matrix M (lower triangle), bv and chi^2 (mrqcof.c:106-136), every
// element over the points in data order; of M and bv the CTA's share, chi^2
// whole.  Residuals once per point; beta's elements are units like alpha's.
__device__ void accumulate_tile_fp64(const DevObject &ob, Smem<PS_FORM_FP64> &s, double *M, double *bv, int np,
                                     int q0, bool conv, double conv_sig, const double *Jrows, const double *ymv,
                                     int rank, int cs)
{
    constexpr int NT = threads_of<PS_FORM_FP64>();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ma = ob.ma, mf = ob.mfit;
    double *wt = s.W;   // [np][mf], reuses the facet-weight tile
    double *dyv = s.pt, *tv = dyv + 32;   // (the points' records have served)
    const double conv_s2 = conv ? 1 / (conv_sig * conv_sig) : 0.0;
    if (warp == kWarpsFp64 - 1 && lane < np) {
        const double dy = (conv ? 0.0 : ob.bright[q0 + lane]) - ymv[lane];
        dyv[lane] = dy;
        tv[lane] = dy * dy * (conv ? conv_s2 : ob.sig2i[q0 + lane]);
    }
    for (int e = tid; e < np * mf; e += NT) {
        const int p = e / mf, j = e - p * mf;
        const double sig2i = conv ? conv_s2 : ob.sig2i[q0 + p];
        wt[p * mf + j] = Jrows[p * ma + ob.free_list[j]] * sig2i * ob.weight[q0 + p];
    }
    __syncthreads();
    if (tid == NT - 1) {
        double c2 = s.misc[M_CHISQ];
#pragma unroll 4
        for (int p = 0; p < np; p++) c2 = fma(tv[p], ob.weight[q0 + p], c2);
        s.misc[M_CHISQ] = c2;
    }
    const int ntri = mf * (mf + 1) / 2;
    for_share(ntri + mf, rank, cs, [&](int e) {
        const double *x, *y;
        double *to;
        int ys;
        if (e < ntri) {
            const int j = tri_row(e), k = e - j * (j + 1) / 2;
            x = wt + j;
            y = Jrows + ob.free_list[k];
            ys = ma;
            to = M + j * mf + k;
        } else {
            x = wt + (e - ntri);
            y = dyv;
            ys = 1;
            to = bv + (e - ntri);
        }
        double acc = *to;
#pragma unroll 4
        for (int p = 0; p < np; p++) acc = fma(x[p * mf], y[p * ys], acc);
        *to = acc;
    });
    __syncthreads();
}

template <bool SPLIT>
__device__ void evaluate_fp64(const DevObject &ob, const FitConfig &cfg, const SlotLayout &L, Smem<PS_FORM_FP64> &s,
                              const double *a, double *M, double *bv, double *scratch, bool fresh)
{
    namespace cgr = cooperative_groups;
    constexpr int NT = threads_of<PS_FORM_FP64>(), NW = NT / 32;
    int rank = 0, cs = 1;
    if constexpr (SPLIT) {
        rank = static_cast<int>(cgr::this_cluster().block_rank());
        cs = static_cast<int>(cgr::this_cluster().num_blocks());
    }
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int C = ob.ncoef, ma = ob.ma, mf = ob.mfit, P = L.P;
    const int RW = rel_row_stride(ma);
    const int ntri = mf * (mf + 1) / 2;

    if (fresh) shape_prologue<PS_FORM_FP64, 1, threads_of<PS_FORM_FP64>()>(ob, s, a);
    else if (tid == 0) s.misc[M_CHISQ] = 0;
    for (int e = tid; e < mf * mf; e += NT) M[e] = 0;
    for (int j = tid; j < mf; j += NT) bv[j] = 0;
    const double omg = a[C + 2];
    __syncthreads();
    const double conv_sig = cfg.conv_sig;

    // A tile's sums (mrqcof.c:51-136).  Jt, yt: the tile's rows and model
    // values (the CTA's own tile, or another CTA's staged in Jst/ymst); the
    // second pass stages its renormalised rows there too, so that s.J, which
    // the other CTAs read during the round, stays as computed.
    // The staging area: stage_cap points' rows and model values.
    const int stage_cap =
        min((static_cast<int>((L.J - L.W) / sizeof(double)) - P * mf) / (ma + 1), P * kRedStride) / P * P;
    double *Jst = s.W + static_cast<size_t>(P) * mf, *ymst = Jst + static_cast<size_t>(stage_cap) * ma;
    auto consume_tile = [&](int lc, int t0, int np, const double *Jt, const double *yt) {
        const int start = ob.lc_start[lc], npts = ob.lc_npts[lc];
        if (!ob.lc_rel[lc]) {
            accumulate_tile_fp64(ob, s, M, bv, np, start + t0, false, conv_sig, Jt, yt, rank, cs);
            return;
        }
        double *dst = scratch + static_cast<size_t>(t0) * RW;
        for (int e = tid; e < np * ma; e += NT) {
            const int p = e / ma, l = e - p * ma;
            dst[static_cast<size_t>(p) * RW + l] = Jt[e];
        }
        if (tid < np) dst[static_cast<size_t>(tid) * RW + ma] = yt[tid];
        for (int l = tid; l < ma; l += NT) {
            double d = t0 == 0 ? 0.0 : s.dave[l];
#pragma unroll 8
            for (int p = 0; p < np; p++) d = d + Jt[p * ma + l];
            s.dave[l] = d;
        }
        // the reference's order (on a warp without column sums, C <= 121)
        if (tid == NT - 1) {
            double av = t0 == 0 ? 0.0 : s.misc[M_AVE];
#pragma unroll 8
            for (int p = 0; p < np; p++) av = av + yt[p];
            s.misc[M_AVE] = av;
        }
        __syncthreads();
        if (t0 + P < npts) return;
        // second pass of the lightcurve (mrqcof.c:90-136), as many tiles at a
        // time as the staging area holds: of the renormalised rows every CTA
        // computes its share of the points for all of the cluster (two
        // divisions per point and one per element: 12 of a tile's 18 kcycles
        // when each CTA computed them all)
        const double ave = s.misc[M_AVE];
        for (int b0 = 0; b0 < npts; b0 += stage_cap) {
            const int nb = min(stage_cap, npts - b0), mine = (nb - rank + cs - 1) / cs;
            const double *src = scratch + static_cast<size_t>(b0) * RW;
            double *coef = s.red;
            if constexpr (SPLIT) cgr::this_cluster().sync();   // every CTA's staging area is free
            for (int i = tid; i < mine; i += NT) {
                const int p = i * cs + rank;
                const double c = ob.sig[start + b0 + p] * npts / ave;
                coef[i] = c;
                const double y = c * src[static_cast<size_t>(p) * RW + ma];
                if constexpr (SPLIT) {
                    for (int r = 0; r < cs; r++) *cgr::this_cluster().map_shared_rank(ymst + p, r) = y;
                } else {
                    ymst[p] = y;
                }
            }
            __syncthreads();
            for (int e = tid; e < mine * ma; e += NT) {
                const int i = e / ma, l = e - i * ma, p = i * cs + rank;
                const double *row = src + static_cast<size_t>(p) * RW;
                const double out = l == 0 ? 0.0 : coef[i] * (row[l] - row[ma] * s.dave[l] / ave);
                if constexpr (SPLIT) {
                    for (int r = 0; r < cs; r++)
                        *cgr::this_cluster().map_shared_rank(Jst + static_cast<size_t>(p) * ma + l, r) = out;
                } else {
                    Jst[static_cast<size_t>(p) * ma + l] = out;
                }
            }
            if constexpr (SPLIT) cgr::this_cluster().sync();
            else __syncthreads();
            for (int u0 = 0; u0 < nb; u0 += P)
                accumulate_tile_fp64(ob, s, M, bv, min(P, nb - u0), start + b0 + u0, false, conv_sig,
                                     Jst + static_cast<size_t>(u0) * ma, ymst + u0, rank, cs);
        }
    };

    // rounds of cs tiles over the real lightcurves, in data order
    int rlc[SPLIT ? kMaxSplit : 1], rt0[SPLIT ? kMaxSplit : 1], rnp[SPLIT ? kMaxSplit : 1];
    int nround = 0, slot = L.phase_tiles;
    auto flush_round = [&]() {
        if constexpr (SPLIT) cgr::this_cluster().sync();   // every CTA's tile of the round is in its shared memory
        for (int k = 0; k < nround; k++) {
            const double *Jt = s.J, *yt = s.ym;
            if constexpr (SPLIT) {
                if (k != rank) {
                    // rank k's tile, read through distributed shared memory
                    const double *rJ = cgr::this_cluster().map_shared_rank(s.J, k);
                    const double *rY = cgr::this_cluster().map_shared_rank(s.ym, k);
                    for (int e = tid; e < rnp[k] * ma; e += NT) Jst[e] = rJ[e];
                    if (tid < rnp[k]) ymst[tid] = rY[tid];
                    __syncthreads();
                    Jt = Jst;
                    yt = ymst;
                }
            }
            consume_tile(rlc[k], rt0[k], rnp[k], Jt, yt);
        }
        if constexpr (SPLIT) cgr::this_cluster().sync();   // the round's tile buffers are free again
        nround = 0;
    };
    const int nreal = ob.n_lc - 1;
    for (int lc = 0; lc < nreal; lc++) {
        const int npts = ob.lc_npts[lc];
        for (int t0 = 0; t0 < npts; t0 += P) {
            const int np = min(P, npts - t0);
            rlc[nround] = lc;
            rt0[nround] = t0;
            rnp[nround] = np;
            if (nround == rank) {
                if (slot == L.phase_tiles) {
                    setup_group_fp64(ob, cfg, L, s, lc, t0, cs, omg);
                    slot = 0;
                }
                tile_rows_fp64(ob, L, s, ob.lc_start[lc] + t0, np, false, slot, fresh);
                slot++;
            }
            if (++nround == cs) flush_round();
        }
    }
    if (nround > 0) flush_round();
    // convexity rows (conv.c:12-29) on every CTA, each accumulating its share
    {
        const int lc = ob.n_lc - 1, start = ob.lc_start[lc], npts = ob.lc_npts[lc];
        for (int t0 = 0; t0 < npts; t0 += P) {
            const int np = min(P, npts - t0);
            tile_rows_fp64(ob, L, s, start + t0, np, true, 0, false);
            accumulate_tile_fp64(ob, s, M, bv, np, start + t0, true, conv_sig, s.J, s.ym, rank, cs);
        }
    }
    // every CTA copies its share of the lower triangle and of bv into the
    // others, then mirrors (mrqcof.c:139-141): the same matrix, solve and
    // decisions everywhere
    if constexpr (SPLIT) {
        for (int r = 0; r < cs; r++) {
            if (r == rank) continue;
            double *rM = cgr::this_cluster().map_shared_rank(M, r), *rb = cgr::this_cluster().map_shared_rank(bv, r);
            for_share(ntri + mf, rank, cs, [&](int e) {
                if (e < ntri) {
                    const int j = tri_row(e), k = e - j * (j + 1) / 2;
                    rM[j * mf + k] = M[j * mf + k];
                } else {
                    rb[e - ntri] = bv[e - ntri];
                }
            });
        }
        cgr::this_cluster().sync();
    }
    for (int e = tid; e < mf * mf; e += NT) {
        const int j = e / mf, k = e - j * mf;
        if (k > j) M[e] = M[k * mf + j];
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// chi^2 alone at parameters a[], FP64 form: of mrqcof.c what decides whether
// a step is accepted.  About half of an LM fit's steps are rejected, and a
// rejected step's alpha and beta are never used, so run_fit takes the trial's
// chi^2 from here and evaluates the derivatives of accepted steps only.
//
// Every value is formed by the operations of evaluate in their order: a
// point's brightness by lane l over the entries l, l + 32, ... of its lit
// list and the same butterfly, the relative lightcurves' sums and chi^2 over
// the points in data order, so chi^2, the area sum and the convexity
// residuals are evaluate's bit for bit.
//
// The points go through in chunks: set-up with a thread per point; a warp
// per pair of points (taken from a counter, lit counts differ) for the
// brightness; residuals.  No barrier inside a chunk's facet work.  The chain
// of chi^2 additions over a chunk runs on the last warp during the next
// chunk's facet work.  Buffers in the W region (unused here).  In a cluster
// every CTA computes its share of the pairs, sends the model values to the
// others and runs the sums itself.
// ---------------------------------------------------------------------------
struct Chi2Plan {
    double *rec;      // [7][cap]: Earth and Sun directions, phase function
    double *ym;       // [2][cap]: model values, then weighted squared residuals
    uint16_t *idx;    // [warps][wcols]: lit lists
    int cap;          // points
};

__device__ inline Chi2Plan chi2_plan(const SlotLayout &L, const Smem<PS_FORM_FP64> &s)
{
    constexpr int NW = threads_of<PS_FORM_FP64>() / 32;
    Chi2Plan c;
    const int lists = (NW * L.wcols * 2 + 15) & ~15;
    c.cap = (static_cast<int>(L.J - L.W) - lists) / (9 * static_cast<int>(sizeof(double)));
    c.rec = s.W;
    c.ym = s.W + static_cast<size_t>(7) * c.cap;
    c.idx = reinterpret_cast<uint16_t *>(s.W + static_cast<size_t>(9) * c.cap);
    return c;
}

// A chunk ends on a tile-independent boundary: kChi2Chunk points, but a
// relative lightcurve is never cut (its sum comes before its residuals).
constexpr int kChi2Chunk = 384;

// Whether the object's longest relative lightcurve fits in a chunk.
__device__ inline bool chi2_fits(const DevObject &ob, const SlotLayout &L, const Smem<PS_FORM_FP64> &s)
{
    const int cap = chi2_plan(L, s).cap;
    return cap >= 32 && ob.max_rel_points <= cap;
}

template <bool SPLIT>
__device__ void chi2_fp64(const DevObject &ob, const FitConfig &cfg, const SlotLayout &L, Smem<PS_FORM_FP64> &s,
                          const double *a)
{
    namespace cgr = cooperative_groups;
    constexpr int NT = threads_of<PS_FORM_FP64>(), NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int rank = 0, cs = 1;
    if constexpr (SPLIT) {
        rank = static_cast<int>(cgr::this_cluster().block_rank());
        cs = static_cast<int>(cgr::this_cluster().num_blocks());
    }
    const int F = ob.nfac, C = ob.ncoef, nreal = ob.n_lc - 1, N = ob.ndata;
    shape_prologue<PS_FORM_FP64, 1, threads_of<PS_FORM_FP64>()>(ob, s, a);
    const Chi2Plan cp = chi2_plan(L, s);
    const int cap = cp.cap, lim = min(cap, kChi2Chunk);
    const double omg = a[C + 2];
    const double *bm = s.bmat;
    const double cls = bm[30], cl = bm[31];
    int *task = reinterpret_cast<int *>(s.misc + M_PIV);
    // convexity residuals (conv.c:12-29)
    if (warp < 3) {
        const double *nc = (warp == 0) ? ob.nx : (warp == 1) ? ob.ny : ob.nz;
        double res = 0;
        for (int i = lane; i < F; i += 32) res = res + s.area[i] * nc[i];
        res = warp_sum(res);
        if (lane == 0) s.misc[M_CHK + warp] = res;
    }
    // chi^2 over the points [q0, q0 + n), their weighted squares in t, added in data order
    double c2 = 0;   // the last warp's lane 0
    auto chain = [&](const double *t, int q0, int n) {
#pragma unroll 8
        for (int i = 0; i < n; i++) c2 = c2 + t[i] * ob.weight[q0 + i];
    };
    int lc0 = 0, q0 = 0, buf = 0, prev_q = 0, prev_n = 0;
    while (q0 < N) {
        // the chunk [q0, q1): whole relative lightcurves, at most lim points
        // (one longer relative lightcurve alone)
        int lc1 = lc0, q1 = q0;
        while (lc1 < nreal) {
            const int end = ob.lc_start[lc1] + ob.lc_npts[lc1];
            if (end - q0 <= lim) {
                q1 = end;
                lc1++;
            } else {
                if (!ob.lc_rel[lc1]) {
                    q1 = q0 + lim;
                } else if (q1 == q0) {
                    q1 = end;
                    lc1++;
                }
                break;
            }
        }
        const int n = q1 - q0, npair = (n + 1) / 2;
        double *ym = cp.ym + static_cast<size_t>(buf) * cap;
        double *rec = cp.rec;
        if (tid == 0) *task = 0;
        // point set-up (bright.c:27-57): the directions and the phase
        // function; of a cluster's points, the CTA's pairs
        const int mine = ((npair - rank + cs - 1) / cs) * 2;
        for (int k = tid; k < mine; k += NT) {
            const int i = ((k >> 1) * cs + rank) * 2 + (k & 1);
            if (i >= n) continue;
            double e[6];
            const double sc = setup_point_light(ob, cfg, q0 + i, omg, bm, e);
#pragma unroll
            for (int c = 0; c < 6; c++) rec[c * cap + i] = e[c];
            rec[6 * cap + i] = sc;
        }
        // A cluster's CTAs store into each other's ym below.  Buffer buf was
        // last read two chunks ago, before the cluster barrier of the chunk in
        // between; in a call's first chunk it may be the one that the call
        // before ended on, which a CTA reads (residuals, the last chain) after
        // that call's last cluster barrier: one more barrier here.
        bool first = false;
        if constexpr (SPLIT) {
            first = q0 == 0;
            if (first) cgr::this_cluster().sync();
        }
        if (!first) __syncthreads();
        if (warp == NW - 1 && lane == 0) chain(cp.ym + static_cast<size_t>(buf ^ 1) * cap, prev_q, prev_n);
        // brightness, a warp per pair of points
        int lit = 0;
        for (;;) {
            int k = 0;
            if (lane == 0) k = atomicAdd(task, 1);
            k = __shfl_sync(0xffffffffu, k, 0) * cs + rank;
            if (k >= npair) break;
            double br[2] = {0.0, 0.0};
            uint16_t *idx = cp.idx + warp * L.wcols;
#pragma unroll 1
            for (int u = 0; u < 2; u++) {
                const int i = 2 * k + u;
                if (i >= n) break;
                const double e1 = rec[i], e2 = rec[cap + i], e3 = rec[2 * cap + i];
                const double f1 = rec[3 * cap + i], f2 = rec[4 * cap + i], f3 = rec[5 * cap + i];
                const int nl = list_lit_fp64(ob, e1, e2, e3, f1, f2, f3, idx);
                lit += nl;
                double b = 0;
#pragma unroll 2
                for (int j = lane; j < nl; j += 32) {
                    const int fi = idx[j];
                    const double nx = ob.nx[fi], ny = ob.ny[fi], nz = ob.nz[fi];
                    const double mu = e1 * nx + e2 * ny + e3 * nz;
                    const double mu0 = f1 * nx + f2 * ny + f3 * nz;
                    const LitTerms<double, PS_FORM_FP64> lt(mu, mu0, cl, cls);
                    b = b + s.area[fi] * lt.sv;
                }
                if (u == 0) br[0] = b;
                else br[1] = b;
                __syncwarp();
            }
            // both sums by one butterfly: lanes 0..15 end with the first
            int id;
            double v = fold_pair(br[0], br[1], 0, 1, 16, lane, id);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            const int i = 2 * k + id;
            if ((lane & 15) == 0 && i < n) {
                const double y = v * rec[6 * cap + i];
                ym[i] = y;
                if constexpr (SPLIT)
                    for (int r = 0; r < cs; r++)
                        if (r != rank) *cgr::this_cluster().map_shared_rank(ym + i, r) = y;
            }
        }
        if (lane == 0) atomicAdd(lit_counter(s.misc), static_cast<unsigned long long>(lit));
        if constexpr (SPLIT) cgr::this_cluster().sync();
        else __syncthreads();
        // residuals (mrqcof.c:90-136): a warp per relative lightcurve, then
        // the absolute lightcurves' points
        for (int lc = lc0 + warp; lc < lc1; lc += NW) {
            if (!ob.lc_rel[lc]) continue;
            const int start = ob.lc_start[lc], npts = ob.lc_npts[lc];
            double *y = ym + (start - q0);
            double ave = 0;
            if (lane == 0)
                for (int p = 0; p < npts; p++) ave = ave + y[p];
            ave = __shfl_sync(0xffffffffu, ave, 0);
            for (int p = lane; p < npts; p += 32) {
                const int q = start + p;
                const double coef = ob.sig[q] * npts / ave;
                const double yr = __dmul_rn(coef, y[p]);
                const double dy = ob.bright[q] - yr;
                y[p] = dy * dy * ob.sig2i[q];
            }
        }
        for (int lc = lc0; lc < nreal && ob.lc_start[lc] < q1; lc++) {
            if (ob.lc_rel[lc]) continue;
            const int lo = max(ob.lc_start[lc], q0), hi = min(ob.lc_start[lc] + ob.lc_npts[lc], q1);
            for (int q = lo + tid; q < hi; q += NT) {
                const double dy = ob.bright[q] - ym[q - q0];
                ym[q - q0] = dy * dy * ob.sig2i[q];
            }
        }
        prev_q = q0;
        prev_n = n;
        q0 = q1;
        lc0 = lc1;
        buf ^= 1;
        __syncthreads();
    }
    if (warp == NW - 1 && lane == 0) {
        chain(cp.ym + static_cast<size_t>(buf ^ 1) * cap, prev_q, prev_n);
        // the convexity rows
        const double sig2i = 1 / (cfg.conv_sig * cfg.conv_sig);
        for (int p = 0; p < 3; p++) {
            const double dy = 0.0 - s.misc[M_CHK + p];
            c2 = c2 + dy * dy * sig2i * ob.weight[N + p];
        }
        s.misc[M_CHISQ] = c2;
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// chi^2 alone at parameters a[], tensor-core paths of the mixed form (the
// counterpart of chi2_fp64: what decides whether a step is accepted).  No
// contraction, no derivative sums, and so no operand tile and no per-tile
// barriers: set-up with a thread per point, brightness with a warp per 16
// points, residuals with a warp per 32-point tile, one thread's ordered sum.
// Each value by evaluate's operations in their order (a point's brightness:
// facet_stage_tc's four lanes and four facet quarters; chi^2: tile sums in
// tile order), so chi^2 is evaluate's bit for bit.
// Buffers in the operand region, eight floats a point: at least kChi2Points, so
// that any relative lightcurve fits (one that did not would never be passed).
// Measured: 3010 fits of 980 points, 288 facets 290 -> 219 ms; 1010 fits with
// 81 coefficients, 512 facets 247 -> 171 ms.
// ---------------------------------------------------------------------------
constexpr int kChi2Bytes = 128 * 65 * sizeof(float);   // of the operand region, at least (make_layout)
constexpr int kChi2Points = kChi2Bytes / 32 & ~31;
static_assert(kChi2Points >= PS_POINTS_MAX, "a relative lightcurve is summed in one chunk");

template <int KU, int NT>
__device__ void chi2_mixed(const DevObject &ob, const FitConfig &cfg, const SlotLayout &L, Smem<PS_FORM_MIXED> &s,
                           const double *a)
{
    constexpr int NW = NT / 32, P = 32;
    constexpr int kTiles = 16 * kRedStride;   // two tile sums each in s.red
    const int tid = team_thread<NT>(), lane = tid & 31, warp = tid >> 5;
    const int F = ob.nfac, C = ob.ncoef, nreal = ob.n_lc - 1, N = ob.ndata;
    shape_prologue<PS_FORM_MIXED, KU, NT>(ob, s, a);
    const int cap = max(static_cast<int>(2 * (L.blo - L.bhi)), kChi2Bytes) / 32 & ~31;
    float *rec = reinterpret_cast<float *>(s.bhi);   // [7][cap] directions, phase function
    float *ym = rec + 7 * cap;                       // [cap] model values
    double *tsum = s.red, *c2sum = s.red + kTiles;
    const double omg = a[C + 2];
    const float cls = s.bmat[30], cl = s.bmat[31];
    const int cq = tc_kpad(F) >> 5;   // 8-facet groups per facet quarter
    int lc0 = 0, q0 = 0;
    while (q0 < N) {
        // the chunk [q0, q1): whole relative lightcurves, absolute ones cut
        // at a tile, at most cap points and kTiles tiles
        int lc1 = lc0, q1 = q0, tiles = 0;
        while (lc1 < nreal) {
            const int st = max(ob.lc_start[lc1], q0), end = ob.lc_start[lc1] + ob.lc_npts[lc1];
            const int nt = (end - st + P - 1) / P;
            if (end - q0 <= cap && tiles + nt <= kTiles) {
                q1 = end;
                tiles += nt;
                lc1++;
                continue;
            }
            if (!ob.lc_rel[lc1]) {
                const int take = min((cap - (st - q0)) / P, kTiles - tiles);
                q1 = st + take * P;
                tiles += take;
            }
            break;
        }
        const int n = q1 - q0;
        for (int i = tid; i < n; i += NT) {
            float pt[32];
            const float4 g0 = ob.geo_f[2 * (q0 + i)], g1 = ob.geo_f[2 * (q0 + i) + 1];
            setup_mixed_phase(ob.tim[q0 + i], omg, cfg.phi0, pt);
            setup_mixed_geo(g0, g1, s.bmat, pt, 0);
            float e[6];
            rotate_directions(pt, e);
#pragma unroll
            for (int c = 0; c < 6; c++) rec[c * cap + i] = e[c];
            rec[6 * cap + i] = pt[24];
        }
        team_sync<NT>();
        const float2 CL = make_float2(cl, cl), CLS = make_float2(cls, cls);
        const int fl = lane & 3;
        // a lane takes two points (one facet load for both: with one point the
        // pass waits for shared memory) and two quarters at a time, four
        // independent chains (3010 fits 168 -> 161 ms)
        for (int g = warp; g * 16 < n; g += NW) {
            float2 E1[2], E2[2], E3[2], F1[2], F2[2], F3[2];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int i = g * 16 + 8 * k + (lane >> 2);
                float e[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                if (i < n) {
#pragma unroll
                    for (int c = 0; c < 6; c++) e[c] = rec[c * cap + i];
                }
                E1[k] = make_float2(e[0], e[0]);
                E2[k] = make_float2(e[1], e[1]);
                E3[k] = make_float2(e[2], e[2]);
                F1[k] = make_float2(e[3], e[3]);
                F2[k] = make_float2(e[4], e[4]);
                F3[k] = make_float2(e[5], e[5]);
            }
            float t[2] = {0.f, 0.f};
#pragma unroll 1
            for (int h0 = 0; h0 < 4; h0 += 2) {
                float2 br[2][2];
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int k = 0; k < 2; k++) br[h][k] = make_float2(0.f, 0.f);
#pragma unroll 1
                for (int kc = 0; kc < cq; kc++) {
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const float4 *fp = s.fac + ((h0 + h) * cq + kc) * 8 + 2 * fl;
                        const float4 fa = fp[0], fb = fp[1];
#pragma unroll
                        for (int k = 0; k < 2; k++) {
                            const LitPair lp(fa, fb, E1[k], E2[k], E3[k], F1[k], F2[k], F3[k]);
                            // the product rounded by itself, as in
                            // facet_stage_tc (which uses it twice): a paired
                            // product is fused into the paired addition,
                            // scalar ones are not
                            const float2 sv = lp.law(CL, CLS);
                            br[h][k] = __fadd2_rn(br[h][k],
                                                  make_float2(__fmul_rn(lp.ax.x, sv.x), __fmul_rn(lp.ax.y, sv.y)));
                        }
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        float v = br[h][k].x + br[h][k].y;
                        v += __shfl_xor_sync(0xffffffffu, v, 1);
                        v += __shfl_xor_sync(0xffffffffu, v, 2);
                        t[k] += v;
                    }
            }
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const int i = g * 16 + 8 * k + (lane >> 2);
                if (fl == 0 && i < n) ym[i] = t[k] * rec[6 * cap + i];
            }
        }
        team_sync<NT>();
        // sums of the relative lightcurves' model values, a tile per warp
        int k = 0;
        for (int lc = lc0; lc < nreal && ob.lc_start[lc] < q1; lc++) {
            const int lo = max(ob.lc_start[lc], q0), hi = min(ob.lc_start[lc] + ob.lc_npts[lc], q1);
            for (int u = lo; u < hi; u += P, k++) {
                if (k % NW != warp || !ob.lc_rel[lc]) continue;
                const double y = warp_sum(u + lane < hi ? static_cast<double>(ym[u + lane - q0]) : 0.0);
                if (lane == 0) tsum[k] = y;
            }
        }
        team_sync<NT>();
        // weighted squared residuals (mrqcof.c:90-136); the sums of a
        // relative lightcurve's tiles are read before they are replaced
        k = 0;
        for (int lc = lc0; lc < nreal && ob.lc_start[lc] < q1; lc++) {
            const int lo = max(ob.lc_start[lc], q0), hi = min(ob.lc_start[lc] + ob.lc_npts[lc], q1);
            const bool rel = ob.lc_rel[lc] != 0;
            const int npts = ob.lc_npts[lc], k0 = k;
            for (int u = lo; u < hi; u += P, k++) {
                if (k % NW != warp) continue;
                double c2 = 0, inv_ave = 0;
                if (rel) {
                    double ave = 0;
                    for (int w = 0; w * P < npts; w++) ave += tsum[k0 + w];
                    inv_ave = 1.0 / ave;
                }
                if (u + lane < hi) {
                    const int q = u + lane;
                    const double yt = static_cast<double>(ym[q - q0]);
                    const double sig2i = ob.sig2i[q], wg = ob.weight[q];
                    double dy;
                    if (rel) {
                        const double coef = ob.sig[q] * npts * inv_ave;
                        // (the wide path stores the renormalised value, the
                        // other one contracts the product into the difference)
                        dy = KU == 3 ? ob.bright[q] - __dmul_rn(coef, yt) : fma(-coef, yt, ob.bright[q]);
                    } else {
                        dy = ob.bright[q] - yt;
                    }
                    c2 = dy * dy * sig2i * wg;
                }
                c2 = warp_sum(c2);
                if (lane == 0) c2sum[k] = c2;
            }
        }
        team_sync<NT>();
        if (tid == 0) {
            double c = s.misc[M_CHISQ];
#pragma unroll 4
            for (int w = 0; w < tiles; w++) c += c2sum[w];
            s.misc[M_CHISQ] = c;
        }
        q0 = q1;
        lc0 = lc1;
        // (the next chunk's set-up writes rec only; its first barrier comes
        // before anything that replaces the sums)
    }
    // convexity rows (conv.c:12-29)
    if (warp >= 1 && warp < 4) {
        const double *nc = (warp == 1) ? ob.nx : (warp == 2) ? ob.ny : ob.nz;
        double res = 0;
        for (int i = lane; i < F; i += 32) res = res + s.area[i] * nc[i];
        res = warp_sum(res);
        if (lane == 0) s.misc[M_CHK + warp - 1] = res;
    }
    team_sync<NT>();
    if (warp == 0) {
        double c2 = 0;
        if (lane < 3) {
            const double sig2i = 1 / (cfg.conv_sig * cfg.conv_sig);
            const double dy = 0.0 - s.misc[M_CHK + lane];
            c2 = dy * dy * sig2i * ob.weight[N + lane];
        }
        c2 = warp_sum(c2);
        if (lane == 0) s.misc[M_CHISQ] += c2;
    }
    team_sync<NT>();
}

// Gauss-Jordan elimination with full pivoting on A (n x n, row-major in
// shared memory) and right-hand side b (gauss_errc.c:9-73).  Only the
// solution is needed by the LM step, so the columns that already hold the
// inverse are not updated and the final column unscrambling is skipped; the
// pivot choices and the solution are those of the full algorithm.
// Returns 0, 1 (no usable pivot: NaN entries) or 2 (zero pivot).
//
// Bound by its serial steps, so a step is two barriers: warps 0 and 1 take
// the pivot's reciprocal and scale the pivot row while the others copy the
// pivot column; then one pass over the columns not yet pivoted (their list:
// every lane busy, half the FP64 instructions of a pass over all) updates the
// rows, swaps the pivot row into place and finds the next pivot.
// The pivot is the largest |a| over unpivoted rows and columns; ties go to
// the last element in row-major order (the reference's >=).  The bits of |a|
// order as its values do (NaN patterns, above +inf's, skipped as v >= 0 skips
// them), so the search compares 64-bit integers, off the FP64 unit.
// wd: gj_doubles(n) doubles and then gj_ints(n) ints of workspace.
// Measured (n = 55, 980 points): ten fits on 4-CTA clusters 68.8 -> 62.8 ms, 400
// fits on one CTA each 548 -> 523 ms.
template <int NT>
__device__ int gauss_jordan(double *A, double *b, int n, double *wd)
{
    int *wi = reinterpret_cast<int *>(wd + gj_doubles(n));
    constexpr int NW = NT / 32;
    constexpr long long kInfBits = 0x7ff0000000000000LL;
    const int tid = team_thread<NT>(), lane = tid & 31, warp = tid >> 5;
    double *prow = wd, *pcol = wd + n;   // scaled pivot row, pivot column; pcol[n]: the scaled pivot row of b
    int *col[2] = {wi, wi + n};          // columns not yet pivoted, in increasing order
    int *flag = wi + 2 * n;              // 1: row and column not yet pivoted
    int *candi = wi + 3 * n;             // candidates of the warps
    long long *candv = reinterpret_cast<long long *>(wd + 2 * n + 1);
    for (int k = tid; k < n; k += NT) {
        col[0][k] = k;
        flag[k] = 1;
    }
    long long bv = -1;
    int bi = -1;
    auto offer = [&](double a, int e) {
        const long long v = __double_as_longlong(a) & 0x7fffffffffffffffLL;
        if (v <= kInfBits && (v > bv || (v == bv && e > bi))) {
            bv = v;
            bi = e;
        }
    };
    for (int e = tid; e < n * n; e += NT) offer(A[e], e);
    for (int step = 0; step < n; step++) {
        const int m = n - step;           // columns not yet pivoted
        const int *cl = col[step & 1];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const long long ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > bv || (ov == bv && oi > bi)) {
                bv = ov;
                bi = oi;
            }
        }
        if (lane == 0) {
            candv[warp] = bv;
            candi[warp] = bi;
        }
        team_sync<NT>();
        // every warp takes the best candidate by itself
        bv = lane < NW ? candv[lane] : -1;
        bi = lane < NW ? candi[lane] : -1;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            const long long ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > bv || (ov == bv && oi > bi)) {
                bv = ov;
                bi = oi;
            }
        }
        const int idx = __shfl_sync(0xffffffffu, bi, 0);
        if (idx < 0) return 1;
        const int irow = idx / n, icol = idx - irow * n;
        // (its bits: a comparison of doubles by every warp holds the FP64 units)
        if (__shfl_sync(0xffffffffu, bv, 0) == 0) return 2;
        // the list without icol (the m - 1 columns still to be pivoted)
        int *cn = col[(step + 1) & 1];
        if (warp < 2) {
            const double pivinv = 1.0 / A[irow * n + icol];
            for (int c = tid; c <= m; c += 64) {
                if (c < m) {
                    const int l = cl[c];
                    if (l != icol) {
                        prow[l] = A[irow * n + l] * pivinv;
                        cn[c - (l > icol ? 1 : 0)] = l;
                    }
                } else {
                    pcol[n] = b[irow] * pivinv;
                }
            }
        } else {
            // the column as the swap of rows irow and icol leaves it
            for (int r = tid - 64; r < n; r += NT - 64) pcol[r] = A[(r == irow ? icol : r) * n + icol];
            if (tid == 64) flag[icol] = 0;
        }
        team_sync<NT>();
        bv = -1;
        bi = -1;
        const int m1 = m - 1;
        const float inv_m1 = m1 > 0 ? 1.0f / static_cast<float>(m1) : 0.f;
        for (int e = tid; e < n * m1; e += NT) {
            // row e / m1 (from FP32, corrected), column number e % m1
            int r = static_cast<int>(static_cast<float>(e) * inv_m1);
            int c = e - r * m1;
            if (c < 0) {
                r--;
                c += m1;
            } else if (c >= m1) {
                r++;
                c -= m1;
            }
            if (r == icol) {
                // the pivot row, unless the thread of row irow swaps it in
                if (irow == icol) A[icol * n + cn[c]] = prow[cn[c]];
                continue;
            }
            const int l = cn[c];
            double v = A[(r == irow ? icol : r) * n + l];
            const double pr = prow[l];
            if (r == irow) A[icol * n + l] = pr;
            v -= pr * pcol[r];
            A[r * n + l] = v;
            if (flag[r]) offer(v, r * n + l);
        }
        // the right-hand side likewise, on the last warps
        const double pb = pcol[n];
        for (int r = NT - 1 - tid; r < n; r += NT) {
            if (r == icol) {
                if (irow == icol) b[icol] = pb;
                continue;
            }
            const double v = b[r == irow ? icol : r];
            if (r == irow) b[icol] = pb;
            b[r] = v - pb * pcol[r];
        }
    }
    team_sync<NT>();
    return 0;
}

// Cholesky factorisation A = L L^T of the damped normal matrix (symmetric
// positive definite; lower triangle used, overwritten by L) and the solve of
// L L^T x = b, in FP64.  The forward substitution runs inside the
// factorisation (b is the bordering column: y_j = b_j / L_jj, then b_i -=
// L_ij y_j with the trailing update).
//
// Columns are taken two at a time, with one pair of look-ahead.  Every FP64
// instruction holds its sub-partition's FP64 unit for the whole warp, so the
// serial chain of a pivot and the bulk of the trailing update run on
// different sub-partitions at the same time.  While pair j is applied to
// the columns beyond pair j + 2 (the workers: warps of sub-partitions 1..3
// but warp 1), warp 0 applies it to the 2 x 2 block of pair j + 2 and to
// its two rows of b and factors the block, and warp 1 applies it to the
// rest of pair j + 2's columns and scales them once warp 0 has published
// the pivot (a named barrier of the two warps) -- one CTA barrier per pair.
// The 2 x 2 pivot takes its two reciprocal square roots (of the leading
// element and of the block's determinant) in one lane-parallel sequence.
// The back substitution runs on warp 0 with b in registers and the rows of
// L pre-scaled by their reciprocal diagonal.  Returns 2 when a pivot is not
// positive (an integer flag: a comparison of doubles by every warp holds the
// FP64 units for 256 cycles a step; two of them in turn, see pivot_flag).  Bound by a pair's chain of dependent FP64
// operations.  Measured (n = 55): the factorisation 74 -> 64 kcycles with the
// flag, the selected loads and the pivot's factors formed by the helper itself.
__device__ inline void chol_pivot_pair(double *A, double *b, int n, int j, double *col, int *flag, int lane)
{
    const bool two = j + 1 < n;
    const double a = A[j * n + j];
    const double bq = two ? A[(j + 1) * n + j] : 0.0;
    const double c = two ? A[(j + 1) * n + j + 1] : 1.0;
    // lane 0: the leading element, lane 1: the determinant a c - bq^2
    // (L11 = sqrt(det / a), so 1 / L11 = a rsqrt(a) rsqrt(det))
    const double x = lane == 1 ? fma(a, c, -(bq * bq)) : a;
    const bool okx = x > 0.0;
    const double r = okx ? rsqrt(x) : 0.0;
    const unsigned okm = __ballot_sync(0xffffffffu, okx);
    const double i0 = __shfl_sync(0xffffffffu, r, 0);
    const double rd = __shfl_sync(0xffffffffu, r, 1);
    // lane 1: l10 = bq / L00, lane 2: y0 = b_j / L00, lane 3: 1 / L11
    const double u = lane == 1 ? bq : lane == 2 ? b[j] : a;
    double v = u * i0;
    if (lane == 3) v *= rd;
    const double l10 = __shfl_sync(0xffffffffu, v, 1);
    const double y0 = __shfl_sync(0xffffffffu, v, 2);
    const double i1 = __shfl_sync(0xffffffffu, v, 3);
    const bool ok = (okm & 1u) && (!two || (okm & 2u));
    if (lane == 0) {
        *flag = ok ? 1 : 0;
        col[j] = i0;
        b[j] = y0;
        if (two) {
            col[j + 1] = i1;
            b[j + 1] = (b[j + 1] - l10 * y0) * i1;
        }
    }
    if (two && lane == 1) A[(j + 1) * n + j] = l10;
    for (int i = j + (two ? 2 : 1) + lane; i < n; i += 32) {
        const double a0 = A[i * n + j] * i0;
        A[i * n + j] = a0;
        if (two) A[i * n + j + 1] = (A[i * n + j + 1] - a0 * l10) * i1;
    }
}

// Named barrier of warps 0 and 1 of a team in the Cholesky solve.
template <int NT>
__device__ inline int helper_barrier()
{
    return NT == kTeamThreads ? 4 + static_cast<int>(threadIdx.x) / kTeamThreads : 1;
}

// The 2 x 2 block [a bq; bq c] of pair (j, j + 1) and its rows bj, bj1 of
// b, already updated, in registers of every lane of warp 0: publishes the two
// reciprocal square roots and arrives on the helper warp's named barrier (the
// helper forms the pivot's factors itself, two dependent operations sooner, and
// scales the columns below), then stores 1/L_jj, 1/L_j+1,j+1 (col), L_j+1,j and
// y (b).
template <int NT>
__device__ inline void chol_pivot_block(double a, double bq, double c, double bj, double bj1, double *A, double *b,
                                        int n, int j, bool two, double *col, double *pub, int *flag, int lane)
{
    const double x = lane == 1 ? fma(a, c, -(bq * bq)) : a;
    const bool okx = x > 0.0;
    if (lane >= 2 && lane < 4) pub[lane] = lane == 2 ? a : bq;
    const double r = okx ? rsqrt(x) : 0.0;
    if (lane < 2) pub[lane] = r;
    // the helper warp may scale the columns now
    asm volatile("bar.arrive %0, 64;" ::"r"(helper_barrier<NT>()) : "memory");
    const unsigned okm = __ballot_sync(0xffffffffu, okx);
    const double i0 = __shfl_sync(0xffffffffu, r, 0);
    const double rd = __shfl_sync(0xffffffffu, r, 1);
    const double u = lane == 1 ? bq : lane == 2 ? bj : a;
    double v = u * i0;
    if (lane == 3) v *= rd;
    const double l10 = __shfl_sync(0xffffffffu, v, 1);
    const double y0 = __shfl_sync(0xffffffffu, v, 2);
    const double i1 = __shfl_sync(0xffffffffu, v, 3);
    const bool ok = (okm & 1u) && (!two || (okm & 2u));
    if (lane == 0) {
        *flag = ok ? 1 : 0;
        col[j] = i0;
        b[j] = y0;
        if (two) {
            col[j + 1] = i1;
            A[(j + 1) * n + j] = l10;
        }
    }
    if (lane == 0 && two) b[j + 1] = (bj1 - l10 * y0) * i1;
}

// The flag of the pair (j, j + 1), one of two: warp 0 stores the next pair's
// while the other warps may still have this pair's to read; the barrier that
// ends the next pair's step comes before this one's place is stored again.
__device__ inline int *pivot_flag(int *flags, int j) { return flags + ((j >> 1) & 1); }

// flags: two ints (pivot_flag).
template <int NT>
__device__ int cholesky_solve(double *A, double *b, int n, double *col, int *flags)
{
    static_assert(NT % 128 == 0 && NT >= 256, "whole warps on every sub-partition");
    const int tid = team_thread<NT>(), lane = tid & 31, warp = tid >> 5;
    // trailing-update workers: the warps of sub-partitions 1..3 but warp 1
    constexpr int kWorkers = (NT / 128 * 3 - 1) * 32;
    const bool worker = (warp & 3) != 0 && warp != 1;
    double *pub = col + n;   // published for the helper: both reciprocal square roots, a, bq
    const int wtid = ((warp >> 2) * 3 + (warp & 3) - 2) * 32 + lane;
    team_sync<NT>();
    if (warp == 0) chol_pivot_pair(A, b, n, 0, col, pivot_flag(flags, 0), lane);
    team_sync<NT>();
    if (*pivot_flag(flags, 0) == 0) return 2;
    for (int j = 0; j + 2 < n; j += 2) {
        // pair (j, j + 1) is factored; b[j], b[j + 1] hold its y
        const bool two = j + 1 < n;
        const int jn = j + 2;
        const bool twon = jn + 1 < n;
        // pair j's L in rows jn, jn + 1 and its y
        const double p0 = A[jn * n + j], p1 = two ? A[jn * n + j + 1] : 0.0;
        const double q0 = twon ? A[(jn + 1) * n + j] : 0.0, q1 = (twon && two) ? A[(jn + 1) * n + j + 1] : 0.0;
        if (warp == 0) {
            // the next pair's 2 x 2 block and rows of b, one value per lane
            // (lane 0: a, 1: bq, 2: c, 3: b_jn, 4: b_jn+1), then its pivot
            // (selected, not branched on)
            const double y0 = b[j], y1 = two ? b[j + 1] : 0.0;
            const bool second = lane == 1 || lane == 2 || lane == 4;   // a value of row jn + 1
            const bool isb = lane == 3 || lane == 4;
            const int row = jn + (twon && second ? 1 : 0);
            const double *at = isb ? b + row : A + row * n + jn + (lane == 2 && twon ? 1 : 0);
            double xv = lane < 5 ? *at : 0.0;
            if (second && !twon) xv = lane == 2 ? 1.0 : 0.0;
            const double u1 = second ? q0 : p0, u2 = second ? q1 : p1;
            const double v1 = isb ? y0 : lane == 2 ? q0 : p0, v2 = isb ? y1 : lane == 2 ? q1 : p1;
            const double xu = xv - u1 * v1 - u2 * v2;
            const double a = __shfl_sync(0xffffffffu, xu, 0);
            const double bq = __shfl_sync(0xffffffffu, xu, 1);
            const double cc = __shfl_sync(0xffffffffu, xu, 2);
            const double bj = __shfl_sync(0xffffffffu, xu, 3);
            const double bj1 = __shfl_sync(0xffffffffu, xu, 4);
            chol_pivot_block<NT>(a, bq, cc, bj, bj1, A, b, n, jn, twon, col, pub, pivot_flag(flags, jn), lane);
        } else if (warp == 1) {
            // the rest of the next pair's columns: update now, scale once
            // warp 0 has published the pivot
            const int i = jn + 2 + lane, i2 = i + 32;
            double c0 = 0, c1 = 0, d0 = 0, d1 = 0;
            if (i < n) {
                const double li0 = A[i * n + j], li1 = two ? A[i * n + j + 1] : 0.0;
                c0 = A[i * n + jn] - li0 * p0 - li1 * p1;
                if (twon) c1 = A[i * n + jn + 1] - li0 * q0 - li1 * q1;
            }
            if (i2 < n) {
                const double li0 = A[i2 * n + j], li1 = two ? A[i2 * n + j + 1] : 0.0;
                d0 = A[i2 * n + jn] - li0 * p0 - li1 * p1;
                if (twon) d1 = A[i2 * n + jn + 1] - li0 * q0 - li1 * q1;
            }
            asm volatile("bar.sync %0, 64;" ::"r"(helper_barrier<NT>()) : "memory");
            // L_jn+1,jn and 1/L_jn+1,jn+1 as warp 0 forms them
            const double i0 = pub[0];
            const double i1 = twon ? pub[2] * i0 * pub[1] : 0.0, l10 = twon ? pub[3] * i0 : 0.0;
            if (i < n) {
                const double a0 = c0 * i0;
                A[i * n + jn] = a0;
                if (twon) A[i * n + jn + 1] = (c1 - a0 * l10) * i1;
            }
            if (i2 < n) {
                const double a0 = d0 * i0;
                A[i2 * n + jn] = a0;
                if (twon) A[i2 * n + jn + 1] = (d1 - a0 * l10) * i1;
            }
            for (int r = i2 + 32; r < n; r += 32) {   // n > 66: the remaining rows, unpipelined
                const double li0 = A[r * n + j], li1 = two ? A[r * n + j + 1] : 0.0;
                const double e0 = A[r * n + jn] - li0 * p0 - li1 * p1;
                const double a0 = e0 * i0;
                A[r * n + jn] = a0;
                if (twon) A[r * n + jn + 1] = (A[r * n + jn + 1] - li0 * q0 - li1 * q1 - a0 * l10) * i1;
            }
        } else if (worker) {
            // apply pair j to the columns beyond the next pair
            const int j2 = j + 4;
            if (j2 < n) {
                const int m = n - j2;
                const int ntri = m * (m + 1) / 2;
                const double y0 = b[j], y1 = two ? b[j + 1] : 0.0;
                for (int e = wtid; e < ntri + m; e += kWorkers) {
                    if (e < ntri) {
                        const int r = tri_row(e);
                        const int cc = e - r * (r + 1) / 2;
                        const int i = j2 + r, k = j2 + cc;
                        double v = A[i * n + k] - A[i * n + j] * A[k * n + j];
                        if (two) v -= A[i * n + j + 1] * A[k * n + j + 1];
                        A[i * n + k] = v;
                    } else {
                        const int i = j2 + (e - ntri);
                        double v = b[i] - A[i * n + j] * y0;
                        if (two) v -= A[i * n + j + 1] * y1;
                        b[i] = v;
                    }
                }
            }
        }
        team_sync<NT>();
        if (*pivot_flag(flags, jn) == 0) return 2;
    }
    // L^T x = y: with the rows of L scaled, L'_jk = L_jk / L_jj (k < j),
    // x = col .* z where z_j = y_j - sum_{i > j} L'_ij z_i
    const int nstrict = n * (n - 1) / 2;
    for (int e = tid; e < nstrict; e += NT) {
        const int r = tri_row(e) + 1;
        const int cc = e - r * (r - 1) / 2;
        A[r * n + cc] *= col[r];
    }
    team_sync<NT>();
    if (warp == 0) {
        if (n <= 96) {
            double z0 = lane < n ? b[lane] : 0.0, z1 = lane + 32 < n ? b[lane + 32] : 0.0,
                   z2 = lane + 64 < n ? b[lane + 64] : 0.0;
            for (int jj = n - 1; jj >= 1; jj--) {
                const int slot = jj >> 5;
                const double own = slot == 0 ? z0 : slot == 1 ? z1 : z2;
                const double zj = __shfl_sync(0xffffffffu, own, jj & 31);
                const double *row = A + jj * n;
                if (lane < jj) z0 -= row[lane] * zj;
                if (lane + 32 < jj) z1 -= row[lane + 32] * zj;
                if (lane + 64 < jj) z2 -= row[lane + 64] * zj;
            }
            if (lane < n) b[lane] = z0 * col[lane];
            if (lane + 32 < n) b[lane + 32] = z1 * col[lane + 32];
            if (lane + 64 < n) b[lane + 64] = z2 * col[lane + 64];
        } else {
            for (int jj = n - 1; jj >= 1; jj--) {
                const double zj = b[jj];
                for (int i = lane; i < jj; i += 32) b[i] -= A[jj * n + i] * zj;
                __syncwarp();
            }
            for (int i = lane; i < n; i += 32) b[i] *= col[i];
        }
    }
    team_sync<NT>();
    return 0;
}

// Learned stop predictor, evaluated by warp 0: standardised features f[10]
// -> 64 GELU -> 64 GELU -> 1, output de-standardised.  Predicts
// log(final rms / rms after kScreenIters iterations).  sh: 64 floats.
__device__ inline float gelu(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }

__device__ float mlp_predict_warp(const float *W, const float *f, float *sh)
{
    const int lane = threadIdx.x & 31;
    float x[kFeat];
#pragma unroll
    for (int i = 0; i < kFeat; i++) x[i] = (f[i] - W[kMlpMu + i]) / W[kMlpSd + i];
    float h1[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int u = lane + 32 * h;
        float z = W[kMlpB1 + u];
#pragma unroll
        for (int i = 0; i < kFeat; i++) z = fmaf(W[kMlpW1 + u * kFeat + i], x[i], z);
        h1[h] = gelu(z);
    }
    sh[lane] = h1[0];
    sh[lane + 32] = h1[1];
    __syncwarp();
    float y = 0.f;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int u = lane + 32 * h;
        float z = W[kMlpB2 + u];
        for (int j = 0; j < kHidden; j++) z = fmaf(W[kMlpW2 + u * kHidden + j], sh[j], z);
        y = fmaf(W[kMlpW3 + u], gelu(z), y);
    }
    y = warp_sum(y) + W[kMlpB3];
    __syncwarp();
    return y * W[kMlpYSd] + W[kMlpYMu];
}

// ---------------------------------------------------------------------------
// One fit (period_search_BOINC.cpp:817-921 with mrqmin.c:11-110).
// ---------------------------------------------------------------------------
// SPLIT: by the CTAs of a cluster (FP64 form).  Inlined, so that the launch's
// structs stay kernel parameters: a call passes them by address, through local
// memory of 1.5 KB a thread, for which the runtime takes 140 MB of device
// memory at the first launch.
template <int FORM, int KU, int NT = threads_of<FORM>(), bool SPLIT = false>
__device__ __forceinline__ void run_fit(const DevObject &ob, const FitConfig &cfg, const SlotLayout &L, Smem<FORM> &s,
                                        typename RealOf<FORM>::T *scratch, int64_t n, int pole, ps_fit *out,
                                        const FitWork &w, long long fidx, TcState &tcs)
{
    constexpr bool kTensor = FORM == PS_FORM_MIXED && (KU == 0 || KU == 3);
    // one model evaluation; fresh = false: chi2 has just run at the same
    // parameters
    auto eval = [&](const double *a, double *M, double *bv, bool fresh) {
        if constexpr (FORM == PS_FORM_FP64) {
            evaluate_fp64<SPLIT>(ob, cfg, L, s, a, M, bv, scratch, fresh);
        } else {
            evaluate_mixed<KU, NT>(ob, cfg, L, s, a, M, bv, scratch, tcs, fresh);
        }
    };
    // chi^2 alone where the form has it (about half of the steps are
    // rejected, and need no more)
    bool lazy = false;
    if constexpr (FORM == PS_FORM_FP64) lazy = chi2_fits(ob, L, s);
    else lazy = kTensor;
    auto chi2 = [&](const double *a) {
        if constexpr (FORM == PS_FORM_FP64) {
            chi2_fp64<SPLIT>(ob, cfg, L, s, a);
        } else if constexpr (kTensor) {
            chi2_mixed<KU, NT>(ob, cfg, L, s, a);
        }
    };
    const int tid = team_thread<NT>();
    const int C = ob.ncoef, ma = ob.ma, mf = ob.mfit;
    const double freq = cfg.freq_start - (n - 1) * cfg.freq_step;
    const double prd = 1 / freq;
    // learned early stop: features after K iterations (accepted chi^2 and
    // lambda every K/4 iterations); the saved state of a resumable fit
    const int K = w.screen_iters > 0 ? w.screen_iters : kScreenIters;
    const int K4 = K >> 2;
    double *st = w.state ? w.state + (w.state_slot ? w.state_slot[fidx] : fidx) * state_stride(ma) : nullptr;
    const bool resume = w.resume && st;
    for (int i = tid; i < ma; i += NT) {
        double v;
        if (resume) v = st[i];
        else if (i < C) v = ob.cg_first[i];
        else if (i == C) v = kDeg2Rad * (90 - c_beta_pole[pole - 1]);
        else if (i == C + 1) v = kDeg2Rad * c_lambda_pole[pole - 1];
        else if (i == C + 2) v = 24 * 2 * kPi / prd;
        else if (i == C + 3) v = cfg.par0;
        else if (i == C + 4) v = cfg.par1;
        else if (i == C + 5) v = cfg.par2;
        else if (i == C + 6) v = cfg.log_cl;
        else v = 1;
        s.cg[i] = v;
        s.atry[i] = v;
    }
    team_sync<NT>();

    double alamda = -1, ochisq = 0, chisq = 0, rchisq = -1;
    double iter_diff = 1e40, dev_old = 1e30, dev_new = 0;
    double chk_acc[3] = {0, 0, 0}, chk_first[3] = {0, 0, 0}, chk_trial[3] = {0, 0, 0};
    double area_first = 0, area_trial = 0, totarea = 0;
    int niter = 0, last_err = 0;
    bool stale = false;   // alpha and beta are not yet those of the accepted step
    // learned early stop: accepted chi^2 and lambda of the first iterations
    double hist[5], lam_hist[4];
    double pred_dev = 0;
    bool screened = false;
    if (resume) {
        // continue where the fit stopped: alpha and beta are those of the
        // accepted parameters, recomputed by one evaluation (the same
        // deterministic evaluation the uninterrupted fit would hold)
        alamda = st[ma];
        ochisq = st[ma + 1];
        chisq = st[ma + 2];
        rchisq = st[ma + 3];
        iter_diff = st[ma + 4];
        dev_old = st[ma + 5];
        dev_new = st[ma + 6];
        for (int c = 0; c < 3; c++) chk_acc[c] = st[ma + 7 + c];
        totarea = st[ma + 10];
        niter = static_cast<int>(st[ma + 11]);
        last_err = static_cast<int>(st[ma + 12]);
        pred_dev = st[ma + 13];
        eval(s.cg, s.alpha, s.beta, true);
        if constexpr (kTensor) {
            if (*s.abort) last_err = kErrTcTimeout;
        }
    }
    while (last_err != kErrTcTimeout &&
           (((niter < cfg.n_iter_max) && (iter_diff > cfg.iter_diff_max)) || (niter < cfg.n_iter_min))) {
        bool accepted = false;
        if (alamda < 0) {
            alamda = cfg.alamda_start;
            eval(s.cg, s.alpha, s.beta, true);
            if constexpr (kTensor) {
                if (*s.abort) {
                    last_err = kErrTcTimeout;
                    break;
                }
            }
            ochisq = s.misc[M_CHISQ];
            hist[0] = ochisq;
            area_first = s.misc[M_AREA];
            for (int c = 0; c < 3; c++) chk_first[c] = s.misc[M_CHK + c];
            totarea = area_first;
        } else if (stale) {
            // alpha and beta of the step accepted last, now that another
            // step is taken from it
            eval(s.cg, s.alpha, s.beta, false);
            if constexpr (kTensor) {
                if (*s.abort) {
                    last_err = kErrTcTimeout;
                    break;
                }
            }
            stale = false;
        }
        for (int e = tid; e < mf * mf; e += NT) {
            const int j = e / mf, k = e - j * mf;
            s.covar[e] = (j == k) ? s.alpha[e] * (1 + alamda) : s.alpha[e];
        }
        for (int j = tid; j < mf; j += NT) s.da[j] = s.beta[j];
        team_sync<NT>();
        int err;
        if constexpr (FORM == PS_FORM_FP64) {
            err = gauss_jordan<NT>(s.covar, s.da, mf, s.col);
        } else {
            // The damped normal matrix is symmetric positive definite: solve
            // it by Cholesky in FP64; if a pivot is not positive (rounding on
            // a nearly singular alpha), redo the step with Gauss-Jordan.
            err = cholesky_solve<NT>(s.covar, s.da, mf, s.col, reinterpret_cast<int *>(s.misc + M_PIV));
            if (err) {
                for (int e = tid; e < mf * mf; e += NT) {
                    const int j = e / mf, k = e - j * mf;
                    s.covar[e] = (j == k) ? s.alpha[e] * (1 + alamda) : s.alpha[e];
                }
                for (int j = tid; j < mf; j += NT) s.da[j] = s.beta[j];
                team_sync<NT>();
                err = gauss_jordan<NT>(s.covar, s.da, mf, s.col);
            }
        }
        team_sync<NT>();
        if (err == 0) {
            for (int j = tid; j < mf; j += NT) {
                const int l = ob.free_list[j];
                s.atry[l] = s.cg[l] + s.da[j];
            }
            team_sync<NT>();
            if (lazy) chi2(s.atry);
            else eval(s.atry, s.covar, s.da, true);
            if constexpr (kTensor) {
                if (*s.abort) {
                    last_err = kErrTcTimeout;
                    break;
                }
            }
            chisq = s.misc[M_CHISQ];
            area_trial = s.misc[M_AREA];
            for (int c = 0; c < 3; c++) chk_trial[c] = s.misc[M_CHK + c];
            totarea = area_trial;
            if (chisq < ochisq) {
                accepted = true;
                stale = lazy;
                if (!lazy) {
                    for (int e = tid; e < mf * mf; e += NT) s.alpha[e] = s.covar[e];
                    for (int j = tid; j < mf; j += NT) s.beta[j] = s.da[j];
                }
                for (int l = tid; l < ma; l += NT) s.cg[l] = s.atry[l];
            } else {
                chisq = ochisq;
            }
        } else {
            last_err = err;
        }
        niter++;
        // The scalar bookkeeping of the step (mrqmin.c:91-107 and
        // period_search_BOINC.cpp:873-892) runs on thread 0 and is broadcast:
        // an FP64 instruction holds the FP64 unit for the whole warp, so
        // every warp computing it would cost 16 times the FP64 time.
        if (tid == 0) {
            if (err == 0) alamda = accepted ? alamda / cfg.alamda_incr : cfg.alamda_incr * alamda;
            if ((niter == 1) || accepted) {
                ochisq = chisq;
                // curv(cg) of the driver: the accepted shape is the trial one;
                // otherwise (first iteration, rejected or failed solve) cg is
                // still the starting vector of the first evaluation.
                const double *src = accepted ? chk_trial : chk_first;
                for (int c = 0; c < 3; c++) chk_acc[c] = src[c];
                totarea = accepted ? area_trial : area_first;
                rchisq = chisq - (chk_acc[0] * chk_acc[0] + chk_acc[1] * chk_acc[1] + chk_acc[2] * chk_acc[2]) *
                                     (cfg.conw_r * cfg.conw_r);
            }
            dev_new = sqrt(rchisq / ob.ndata);
            if (dev_old - dev_new > 1e-10) {
                iter_diff = dev_old - dev_new;
                dev_old = dev_new;
            }
            s.misc[M_LM] = alamda;
            s.misc[M_LM + 1] = ochisq;
            s.misc[M_LM + 2] = dev_new;
            s.misc[M_LM + 3] = iter_diff;
        }
        team_sync<NT>();
        alamda = s.misc[M_LM];
        ochisq = s.misc[M_LM + 1];
        dev_new = s.misc[M_LM + 2];
        iter_diff = s.misc[M_LM + 3];
        if (!resume && niter <= K && niter % K4 == 0) {
            hist[niter / K4] = ochisq;
            lam_hist[niter / K4 - 1] = alamda;
        }
        // trajectory records: the rms after 8, 16 and 32 iterations as well
        if (w.traj && tid == 0 && (niter == 8 || niter == 16 || niter == 32))
            w.traj[static_cast<size_t>(fidx) * kTrajFloats + (niter == 8 ? 13 : niter == 16 ? 14 : 15)] =
                static_cast<float>(dev_new);
        if (!resume && niter == K && (w.traj || w.mlp)) {
            // features and prediction on warp 0 only (FP64 logarithms)
            if (tid < 32) {
                float f[kFeat];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    f[i] = static_cast<float>(log(hist[i + 1] / hist[0]));
                    f[4 + i] = static_cast<float>(log10(lam_hist[i]));
                }
                f[8] = static_cast<float>(log(static_cast<double>(ob.ndata)));
                f[9] = static_cast<float>(log(prd));
                if (w.traj && tid == 0) {
                    float *rec = w.traj + static_cast<size_t>(fidx) * kTrajFloats;
                    for (int i = 0; i < kFeat; i++) rec[i] = f[i];
                    rec[10] = static_cast<float>(dev_new);
                }
                if (w.mlp && w.iter_limit == K) {
                    const float y = mlp_predict_warp(w.mlp, f, reinterpret_cast<float *>(s.pt));
                    if (tid == 0) pred_dev = dev_new * exp(static_cast<double>(y));
                }
            }
            team_sync<NT>();
        }
        if (w.iter_limit > 0 && niter >= w.iter_limit) {
            screened = true;
            if (st) {
                // save the state for a later resume (thread 0 holds the
                // prediction; every thread holds the broadcast scalars)
                for (int i = tid; i < ma; i += NT) st[i] = s.cg[i];
                if (tid == 0) {
                    st[ma] = alamda;
                    st[ma + 1] = ochisq;
                    st[ma + 2] = chisq;
                    st[ma + 3] = rchisq;
                    st[ma + 4] = iter_diff;
                    st[ma + 5] = dev_old;
                    st[ma + 6] = dev_new;
                    for (int c = 0; c < 3; c++) st[ma + 7 + c] = chk_acc[c];
                    st[ma + 10] = totarea;
                    st[ma + 11] = niter;
                    st[ma + 12] = last_err;
                    st[ma + 13] = pred_dev;
                }
            }
            break;
        }
    }
    if (w.traj && tid == 0) {
        float *rec = w.traj + static_cast<size_t>(fidx) * kTrajFloats;
        rec[11] = static_cast<float>(dev_new);
        rec[12] = static_cast<float>(niter);
    }
    if (tid == 0) {
        ps_fit r;
        r.dev = dev_new;
        r.dark = sqrt(chk_acc[0] * chk_acc[0] + chk_acc[1] * chk_acc[1] + chk_acc[2] * chk_acc[2]);
        r.totarea = totarea;
        r.period_h = 24 * (2 * kPi / s.cg[C + 2]);
        r.lambda_deg = kRad2Deg * s.cg[C + 1];
        r.beta_deg = 90 - kRad2Deg * s.cg[C];
        r.chisq = chisq;
        r.niter = niter;
        r.err_code = last_err;
        r.pred_dev = pred_dev;
        r.screened = screened ? 1 : 0;
        r.reserved = 0;
        if (out) *out = r;
    }
    team_sync<NT>();
}

template <int FORM, int KU>
__global__ void __launch_bounds__(threads_of<FORM>(), 1)
    fit_kernel(DevObject ob, FitConfig cfg, FitWork w, int P, int dsph_smem)
{
    using R = typename RealOf<FORM>::T;
    constexpr int NT = threads_of<FORM>();
    extern __shared__ __align__(16) char smem[];
    const SlotLayout L = make_layout(FORM, ob.ma, ob.mfit, ob.nfac, ob.ncoef, P, dsph_smem, w.rel_rows);
    Smem<FORM> s = carve<FORM>(smem, L);
    constexpr bool kTensor = FORM == PS_FORM_MIXED && (KU == 0 || KU == 3);
    if (s.dsph)
        for (int e = threadIdx.x; e < ob.nfac * ob.ncoef; e += NT) s.dsph[e] = ob.dsph_f[e];
    TcState tcs;
    if constexpr (kTensor) tc_setup<NT, KU == 3>(ob, s, s, tcs);
    // the wide tensor-core path keeps the slot's normal matrix in global memory
    if (L.dsph_smem == kBasisTensorWide) s.alpha = w.alpha_g + static_cast<size_t>(blockIdx.x) * w.alpha_stride;
    R *scratch = L.rels ? reinterpret_cast<R *>(smem + L.rels)
                        : reinterpret_cast<R *>(w.scratch + static_cast<size_t>(blockIdx.x) * w.scratch_stride);
    if (FORM == PS_FORM_FP64 && threadIdx.x == 0) *lit_counter(s.misc) = 0;
    __shared__ long long next;
    for (;;) {
        if (threadIdx.x == 0) next = static_cast<long long>(atomicAdd(w.queue, 1ULL));
        __syncthreads();
        const long long f = next;
        __syncthreads();
        if (f >= w.nfits) break;
        if constexpr (kTensor) {
            if (*s.abort) break;
        }
        int64_t n;
        int pole;
        if (w.period_index) {
            n = w.period_index[f];
            pole = w.pole[f];
        } else {
            n = w.n_lo + f / PS_N_POLES;
            pole = static_cast<int>(f % PS_N_POLES) + 1;
        }
        run_fit<FORM, KU>(ob, cfg, L, s, scratch, n, pole, w.out + f, w, f, tcs);
    }
    if constexpr (kTensor) tc_teardown<NT>(s, tcs, ob.nfac, ob.mfit);
    if (FORM == PS_FORM_FP64 && threadIdx.x == 0 && w.lit) atomicAdd(w.lit, *lit_counter(s.misc));
}

// Two fits of the mixed form's tensor-core path side by side on one SM: the
// CTA's two teams of kTeamThreads threads each run fits from the queue, with
// their own slot of shared memory, barriers and accumulators; the basis in
// Tensor Memory is common.  One fit alone leaves the SM idle two cycles of
// three (barriers, FP64 and MMA latency); two teams fill each other's gaps.
// A team's kept normal matrix lies in global memory and alpha's operands over
// the contraction's, so that two slots fit the shared memory.  A fit's
// results do not depend on which kernel runs it.
// Measured (980 points, 288 facets): 304 fits 22.8 ms as two launches of one per
// SM, 18.2 ms here; 3010 fits 217 -> 171 ms; 1510 fits of 817 relative points
// 126 -> 94 ms.  Issue slots 33 -> 45 % busy; what is left is FP64 and
// shared-memory latency and the barriers (stalls per issue: wait 2.3, barrier
// 1.6, short scoreboard 1.5).
__global__ void __launch_bounds__(threads_of<PS_FORM_MIXED>(), 1)
    fit_kernel_pair(DevObject ob, FitConfig cfg, FitWork w)
{
    constexpr int NT = kTeamThreads, kTeams = kPairFits;
    extern __shared__ __align__(16) char smem[];
    const SlotLayout L =
        make_layout(PS_FORM_MIXED, ob.ma, ob.mfit, ob.nfac, ob.ncoef, 32, kBasisTensor, w.rel_rows, true);
    const int team = threadIdx.x / NT, slot = blockIdx.x * kTeams + team;
    Smem<PS_FORM_MIXED> s0 = carve<PS_FORM_MIXED>(smem, L), s = carve<PS_FORM_MIXED>(smem + team * L.bytes, L);
    TcState tcs;
    tc_setup<NT>(ob, s0, s, tcs);
    s.alpha = w.alpha_g + static_cast<size_t>(slot) * w.alpha_stride;
    float *scratch = L.rels ? reinterpret_cast<float *>(smem + team * L.bytes + L.rels)
                            : reinterpret_cast<float *>(w.scratch + static_cast<size_t>(slot) * w.scratch_stride);
    __shared__ long long next[kTeams];
    for (;;) {
        if (team_thread<NT>() == 0) next[team] = static_cast<long long>(atomicAdd(w.queue, 1ULL));
        team_sync<NT>();
        const long long f = next[team];
        team_sync<NT>();
        if (f >= w.nfits || *s.abort) break;
        const int64_t n = w.period_index ? w.period_index[f] : w.n_lo + f / PS_N_POLES;
        const int pole = w.period_index ? w.pole[f] : static_cast<int>(f % PS_N_POLES) + 1;
        run_fit<PS_FORM_MIXED, 0, NT>(ob, cfg, L, s, scratch, n, pole, w.out + f, w, f, tcs);
    }
    tc_teardown<NT>(s, tcs, ob.nfac, ob.mfit);
}

// FP64 fits, each spread over a thread-block cluster (evaluate_fp64): the
// cluster's leader takes fits from the work counter and hands every fit to
// all of the cluster's CTAs, which run the same LM loop together; the
// leader writes the result.  Bit-identical to fit_kernel<FP64>.
__global__ void __launch_bounds__(threads_of<PS_FORM_FP64>(), 1)
    fit_kernel_split(DevObject ob, FitConfig cfg, FitWork w, int P)
{
    namespace cgr = cooperative_groups;
    cgr::cluster_group cl = cgr::this_cluster();
    const int rank = static_cast<int>(cl.block_rank()), cs = static_cast<int>(cl.num_blocks());
    extern __shared__ __align__(16) char smem[];
    const SlotLayout L = make_layout(PS_FORM_FP64, ob.ma, ob.mfit, ob.nfac, ob.ncoef, P, 0, w.rel_rows);
    Smem<PS_FORM_FP64> s = carve<PS_FORM_FP64>(smem, L);
    TcState tcs;
    double *scratch = L.rels ? reinterpret_cast<double *>(smem + L.rels)
                             : w.scratch + static_cast<size_t>(blockIdx.x) * w.scratch_stride;
    if (threadIdx.x == 0) *lit_counter(s.misc) = 0;
    __shared__ long long next;
    cl.sync();   // every CTA of the cluster runs: its shared memory may be written
    for (;;) {
        if (rank == 0 && threadIdx.x == 0) {
            const long long f = static_cast<long long>(atomicAdd(w.queue, 1ULL));
            for (int r = 0; r < cs; r++) *cl.map_shared_rank(&next, r) = f;
        }
        cl.sync();
        const long long f = next;
        cl.sync();
        if (f >= w.nfits) break;
        int64_t n;
        int pole;
        if (w.period_index) {
            n = w.period_index[f];
            pole = w.pole[f];
        } else {
            n = w.n_lo + f / PS_N_POLES;
            pole = static_cast<int>(f % PS_N_POLES) + 1;
        }
        run_fit<PS_FORM_FP64, 1, threads_of<PS_FORM_FP64>(), true>(ob, cfg, L, s, scratch, n, pole,
                                                                   rank == 0 ? w.out + f : nullptr, w, f, tcs);
    }
    if (threadIdx.x == 0 && w.lit) atomicAdd(w.lit, *lit_counter(s.misc));
}

// One FP64 evaluation spread over one thread-block cluster, bit-identical to
// eval_kernel<FP64>'s.
__global__ void __launch_bounds__(threads_of<PS_FORM_FP64>(), 1)
    eval_kernel_split(DevObject ob, FitConfig cfg, const double *cg, double *alpha, double *beta, double *chisq,
                      double *area, double *scratch, size_t scratch_stride, int P, int rel_rows)
{
    constexpr int NT = threads_of<PS_FORM_FP64>();
    extern __shared__ __align__(16) char smem[];
    const SlotLayout L = make_layout(PS_FORM_FP64, ob.ma, ob.mfit, ob.nfac, ob.ncoef, P, 0, rel_rows);
    Smem<PS_FORM_FP64> s = carve<PS_FORM_FP64>(smem, L);
    for (int i = threadIdx.x; i < ob.ma; i += NT) s.cg[i] = cg[i];
    if (threadIdx.x == 0) *lit_counter(s.misc) = 0;
    __syncthreads();
    double *rows = L.rels ? reinterpret_cast<double *>(smem + L.rels)
                          : scratch + static_cast<size_t>(blockIdx.x) * scratch_stride;
    evaluate_fp64<true>(ob, cfg, L, s, s.cg, s.alpha, s.beta, rows, true);
    if (blockIdx.x != 0) return;   // the last remote accesses lie before evaluate_fp64's last cluster barrier
    const int mf = ob.mfit;
    for (int e = threadIdx.x; e < mf * mf; e += NT) alpha[e] = s.alpha[e];
    for (int j = threadIdx.x; j < mf; j += NT) beta[j] = s.beta[j];
    if (area)
        for (int i = threadIdx.x; i < ob.nfac; i += NT) area[i] = s.area[i];
    if (threadIdx.x == 0) *chisq = s.misc[M_CHISQ];
}

template <int FORM, int KU>
__global__ void __launch_bounds__(threads_of<FORM>(), 1) eval_kernel(DevObject ob, FitConfig cfg, const double *cg, double *alpha,
                                                        double *beta, double *chisq, double *area, double *scratch,
                                                        int P, int dsph_smem, int rel_rows)
{
    using R = typename RealOf<FORM>::T;
    constexpr int NT = threads_of<FORM>();
    extern __shared__ __align__(16) char smem[];
    const SlotLayout L = make_layout(FORM, ob.ma, ob.mfit, ob.nfac, ob.ncoef, P, dsph_smem, rel_rows);
    Smem<FORM> s = carve<FORM>(smem, L);
    constexpr bool kTensor = FORM == PS_FORM_MIXED && (KU == 0 || KU == 3);
    if (s.dsph)
        for (int e = threadIdx.x; e < ob.nfac * ob.ncoef; e += NT) s.dsph[e] = ob.dsph_f[e];
    TcState tcs;
    if constexpr (kTensor) tc_setup<NT, KU == 3>(ob, s, s, tcs);
    for (int i = threadIdx.x; i < ob.ma; i += NT) s.cg[i] = cg[i];
    if (FORM == PS_FORM_FP64 && threadIdx.x == 0) *lit_counter(s.misc) = 0;
    // the wide tensor-core path accumulates straight into the output matrix
    if (L.dsph_smem == kBasisTensorWide) s.alpha = alpha;
    __syncthreads();
    R *rows = L.rels ? reinterpret_cast<R *>(smem + L.rels) : reinterpret_cast<R *>(scratch);
    if constexpr (FORM == PS_FORM_FP64) evaluate_fp64<false>(ob, cfg, L, s, s.cg, s.alpha, s.beta, rows, true);
    else evaluate_mixed<KU, NT>(ob, cfg, L, s, s.cg, s.alpha, s.beta, rows, tcs);
    if constexpr (kTensor) {
        const bool aborted = *s.abort != 0;
        tc_teardown<NT>(s, tcs, ob.nfac, ob.mfit);
        if (aborted) {
            if (threadIdx.x == 0) *chisq = NAN;
            return;
        }
    }
    const int mf = ob.mfit;
    if (L.dsph_smem != kBasisTensorWide)
        for (int e = threadIdx.x; e < mf * mf; e += NT) alpha[e] = s.alpha[e];
    for (int j = threadIdx.x; j < mf; j += NT) beta[j] = s.beta[j];
    if (area)
        for (int i = threadIdx.x; i < ob.nfac; i += NT) area[i] = s.area[i];
    if (threadIdx.x == 0) *chisq = s.misc[M_CHISQ];
}

}  // namespace
}  // namespace psg
