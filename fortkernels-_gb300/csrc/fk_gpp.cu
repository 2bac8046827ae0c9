// fk_gpp.cu -- GPP self-energy sum on sm_103a.
//
// Reference: the n1 x my_igp x ig x iw loop nest of BGW-Kernels/gppKer.cpp:
// 303-439 (ssxt_scht_solver :19-65, flagOCC_solver :130-159, noflag block
// :349-413, accumulation :416-439).
//
// Structure.  Every factor of a GPP term except the band pair product
//     conj(aqsmtemp[n1][igp]) * aqsntemp[n1][ig]
// depends only on (my_igp, ig, iw).  The kernels therefore
//   1. build, once per (my_igp, ig), the three branch-resolved factors
//      D[my_igp*3+iw][ig] = mask(wdiffr > limittwo && delwr < limitone)
//                           * delw * I_eps                     (prep kernel),
//      and contract the flagOCC bands (n1 < nvband: sch and ssx) right there;
//   2. contract the noflag bands as a complex GEMM, aqsntemp x D^T, whose
//      epilogue applies 0.5*vcoul[igp]*conj(aqsmtemp[n1][igp]) and reduces
//      each row to its three iw sums (fk_gemm.cuh);
//   3. add all partials in a fixed order (finalize kernels).
// FP64 path: each branch is taken exactly as in the reference's C++: an element near
// a threshold follows the reference's expression sequence with round-to-nearest FP64
// operations (no contraction), as every element of the half and real-valued sums does;
// clear of the thresholds the full sum's prep decides in FP32 and forms its values with
// FMAs and a reciprocal refined to FP64 (prep64_kernel).  The contraction runs on
// the tensor cores by digit products (fk_tc64.cuh), or on FP64 DMMA where
// there is no room for their images or the digits are too coarse.  Mixed path: the branch quantities are evaluated in FP32 from an
// FP64 wdiff and re-evaluated with the exact FP64 sequence whenever a test
// value lies within a relative guard band of its threshold, so branch
// decisions remain those of the FP64 sequence; the bulk products run in FP32
// with compensated accumulation.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <new>

#include "fk_branch.h"
#include "fk_gemm.cuh"
#include "fk_internal.h"
#include "fk_tc64.cuh"
#include "fk_tc_contract.cuh"

namespace fk {
namespace {

constexpr int PREP_THREADS = 256;
constexpr int PREP_TILE = 2 * PREP_THREADS;  // plane waves per chunk of the FP64 half-sum and real preps
constexpr int NVC = 2;  // flag bands contracted per prep pass
constexpr double TO1 = 1e-6;
constexpr float GUARD = 1e-5f;  // relative guard band of the FP32 branch tests
constexpr int GPP_COLS = 21;    // igp columns per 64-wide tensor-core n-tile (63 used)
// error estimate of the mixed path: C of C * 2^-24 * sqrt(sum |term|^2), set
// above the largest ratio |mixed - FP64| / (2^-24 * bound) measured over the
// GPU tests' inputs with a margin (est_* kernels)
constexpr double GPP_EST_C = 64.0;

struct PrepArgs {
    int nb, nv, nc, ng;
    const double2 *aqsn, *eps, *wt;
    const double* wx;
    const int* igp;
    void* D;     // FP64: [3*ng][nc] double2; mixed: pre-split B image (fk_tc_contract.cuh); nullptr = not needed
    int kstages; // mixed: k-stages per n-tile in the image
    double2* F;  // [nch][nv][ng][3][2]  (sch, ssx) flag-band sums over the chunk
    int nch;
    int tile;    // plane waves per chunk (mixed: a multiple of the 32-wide k-stage)
    int n1base;  // first flag band handled by this pass
    int ch0;     // first chunk of this launch (blockIdx.x counts from it)
    // half-sum mode (FK_GPP_HALF_SUM)
    const double2* aqsm;  // full [nb][nc] (half sum); the weights' source (set-up, below)
    const int* brk;       // [ng][HALF_CHUNKS]: first ig whose |Omega2| < 1e-6 in each chunk (half_brk: the flag bands stop there)
    // Set-up folded into the first pass (setup != 0): the column map is computed
    // from inv/indinv rather than read from igp, and the first chunk of each
    // column writes igp/acol, the epilogue weights W (mixed) and, in the last
    // column of a tensor-core tile, the image's padding rows; block (0, 0)
    // clears the reduction's completion counter and the error word.
    int setup;
    const int *inv, *indinv;
    int* igp_out;
    int* acol_out;
    int compact;          // aqsm holds column my_igp at position my_igp (stride ldm)
    long ldm;
    const double* vcoul;
    float2* W;            // [ng][M] 0.5*vcoul*conj(aqsm[nv+m][igp]) in FP32, or nullptr
    int M;
    int* counter;
    double2* wf;          // [nv][ng][2] flag-band weights (sch: 0.5*vcoul*conj(aqsm), ssx: occ*vcoul*conj(aqsm)), or nullptr
    int asx_neg;          // physics mode: the ssx weight is -occ*vcoul*conj(aqsm) (asxtemp subtracted)
    float* est;           // error estimate (EST prep): [nch][ng][3][6] magnitudes of the chunk's values
    int wm0 = -1;         // first band of the weight table W (-1: nvband)
    int* err = nullptr;   // the contraction's error word, cleared by block (0, 0), or nullptr
};

// The set-up work of block (ch, my_igp) other than the image padding.
FK_DEV int prep_setup(const PrepArgs& p, int ch, int my_igp) {
    if (!p.setup) return p.igp[my_igp];
    const int igp = gpp_igp_of(my_igp, p.nc, p.inv, p.indinv);
    if (ch == 0) {
        const int acol = igp < 0 ? -1 : (p.compact ? my_igp : igp);
        if (threadIdx.x == 0) {
            p.igp_out[my_igp] = igp;
            p.acol_out[my_igp] = acol;
            if (my_igp == 0 && p.counter) *p.counter = 0;
            if (my_igp == 0 && p.err) *p.err = 0;
        }
        if (p.wf)
            for (int n1 = threadIdx.x; n1 < p.nv; n1 += blockDim.x) {
                double2 a = make_double2(0.0, 0.0), b = a;
                if (igp >= 0) {
                    const double2 cm = cconj(p.aqsm[(long)n1 * p.ldm + acol]);
                    // asxtemp += ssx*occ*vcoul (BGW-Kernels/gppKer.cpp:419); the Fortran
                    // subtracts it (gppkernel.deslippe.09.30.2014.f90:393)
                    const double occ = p.asx_neg ? -1.0 : 1.0;
                    a = cscale(cm, 0.5 * p.vcoul[igp]);
                    b = cscale(cm, occ * p.vcoul[igp]);
                }
                p.wf[((long)n1 * p.ng + my_igp) * 2 + 0] = a;
                p.wf[((long)n1 * p.ng + my_igp) * 2 + 1] = b;
            }
    }
    if (p.W) {
        // the column's epilogue weights, rows split evenly over its chunks
        const int acol = igp < 0 ? -1 : (p.compact ? my_igp : igp);
        const int m0 = (int)((long)p.M * ch / p.nch), m1 = (int)((long)p.M * (ch + 1) / p.nch);
        const int w0 = p.wm0 < 0 ? p.nv : p.wm0;
        for (int m = m0 + threadIdx.x; m < m1; m += blockDim.x)
            p.W[(long)my_igp * p.M + m] =
                igp >= 0 ? tcx::weight_w1(p.aqsm[(long)(w0 + m) * p.ldm + acol], 0.5 * p.vcoul[igp])
                         : make_float2(0.f, 0.f);
    }
    return igp;
}

// ---------------------------------------------------------------- FP64 exact
struct Branch64 {
    double2 delw;
    bool A, B;
};
// ssxt_scht_solver's branch quantities, BGW-Kernels/gppKer.cpp:30-38.
FK_DEV Branch64 branch64(double wxt, double2 wt) {
    const double limitone = 1.0 / (TO1 * 4.0);
    const double limittwo = 0.5 * 0.5;
    double2 wdiff = make_double2(__dsub_rn(wxt, wt.x), -wt.y);
    double rden = __ddiv_rn(1.0, cnorm2(wdiff));
    Branch64 b;
    b.delw = cscale(cmul(wt, cconj(wdiff)), rden);
    double delwr = cnorm2(b.delw);
    double wdiffr = cnorm2(wdiff);
    b.A = (wdiffr > limittwo) && (delwr < limitone);
    b.B = delwr > TO1;
    return b;
}
// ssx of ssxt_scht_solver, BGW-Kernels/gppKer.cpp:38-58.  phys: the Fortran
// branch A, cden = wxt**2 - wtilde2 (gppkernel.deslippe.09.30.2014.f90:302-305).
FK_DEV double2 ssx64(const Branch64& b, double wxt, double2 wt2, double2 Omega2, bool phys = false) {
    if (b.A && phys) {
        const double2 cd = make_double2(__dsub_rn(__dmul_rn(wxt, wxt), wt2.x), __dsub_rn(0.0, wt2.y));
        const double rd = __ddiv_rn(1.0, cnorm2(cd));
        return cscale(cmul(Omega2, cconj(cd)), rd);
    }
    if (b.A) {
        double w2 = __dmul_rn(wxt, wxt);
        double rd = __ddiv_rn(1.0, __dmul_rn(w2, w2));
        double2 t = make_double2(__dsub_rn(__dmul_rn(Omega2.x, w2), __dmul_rn(Omega2.y, -0.0)),
                                 __dadd_rn(__dmul_rn(Omega2.x, -0.0), __dmul_rn(Omega2.y, w2)));
        return cscale(t, rd);
    }
    if (b.B) {
        double2 c = cmul(cscale(wt2, 4.0), make_double2(__dadd_rn(b.delw.x, 0.5), b.delw.y));
        double rd = __ddiv_rn(1.0, cnorm2(c));
        double2 negO = make_double2(-Omega2.x, -Omega2.y);
        return cmul(cscale(cmul(negO, cconj(c)), rd), b.delw);
    }
    return make_double2(0.0, 0.0);
}
// The Fortran sexcut test (gppkernel.deslippe.09.30.2014.f90:319-320): ssx is
// dropped when wxt < 0 and |ssx| > sexcut*|I_eps| (the C++ test, abs(wxt) < 0 at
// BGW-Kernels/gppKer.cpp:60-61, never fires).
FK_DEV double2 sexcut64(double2 ssx, double wxt, double2 ep) {
    return (wxt < 0.0 && hypot(ssx.x, ssx.y) > 4.0 * hypot(ep.x, ep.y)) ? make_double2(0.0, 0.0) : ssx;
}

// Fixed-order block sum of NV values per thread; thread v < NV of the block
// receives the total of value v.  Deterministic: shuffle tree, then warps in order.
template <int NV>
FK_DEV void block_sum(double2 (&v)[NV], double2* sm /* [8][NV] */) {
#pragma unroll
    for (int i = 0; i < NV; ++i)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            v[i].x += __shfl_down_sync(0xffffffffu, v[i].x, off);
            v[i].y += __shfl_down_sync(0xffffffffu, v[i].y, off);
        }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
#pragma unroll
        for (int i = 0; i < NV; ++i) sm[warp * NV + i] = v[i];
    __syncthreads();
    if (threadIdx.x < NV) {
        double2 s = make_double2(0.0, 0.0);
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s = cadd(s, sm[w * NV + threadIdx.x]);
        v[threadIdx.x] = s;
    }
}

// Fixed-order block sum of FP32 values carried as float-float pairs (TwoSum
// at every level, across the warps too); thread v < NV of the block widens
// its pair to FP64 once.  FP32 instructions everywhere but that last step:
// the FP64 pipe of GB300 takes ~16 cycles per warp instruction.
template <int NV>
FK_DEV void block_sum_ff(float2 (&v)[NV], double2* sm /* [8][NV] */, double2 (&out)[NV]) {
    float2 lo[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) lo[i] = make_float2(0.f, 0.f);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const float hx = __shfl_down_sync(0xffffffffu, v[i].x, off), hy = __shfl_down_sync(0xffffffffu, v[i].y, off);
            const float lx = __shfl_down_sync(0xffffffffu, lo[i].x, off), ly = __shfl_down_sync(0xffffffffu, lo[i].y, off);
            ff32 a{v[i].x, lo[i].x + lx}, b{v[i].y, lo[i].y + ly};
            ff_add(a, hx);
            ff_add(b, hy);
            v[i] = make_float2(a.hi, b.hi);
            lo[i] = make_float2(a.lo, b.lo);
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float4* sm4 = reinterpret_cast<float4*>(sm);  // [warp][NV] (hi.x, hi.y, lo.x, lo.y)
    if (lane == 0)
#pragma unroll
        for (int i = 0; i < NV; ++i) sm4[warp * NV + i] = make_float4(v[i].x, v[i].y, lo[i].x, lo[i].y);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NV; ++i) out[i] = make_double2(0.0, 0.0);
    if (threadIdx.x < NV) {
        ff32 a{0.f, 0.f}, b{0.f, 0.f};
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            const float4 q = sm4[w * NV + threadIdx.x];
            a.lo += q.z;
            b.lo += q.w;
            ff_add(a, q.x);
            ff_add(b, q.y);
        }
        const double2 s = make_double2((double)a.hi + (double)a.lo, (double)b.hi + (double)b.lo);
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (i == (int)threadIdx.x) out[i] = s;
    }
}

// |v| >= 2^60, an infinity or NaN: squares and products of two such no longer fit FP32
FK_DEV bool large(double v) { return (((unsigned)__double2hiint(v) >> 20) & 0x7ffu) >= 1023u + 60u; }

// Sums of N <= 16 values over a block of 256 threads, in a fixed order: in each
// step a lane hands half of its values to its partner and adds the partner's
// half of the others (8 + 4 + 2 + 1 + 1 additions instead of a five-level tree
// per value), then the warps are added in order.  Thread v < N receives value v.
template <int N>
FK_DEV double block_sum_scatter(double (&v)[16], double* sm /* [8][16] */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int w = 8; w >= 1; w >>= 1) {
        const bool up = (lane & w) != 0;  // this lane keeps the upper half of its 2w values
#pragma unroll
        for (int i = 0; i < w; ++i) {
            const double give = up ? v[i] : v[i + w], keep = up ? v[i + w] : v[i];
            v[i] = __dadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, w));
        }
    }
    // lane l (of 16) holds value l; the two halves of the warp
    v[0] = __dadd_rn(v[0], __shfl_xor_sync(0xffffffffu, v[0], 16));
    if (lane < 16) sm[warp * 16 + lane] = v[0];
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x < N)
        for (int w = 0; w < PREP_THREADS / 32; ++w) s = __dadd_rn(s, sm[w * 16 + threadIdx.x]);
    return s;
}

// One (igp, ig, iw) element by the reference's FP64 sequence: the value delw*I_eps,
// sch and ssx, and the noflag mask.  Out of line: the common path keeps its registers.
struct Element64 {
    double2 dv, sch, ssx;
    int A;
};
template <int Q>
__device__ __noinline__ Element64 element64(double wxt, double2 wt, double2 ep, double2 eq, int flags) {
    const Branch64 b = branch64(wxt, wt);
    Element64 r;
    r.A = b.A;
    r.dv = cmul(b.delw, ep);
    r.sch = r.ssx = make_double2(0.0, 0.0);
    if (flags) {
        const double2 wt2 = cmul(wt, wt);
        if (b.A) r.sch = cmul(b.delw, eq);
        r.ssx = ssx64(b, wxt, wt2, cmul(wt2, ep), Q == 2);
        if (Q == 2) r.ssx = sexcut64(r.ssx, wxt, ep);
    }
    return r;
}

// FP64 prep of chunk ch (tile plane waves) of column my_igp.  Q = 0:
// BGW-Kernels/gppKer.cpp; 1: root gppKer.cpp semantics; 2: the Fortran source's
// (physics mode).  SCH = false: the flag bands' sch sums go through the contraction
// (rows from band 0), only the ssx sums are kept here.
// Bound by the FP64 pipe (64 cycles per warp instruction on each sub-partition),
// so the common path spends few FP64 instructions: the branch tests run in FP32
// on |wdiff|^2 (from its FP64 value) and |wt|^2/|wdiff|^2, any element within a
// relative 1e-5 of a threshold, out of FP32's comfortable range or with a value
// that is not finite takes the reference's sequence (element64), as do the rare branches of ssx; the
// value wt*I_eps*conj(wdiff)/|wdiff|^2 needs ten (the reciprocal: an FP32 one and
// two Newton steps, r += r(1 - n r), relative error 2^-23 -> 2^-46 -> 2^-53), and
// ssx = Omega2/wx^2 six per element and band plus two per frequency.  512 x 2 x
// 32768 x 20: 339 us with the reference's sequence for every element.
template <int Q, bool SCH>
__global__ void __launch_bounds__(PREP_THREADS, 2) prep64_kernel(PrepArgs p) {
    __shared__ double sm[8 * 16];
    const int my_igp = blockIdx.y, ch = blockIdx.x, tid = threadIdx.x;
    const int igp = prep_setup(p, ch, my_igp);
    const int nflag = min(NVC, p.nv - p.n1base);
    const bool flags = nflag > 0 && igp >= 0;
    const bool all_exact = Q != 0 && flags;
    const float limitone = 250000.0f, limittwo = 0.25f, to1 = 1e-6f;
    double2 sx[NVC * 3], sc[SCH ? NVC * 3 : 1];
#pragma unroll
    for (int i = 0; i < NVC * 3; ++i) {
        sx[i] = make_double2(0.0, 0.0);
        if (SCH) sc[i] = make_double2(0.0, 0.0);
    }
    double wx[3], iw2[3];
    bool wok[3];
#pragma unroll
    for (int iw = 0; iw < 3; ++iw) {
        wx[iw] = p.wx[iw];
        const double w2 = wx[iw] * wx[iw];
        iw2[iw] = 1.0 / w2;
        // |wdiff|^2 stays a number of FP32 (wtilde below 2^60), and (wx^2)^2, by which the sequence
        // divides, a normal number
        wok[iw] = w2 > 1e-140 && w2 < 1e36;
    }
    const double2* wrow = p.wt + (long)my_igp * p.nc;
    const double2* erow = p.eps + (long)my_igp * p.nc;
    double2* D = reinterpret_cast<double2*>(p.D);
    const int ig_end = min(p.nc, (ch + 1) * p.tile);
    auto infinite = [](double v) { return ((unsigned)__double2hiint(v) & 0x7ff00000u) == 0x7ff00000u; };  // or NaN
    for (int ig = ch * p.tile + tid; ig < ig_end; ig += PREP_THREADS) {
        const double2 wt = wrow[ig], ep = erow[ig];
        double2 eq = ep, an[NVC], pn[NVC];
        bool bad = false;  // an occupied band's value is not finite: the sequence adds it times a zero ssx, too
        if (Q == 1 && flags) eq = p.eps[(long)my_igp * p.ng + ig];  // gppKer.cpp:139
        if (flags) {
            // aqsntemp*Omega2 of the pass's bands
            const double2 w2 = make_double2(fma(wt.x, wt.x, -(wt.y * wt.y)), (wt.x + wt.x) * wt.y);
            const double2 om = make_double2(fma(w2.x, ep.x, -(w2.y * ep.y)), fma(w2.x, ep.y, w2.y * ep.x));
#pragma unroll
            for (int j = 0; j < NVC; ++j) {
                an[j] = j < nflag ? p.aqsn[(long)(p.n1base + j) * p.nc + ig] : make_double2(0.0, 0.0);
                bad = bad || infinite(an[j].x) || infinite(an[j].y);
                pn[j] = make_double2(fma(an[j].x, om.x, -(an[j].y * om.y)), fma(an[j].x, om.y, an[j].y * om.x));
            }
        }
        const bool weird = all_exact || bad || large(wt.x) || large(wt.y) || large(ep.x) || large(ep.y);
        const float2 wf = c64_to_f32(wt);
        const float wsq = wf.x * wf.x + wf.y * wf.y;
        const double y2 = wt.y * wt.y;
        const double2 a = make_double2(fma(wt.x, ep.x, -(wt.y * ep.y)), fma(wt.x, ep.y, wt.y * ep.x));
        const double cx = -(a.y * wt.y), cy = a.x * wt.y;
#pragma unroll
        for (int iw = 0; iw < 3; ++iw) {
            const double wd = __dsub_rn(wx[iw], wt.x);
            const double n = fma(wd, wd, y2);
            const float nf = f64_to_f32_bits(n), rf = __frcp_rn(nf), dr = wsq * rf;
            const bool amb = weird || !wok[iw] || !(nf > 1e-30f) || !(nf < 1e30f) || !(dr < 1e30f) ||
                             fabsf(nf - limittwo) <= limittwo * GUARD || fabsf(dr - limitone) <= limitone * GUARD ||
                             (flags && fabsf(dr - to1) <= to1 * GUARD);
            bool A = nf > limittwo && dr < limitone;
            // the sequence itself: near a threshold, or ssx of the branches but the common one
            const bool seq = amb || (flags && !A && dr > to1);
            double2 dv;
            if (seq) {
                const Element64 x = element64<Q>(wx[iw], wt, ep, eq, flags);
                A = x.A != 0;
                dv = x.dv;
                if (flags)
#pragma unroll
                    for (int j = 0; j < NVC; ++j) {
                        cfma(sx[j * 3 + iw], an[j], x.ssx);
                        if (SCH) cfma(sc[SCH ? j * 3 + iw : 0], an[j], x.sch);
                    }
            } else {
                double r = f32_to_f64_bits(rf);
                r = fma(r, fma(-n, r, 1.0), r);
                r = fma(r, fma(-n, r, 1.0), r);
                dv = make_double2(fma(a.x, wd, cx) * r, fma(a.y, wd, cy) * r);
                if (flags && A)
#pragma unroll
                    for (int j = 0; j < NVC; ++j) {
                        sx[j * 3 + iw].x = fma(pn[j].x, iw2[iw], sx[j * 3 + iw].x);
                        sx[j * 3 + iw].y = fma(pn[j].y, iw2[iw], sx[j * 3 + iw].y);
                        if (SCH) cfma(sc[SCH ? j * 3 + iw : 0], an[j], dv);
                    }
            }
            if (D) {
                const bool keep = igp >= 0 && (Q == 1 || A);
                D[((long)my_igp * 3 + iw) * p.nc + ig] = keep ? dv : make_double2(0.0, 0.0);
            }
        }
    }
    if (nflag <= 0) return;
    // F[..][iw * 2 + kind], kind 0 sch, 1 ssx
    double* F = (double*)(p.F + ((long)ch * p.nv * p.ng) * 6);
    auto put = [&](double2(&s)[NVC * 3], int kind) {
        double v[16];
#pragma unroll
        for (int i = 0; i < NVC * 3; ++i) {
            v[2 * i] = s[i].x;
            v[2 * i + 1] = s[i].y;
        }
#pragma unroll
        for (int i = NVC * 6; i < 16; ++i) v[i] = 0.0;
        const double x = block_sum_scatter<NVC * 6>(v, sm);
        const int j = tid / 6, q = tid % 6;  // band, (frequency, re or im)
        if (tid < nflag * 6)
            F[(((long)(p.n1base + j) * p.ng + my_igp) * 6 + (q >> 1) * 2 + kind) * 2 + (q & 1)] = x;
    };
    put(sx, 1);
    if constexpr (SCH) {
        __syncthreads();  // sm is reused
        put(sc, 0);
    }
}

// ------------------------------------------------------ half sum (gppsum == 1)
// gppKerSeq.cpp with gppsum == 1: for column igp the sum over ig runs below
// igp.  Every term of a band n1 >= nvband is
//   conj(aqsm[n1][igp]) aqsn[n1][ig] sch + aqsm[n1][igp] conj(aqsm[n1][ig]) conj(sch)
// with sch = mask' * (wtilde / (wx - wtilde)) * I_eps and the inverted mask
// mask' = |wdiff|^2 < limittwo || |delw|^2 > limitone (noflagOCC_solver :206-242).
// The driver's blocks (:430-447) take ig < igp-1 except ig = 511 mod 512, and
// add the diagonal ig = igp (first term only) when igp is a multiple of 512.
// The second term summed over ig is aqsm[n1][igp] conj(sum_ig aqsm[n1][ig] sch):
// the same contraction with A = aqsmtemp, conjugated.  Occupied bands follow
// flagOCC_solver (:90-139), which stops at the first ig with |Omega2| < to1.

// complex division a * conj(b) / |b|^2, round-to-nearest FP64
FK_DEV double2 cdiv_rn(double2 a, double2 b) {
    const double n = __dadd_rn(__dmul_rn(b.x, b.x), __dmul_rn(b.y, b.y));
    return make_double2(__ddiv_rn(__dadd_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)), n),
                        __ddiv_rn(__dsub_rn(__dmul_rn(a.y, b.x), __dmul_rn(a.x, b.y)), n));
}

// D'(my_igp, iw, ig) of the half sum (without the block membership test)
FK_DEV double2 half_sch(double wxt, double2 wt, double2 eps) {
    const double limitone = 1.0 / (1e-6 * 4.0), limittwo = 0.25;
    const double2 wdiff = make_double2(__dsub_rn(wxt, wt.x), 0.0 - wt.y);
    const double2 delw = cdiv_rn(wt, wdiff);
    const double delw2 = cnorm2(delw), wdiffr = cnorm2(wdiff);
    const bool on = fabs(wdiffr) < limittwo || delw2 > limitone;
    return on ? cmul(delw, eps) : make_double2(0.0, 0.0);
}

// ig takes part in column igp's noflag sum (the reference program's 512-wide blocks)
FK_DEV bool half_member(int ig, int igp) { return ig < igp - 1 && (ig & 511) != 511; }

// The first ig < igp with |wtilde^2 * I_eps| < to1 is found chunk by chunk (half_break: the
// smallest hit of one chunk of the column, or a value above every igp).  The test runs in FP32
// on |Omega2|^2 against to1^2; inside a relative guard band of 1e-5 around it (the FP32 error
// is ~1e-7) and for values out of FP32's range the FP64 test decides, so every decision is
// the FP64 one.
constexpr int HALF_CHUNKS = 64;
__device__ __noinline__ bool half_break64(double2 w, double2 ep) {
    const double2 o = cmul(cmul(w, w), ep);
    return hypot(o.x, o.y) < 1e-6;
}
// One block; every thread calls it.
FK_DEV void half_break(int nc, int igp, int chunk, const double2* wt, const double2* eps, int* out) {
    const int span = ceil_div(nc, HALF_CHUNKS), g1 = min(igp, (chunk + 1) * span);
    int first = 0x7fffffff;
    for (int ig = chunk * span + threadIdx.x; ig < g1; ig += blockDim.x) {
        const double2 w64 = wt[ig], e64 = eps[ig];
        const float2 w = c64_to_f32(w64), o = cmulf(cmulf(w, w), c64_to_f32(e64));
        const float o2 = o.x * o.x + o.y * o.y;
        bool hit = o2 < 1e-12f;
        if (large(w64.x) || large(w64.y) || large(e64.x) || large(e64.y) || !(o2 < 1e30f) || !(o2 > 1e-36f) ||
            fabsf(o2 - 1e-12f) <= 1e-12f * GUARD)
            hit = half_break64(w64, e64);
        if (hit) first = min(first, ig);
    }
    __shared__ int sm[8];
    first = __reduce_min_sync(0xffffffffu, first);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = first;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) first = min(first, sm[w]);
        *out = first;
    }
}
// The first hit of column my_igp (whole warps call it).
FK_DEV int half_brk(const int* brk, int my_igp) {
    const int* b = brk + (long)my_igp * HALF_CHUNKS;
    int v = 0x7fffffff;
    for (int i = threadIdx.x & 31; i < HALF_CHUNKS; i += 32) v = min(v, b[i]);
    return __reduce_min_sync(0xffffffffu, v);
}

// What the half and the real-valued sum need before their preps, in one launch: the
// column map, the epilogue weights W (rows nv.. of aqsmtemp), the image's padding, the
// cleared counter and error word; the half sum's break table and its diagonal values
// sch(igp) of the columns on a block edge (igp % 512 == 0, else 0); the real-valued
// sum's aqsmtemp columns as complex (value, 0), [nb][ng] (the weights' source).
// As separate launches these were four to six kernels of 3 to 5 us, with a gap of 2 to
// 3 us behind each.  512 x 32768 x 20: half sum 199 -> 175 us, real-valued 163 -> 146 us.
struct SetupArgs {
    int nb, nv, nc, ng;
    const int *inv, *indinv;
    int *igp, *acol;
    const double* vcoul;
    float2* W;                // [ng][nb - nv], or nullptr
    int *counter, *err;       // err: or nullptr
    uint8_t* img;             // the image to pad, or nullptr
    int NT, kstages, K;
    const double2* aqsm;      // half sum (complex, all columns)
    const double2 *eps, *wt;
    const double* wx;
    int* brk;
    double2* schd;
    const double* aqsm_re;    // real-valued sum
    double2* ac;
};
constexpr int SETUP_THREADS = 128;
__host__ __device__ inline int setup_row_blocks(int nb) { return (nb + SETUP_THREADS - 1) / SETUP_THREADS; }
__global__ void __launch_bounds__(SETUP_THREADS) setup_kernel(SetupArgs a) {
    const int nr = setup_row_blocks(a.nb), b = blockIdx.x, tid = threadIdx.x;
    if (b >= nr * a.ng) {
        int s = b - nr * a.ng;
        if (a.brk) {
            if (s < HALF_CHUNKS * a.ng) {
                const int h = s / HALF_CHUNKS, c = s % HALF_CHUNKS;
                half_break(a.nc, gpp_igp_of(h, a.nc, a.inv, a.indinv), c, a.wt + (long)h * a.nc, a.eps + (long)h * a.nc, a.brk + s);
                return;
            }
            s -= HALF_CHUNKS * a.ng;
        }
        tcx::img_pad_stage<64>(a.img, s / a.NT, s % a.NT, a.NT, a.kstages, a.ng, GPP_COLS, a.K);
        return;
    }
    const int h = b / nr, n = (b % nr) * SETUP_THREADS + tid;
    const int g = gpp_igp_of(h, a.nc, a.inv, a.indinv);
    if (b % nr == 0) {
        if (tid == 0) {
            a.igp[h] = g;
            a.acol[h] = g < 0 ? -1 : (a.ac ? h : g);
            if (h == 0) {
                *a.counter = 0;
                if (a.err) *a.err = 0;
            }
        }
        if (a.schd && tid < 3)
            a.schd[h * 3 + tid] = g > 0 && (g & 511) == 0
                                      ? half_sch(a.wx[tid], a.wt[(long)h * a.nc + g], a.eps[(long)h * a.nc + g])
                                      : make_double2(0.0, 0.0);
    }
    if (n >= a.nb) return;
    double2 am = make_double2(0.0, 0.0);
    if (a.ac) {
        if (g >= 0) am.x = a.aqsm_re[(long)n * a.nc + g];
        a.ac[(long)n * a.ng + h] = am;
    } else if (g >= 0) {
        am = a.aqsm[(long)n * a.nc + g];
    }
    if (a.W && n >= a.nv)
        a.W[(long)h * (a.nb - a.nv) + n - a.nv] = g >= 0 ? tcx::weight_w1(am, 0.5 * a.vcoul[g]) : make_float2(0.f, 0.f);
}
inline void launch_setup(const SetupArgs& a, cudaStream_t st) {
    const int blocks = setup_row_blocks(a.nb) * a.ng + (a.brk ? HALF_CHUNKS * a.ng : 0) + (a.img ? a.kstages * a.NT : 0);
    setup_kernel<<<blocks, SETUP_THREADS, 0, st>>>(a);
}

// The flag-band terms of one (ig, iw): sch and ssx of flagOCC_solver (gppsum == 1)
FK_DEV void half_flag_terms(double wxt, double2 wt, double2 eps, double2& sch, double2& ssx) {
    const double to1 = 1e-6, gamma = 0.5;
    const double2 wt2 = cmul(wt, wt), Omega2 = cmul(wt2, eps);
    const double2 halfinv = cdiv_rn(make_double2(0.5, 0.0), wt);
    const double2 wmw = make_double2(__dsub_rn(wxt, wt.x), 0.0 - wt.y);
    const double2 delw = cmul(wmw, halfinv);
    const double ad = hypot(delw.x, delw.y);
    if (hypot(wmw.x, wmw.y) < gamma || __dmul_rn(ad, ad) < to1) {
        sch = make_double2(0.0, 0.0);
        ssx = hypot(wt.x, wt.y) > to1
                  ? cdiv_rn(make_double2(0.0 - Omega2.x, 0.0 - Omega2.y),
                            cmul(cscale(wt2, 4.0), make_double2(__dadd_rn(1.0, delw.x), delw.y)))
                  : make_double2(0.0, 0.0);
    } else {
        sch = cdiv_rn(cmul(wt, eps), wmw);
        ssx = cdiv_rn(Omega2, make_double2(__dsub_rn(__dmul_rn(wxt, wxt), wt2.x), 0.0 - wt2.y));
    }
}

// Prep of the half sum, FP64 path: D' as FP64 rows; flag bands n1base ..
// n1base+NVC-1 accumulate, per (iw, sch/ssx), S1 = sum_ig aqsn[n1][ig] x and
// S2 = sum_ig aqsm[n1][ig] x (S2 without ig = igp-1) over ig < brk:
// F[ch][n1][my_igp][12], entry ((iw*2 + kind)*2 + part).
__global__ void __launch_bounds__(PREP_THREADS) prep_half_kernel(PrepArgs p) {
    __shared__ double2 sm[8 * NVC * 12];
    const int my_igp = blockIdx.y, ch = p.ch0 + blockIdx.x, tid = threadIdx.x;
    const int igp = p.igp[my_igp];
    const int nflag = min(NVC, p.nv - p.n1base);
    const int stop = igp < 0 ? 0 : min(igp, half_brk(p.brk, my_igp));
    double2 acc[NVC * 12];
#pragma unroll
    for (int i = 0; i < NVC * 12; ++i) acc[i] = make_double2(0.0, 0.0);
    const double2* wrow = p.wt + (long)my_igp * p.nc;
    const double2* erow = p.eps + (long)my_igp * p.nc;
    for (int ig = ch * p.tile + tid; ig < min(p.nc, (ch + 1) * p.tile); ig += PREP_THREADS) {
        const double2 wt = wrow[ig], ep = erow[ig];
#pragma unroll
        for (int iw = 0; iw < 3; ++iw) {
            const double wxt = p.wx[iw];
            if (p.D) {
                const double2 dv = (igp >= 0 && half_member(ig, igp)) ? half_sch(wxt, wt, ep) : make_double2(0.0, 0.0);
                ((double2*)p.D)[((long)my_igp * 3 + iw) * p.nc + ig] = dv;
            }
            if (nflag > 0 && ig < stop) {
                double2 sch, ssx;
                half_flag_terms(wxt, wt, ep, sch, ssx);
#pragma unroll
                for (int j = 0; j < NVC; ++j)
                    if (j < nflag) {
                        const long row = (long)(p.n1base + j) * p.nc + ig;
                        const double2 an = p.aqsn[row], am = p.aqsm[row];
                        double2* a = acc + j * 12 + iw * 4;
                        cfma(a[0], an, sch);
                        cfma(a[2], an, ssx);
                        if (ig != igp - 1) {
                            cfma(a[1], am, sch);
                            cfma(a[3], am, ssx);
                        }
                    }
            }
        }
    }
    if (nflag <= 0) return;
    block_sum<NVC * 12>(acc, sm);
    if (tid < nflag * 12) {
        const int j = tid / 12, r = tid % 12;
        p.F[(((long)ch * p.nv + p.n1base + j) * p.ng + my_igp) * 12 + r] = acc[tid];
    }
}

// Mixed-precision prep of the half sum: prep_half_kernel's outputs, D' as the pre-split image,
// with the branch quantities in FP32 from an FP64 wx - wtilde; inside a relative
// guard band of 1e-5 around a threshold (or outside FP32's comfortable range)
// the FP64 sequence decides and supplies the values, so every branch is the
// FP64 one.  Flag-band sums in FP32 float-float (block_sum_ff).
__device__ __noinline__ double2 half_sch_rare(double wxt, double2 wt, double2 eps) { return half_sch(wxt, wt, eps); }
__device__ __noinline__ void half_flag_rare(double wxt, double2 wt, double2 eps, float2& sch, float2& ssx) {
    double2 a, b;
    half_flag_terms(wxt, wt, eps, a, b);
    sch = c64_to_f32(a);
    ssx = c64_to_f32(b);
}
FK_DEV float2 cdivf(float2 a, float2 b) {
    const float r = __frcp_rn(b.x * b.x + b.y * b.y);
    return make_float2((a.x * b.x + a.y * b.y) * r, (a.y * b.x - a.x * b.y) * r);
}

__global__ void __launch_bounds__(PREP_THREADS, 2) prep_half_mixed_kernel(PrepArgs p) {
    __shared__ double2 sm[8 * NVC * 12];
    const int my_igp = blockIdx.y, ch = p.ch0 + blockIdx.x, tid = threadIdx.x;
    const int igp = p.igp[my_igp];
    const int nflag = min(NVC, p.nv - p.n1base);
    const int stop = igp < 0 ? 0 : min(igp, half_brk(p.brk, my_igp));
    const float limitone = 250000.0f, limittwo = 0.25f, to1 = 1e-6f, to1sq = 1e-12f;
    float2 acc[NVC * 12];
#pragma unroll
    for (int i = 0; i < NVC * 12; ++i) acc[i] = make_float2(0.f, 0.f);
    double wx64[3];
    float wxsq[3];
#pragma unroll
    for (int iw = 0; iw < 3; ++iw) {
        wx64[iw] = p.wx[iw];
        const float wf = f64_to_f32_bits(wx64[iw]);
        wxsq[iw] = wf * wf;
    }
    const double2* wrow = p.wt + (long)my_igp * p.nc;
    const double2* erow = p.eps + (long)my_igp * p.nc;
    for (int ig = ch * p.tile + tid; ig < min(p.nc, (ch + 1) * p.tile); ig += PREP_THREADS) {
        const double2 wt64 = wrow[ig], ep64 = erow[ig];
        const float2 wt = c64_to_f32(wt64), ep = c64_to_f32(ep64);
        const bool member = igp >= 0 && half_member(ig, igp);
        const bool flag = nflag > 0 && ig < stop;
        float2 wt2 = make_float2(0.f, 0.f), Om = wt2, hinv = wt2;
        float wtsq = 0.f;
        float2 an[NVC], am[NVC];
        if (flag) {
            wt2 = cmulf(wt, wt);
            Om = cmulf(wt2, ep);
            wtsq = wt.x * wt.x + wt.y * wt.y;
            const float r = __frcp_rn(wtsq);
            hinv = make_float2(0.5f * wt.x * r, -0.5f * wt.y * r);  // 0.5 / wtilde
#pragma unroll
            for (int j = 0; j < NVC; ++j) {
                const long row = (long)(p.n1base + j) * p.nc + ig;
                an[j] = j < nflag ? c64_to_f32(p.aqsn[row]) : make_float2(0.f, 0.f);
                am[j] = j < nflag ? c64_to_f32(p.aqsm[row]) : make_float2(0.f, 0.f);
            }
        }
#pragma unroll
        for (int iw = 0; iw < 3; ++iw) {
            const float2 wdiff = make_float2(f64_to_f32_bits(__dsub_rn(wx64[iw], wt64.x)), -wt.y);
            const float wdiffr = wdiff.x * wdiff.x + wdiff.y * wdiff.y;
            if (p.D) {
                float2 dv = make_float2(0.f, 0.f);
                if (member) {
                    const float2 delw = cdivf(wt, wdiff);
                    const float delw2 = delw.x * delw.x + delw.y * delw.y;
                    const bool amb = !(wdiffr > 1e-30f) || !(delw2 < 1e30f) ||
                                     fabsf(wdiffr - limittwo) <= limittwo * GUARD ||
                                     fabsf(delw2 - limitone) <= limitone * GUARD;
                    if (__any_sync(__activemask(), amb) && amb) dv = c64_to_f32(half_sch_rare(wx64[iw], wt64, ep64));
                    else if (wdiffr < limittwo || delw2 > limitone) dv = cmulf(delw, ep);
                }
                const int nt = my_igp / GPP_COLS, row = (my_igp % GPP_COLS) * 3 + iw;
                tcx::bimg_store<64>((uint8_t*)p.D + (long)nt * p.kstages * tcx::Cfg<64>::B_BYTES, p.kstages, row, ig,
                                    dv.x, dv.y);
            }
            if (flag) {
                // flagOCC_solver (gppsum = 1): wmw = wdiff, delw = wmw * 0.5/wtilde
                const float2 delw = cmulf(wdiff, hinv);
                const float ad2 = delw.x * delw.x + delw.y * delw.y;
                const bool amb = !(wtsq > 1e-30f) || !(wdiffr > 1e-30f) || !(ad2 < 1e30f) || !(wtsq < 1e30f) ||
                                 fabsf(wdiffr - limittwo) <= limittwo * GUARD || fabsf(ad2 - to1) <= to1 * GUARD ||
                                 fabsf(wtsq - to1sq) <= to1sq * GUARD;
                float2 sch, ssx;
                if (__any_sync(__activemask(), amb) && amb) {
                    half_flag_rare(wx64[iw], wt64, ep64, sch, ssx);
                } else if (wdiffr < limittwo || ad2 < to1) {
                    sch = make_float2(0.f, 0.f);
                    ssx = wtsq > to1sq ? cdivf(make_float2(-Om.x, -Om.y),
                                               cmulf(make_float2(4.f * wt2.x, 4.f * wt2.y),
                                                     make_float2(1.f + delw.x, delw.y)))
                                       : make_float2(0.f, 0.f);
                } else {
                    sch = cdivf(cmulf(wt, ep), wdiff);
                    ssx = cdivf(Om, make_float2(wxsq[iw] - wt2.x, -wt2.y));
                }
#pragma unroll
                for (int j = 0; j < NVC; ++j) {
                    float2* a = acc + j * 12 + iw * 4;
                    cfmaf(a[0], an[j], sch);
                    cfmaf(a[2], an[j], ssx);
                    if (ig != igp - 1) {
                        cfmaf(a[1], am[j], sch);
                        cfmaf(a[3], am[j], ssx);
                    }
                }
            }
        }
    }
    if (nflag <= 0) return;
    double2 accd[NVC * 12];
    block_sum_ff<NVC * 12>(acc, sm, accd);
    if (tid < nflag * 12) {
        const int j = tid / 12, r = tid % 12;
#pragma unroll
        for (int i = 0; i < NVC * 12; ++i)
            if (i == tid) p.F[(((long)ch * p.nv + p.n1base + j) * p.ng + my_igp) * 12 + r] = accd[i];
    }
}

// ------------------------------------------------------------ mixed (guarded)
// Exact FP64 re-evaluation of one (igp, ig, iw) element whose FP32 branch
// quantities fell inside a guard band.  Kept out of line so that the compiler
// does not if-convert it into the common path (it is rare; inlined and
// predicated it would run on GB300's narrow FP64 pipe for every element), and
// returned by value so that the caller's variables stay in registers.
struct Exact {
    float2 dv, sch, ssx;
    int A, B;
};
__device__ __noinline__ Exact exact_element(double wxt, double2 wt64, double2 ep64, double2 eq64, int need_ssx,
                                            int phys) {
    const Branch64 b = branch64(wxt, wt64);
    Exact r;
    r.A = b.A;
    r.B = b.B;
    r.dv = c64_to_f32(cmul(b.delw, ep64));
    r.sch = b.A ? c64_to_f32(cmul(b.delw, eq64)) : make_float2(0.f, 0.f);
    r.ssx = make_float2(0.f, 0.f);
    if (need_ssx) {
        const double2 wt2d = cmul(wt64, wt64);
        double2 x = ssx64(b, wxt, wt2d, cmul(wt2d, ep64), phys != 0);
        if (phys) x = sexcut64(x, wxt, ep64);
        r.ssx = c64_to_f32(x);
    }
    return r;
}

// Block (ch, my_igp) covers plane waves [ch*tile, (ch+1)*tile) of column
// my_igp; the chunk count is chosen so that all blocks are resident at once
// (no tail wave).  Each thread walks its elements with the next element's
// inputs already loading while the current one is evaluated.
// Writes D straight into the pre-split BF16 image consumed by the tensor-core
// contraction (column j = my_igp*3 + iw lives in n-tile j / GPP_COLS).
// EST: also the magnitudes the error estimate needs, per frequency iw over the
// block's elements: sum and max of |D|^2 (the image values), |sch|^2 and
// |ssx|^2 (the flag-band factors), written to p.est[ch][my_igp][iw][6].
// SCH = false: the flag bands' sch sums are left to the contraction (their
// terms are the image's products: sch = D where the mask holds, for the C++
// and Fortran variants), and only the ssx sums are kept (F's odd entries).
// The ALU pipe bounds the kernel (72% busy at 440 instructions per element): the
// elements clear of every threshold skip the branch logic by one four-test check,
// and the image addresses are formed once per thread.  512 x 2 x 32768 x 1638: 921 ->
// 840 us; x 20: 20.5 -> 18.7 us.  Measured slower: the pieces staged in shared memory
// and stored as 16-byte chunks (1092 us: a barrier per 256 elements).
template <int Q, int BN, bool EST = false, bool SCH = true>
FK_DEV void prep_mixed_item(const PrepArgs& p, int ch, int my_igp, double2* sm) {
    constexpr int NK = SCH ? 2 : 1;  // kinds accumulated per (band, iw): sch and ssx, or ssx
    const int tid = threadIdx.x;
    const int nflag = min(NVC, p.nv - p.n1base);
    const int igp = prep_setup(p, ch, my_igp);
    const bool flags = nflag > 0 && igp >= 0;
    const float limitone = 250000.0f, limittwo = 0.25f, to1 = 1e-6f;
    uint8_t* D = reinterpret_cast<uint8_t*>(p.D);
    float iw2[3];
    double wx64[3];
#pragma unroll
    for (int iw = 0; iw < 3; ++iw) {
        wx64[iw] = p.wx[iw];
        const float wxf = f64_to_f32_bits(wx64[iw]);
        iw2[iw] = 1.0f / (wxf * wxf);
    }
    const double2* wrow = p.wt + (long)my_igp * p.nc;
    const double2* erow = p.eps + (long)my_igp * p.nc;
    const int ig_end = min(p.nc, (ch + 1) * p.tile);
    float2 acc[NVC * 3 * NK];
#pragma unroll
    for (int i = 0; i < NVC * 3 * NK; ++i) acc[i] = make_float2(0.f, 0.f);
    float es[EST ? 18 : 1];
#pragma unroll
    for (int i = 0; i < (EST ? 18 : 1); ++i) es[i] = 0.f;
    // inputs of the next element
    double2 wt_n = make_double2(0.0, 0.0), ep_n = wt_n, an_n[NVC];
    auto load = [&](int ig) {
        wt_n = wrow[ig];
        ep_n = erow[ig];
#pragma unroll
        for (int j = 0; j < NVC; ++j)
            an_n[j] = (flags && j < nflag) ? p.aqsn[(long)(p.n1base + j) * p.nc + ig] : make_double2(0.0, 0.0);
    };
    int ig = ch * p.tile + tid;
    // the thread's place within an image stage is the same in every group of 256 plane
    // waves (the chunk starts on a stage): its byte offsets of the three rows are formed
    // once, and the stage pointer advances by eight stages
    constexpr long STAGE_B = (long)BN * tcx::NSUB * 64;
    uint8_t* stage = D ? D + ((long)(my_igp / GPP_COLS) * p.kstages + ig / tcx::BK) * STAGE_B : nullptr;
    uint32_t place[3];
#pragma unroll
    for (int iw = 0; iw < 3; ++iw) place[iw] = tc::sw64_offset((my_igp % GPP_COLS) * 3 + iw, tid % tcx::BK);
    if (ig < ig_end) load(ig);
    for (; ig < ig_end; ig += PREP_THREADS, stage += PREP_THREADS / tcx::BK * STAGE_B) {
        const double2 wt64 = wt_n, ep64 = ep_n;
        float2 an[NVC];
#pragma unroll
        for (int j = 0; j < NVC; ++j) an[j] = c64_to_f32(an_n[j]);
        if (ig + PREP_THREADS < ig_end) load(ig + PREP_THREADS);
        const float2 wt = c64_to_f32(wt64), ep = c64_to_f32(ep64);
        float2 wt2 = make_float2(0.f, 0.f), Om = wt2, eq = ep;
        double2 eq64 = ep64;
        if (nflag > 0) {
            wt2 = cmulf(wt, wt);
            Om = cmulf(wt2, ep);
            if (Q == 1) {
                eq64 = p.eps[(long)my_igp * p.ng + ig];
                eq = c64_to_f32(eq64);
            }
        }
#pragma unroll
        for (int iw = 0; iw < 3; ++iw) {
            // wdiff from an FP64 subtraction: keeps full relative accuracy next to the pole
            const float wdr = f64_to_f32_bits(__dsub_rn(wx64[iw], wt64.x)), wdi = -wt.y;
            const float wdiffr = wdr * wdr + wdi * wdi;
            const float rden = __frcp_rn(wdiffr);
            float2 delw = cmulf(wt, make_float2(wdr, -wdi));
            delw.x *= rden;
            delw.y *= rden;
            const float delwr = delw.x * delw.x + delw.y * delw.y;
            bool A, B;
            float2 dv, sch, ssx;
            // clear of every threshold and guard band: both tests hold (the common case)
            const bool clear = Q != 2 && wdiffr > 0.26f && wdiffr < 1e30f && delwr > 1.1e-6f && delwr < 2.4e5f;
            if (clear) {
                A = B = true;
                dv = cmulf(delw, ep);
                sch = Q == 1 ? cmulf(delw, eq) : dv;
                ssx = make_float2(Om.x * iw2[iw], Om.y * iw2[iw]);
            } else {
                const bool amb = !(wdiffr > 1e-30f) || !(delwr < 1e30f) ||
                                 fabsf(wdiffr - limittwo) <= limittwo * GUARD ||
                                 fabsf(delwr - limitone) <= limitone * GUARD || fabsf(delwr - to1) <= to1 * GUARD;
                // physics mode: elements whose Fortran quantities are ill-conditioned in
                // FP32 (wx^2 - wtilde^2 near 0) or whose sexcut test lies within the guard
                // band go to the exact sequence as well
                bool amb2 = false;
                if (__any_sync(__activemask(), amb) && amb) {
                    // exact FP64 sequence for this element (rare)
                    const Exact x = exact_element(wx64[iw], wt64, ep64, eq64, nflag > 0, Q == 2);
                    A = x.A != 0;
                    B = x.B != 0;
                    dv = x.dv;
                    sch = x.sch;
                    ssx = x.ssx;
                } else {
                    A = (wdiffr > limittwo) && (delwr < limitone);
                    B = delwr > to1;
                    dv = cmulf(delw, ep);
                    sch = A ? cmulf(delw, eq) : make_float2(0.f, 0.f);
                    if (A && Q == 2) {
                        // cden = wx^2 - wtilde^2 = (wx - wtilde)(wx + wtilde), each factor from an
                        // FP64 subtraction / addition (gppkernel.deslippe.09.30.2014.f90:302-305)
                        const float wsr = f64_to_f32_bits(__dadd_rn(wx64[iw], wt64.x));
                        const float2 cd = cmulf(make_float2(wdr, wdi), make_float2(wsr, wt.y));
                        const float cd2 = cd.x * cd.x + cd.y * cd.y;
                        amb2 = !(cd2 > 1e-30f);
                        const float rd = __frcp_rn(cd2);
                        const float2 t = cmulf(Om, make_float2(cd.x, -cd.y));
                        ssx = make_float2(t.x * rd, t.y * rd);
                    } else if (A) {
                        ssx = make_float2(Om.x * iw2[iw], Om.y * iw2[iw]);
                    } else if (B) {
                        float2 c = cmulf(make_float2(4.f * wt2.x, 4.f * wt2.y), make_float2(delw.x + 0.5f, delw.y));
                        float rd = __frcp_rn(c.x * c.x + c.y * c.y);
                        float2 t = cmulf(make_float2(-Om.x, -Om.y), make_float2(c.x, -c.y));
                        ssx = cmulf(make_float2(t.x * rd, t.y * rd), delw);
                    } else {
                        ssx = make_float2(0.f, 0.f);
                    }
                    if (Q == 2 && wx64[iw] < 0.0) {
                        // the Fortran sexcut test, |ssx| > 4|I_eps| (f90:319-320), in squares
                        const float a2 = ssx.x * ssx.x + ssx.y * ssx.y, c2 = 16.f * (ep.x * ep.x + ep.y * ep.y);
                        const bool near = !(a2 < 1e30f) || fabsf(a2 - c2) <= c2 * (4.f * GUARD);
                        amb2 = amb2 || near;
                        if (!near && a2 > c2) ssx = make_float2(0.f, 0.f);
                    }
                }
                if (Q == 2 && nflag > 0 && __any_sync(__activemask(), amb2) && amb2) {
                    const Exact x = exact_element(wx64[iw], wt64, ep64, eq64, nflag > 0, 1);
                    A = x.A != 0;
                    B = x.B != 0;
                    dv = x.dv;
                    sch = x.sch;
                    ssx = x.ssx;
                }
            }
            if constexpr (EST) {
                if (igp >= 0) {
                    const float d2 = (Q == 1 || A) ? dv.x * dv.x + dv.y * dv.y : 0.f;
                    const float c2 = sch.x * sch.x + sch.y * sch.y, x2 = ssx.x * ssx.x + ssx.y * ssx.y;
                    es[iw * 6 + 0] += d2;
                    es[iw * 6 + 1] = fmaxf(es[iw * 6 + 1], d2);
                    if (nflag > 0) {
                        es[iw * 6 + 2] += c2;
                        es[iw * 6 + 3] = fmaxf(es[iw * 6 + 3], c2);
                        es[iw * 6 + 4] += x2;
                        es[iw * 6 + 5] = fmaxf(es[iw * 6 + 5], x2);
                    }
                }
            }
            if (D) {
                // every element of the image is written (zero where the term is masked)
                const bool keep = igp >= 0 && (Q == 1 || A);
                tcx::bimg_store_at<BN>(stage + place[iw], keep ? dv.x : 0.f, keep ? dv.y : 0.f);
            }
#pragma unroll
            for (int j = 0; j < NVC; ++j) {
                if (SCH) cfmaf(acc[(j * 3 + iw) * NK + 0], an[j], sch);
                cfmaf(acc[(j * 3 + iw) * NK + NK - 1], an[j], ssx);
            }
        }
    }
    if (p.setup && D) {
        // zeros of the image that no column writes: the padding rows of this
        // column's tile (the chunk's k-range split evenly over the tile's
        // columns) and, in the last chunk, k from ncouls to the end of the last
        // k-stage
        const int c = my_igp % GPP_COLS, nt = my_igp / GPP_COLS;
        const bool lastcol = c == GPP_COLS - 1 || my_igp == p.ng - 1;
        const int ncols = min(GPP_COLS, p.ng - nt * GPP_COLS), rp = 3 * ncols;  // first padding row
        uint8_t* tile = D + (long)nt * p.kstages * tcx::Cfg<BN>::B_BYTES;
        const int kend = p.kstages * tcx::BK;
        if (rp < BN) {
            const int k0 = ch * p.tile, k1 = min(p.nc, (ch + 1) * p.tile);
            const int ka = k0 + (int)((long)(k1 - k0) * c / ncols), kb = k0 + (int)((long)(k1 - k0) * (c + 1) / ncols);
            for (int k = ka + tid; k < kb; k += PREP_THREADS)
                for (int r = rp; r < BN; ++r) tcx::bimg_store<BN>(tile, p.kstages, r, k, 0.f, 0.f);
        }
        if ((ch + 1) * p.tile >= p.nc)
            for (int k = p.nc + tid; k < kend; k += PREP_THREADS)
                for (int r = 3 * c; r < (lastcol ? BN : 3 * c + 3); ++r) tcx::bimg_store<BN>(tile, p.kstages, r, k, 0.f, 0.f);
    }
    if constexpr (EST) {
        // sums (even q) and maxima (odd q) over the block: warps, then the eight warps in order
        __shared__ float esm[8][18];
#pragma unroll
        for (int q = 0; q < 18; ++q)
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                const float o = __shfl_down_sync(0xffffffffu, es[q], off);
                es[q] = (q & 1) ? fmaxf(es[q], o) : es[q] + o;
            }
        if ((tid & 31) == 0)
#pragma unroll
            for (int q = 0; q < 18; ++q) esm[tid >> 5][q] = es[q];
        __syncthreads();
        if (tid < 18) {
            float v = 0.f;
            for (int w = 0; w < PREP_THREADS / 32; ++w) v = (tid & 1) ? fmaxf(v, esm[w][tid]) : v + esm[w][tid];
            p.est[((long)ch * p.ng + my_igp) * 18 + tid] = v;
        }
    }
    if (nflag <= 0) return;
    double2 accd[NVC * 3 * NK];
    block_sum_ff<NVC * 3 * NK>(acc, sm, accd);
    if (tid < nflag * 3 * NK) {
        // F[..][iw * 2 + kind] (kind 0 sch, 1 ssx)
        const int j = tid / (3 * NK), q = tid % (3 * NK), r = SCH ? q : 2 * q + 1;
#pragma unroll
        for (int i = 0; i < NVC * 3 * NK; ++i)
            if (i == tid) p.F[(((long)ch * p.nv + p.n1base + j) * p.ng + my_igp) * 6 + r] = accd[i];
    }
}

template <int Q, int BN, bool EST = false, bool SCH = true>
__global__ void __launch_bounds__(PREP_THREADS, 2) prep_mixed_kernel(PrepArgs p) {
    __shared__ double2 sm[8 * NVC * 6];
    prep_mixed_item<Q, BN, EST, SCH>(p, p.ch0 + blockIdx.x, blockIdx.y, sm);
}

// ------------------------------------------------------------ error estimate
// A-priori estimate of the mixed path's absolute error (fk_gpp_error_estimate).
// Each output is a sum of terms w * a * x (w the band-column weight, a an
// aqsntemp element, x a D / sch / ssx value).  Every term carries a few FP32
// roundings (operands, the FP32 branch factors, the tensor cores' truncating
// FP32 accumulation, the FP32 epilogue) of random sign, so the error is about
// C * 2^-24 * sqrt(sum of |term|^2).  The sum over ig of |a|^2 |x|^2 is bounded
// by min(|a_n|_2^2 |x_j|_inf^2, |a_n|_inf^2 |x_j|_2^2) for band n and column
// j = (my_igp, iw), which needs only the row norms below and the prep's column
// magnitudes; the estimate is therefore at least C * 2^-24 * rss.

// an[n] = (sum_ig |aqsn[n][ig]|^2, max_ig |aqsn[n][ig]|^2), one block per band.
__global__ void __launch_bounds__(256) est_rows_kernel(int nc, const double2* aqsn, float2* an) {
    const double2* row = aqsn + (long)blockIdx.x * nc;
    float s = 0.f, m = 0.f;
    for (int ig = threadIdx.x; ig < nc; ig += 256) {
        const float2 a = c64_to_f32(row[ig]);
        const float a2 = a.x * a.x + a.y * a.y;
        s += a2;
        m = fmaxf(m, a2);
    }
    __shared__ float sm[8][2];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        s += __shfl_down_sync(0xffffffffu, s, off);
        m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, off));
    }
    if ((threadIdx.x & 31) == 0) {
        sm[threadIdx.x >> 5][0] = s;
        sm[threadIdx.x >> 5][1] = m;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) {
            s += sm[w][0];
            m = fmaxf(m, sm[w][1]);
        }
        an[blockIdx.x] = make_float2(s, m);
    }
}

// Per band n, per iw: the bound of sum |term|^2 of its achtemp terms (bands
// n >= nvband: D columns; occupied bands: sch) and, occupied bands, of its
// asxtemp terms (ssx), into eb[n][6].  One block of 128 threads per band, the
// threads taking columns; the column magnitudes are first reduced over the
// prep's chunks.
__global__ void __launch_bounds__(128) est_bands_kernel(int nv, int ng, int nch, const float* est, const float2* an,
                                                        const double2* aqsm, long ldm, const int* igp,
                                                        const int* acol, const double* vcoul, double* eb) {
    const int n = blockIdx.x;
    const float2 a = an[n];
    double v[6] = {0, 0, 0, 0, 0, 0};
    for (int h = threadIdx.x; h < ng; h += 128) {
        const int g = igp[h];
        if (g < 0) continue;
        const double2 am = aqsm[(long)n * ldm + acol[h]];
        const double w2 = (am.x * am.x + am.y * am.y) * vcoul[g] * vcoul[g];
#pragma unroll
        for (int iw = 0; iw < 3; ++iw) {
            float c[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int ch = 0; ch < nch; ++ch) {
                const float* e = est + ((long)ch * ng + h) * 18 + iw * 6;
#pragma unroll
                for (int q = 0; q < 6; ++q) c[q] = (q & 1) ? fmaxf(c[q], e[q]) : c[q] + e[q];
            }
            const int o = n < nv ? 2 : 0;  // occupied bands: sch; the others: the image values
            const double t = fmin((double)a.x * c[o + 1], (double)a.y * c[o]);
            v[iw] += 0.25 * w2 * t;  // achtemp weight 0.5 vcoul conj(aqsm)
            if (n < nv) v[3 + iw] += w2 * fmin((double)a.x * c[5], (double)a.y * c[4]);  // asxtemp: vcoul conj(aqsm)
        }
    }
    __shared__ double sm[4][6];
#pragma unroll
    for (int q = 0; q < 6; ++q)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v[q] += __shfl_down_sync(0xffffffffu, v[q], off);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int q = 0; q < 6; ++q) sm[threadIdx.x >> 5][q] = v[q];
    __syncthreads();
    if (threadIdx.x < 6) eb[(long)n * 6 + threadIdx.x] = sm[0][threadIdx.x] + sm[1][threadIdx.x] + sm[2][threadIdx.x] + sm[3][threadIdx.x];
}

// out[0] = achtemp, out[1] = asxtemp (max over iw), out[2] = acht_n1_loc (max
// over bands; its component is iw = 2): scale * sqrt(bound), bands added in a
// fixed order.  One block of 256 threads.
__global__ void __launch_bounds__(256) est_total_kernel(int nb, const double* eb, double scale, double* out) {
    double v[6] = {0, 0, 0, 0, 0, 0}, mx = 0.0;
    for (int n = threadIdx.x; n < nb; n += 256) {
#pragma unroll
        for (int q = 0; q < 6; ++q) v[q] += eb[(long)n * 6 + q];
        mx = fmax(mx, eb[(long)n * 6 + 2]);
    }
    __shared__ double sm[8][7];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
        for (int q = 0; q < 6; ++q) v[q] += __shfl_down_sync(0xffffffffu, v[q], off);
        mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, off));
    }
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int q = 0; q < 6; ++q) sm[threadIdx.x >> 5][q] = v[q];
        sm[threadIdx.x >> 5][6] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t[7] = {0, 0, 0, 0, 0, 0, 0};
        for (int w = 0; w < 8; ++w)
            for (int q = 0; q < 7; ++q) t[q] = q == 6 ? fmax(t[q], sm[w][q]) : t[q] + sm[w][q];
        out[0] = scale * sqrt(fmax(fmax(t[0], t[1]), t[2]));
        out[1] = scale * sqrt(fmax(fmax(t[3], t[4]), t[5]));
        out[2] = scale * sqrt(t[6]);
    }
}

// ------------------------------------------------------------------ finalize
// Warp-level fixed-order sum of NV double2 values (shuffle tree).
template <int NV>
FK_DEV void warp_sum(double2 (&v)[NV]) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            v[i].x += __shfl_down_sync(0xffffffffu, v[i].x, off);
            v[i].y += __shfl_down_sync(0xffffffffu, v[i].y, off);
        }
}

// Fixed shuffle tree: lane 0 receives the sum of the 32 lanes' values.
FK_DEV double2 warp_tree(double2 v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        v.x = __dadd_rn(v.x, __shfl_down_sync(0xffffffffu, v.x, off));
        v.y = __dadd_rn(v.y, __shfl_down_sync(0xffffffffu, v.y, off));
    }
    return v;
}

// Per-band sums into rows[n1][8] = {sch iw0..2, ssx iw0..2, stat, 0}.  Bands
// n1 >= nvband add the contraction's k-slice partials P[slot][m][3]
// (rows_band_warp, below).  Occupied bands n1 < nvband, one block per (band,
// component c of 7; rows_flag_block): for c < 6, over columns my_igp, the chunk
// partials of the prep F[ch][n1][my_igp][6] times the reference's weight
// (sch: 0.5*vcoul*conj(aqsm), BGW-Kernels/gppKer.cpp:346,421; ssx:
// occ*vcoul*conj(aqsm), :419), the threads taking (chunk, column) items and a
// fixed tree adding them (deterministic); c == 6: the static-remainder partials
// S[slot][n1].
constexpr int ROWS_THREADS = 128;
struct RowsArgs {
    int nb, nv, ng, nslots;
    const double2* P;
    int nslots_s;
    const double2* S;
    int nch;
    const double2* F;
    long ldm;
    const double2* aqsm;
    const double* vcoul;
    const int *igp, *acol;
    double2* rows;
    // half-sum mode: partials of the A = aqsmtemp contraction, diagonal values, aqsntemp
    const double2* P2;
    const double2* schd;  // [ng][3]
    const double2* aqsn;  // [nb][nc]
    int nc;
    bool re_only;         // real-valued sum: the contraction partials carry it in their real parts
    double* out_re = nullptr;  // its results [achtemp 3 | asxtemp 3 | acht_n1_loc nb], in place of out
    // totals folded in: the last block to finish (counter, zero at entry) writes out
    int* counter;
    double2* out;
    const double2* wf;    // flag-band weights from the prep ([nv][ng][2]), or nullptr
    int m0 = -1;          // first band of the contraction partials P (-1: nvband)
    bool fsch = false;    // occupied bands' sch components from P (rows from m0 = 0), not from F
};

// Bound: the round trips to memory of a thread's items, one after another.  Over one
// warp, column by column, 1638 columns took 51 of them and the kernel 119 us at
// 512 x 2 x 32768 x 1638 (now 21 us); eight items are in flight at a time.
FK_DEV void rows_flag_block(const RowsArgs& ra, int n1, int c, int tid) {
    constexpr int T = ROWS_THREADS;
    const int nb = ra.nb, nv = ra.nv, ng = ra.ng, nslots_s = ra.nslots_s, nch = ra.nch;
    const double2 *S = ra.S, *F = ra.F, *aqsm = ra.aqsm;
    const long ldm = ra.ldm;
    const double* vcoul = ra.vcoul;
    const int *igp = ra.igp, *acol = ra.acol;
    double2* rows = ra.rows;
    double2 v = make_double2(0.0, 0.0);
    if (c == 6) {
        if (S && tid < nslots_s) v = ordered_sum(S + (long)tid * nb + n1, (long)T * nb, (nslots_s - tid + T - 1) / T);
    } else if (ra.fsch && c < 3) {
        // the band's sch component from the contraction: its k-slice partials in slot order
        const int m0 = ra.m0 < 0 ? nv : ra.m0;
        const long M = nb - m0, m = n1 - m0;
        if (tid < ra.nslots) v = ordered_sum(ra.P + ((long)tid * M + m) * 3 + c, (long)T * M * 3, (ra.nslots - tid + T - 1) / T);
    } else if (ra.P2) {
        // half sum, occupied band: weight * (cm S1 + conj(cm S2)) per column
        const int kind = c / 3, r = ((c % 3) * 2 + kind) * 2;
        const double occ = 1.0;
        for (long i = tid; i < (long)nch * ng; i += T) {  // item i = (chunk i / ng, column i % ng)
            const long k = i / ng, h = i - k * ng;
            const int g = igp[h];
            if (g < 0) continue;
            const double2* x = F + ((k * nv + n1) * ng + h) * 12 + r;
            const double2 s1 = x[0], s2 = x[1], cm = cconj(aqsm[(long)n1 * ldm + acol[h]]);
            v = cadd(v, cscale(cadd(cmul(cm, s1), cconj(cmul(cm, s2))), kind ? occ * vcoul[g] : 0.5 * vcoul[g]));
        }
    } else if (ra.wf) {
        // weights from the prep; item i = (chunk i / ng, column i % ng)
        constexpr int U = 8;
        const int kind = c / 3, r = (c % 3) * 2 + kind;  // kind 0: sch, 1: ssx
        const long items = (long)nch * ng;
        for (long i0 = tid; i0 < items; i0 += U * T) {
            double2 w[U], x[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {  // clamped indices: every load reads a valid address
                const long i = min(i0 + u * T, items - 1), k = i / ng, h = i - k * ng;
                w[u] = ra.wf[((long)n1 * ng + h) * 2 + kind];
                x[u] = F[((k * nv + n1) * ng + h) * 6 + r];
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (i0 + u * T < items) v = cadd(v, cmul(w[u], x[u]));
        }
    } else {
        const int kind = c / 3, r = (c % 3) * 2 + kind;  // kind 0: sch, 1: ssx
        const double occ = 1.0;
        for (long i = tid; i < (long)nch * ng; i += T) {
            const long k = i / ng, h = i - k * ng;
            const int g = igp[h];
            if (g < 0) continue;
            const double2 sum = F[((k * nv + n1) * ng + h) * 6 + r];
            const double2 cm = cconj(aqsm[(long)n1 * ldm + acol[h]]);
            v = cadd(v, cscale(cmul(cm, sum), kind ? occ * vcoul[g] : 0.5 * vcoul[g]));
        }
    }
    // a component with no terms (stat without S) skips the tree
    __shared__ double2 part[T / 32];
    if (c != 6 || S) {
        v = warp_tree(v);
        if ((tid & 31) == 0) part[tid >> 5] = v;
        __syncthreads();
        if (tid == 0)
            for (int w = 1; w < T / 32; ++w) v = cadd(v, part[w]);
    }
    if (tid == 0) {
        rows[(long)n1 * 8 + c] = v;
        if (c == 2 && ra.out) ra.out[7 + n1] = v;  // acht_n1_loc
        if (c == 2 && ra.out_re) ra.out_re[6 + n1] = v.x;
    }
    __syncthreads();  // part is reused by the block's next task
}

// Bands n1 >= nvband, one warp per band.  GB300's FP64 pipe retires one warp
// instruction per 64 cycles on each SM sub-partition, whatever the
// instruction-level parallelism, so the sums are laid out to need few FP64
// warp instructions per warp: lane 5p + s (p < 6: component p/2, real or
// imaginary part p%2; s < 5) adds slots s, s+5, s+10, .. of its part, and
// four shuffles add the five splits; lanes 30 and 31 hold the static
// remainder's parts.  Blocks are four warps (four bands, one per
// sub-partition); warp 0 then writes the block's partial totals (eight
// parts: components 0..2 and 6), so the totals read one value per four bands.
// The rows buffer is [nb][8] band rows, then [band blocks][8] partials.
__host__ __device__ inline int rows_flag_blocks(int nv) { return nv * 7; }
__host__ __device__ inline int rows_band_blocks(int nb, int nv) { return (nb - nv + 3) / 4; }
__host__ __device__ inline int rows_blocks(int nb, int nv) { return rows_flag_blocks(nv) + rows_band_blocks(nb, nv); }
__host__ __device__ inline size_t rows_bytes(int nb) {
    return ((size_t)nb * 8 + 4 * (size_t)((nb + 3) / 4)) * sizeof(double2);
}

FK_DEV double part_of(double2 v, int im) { return im ? v.y : v.x; }

// sum over slots k = s, s+5, .. < nslots (ascending) of part im of P[k][m][c]
FK_DEV double split_sum(const double2* P, long M, long m, int c, int im, int nslots, int s) {
    double v = 0.0;
    for (int k0 = s; k0 < nslots; k0 += 5 * 8) {
        double a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = part_of(P[((long)min(k0 + 5 * i, nslots - 1) * M + m) * 3 + c], im);
#pragma unroll
        for (int i = 0; i < 8; ++i) v = __dadd_rn(v, k0 + 5 * i < nslots ? a[i] : 0.0);  // unconditional: see ordered_sum
    }
    return v;
}

FK_DEV void rows_band_warp(const RowsArgs& ra, int n1, int lane, double* parts) {
    const int m0 = ra.m0 < 0 ? ra.nv : ra.m0;
    const long M = ra.nb - m0, m = n1 - m0;
    const int p = lane / 5, s = lane % 5, c = p >> 1, im = p & 1;
    double a = 0.0, b = 0.0, d = 0.0;  // this split's contraction sum, A = aqsmtemp sum, diagonal terms
    if (lane < 30) {
        if (!(ra.re_only && im)) a = split_sum(ra.P, M, m, c, im, ra.nslots, s);
        if (ra.P2) {
            // half sum: the A = aqsmtemp contraction and the diagonal terms of the
            // columns on 512-wide block edges (split s: columns s, s+5, ..)
            b = split_sum(ra.P2, M, m, c, im, ra.nslots, s);
            for (int h = s; h < ra.ng; h += 5) {
                const int g = ra.igp[h];
                if (g <= 0 || (g & 511)) continue;
                const double2 am = cmul(cconj(ra.aqsm[(long)n1 * ra.ldm + ra.acol[h]]), ra.aqsn[(long)n1 * ra.nc + g]);
                d = __dadd_rn(d, part_of(cscale(cmul(am, ra.schd[h * 3 + c]), 0.5 * ra.vcoul[g]), im));
            }
        }
    }
    if (ra.S) {
        // static remainder: the lanes take slots, a fixed tree adds them; lane 30 keeps
        // the real, lane 31 the imaginary part
        double2 v = make_double2(0.0, 0.0);
        if (lane < ra.nslots_s) v = ordered_sum(ra.S + (long)lane * ra.nb + n1, 32L * ra.nb, (ra.nslots_s - lane + 31) / 32);
        v = warp_tree(v);
        v.x = __shfl_sync(0xffffffffu, v.x, 0);
        v.y = __shfl_sync(0xffffffffu, v.y, 0);
        if (lane >= 30) a = part_of(v, lane - 30);
    }
    // lane 5p adds the other four splits of part p, in split order (the
    // shuffles read the unmodified split sums a0, b0, d0)
    const int base = (lane < 30 ? p : 0) * 5;
    const double a0 = a, b0 = b, d0 = d;
#pragma unroll
    for (int i = 1; i < 5; ++i) {
        const double ai = __shfl_sync(0xffffffffu, a0, base + i);
        const double bi = __shfl_sync(0xffffffffu, b0, base + i);
        const double di = __shfl_sync(0xffffffffu, d0, base + i);
        if (lane < 30 && s == 0) {
            a = __dadd_rn(a, ai);
            if (ra.P2) {
                b = __dadd_rn(b, bi);
                d = __dadd_rn(d, di);
            }
        }
    }
    double* row = (double*)(ra.rows + (long)n1 * 8);
    if (lane < 30 && s == 0) {
        double v = a;
        if (ra.P2) v = __dadd_rn(__dadd_rn(v, im ? -b : b), d);  // + conj(A = aqsmtemp sum) + diagonal
        row[2 * c + im] = v;
        parts[p] = v;
        if (c == 2 && ra.out) ((double*)(ra.out + 7 + n1))[im] = v;  // acht_n1_loc
        if (c == 2 && ra.out_re && !im) ra.out_re[6 + n1] = v;
    }
    if (lane >= 30) {
        row[12 + lane - 30] = a;  // component 6
        parts[6 + lane - 30] = a;
    }
    if (lane < 6) row[6 + lane] = 0.0;  // ssx (3..5): occupied bands only
}

// Block task i of a request's rows: flag blocks (one occupied-band component
// each), then band blocks (four bands each).  Every
// thread of the block calls it with the same i.
FK_DEV void rows_block(const RowsArgs& ra, int i, int tid) {
    const int warp = tid >> 5, lane = tid & 31, nfb = rows_flag_blocks(ra.nv);
    if (i < nfb) {
        rows_flag_block(ra, i / 7, i % 7, tid);
        return;
    }
    const int bb = i - nfb, n0 = ra.nv + bb * 4;
    __shared__ double parts[4][8];  // the block's bands' values of the eight parts
    if (n0 + warp < ra.nb) rows_band_warp(ra, n0 + warp, lane, parts[warp]);
    __syncthreads();
    if (tid < 8) {
        // the four bands' partial totals of part tid (component tid/2 for tid < 6, else 6)
        double v = 0.0;
        for (int b = 0; b < 4 && n0 + b < ra.nb; ++b) v = __dadd_rn(v, parts[b][tid]);
        ((double*)(ra.rows + (long)ra.nb * 8 + (long)bb * 4))[tid] = v;
    }
    __syncthreads();  // parts is reused by the block's next task
}

// Totals by one block of ROWS_THREADS: thread 16q + s (q < 8: part q of
// components 0..2 and 6) adds items s, s+16, .. of the part's list -- the
// occupied bands' rows, then the band blocks' partials -- and four shuffles
// add the sixteen splits; the ssx parts (occupied bands only) by threads 0..5.
// out = [achtemp 3 | asxtemp 3 | achstemp | acht_n1_loc nb] (acht_n1_loc is
// written by the band warps).
FK_DEV void totals_block(int nb, int nv, const double2* rows, double2* out, double* out_re = nullptr) {
    constexpr int B = 12;  // items in flight per thread: one round trip up to 16*B items
    const int t = threadIdx.x, q = t >> 4, s = t & 15;
    const int c = q < 6 ? q >> 1 : 6, im = q & 1;
    const long items = nv + rows_band_blocks(nb, nv);
    const double* part = (const double*)(rows + (long)nb * 8);
    // ssx (components 3..5, occupied bands only): threads 0..5, loaded with the first batch
    const int nx = t < 6 ? nv : 0;
    double v = 0.0, w = 0.0;
    for (long i0 = s, x0 = 0; i0 < items || x0 < nx; i0 += 16 * B, x0 += B) {
        double a[B], x[B];
#pragma unroll
        for (int j = 0; j < B; ++j) {  // clamped indices: every load reads a valid address
            const long i = min(i0 + 16 * j, items - 1);
            a[j] = *(i < nv ? (const double*)(rows + i * 8 + c) + im : part + (i - nv) * 8 + q);
        }
        if (nx)  // threads 0..5 only (their component 3 + t/2 exists in every row)
#pragma unroll
            for (int j = 0; j < B; ++j) x[j] = part_of(rows[min(x0 + j, (long)nx - 1) * 8 + 3 + (t >> 1)], t & 1);
#pragma unroll
        for (int j = 0; j < B; ++j) v = __dadd_rn(v, i0 + 16 * j < items ? a[j] : 0.0);  // unconditional: see ordered_sum
        if (nx)
#pragma unroll
            for (int j = 0; j < B; ++j) w = __dadd_rn(w, x0 + j < nx ? x[j] : 0.0);
    }
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) v = __dadd_rn(v, __shfl_down_sync(0xffffffffu, v, off));
    if (out_re) {
        if (s == 0 && c < 3 && !im) out_re[c] = v;
        if (t < 6 && !(t & 1)) out_re[3 + (t >> 1)] = w;
        return;
    }
    double* o = (double*)out;
    if (s == 0) o[2 * c + im] = v;
    if (t < 6) o[6 + t] = w;
}

__global__ void __launch_bounds__(ROWS_THREADS) rows_kernel(RowsArgs ra) {
    rows_block(ra, blockIdx.x, threadIdx.x);
    if (!ra.counter) return;
    // the last block to finish adds the bands (totals_block, fixed order): the
    // barrier orders the block's row writes before thread 0's count, a
    // device-scope release; the last block's count also acquires the others'
    __shared__ int last;
    __syncthreads();
    if (threadIdx.x == 0) {
        int old;
        asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(old) : "l"(ra.counter) : "memory");
        last = old == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    totals_block(ra.nb, ra.nv, ra.rows, ra.out, ra.out_re);
    if (threadIdx.x == 0) *ra.counter = 0;
}


// The mixed-precision contraction of fk_gpp runs on CTA pairs, except in the
// pipelined host path (one launch per row block), the half sum, the served
// steps and the real-valued sum, which keep the single-CTA kernel.
// A request with one n-tile of columns (ngpown <= 21) streams aqsntemp once at
// the HBM rate, where the single-CTA kernel is the faster one (measured: the call takes
// 96 us against 103 at 512 x 2 x 32768 x 20); with more n-tiles the tensor work dominates.
inline bool gpp_pair(const GppDev& r, bool pipelined) {
    return r.prec == FK_MIXED && !pipelined && !(r.flags & FK_GPP_HALF_SUM) && r.ng > 21;
}

struct Plan {
    int nch, tile, passes;
    int pipe_sub, pipe_chunks;   // pipelined host path: prep chunks (= k-slices) per k-chunk, k-chunks
    int BN, kstages, units;      // tensor-core contraction (mixed)
    int MT, NT, KS, kchunk;      // main contraction
    int MTs, NTs, KSs, kchunks;  // static remainder contraction
    bool mixed;
    bool fsch;  // the occupied bands' sch sums through the contraction (its rows start at band 0)
    int m0;     // first band of the contraction: 0 with fsch, else nvband
    // CTA pairs over four or more n-tiles: aqsntemp split into BF16 pieces once (an A
    // image) instead of by the converter warps of every n-tile's units
    bool apre;
    size_t bytesD, bytesF, bytesP, bytesS, bytesRows, bytesIgp, bytesW, bytesAimg;
    // FP64 on the tensor cores (fk_tc64.cuh): the main and the static remainder contraction, and their workspace
    bool tc64;
    tc64::Plan z, zs;
    size_t zA, zB, zEa, zEb, zW, zG;
    size_t bytesZ() const { return tc64 ? zA + zB + zEa + zEb + zW + zG + 6 * 256 : 0; }
};

// fk_gpp's mixed path and its FP64 path on the tensor cores (not the half sum, not
// the root file's flag-band I_eps indexing, whose sch differs from the image's values) contracts the occupied
// bands too: their sch terms are the image's products.
inline bool gpp_fsch(const GppDev& r) {
    return (r.prec == FK_MIXED || r.tc64) && !(r.flags & (FK_GPP_HALF_SUM | FK_GPP_ROOT_QUIRKS));
}

// k-slice count for the persistent tensor-core kernel: the fewest slices
// whose unit count fills the SMs evenly (tail waste <= 8%), with slices of at
// least 256 k-values.
void pick_split_tc(int tiles, int K, int sms, int& KS, int& kchunk) {
    const int kmax = std::max(1, K / 256);
    int best = 1;
    double best_cost = 1e30;
    for (int ks = 1; ks <= std::min(kmax, 256); ++ks) {
        const long units = (long)tiles * ks;
        const long waves = (units + sms - 1) / sms;
        const double eff = (double)units / (double)(waves * sms);
        const double cost = (1.0 / eff) * (1.0 + 0.002 * ks);  // mild preference for fewer slices
        if (cost < best_cost - 1e-9) { best_cost = cost; best = ks; }
        if (eff > 0.92 && units >= sms) break;
    }
    kchunk = ((K + best - 1) / best + tcx::BK - 1) / tcx::BK * tcx::BK;
    KS = (K + kchunk - 1) / kchunk;
}

void pick_split(int tiles, int K, int target, int& KS, int& kchunk) {
    KS = std::max(1, std::min((target + tiles - 1) / tiles, std::max(1, K / 256)));
    kchunk = ((K + KS - 1) / KS + 15) / 16 * 16;
    KS = (K + kchunk - 1) / kchunk;
}

constexpr int PIPE_CHUNKS = 8;  // row blocks of the pipelined host path at most (events 0..7 of Ctx::pipe_ev)

// pair: the contraction runs on CTA pairs (tc_contract_pair_kernel): MT counts
// 256-row tiles and the k-split fills the SM pairs
Plan make_plan(const Ctx& c, const GppDev& r, int ks_override = 0, bool pipelined = false, bool pair = false,
               bool fsch = false) {
    Plan p{};
    p.mixed = r.prec == FK_MIXED;
    if (!p.mixed && r.tc64) {
        // FP64 on the tensor cores, where a split of both contractions exists
        const int M = r.nb - (fsch ? 0 : r.nv);
        if (M > 0) {
            p.z = tc64::make_plan(M, 3 * r.ng, r.nc, 1, c.sms / 2);
            if (r.flags & FK_GPP_ACHSTEMP) p.zs = tc64::make_plan(r.nb, r.ng, r.nc, 1, c.sms / 2);
            p.tc64 = p.z.KS && (p.zs.KS || !(r.flags & FK_GPP_ACHSTEMP));
        }
    }
    p.fsch = fsch && (p.mixed || p.tc64);
    p.m0 = p.fsch ? 0 : r.nv;
    p.pipe_sub = p.pipe_chunks = 0;
    if (r.prec == FK_MIXED) {
        // one wave: chunks x ngpown blocks fill the resident block slots
        int per_sm = 0;
        void (*kprep)(PrepArgs) = p.fsch ? prep_mixed_kernel<0, 64, false, false> : prep_mixed_kernel<0, 64>;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kprep, PREP_THREADS, 0) != cudaSuccess || per_sm < 1)
            per_sm = 1;
        // chunks in whole k-stages (a warp's 32 plane waves fill whole image rows),
        // so that the last chunk is not much shorter than the others
        const int nch = std::max(1, per_sm * c.sms / r.ng);
        p.tile = ceil_div(ceil_div(r.nc, nch), tcx::BK) * tcx::BK;
        p.nch = ceil_div(r.nc, p.tile);
    } else {
        // one wave of resident blocks (two per SM; one beside the digit conversion of
        // aqsntemp, which takes the rest of the registers); each chunk is one partial per
        // flag band and column for the band reduction
        const int nch = std::max(1, (p.tc64 ? 1 : 2) * c.sms / r.ng);
        p.tile = ceil_div(ceil_div(r.nc, nch), PREP_THREADS) * PREP_THREADS;
        p.nch = ceil_div(r.nc, p.tile);
    }
    const bool half = (r.flags & FK_GPP_HALF_SUM) != 0;
    if (half) {
        // FP64: tiles of the FP64 prep; mixed: chunks of one resident wave (two
        // blocks per SM), so that the band reduction adds few chunk partials
        p.tile = r.prec == FK_MIXED
                     ? ceil_div(ceil_div(r.nc, std::max(1, 2 * c.sms / r.ng)), PREP_THREADS) * PREP_THREADS
                     : PREP_TILE;
        p.nch = ceil_div(r.nc, p.tile);
    }
    p.passes = std::max(1, ceil_div(r.nv, NVC));
    const int M = r.nb - p.m0, N = 3 * r.ng;
    if (p.mixed) {
        p.BN = 64;
        p.kstages = ceil_div(r.nc, tcx::BK);
        p.MT = ceil_div(std::max(M, 1), (pair ? 2 : 1) * tcx::BM);
        p.NT = ceil_div(r.ng, GPP_COLS);
        pick_split_tc(p.MT * p.NT, r.nc, pair ? c.sms / 2 : c.sms, p.KS, p.kchunk);
        if (ks_override > 0) {
            const int ks = std::min(ks_override, std::max(1, ceil_div(r.nc, tcx::BK)));
            p.kchunk = ceil_div(ceil_div(r.nc, ks), tcx::BK) * tcx::BK;
            p.KS = ceil_div(r.nc, p.kchunk);
        }
        if (pipelined) {
            // one launch per row block of pipe_sub m-tiles: enough k-slices for that block to fill the GPU
            p.pipe_sub = ceil_div(p.MT, PIPE_CHUNKS);
            p.pipe_chunks = ceil_div(p.MT, p.pipe_sub);
            const int ks = std::max(1, std::min(c.sms / std::max(1, p.pipe_sub * p.NT), r.nc / 256));
            p.kchunk = ceil_div(ceil_div(r.nc, ks), tcx::BK) * tcx::BK;
            p.KS = ceil_div(r.nc, p.kchunk);
            p.units = p.MT * p.NT * p.KS;
        }
        p.units = p.MT * p.NT * p.KS;
        p.apre = pair && !pipelined && p.NT >= 4;
        p.bytesAimg = p.apre ? (size_t)2 * p.MT * p.kstages * tcx::Cfg<64, false, true>::A_BYTES : 0;
    } else {
        p.MT = ceil_div(std::max(M, 1), d64::BM);
        p.NT = ceil_div(N, d64::BN);
        pick_split(p.MT * p.NT, r.nc, c.sms * 2, p.KS, p.kchunk);
        if (p.tc64) {
            p.NT = 2 * p.z.NT;  // its partial slots: the re and im half of each 64-wide n-tile
            p.KS = p.z.KS;
            p.zA = p.z.bytesA;
            p.zB = p.z.bytesB;
            p.zEa = p.z.bytesEa;
            p.zEb = p.z.bytesEb;
            p.zW = (size_t)r.ng * M * sizeof(double2);
            p.zG = p.z.guard_bytes(M, 3, 1);
        }
    }
    const int BM = p.mixed ? f32::BM : d64::BM, BN = p.mixed ? f32::BN : d64::BN;
    p.MTs = ceil_div(r.nb, BM);
    p.NTs = ceil_div(r.ng, BN);
    if (p.mixed) {
        // one block per SM (its registers): the k-slices that fill one wave, of at least
        // 64 k-values; the FP32 sums run over 16-wide k-steps whatever the slice
        const int ks = std::max(1, std::min(c.sms / std::max(1, p.MTs * p.NTs), std::max(1, r.nc / 64)));
        p.kchunks = ceil_div(ceil_div(r.nc, ks), 16) * 16;
        p.KSs = ceil_div(r.nc, p.kchunks);
    } else {
        pick_split(p.MTs * p.NTs, r.nc, c.sms * 2, p.KSs, p.kchunks);
    }
    if (p.tc64 && (r.flags & FK_GPP_ACHSTEMP)) {
        p.NTs = 2 * p.zs.NT;
        p.KSs = p.zs.KS;
        p.zA = std::max(p.zA, p.zs.bytesA);
        p.zB = std::max(p.zB, p.zs.bytesB);
        p.zEa = std::max(p.zEa, p.zs.bytesEa);
        p.zEb = std::max(p.zEb, p.zs.bytesEb);
        p.zW = (size_t)r.ng * r.nb * sizeof(double2);
        p.zG = std::max(p.zG, p.zs.guard_bytes(r.nb, 1, 1));
    }
    p.bytesD = M <= 0 ? 0
               : p.mixed ? (size_t)p.NT * p.kstages * tcx::Cfg<64>::B_BYTES
                         : (size_t)N * r.nc * sizeof(double2);
    p.bytesW = (p.mixed && M > 0) ? (size_t)M * r.ng * sizeof(float2) : 0;
    p.bytesF = (size_t)p.nch * std::max(r.nv, 1) * r.ng * (half ? 12 : 6) * sizeof(double2);
    p.bytesP = M > 0 ? (size_t)p.KS * p.NT * M * 3 * sizeof(double2) : 0;
    p.bytesS = (r.flags & FK_GPP_ACHSTEMP) ? (size_t)p.KSs * p.NTs * r.nb * sizeof(double2) : 0;
    p.bytesRows = rows_bytes(r.nb);
    p.bytesIgp = 2 * (size_t)r.ng * sizeof(int);  // igp, acol
    return p;
}

// FP64 on the tensor cores: takes its workspace / runs one contraction.
bool take_tc64(Ctx& c, const Plan& p, tc64::Bufs& b) {
    if (!p.tc64) return true;
    b.A = (uint8_t*)c.ws.take(p.zA);
    b.B = (uint8_t*)c.ws.take(p.zB);
    b.ea = (int*)c.ws.take(p.zEa);
    b.eb = (int*)c.ws.take(p.zEb);
    b.W1 = (double2*)c.ws.take(p.zW);
    b.W2 = nullptr;
    b.planes = 1;
    b.guard_bytes = p.zG;
    b.guard = (uint8_t*)c.ws.take(p.zG);
    return b.A && b.B && b.ea && b.eb && b.W1 && b.guard;
}
template <int EPI>
cudaError_t run_tc64(Ctx& c, const ContractArgs& a, const tc64::Plan& z, const tc64::Bufs& b, bool have_a = false,
                     bool re_only = false) {
    tc64::enqueue_weights(c, a, EPI == EPI_GPP ? a.N / 3 : a.N, b, false);
    const cudaError_t e = have_a ? cudaSuccess : tc64::enqueue_a(c, a, z, b);
    if (e == cudaSuccess) tc64::enqueue<EPI>(c, a, z, b, tc64::one_plane(z), 0, re_only);
    return e;
}

struct CudaApi {
    using Stream = cudaStream_t;
    using Event = cudaEvent_t;
    using Error = cudaError_t;
    Error record(Event e, Stream s) { return cudaEventRecord(e, s); }
    Error wait(Stream s, Event e) { return cudaStreamWaitEvent(s, e, 0); }
    Error synchronize(Stream s) { return cudaStreamSynchronize(s); }
    bool capturing(Stream s) {
        cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
        return cudaStreamIsCapturing(s, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone;
    }
    void clear() { cudaGetLastError(); }
};
// (no side stream: none yet, and the caller captures)
struct SideBranch : Branch<CudaApi> {
    explicit SideBranch(Ctx& c)
        : Branch(CudaApi{}, c.stream, side_ready(c) == FK_OK ? c.copy_stream : nullptr, c.pipe_ev[0], c.pipe_ev[1]) {}
};

template <class K>
cudaError_t set_smem(K kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// ----------------------------------------------------- real-valued sum (gppKer_real.cpp)
// The real driver's noflag blocks (gppKer_real.cpp:341-383) keep one scha[512]
// per (n1, my_igp) across blocks and frequencies and assign scha[ig] only
// where the mask holds; every block sum adds all of scha[0 .. igend).  The
// mask and delw*I_eps depend on (my_igp, iw, ig) alone, so for each block
// offset j the value in scha[j] at any step comes from a source element
// (g = 512*b' + j, iw') fixed by the inputs, and
//   sch_array[iw] = 0.5 * aqsm[n1][igp] * sum_g aqsn[n1][g] * E[my_igp][iw][g]
// where E[iw][g] adds D(g, iw') once for every block sum of frequency iw that
// found (g, iw') in scha[j].  The prep evaluates the mask and D; the carry
// kernel replays the reference program's sequence per (my_igp, j) and writes E.
//
// A real dot product is the real part of a complex one over half the length:
// with a[k] = A[2k] + i A[2k+1] (the row of doubles read as complex pairs, in
// place) and b[k] = E[2k] - i E[2k+1], Re(a[k] b[k]) = A[2k] E[2k] + A[2k+1] E[2k+1].
// So E is written in that pair form and the complex contraction engines run
// unchanged over ncouls/2 (rounded up) pairs; the per-band reduction keeps
// the real part.

struct RealPrepArgs {
    int nb, nv, nc, ng;
    const double *aqsn, *eps, *wt, *wx;
    long lda;          // row stride of aqsn
    const int* igp;
    double* Dv;        // [ng][3][nc] delw*I_eps of every element; nullptr = not written by this pass
    uint8_t* mask;     // [ng][nc] bit iw: the noflag mask of (iw, ig)
    double2* F;        // [nch][nv][ng][6] flag-band (sch, ssx) sums, as (value, 0)
    int nch, n1base;
    int tile;          // plane waves per chunk (a multiple of PREP_THREADS)
};

// Per element: the noflag mask and value (gppKer_real.cpp:351-366) and, for
// the flag bands of this pass, ssxt_scht_solver's sch and ssx (:17-63) times
// aqsn[n1][ig] (flagOCC_solver :124-153), FP64 round-to-nearest without
// contraction so that every branch matches the reference's.
__global__ void __launch_bounds__(PREP_THREADS) real_prep_kernel(RealPrepArgs p) {
    __shared__ double2 sm[8 * NVC * 6];
    const int my_igp = blockIdx.y, ch = blockIdx.x, tid = threadIdx.x;
    const int igp = p.igp[my_igp];
    const int nflag = igp < 0 ? 0 : min(NVC, p.nv - p.n1base);
    const double to1 = 1e-6, limitone = 1.0 / (to1 * 4.0), limittwo = 0.25;
    double2 acc[NVC * 6];
#pragma unroll
    for (int i = 0; i < NVC * 6; ++i) acc[i] = make_double2(0.0, 0.0);
    for (int ig = ch * p.tile + tid; ig < min(p.nc, (ch + 1) * p.tile); ig += PREP_THREADS) {
        const double w = p.wt[(long)my_igp * p.nc + ig], ep = p.eps[(long)my_igp * p.nc + ig];
        const double w2 = __dmul_rn(w, w), Om = __dmul_rn(w2, ep);
        int bits = 0;
#pragma unroll
        for (int iw = 0; iw < 3; ++iw) {
            const double wxt = p.wx[iw];
            const double wdiff = __dsub_rn(wxt, w);
            const double rden = __ddiv_rn(1.0, __dmul_rn(wdiff, wdiff));
            const double delw = __dmul_rn(__dmul_rn(w, wdiff), rden);
            const double delwr = __dmul_rn(delw, delw), wdiffr = __dmul_rn(wdiff, wdiff);
            const bool A = wdiffr > limittwo && delwr < limitone;
            if (p.Dv) {
                p.Dv[((long)my_igp * 3 + iw) * p.nc + ig] = __dmul_rn(delw, ep);
                bits |= (int)A << iw;
            }
            if (nflag > 0) {
                double sch = 0.0, ssx = 0.0;
                if (A) {
                    sch = __dmul_rn(delw, ep);
                    const double cden = __dmul_rn(wxt, wxt);
                    ssx = __dmul_rn(__dmul_rn(Om, cden), __ddiv_rn(1.0, __dmul_rn(cden, cden)));
                } else if (delwr > to1) {
                    const double cden = __dmul_rn(__dmul_rn(4.0, w2), __dadd_rn(delw, 0.5));
                    ssx = __dmul_rn(__dmul_rn(__dmul_rn(0.0 - Om, cden), __ddiv_rn(1.0, __dmul_rn(cden, cden))), delw);
                }
#pragma unroll
                for (int j = 0; j < NVC; ++j)
                    if (j < nflag) {
                        const double an = p.aqsn[(long)(p.n1base + j) * p.lda + ig];
                        acc[(j * 3 + iw) * 2 + 0].x = __dadd_rn(acc[(j * 3 + iw) * 2 + 0].x, __dmul_rn(an, sch));
                        acc[(j * 3 + iw) * 2 + 1].x = __dadd_rn(acc[(j * 3 + iw) * 2 + 1].x, __dmul_rn(an, ssx));
                    }
            }
        }
        if (p.Dv) p.mask[(long)my_igp * p.nc + ig] = (uint8_t)bits;
    }
    if (p.nv - p.n1base <= 0) return;
    block_sum<NVC * 6>(acc, sm);
    const int nf = min(NVC, p.nv - p.n1base);
    if (tid < nf * 6) {
        const int j = tid / 6, r = tid % 6;
        p.F[(((long)ch * p.nv + p.n1base + j) * p.ng + my_igp) * 6 + r] = acc[tid];
    }
}

// Mixed precision: the branch quantities of real_prep_kernel in FP32 from an FP64
// wx - wtilde, the FP64 sequence inside a relative guard band of 1e-5 around
// every threshold (so every branch is the FP64 one), flag-band sums in FP32
// float-float.  Dv and the mask mean what they mean in the FP64 kernel.
struct RealTerm {
    double dv, sch, ssx;
    int A;
};
__device__ __noinline__ RealTerm real_term_rare(double wxt, double w, double ep) {
    const double to1 = 1e-6, limitone = 1.0 / (to1 * 4.0), limittwo = 0.25;
    const double w2 = __dmul_rn(w, w), Om = __dmul_rn(w2, ep);
    const double wdiff = __dsub_rn(wxt, w);
    const double rden = __ddiv_rn(1.0, __dmul_rn(wdiff, wdiff));
    const double delw = __dmul_rn(__dmul_rn(w, wdiff), rden);
    const double delwr = __dmul_rn(delw, delw), wdiffr = __dmul_rn(wdiff, wdiff);
    RealTerm t;
    t.A = wdiffr > limittwo && delwr < limitone;
    t.dv = __dmul_rn(delw, ep);
    t.sch = 0.0;
    t.ssx = 0.0;
    if (t.A) {
        t.sch = t.dv;
        const double cden = __dmul_rn(wxt, wxt);
        t.ssx = __dmul_rn(__dmul_rn(Om, cden), __ddiv_rn(1.0, __dmul_rn(cden, cden)));
    } else if (delwr > to1) {
        const double cden = __dmul_rn(__dmul_rn(4.0, w2), __dadd_rn(delw, 0.5));
        t.ssx = __dmul_rn(__dmul_rn(__dmul_rn(0.0 - Om, cden), __ddiv_rn(1.0, __dmul_rn(cden, cden))), delw);
    }
    return t;
}

// The chunks make one wave of four blocks per SM (make_real_plan): 64 registers.  At 78,
// three blocks, the wave was not one: 44 us at 512 x 32768 x 20, now 32 (the call 129 -> 117).
__global__ void __launch_bounds__(PREP_THREADS, 4) real_prep_mixed_kernel(RealPrepArgs p) {
    __shared__ double2 sm[8 * NVC * 6];
    const int my_igp = blockIdx.y, ch = blockIdx.x, tid = threadIdx.x;
    const int igp = p.igp[my_igp];
    const int nflag = igp < 0 ? 0 : min(NVC, p.nv - p.n1base);
    const float to1 = 1e-6f, limitone = 250000.0f, limittwo = 0.25f;
    float2 acc[NVC * 6];
#pragma unroll
    for (int i = 0; i < NVC * 6; ++i) acc[i] = make_float2(0.f, 0.f);
    double wx64[3];
    float wxsq[3];
#pragma unroll
    for (int iw = 0; iw < 3; ++iw) {
        wx64[iw] = p.wx[iw];
        const float wf = f64_to_f32_bits(wx64[iw]);
        wxsq[iw] = wf * wf;
    }
    for (int ig = ch * p.tile + tid; ig < min(p.nc, (ch + 1) * p.tile); ig += PREP_THREADS) {
        const double w64 = p.wt[(long)my_igp * p.nc + ig], ep64 = p.eps[(long)my_igp * p.nc + ig];
        const float w = f64_to_f32_bits(w64), ep = f64_to_f32_bits(ep64);
        const float w2 = w * w, Om = w2 * ep;
        float an[NVC];
#pragma unroll
        for (int j = 0; j < NVC; ++j) an[j] = j < nflag ? f64_to_f32_bits(p.aqsn[(long)(p.n1base + j) * p.lda + ig]) : 0.f;
        int bits = 0;
#pragma unroll
        for (int iw = 0; iw < 3; ++iw) {
            const double wd64 = __dsub_rn(wx64[iw], w64);
            const float wdiff = f64_to_f32_bits(wd64);
            const float wdiffr = wdiff * wdiff;
            const float delw = __fdiv_rn(w, wdiff);  // = w*wdiff/wdiff^2, correctly rounded
            const float delwr = delw * delw;
            const bool amb = !(wdiffr > 1e-30f) || !(delwr < 1e30f) || fabsf(wdiffr - limittwo) <= limittwo * GUARD ||
                             fabsf(delwr - limitone) <= limitone * GUARD ||
                             (nflag > 0 && fabsf(delwr - to1) <= to1 * GUARD);
            bool A;
            float dv, sch = 0.f, ssx = 0.f;
            double dv64;
            if (__any_sync(__activemask(), amb) && amb) {
                const RealTerm t = real_term_rare(wx64[iw], w64, ep64);
                A = t.A != 0;
                dv64 = t.dv;
                dv = f64_to_f32_bits(t.dv);
                sch = f64_to_f32_bits(t.sch);
                ssx = f64_to_f32_bits(t.ssx);
            } else {
                A = wdiffr > limittwo && delwr < limitone;
                // the value to FP64 accuracy (it is summed, then rounded once for the
                // tensor cores): one FP64 correction of the FP32 quotient w / wdiff
                double q = f32_to_f64_bits(delw);
                q = __fma_rn(__fma_rn(-q, wd64, w64), f32_to_f64_bits(__frcp_rn(wdiff)), q);
                dv64 = __dmul_rn(q, ep64);
                dv = f64_to_f32_bits(dv64);
                if (A) {
                    sch = dv;
                    ssx = __fdiv_rn(Om, wxsq[iw]);
                } else if (delwr > to1) {
                    const float cden = 4.f * w2 * (delw + 0.5f);
                    ssx = __fdiv_rn(-Om * delw, cden);
                }
            }
            if (p.Dv) {
                p.Dv[((long)my_igp * 3 + iw) * p.nc + ig] = dv64;
                bits |= (int)A << iw;
            }
#pragma unroll
            for (int j = 0; j < NVC; ++j) {
                acc[(j * 3 + iw) * 2 + 0].x = fmaf(an[j], sch, acc[(j * 3 + iw) * 2 + 0].x);
                acc[(j * 3 + iw) * 2 + 1].x = fmaf(an[j], ssx, acc[(j * 3 + iw) * 2 + 1].x);
            }
        }
        if (p.Dv) p.mask[(long)my_igp * p.nc + ig] = (uint8_t)bits;
    }
    if (p.nv - p.n1base <= 0) return;
    double2 accd[NVC * 6];
    block_sum_ff<NVC * 6>(acc, sm, accd);
    const int nf = min(NVC, p.nv - p.n1base);
    if (tid < nf * 6) {
        const int j = tid / 6, r = tid % 6;
#pragma unroll
        for (int i = 0; i < NVC * 6; ++i)
            if (i == tid) p.F[(((long)ch * p.nv + p.n1base + j) * p.ng + my_igp) * 6 + r] = accd[i];
    }
}

struct RealCarryArgs {
    int nc, ng;
    long K2;             // complex pairs per row of the operand
    const int* igp;
    const double* Dv;
    const uint8_t* mask;
    int carry;           // 1: the reference program's stale scha; 0: a masked term contributes 0
    double* D64;         // FP64 operand rows [3*ng][2*K2] (pair form), or nullptr
    uint8_t* img;        // mixed: the pre-split B image, or nullptr
    int kstages;
};

// At block offset j the reference program's block sums happen at times t = 3*b + iw
// (block b, frequency iw) for the blocks that reach j; the source of scha[j]
// changes at the times whose mask bit is set.  A source (g, iw') set at t0 and
// replaced at t1 adds D(g, iw') to E[iw][g] once for every t in [t0, t1) with
// t = iw (mod 3), so
//   E[iw][g] = sum over set bits iw' of g's mask of D(g, iw') * #{t in [t0, t1): t = iw mod 3},
// t1 being the next set bit of the same block, else the first set time of a
// later block at the same offset.  E of an element thus depends on its own
// mask and values and on that first later set time only: one thread per
// element, looking ahead through the masks of the later blocks (usually one).
// Bound: FP64 instructions (64 cycles each).  The usual element has one source per iw
// that lasts one time, and needs none; signs and counts are formed in FP32.
// 512 x 32768 x 20 mixed: 30 -> 13 us.
template <int IMG>
__global__ void real_carry_kernel(RealCarryArgs a) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long)a.ng * a.nc) return;
    const int my_igp = (int)(t / a.nc), g = (int)(t % a.nc);
    auto put = [&](int iw, int gg, double v) {
        if (IMG) {
            const int nt = my_igp / GPP_COLS, row = (my_igp % GPP_COLS) * 3 + iw;
            const float f = f64_to_f32_bits(v);
            tcx::bimg_store_part<64>(a.img + (long)nt * a.kstages * tcx::Cfg<64>::B_BYTES, row, gg >> 1, gg & 1,
                                     (gg & 1) ? 0.f - f : f);
        } else {
            a.D64[((long)my_igp * 3 + iw) * 2 * a.K2 + gg] = (gg & 1) ? 0.0 - v : v;
        }
    };
    const uint8_t* mrow = a.mask + (long)my_igp * a.nc;
    const int m = a.igp[my_igp] >= 0 ? mrow[g] : 0;
    double e[3] = {0.0, 0.0, 0.0};
    if (m) {
        double dv[3];
#pragma unroll
        for (int iw = 0; iw < 3; ++iw) dv[iw] = a.Dv[((long)my_igp * 3 + iw) * a.nc + g];
        if (!a.carry) {
#pragma unroll
            for (int iw = 0; iw < 3; ++iw) e[iw] = ((m >> iw) & 1) ? dv[iw] : 0.0;
        } else {
            const int j = g & 511, b = g >> 9;
            int tnext = 3 * ((a.nc - j + 511) / 512);  // no later set time: the end of offset j's blocks
            for (int g2 = g + 512; g2 < a.nc; g2 += 512) {
                const int m2 = mrow[g2];
                if (m2) {
                    tnext = 3 * (g2 >> 9) + __ffs(m2) - 1;
                    break;
                }
            }
            auto upto = [](int T, int iw) { return (T - iw + 2) / 3; };  // #{t < T : t = iw mod 3}
            int touched = 0;
#pragma unroll
            for (int ws = 0; ws < 3; ++ws) {
                if (!((m >> ws) & 1)) continue;
                const int t0 = 3 * b + ws, later = m >> (ws + 1);
                const int t1 = later ? t0 + __ffs(later) : tnext;
#pragma unroll
                for (int iw = 0; iw < 3; ++iw) {
                    const int n = upto(t1, iw) - upto(t0, iw);
                    // e[iw] still 0: 1 * D + 0 is D, and the first term needs no addition
                    if (n == 1 && !(touched >> iw & 1)) e[iw] = dv[ws];
                    else if (n) e[iw] = __fma_rn(f32_to_f64_bits((float)n), dv[ws], e[iw]);
                    touched |= (n ? 1 : 0) << iw;
                }
            }
        }
    }
#pragma unroll
    for (int iw = 0; iw < 3; ++iw) put(iw, g, e[iw]);
    // odd ncouls: the imaginary half of the last pair has no element behind it
    if ((a.nc & 1) && g == a.nc - 1)
        for (int iw = 0; iw < 3; ++iw) put(iw, a.nc, 0.0);
}

}  // namespace

size_t gpp_workspace(const Ctx& c, const GppDev& r, bool pipelined) {
    Plan p = make_plan(c, r, 0, pipelined, gpp_pair(r, pipelined), gpp_fsch(r));
    const size_t half = (r.flags & FK_GPP_HALF_SUM) ? p.bytesP + (size_t)r.ng * (4 * HALF_CHUNKS + 3 * sizeof(double2)) + 768 : 0;
    const size_t wf = (size_t)r.nv * r.ng * 2 * sizeof(double2);
    // the error estimate's column magnitudes, row norms and band bounds (when on)
    const size_t est = (c.est_on && p.mixed)
                           ? (size_t)p.nch * r.ng * 18 * sizeof(float) + (size_t)r.nb * (sizeof(float2) + 6 * sizeof(double)) + 768
                           : 0;
    return p.bytesD + p.bytesF + p.bytesP + p.bytesS + p.bytesRows + p.bytesIgp + p.bytesW + p.bytesAimg + half + wf + est +
           p.bytesZ() + 16 * 256;
}

int gpp_pipe_chunks(const Ctx& c, const GppDev& r) { return make_plan(c, r, 0, true, false, gpp_fsch(r)).pipe_chunks; }

fk_status side_ready(Ctx& c) {
    if (!c.copy_stream) {
        // not created while the caller captures the stream
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(c.stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
            cudaGetLastError();
            return FK_ENOTSUP;
        }
        if (cudaStreamCreateWithFlags(&c.copy_stream, cudaStreamNonBlocking) != cudaSuccess)
            return cuda_fail(c, cudaGetLastError(), "pipeline: copy stream");
    }
    for (auto& e : c.pipe_ev)
        if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess)
            return cuda_fail(c, cudaGetLastError(), "pipeline: events");
    return FK_OK;
}

fk_status pipe_begin(Ctx& c) {
    const fk_status s = side_ready(c);
    if (s != FK_OK) return s;
    // the destinations are free once the work queued before this call is done
    cudaError_t e = cudaEventRecord(c.pipe_ev[PIPE_FREE], c.stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(c.copy_stream, c.pipe_ev[PIPE_FREE], 0);
    return e == cudaSuccess ? FK_OK : cuda_fail(c, e, "pipeline: start");
}

fk_status gpp_pipe_copy(Ctx& c, const GppDev& r, const GppPipe* pipe, int q0, int q1) {
    const Plan p = make_plan(c, r, 0, true, false, gpp_fsch(r));
    const size_t rowb = (size_t)r.nc * sizeof(double2);
    for (int q = q0; q < std::min(q1, p.pipe_chunks); ++q) {
        // rows of m-tiles q*pipe_sub .. (from band m0); block 0 also carries the flag bands 0 .. nvband-1
        const long r0 = q == 0 ? 0 : p.m0 + (long)q * p.pipe_sub * tcx::BM;
        const long r1 = std::min((long)r.nb, p.m0 + (long)(q + 1) * p.pipe_sub * tcx::BM);
        cudaError_t e = cudaMemcpyAsync(pipe->aqsn_d + r0 * r.nc, pipe->aqsn + r0 * r.nc, (size_t)(r1 - r0) * rowb,
                                        cudaMemcpyHostToDevice, c.copy_stream);
        if (e == cudaSuccess) e = cudaEventRecord(c.pipe_ev[q], c.copy_stream);
        if (e != cudaSuccess) return cuda_fail(c, e, "gpp: block copy");
        c.h2d_bytes += (size_t)(r1 - r0) * rowb;
    }
    return FK_OK;
}

// The half-sum mode (FK_GPP_HALF_SUM): prep in FP64, then the contraction of
// the image with A = aqsntemp (partials P) and with A = aqsmtemp (partials P2).
fk_status gpp_run_half(Ctx& c, const GppDev& r) {
    const Plan p = make_plan(c, r);
    cudaStream_t st = c.stream;
    const int M = r.nb - r.nv;
    int* igp = (int*)c.ws.take(p.bytesIgp);
    int* acol = igp ? igp + r.ng : nullptr;
    void* D = p.bytesD ? c.ws.take(p.bytesD) : nullptr;
    double2* F = (double2*)c.ws.take(p.bytesF);
    double2* P = p.bytesP ? (double2*)c.ws.take(p.bytesP) : nullptr;
    double2* P2 = p.bytesP ? (double2*)c.ws.take(p.bytesP) : nullptr;
    double2* rows = (double2*)c.ws.take(p.bytesRows);
    float2* W = p.bytesW ? (float2*)c.ws.take(p.bytesW) : nullptr;
    int* brk = (int*)c.ws.take((size_t)r.ng * HALF_CHUNKS * sizeof(int));
    double2* schd = (double2*)c.ws.take((size_t)r.ng * 3 * sizeof(double2));
    int* counter = (int*)c.ws.take(sizeof(int));
    tc64::Bufs zb{};
    if (!take_tc64(c, p, zb)) return fail(c, FK_ENOMEM, "workspace too small for GPP request");
    if (!igp || !F || !rows || !brk || !schd || !counter || (p.bytesD && !D) || (p.bytesP && (!P || !P2)) || (p.bytesW && !W))
        return fail(c, FK_ENOMEM, "workspace too small for GPP request");
    if (r.aqsm_compact || r.ldm != r.nc) return fail(c, FK_EINVAL, "gpp: the half sum needs all of aqsmtemp");
    c.launches = 0;
    phase_mark(c, 1);
    SetupArgs sa{};
    sa.nb = r.nb; sa.nv = r.nv; sa.nc = r.nc; sa.ng = r.ng;
    sa.inv = r.inv; sa.indinv = r.indinv; sa.igp = igp; sa.acol = acol; sa.vcoul = r.vcoul;
    sa.W = p.mixed && M > 0 ? W : nullptr;
    sa.counter = counter;
    sa.err = (p.mixed || p.tc64) && D ? c.errword : nullptr;
    if (p.mixed && D && tcx::img_needs_pad(64, r.ng, GPP_COLS, r.nc)) sa.img = (uint8_t*)D;
    sa.NT = p.NT; sa.kstages = p.kstages; sa.K = r.nc;
    sa.aqsm = r.aqsm; sa.eps = r.eps; sa.wt = r.wt; sa.wx = r.wx; sa.brk = brk; sa.schd = schd;
    launch_setup(sa, st);
    ++c.launches;
    for (int pass = 0; pass < p.passes; ++pass) {
        PrepArgs a{r.nb, r.nv, r.nc, r.ng, r.aqsn, r.eps, r.wt, r.wx, igp, (pass == 0 && M > 0) ? D : nullptr,
                   p.kstages, F, p.nch, p.tile, pass * NVC, 0, r.aqsm, brk};
        if (p.mixed) prep_half_mixed_kernel<<<dim3(p.nch, r.ng), PREP_THREADS, 0, st>>>(a);
        else prep_half_kernel<<<dim3(p.nch, r.ng), PREP_THREADS, 0, st>>>(a);
        ++c.launches;
    }
    phase_mark(c, 2);
    for (int pass = 0; pass < 2 && M > 0; ++pass) {
        const double2* A = pass == 0 ? r.aqsn : r.aqsm;
        ContractArgs a{};
        a.A = A; a.lda = r.nc; a.m0 = r.nv; a.M = M;
        a.B = D; a.ldb = r.nc; a.bstride = 0; a.N = 3 * r.ng; a.K = r.nc;
        a.KS = p.KS; a.kchunk = p.kchunk; a.batches = 1; a.batch_plane = nullptr;
        a.aqsm = r.aqsm; a.ldm = r.ldm; a.vcoul = r.vcoul; a.igp = igp; a.acol = acol; a.wscale = 0.5; a.G = 3;
        a.P = pass == 0 ? P : P2;
        if (p.mixed) {
            tcx::TcArgs t{};
            t.c = a;
            t.Bimg = (const uint8_t*)D;
            t.W1 = W; t.W2 = nullptr; t.ldw = M; t.gpp_cols = GPP_COLS; t.Aimg = nullptr; t.vcol = nullptr;
            t.kstages_total = p.kstages;
            t.MT = p.MT; t.NT = p.NT; t.units = p.units;
            t.err = c.errword;
            t.wait_limit = c.wait_limit;
            if (tcx::encode_rows_map(&t.amap, A, r.nc, r.nc, r.nb) != cudaSuccess)
                return fail(c, FK_ECUDA, "gpp: cannot describe an input as a tensor map (needs a 16-byte aligned array)");
            auto k = tcx::tc_contract_kernel<EPI_GPP, 64, false>;
            set_smem(k, tcx::Cfg<64>::SMEM);
            kernel_begin(c);
            k<<<std::min(p.units, c.sms), tcx::THREADS, tcx::Cfg<64>::SMEM, st>>>(t);
            kernel_end(c);
        } else if (p.tc64) {
            const cudaError_t e = run_tc64<EPI_GPP>(c, a, p.z, zb);
            if (e != cudaSuccess) return cuda_fail(c, e, "gpp: digits");
            continue;
        } else {
            auto k = d64::contract_kernel<EPI_GPP>;
            set_smem(k, d64::SMEM);
            kernel_begin(c);
            k<<<dim3(p.MT, p.NT * p.KS), d64::THREADS, d64::SMEM, st>>>(a, d64::Redo{});
            kernel_end(c);
        }
        ++c.launches;
    }
    phase_mark(c, 3);
    RowsArgs ra{r.nb, r.nv, r.ng, P ? p.KS * p.NT : 0, P, 0, nullptr, p.nch, F, r.ldm, r.aqsm, r.vcoul, igp, acol, rows};
    ra.P2 = P2 ? P2 : (const double2*)F;  // non-null selects the half sum even without contraction partials
    ra.schd = schd;
    ra.aqsn = r.aqsn;
    ra.nc = r.nc;
    ra.counter = counter;  // the last block also writes the totals
    ra.out = r.out;
    rows_kernel<<<rows_blocks(r.nb, r.nv), ROWS_THREADS, 0, st>>>(ra);
    ++c.launches;
    phase_mark(c, 4);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FK_OK : cuda_fail(c, e, "gpp kernels (half sum)");
}

fk_status gpp_run(Ctx& c, const GppDev& r, const GppPipe* pipe) {
    if (r.flags & FK_GPP_HALF_SUM) return pipe ? fail(c, FK_EINVAL, "gpp: no pipelined half sum") : gpp_run_half(c, r);
    const Plan p = make_plan(c, r, 0, pipe != nullptr, gpp_pair(r, pipe != nullptr), gpp_fsch(r));
    if (pipe && !p.pipe_chunks) return fail(c, FK_EINVAL, "gpp: pipelined staging needs the mixed path");
    cudaStream_t st = c.stream;
    int* igp = (int*)c.ws.take(p.bytesIgp);
    int* acol = igp + r.ng;
    void* D = p.bytesD ? c.ws.take(p.bytesD) : nullptr;
    double2* F = (double2*)c.ws.take(p.bytesF);
    double2* P = p.bytesP ? (double2*)c.ws.take(p.bytesP) : nullptr;
    double2* S = p.bytesS ? (double2*)c.ws.take(p.bytesS) : nullptr;
    double2* rows = (double2*)c.ws.take(p.bytesRows);
    float2* W = p.bytesW ? (float2*)c.ws.take(p.bytesW) : nullptr;
    int* counter = (int*)c.ws.take(sizeof(int));
    double2* wf = r.nv > 0 ? (double2*)c.ws.take((size_t)r.nv * r.ng * 2 * sizeof(double2)) : nullptr;
    // error estimate: the prep's column magnitudes, the bands' row norms and bounds
    const bool est = c.est_on && p.mixed && c.est_dev;
    float* estE = est ? (float*)c.ws.take((size_t)p.nch * r.ng * 18 * sizeof(float)) : nullptr;
    float2* estA = est ? (float2*)c.ws.take((size_t)r.nb * sizeof(float2)) : nullptr;
    double* estB = est ? (double*)c.ws.take((size_t)r.nb * 6 * sizeof(double)) : nullptr;
    uint8_t* Aimg = p.bytesAimg ? (uint8_t*)c.ws.take(p.bytesAimg) : nullptr;
    if (!igp || !F || !rows || !counter || (p.bytesD && !D) || (p.bytesP && !P) || (p.bytesS && !S) ||
        (p.bytesW && !W) || (r.nv > 0 && !wf) || (est && (!estE || !estA || !estB)) || (p.bytesAimg && !Aimg))
        return fail(c, FK_ENOMEM, "workspace too small for GPP request");
    tc64::Bufs zb{};
    if (!take_tc64(c, p, zb)) return fail(c, FK_ENOMEM, "workspace too small for GPP request");
    if (p.tc64 && D) {  // (mixed: the prep clears it)
        cudaError_t e = cudaMemsetAsync(c.errword, 0, sizeof(int), st);  // bounded-wait status
        if (e != cudaSuccess) return cuda_fail(c, e, "gpp: error word");
    }
    // prep variant: 0 = BGW-Kernels/gppKer.cpp, 1 = root gppKer.cpp, 2 = the Fortran source
    const int Q = (r.flags & FK_GPP_ROOT_QUIRKS) ? 1 : (r.flags & FK_GPP_PHYSICS) ? 2 : 0;
    const int M = r.nb - p.m0;  // contraction rows: bands m0 .. nb-1
    c.launches = 0;
    // the first prep pass also maps the columns, writes the epilogue weights and
    // the image's padding, and clears the reduction's counter
    auto prep_args = [&](int pass) {
        PrepArgs a{r.nb, r.nv, r.nc, r.ng, r.aqsn, r.eps, r.wt, r.wx, igp, pass == 0 ? D : nullptr, p.kstages,
                   F, p.nch, p.tile, pass * NVC, 0};
        if (pass == 0) {
            a.setup = 1;
            a.inv = r.inv; a.indinv = r.indinv;
            a.igp_out = igp; a.acol_out = acol;
            a.compact = r.aqsm_compact ? 1 : 0;
            a.aqsm = r.aqsm; a.ldm = r.ldm; a.vcoul = r.vcoul;
            a.W = (p.mixed && M > 0) ? W : nullptr;
            a.M = M;
            a.wm0 = p.m0;
            a.err = p.mixed && D ? c.errword : nullptr;
            a.counter = counter;
            a.wf = wf;
            a.asx_neg = Q == 2;
            a.est = estE;
        }
        return a;
    };
    auto launch_prep = [&](const PrepArgs& a, dim3 grid) {
        if (p.mixed && p.fsch) {
            // the flag bands' ssx sums only (their sch terms go through the contraction);
            // fsch excludes the root file's variant (Q == 1)
            if (a.est) {
                if (Q == 2) prep_mixed_kernel<2, 64, true, false><<<grid, PREP_THREADS, 0, st>>>(a);
                else prep_mixed_kernel<0, 64, true, false><<<grid, PREP_THREADS, 0, st>>>(a);
            } else {
                if (Q == 2) prep_mixed_kernel<2, 64, false, false><<<grid, PREP_THREADS, 0, st>>>(a);
                else prep_mixed_kernel<0, 64, false, false><<<grid, PREP_THREADS, 0, st>>>(a);
            }
        } else if (p.mixed && a.est) {
            if (Q == 1) prep_mixed_kernel<1, 64, true><<<grid, PREP_THREADS, 0, st>>>(a);
            else if (Q == 2) prep_mixed_kernel<2, 64, true><<<grid, PREP_THREADS, 0, st>>>(a);
            else prep_mixed_kernel<0, 64, true><<<grid, PREP_THREADS, 0, st>>>(a);
        } else if (p.mixed) {
            if (Q == 1) prep_mixed_kernel<1, 64><<<grid, PREP_THREADS, 0, st>>>(a);
            else if (Q == 2) prep_mixed_kernel<2, 64><<<grid, PREP_THREADS, 0, st>>>(a);
            else prep_mixed_kernel<0, 64><<<grid, PREP_THREADS, 0, st>>>(a);
        } else {
            auto k = p.fsch ? (Q == 2 ? prep64_kernel<2, false> : prep64_kernel<0, false>)
                            : (Q == 1 ? prep64_kernel<1, true> : Q == 2 ? prep64_kernel<2, true> : prep64_kernel<0, true>);
            // blocks of the digit conversion share the SM with it (p.tc64): the same split of
            // the SM's memory between L1 and shared memory
            if (p.tc64) cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
            k<<<grid, PREP_THREADS, 0, st>>>(a);
        }
        ++c.launches;
    };

    phase_mark(c, 1);
    if (pipe && cudaStreamWaitEvent(st, c.pipe_ev[PIPE_READY], 0) != cudaSuccess)
        return cuda_fail(c, cudaGetLastError(), "gpp: waiting for the small inputs");
    // pipelined host path: the prep waits for row block 0 (the flag bands), each
    // block's contraction for its own copy
    if (pipe) {
        if (cudaStreamWaitEvent(st, c.pipe_ev[0], 0) != cudaSuccess)
            return cuda_fail(c, cudaGetLastError(), "gpp: waiting for a block");
        for (int pass = 0; pass < p.passes; ++pass) launch_prep(prep_args(pass), dim3(p.nch, r.ng));
        if (p.mixed && M > 0) {
            ContractArgs a{};
            a.A = r.aqsn; a.lda = r.nc; a.m0 = p.m0; a.M = M;
            a.B = D; a.ldb = r.nc; a.bstride = 0; a.N = 3 * r.ng; a.K = r.nc;
            a.KS = p.KS; a.kchunk = p.kchunk; a.batches = 1; a.batch_plane = nullptr;
            a.aqsm = r.aqsm; a.ldm = r.ldm; a.vcoul = r.vcoul; a.igp = igp; a.acol = acol; a.wscale = 0.5; a.G = 3;
            a.P = P;
            tcx::TcArgs t{};
            t.c = a;
            t.Bimg = (const uint8_t*)D;
            t.W1 = W; t.W2 = nullptr; t.ldw = M; t.gpp_cols = GPP_COLS; t.Aimg = nullptr; t.vcol = nullptr;
            t.kstages_total = p.kstages;
            t.NT = p.NT;
            t.err = c.errword;
            t.wait_limit = c.wait_limit;
            if (tcx::encode_rows_map(&t.amap, r.aqsn, r.nc, r.nc, r.nb) != cudaSuccess)
                return fail(c, FK_ECUDA, "gpp: cannot describe aqsntemp as a tensor map");
            set_smem(tcx::tc_contract_kernel<EPI_GPP, 64, false>, tcx::Cfg<64>::SMEM);
            for (int q = 0; q < p.pipe_chunks; ++q) {
                if (q > 0 && cudaStreamWaitEvent(st, c.pipe_ev[q], 0) != cudaSuccess)
                    return cuda_fail(c, cudaGetLastError(), "gpp: waiting for a block");
                t.mt0 = q * p.pipe_sub;
                t.MT = std::min(p.MT, t.mt0 + p.pipe_sub) - t.mt0;
                t.units = t.MT * p.NT * p.KS;
                kernel_begin(c);
                tcx::tc_contract_kernel<EPI_GPP, 64, false>
                    <<<std::min(t.units, c.sms), tcx::THREADS, tcx::Cfg<64>::SMEM, st>>>(t);
                kernel_end(c);
                ++c.launches;
            }
        }
    }
    // FP64: aqsntemp's digits (bound by memory) beside the prep (by the FP64 pipe).
    // 512 x 32768 x 20: the prep takes 103 us at one block per SM instead of 98 at two, the
    // digits hide behind it, the call goes from 435 to 409 us.
    if (p.tc64) {
        SideBranch br(c);
        cudaError_t ea = cudaSuccess;
        ContractArgs a{};
        a.A = r.aqsn; a.lda = r.nc; a.m0 = p.m0; a.M = M; a.K = r.nc;
        for (int pass = 0; pass < p.passes; ++pass) launch_prep(prep_args(pass), dim3(p.nch, r.ng));
        br.run([&] { ea = tc64::enqueue_a(c, a, p.z, zb); });
        const cudaError_t ej = br.join();
        if (ea != cudaSuccess || ej != cudaSuccess) return cuda_fail(c, ea != cudaSuccess ? ea : ej, "gpp: digits");
    }
    for (int pass = 0; pass < p.passes && !pipe && !p.tc64; ++pass) launch_prep(prep_args(pass), dim3(p.nch, r.ng));
    phase_mark(c, 2);
    // mixed: the static remainder beside the main contraction (both need the prep's set-up
    // only): 130 x 4099 x 70 98 -> 95 us
    std::unique_ptr<SideBranch> stat;
    if (S && p.mixed && M > 0 && !pipe && !c.profiling) stat.reset(new (std::nothrow) SideBranch(c));
    if (M > 0 && !pipe) {
        ContractArgs a{};
        a.A = r.aqsn; a.lda = r.nc; a.m0 = p.m0; a.M = M;
        a.B = D; a.ldb = r.nc; a.bstride = 0; a.N = 3 * r.ng; a.K = r.nc;
        a.KS = p.KS; a.kchunk = p.kchunk; a.batches = 1; a.batch_plane = nullptr;
        a.aqsm = r.aqsm; a.ldm = r.ldm; a.vcoul = r.vcoul; a.igp = igp; a.acol = acol; a.wscale = 0.5; a.G = 3; a.P = P;
        dim3 grid(p.MT, p.NT * p.KS);
        if (p.mixed) {
            tcx::TcArgs t{};
            t.c = a;
            t.Bimg = (const uint8_t*)D;
            t.W1 = W; t.W2 = nullptr; t.ldw = M; t.gpp_cols = GPP_COLS; t.Aimg = nullptr; t.vcol = nullptr;
            t.kstages_total = p.kstages;
            t.MT = p.MT; t.NT = p.NT; t.units = p.units;
            t.err = c.errword;
            t.wait_limit = c.wait_limit;
            if (tcx::encode_rows_map(&t.amap, r.aqsn, r.nc, r.nc, r.nb) != cudaSuccess)
                return fail(c, FK_ECUDA, "gpp: cannot describe aqsntemp as a tensor map (needs a 16-byte aligned array)");
            if (gpp_pair(r, false)) {
                auto k = p.apre ? tcx::tc_contract_pair_apre_kernel<EPI_GPP, 64>
                                : tcx::tc_contract_pair_kernel<EPI_GPP, 64, false>;
                const size_t smem = p.apre ? tcx::Cfg<64, false, true, true>::SMEM : tcx::Cfg<64, false, true>::SMEM;
                static const int pairs = tcx::resident_pairs(tcx::tc_contract_pair_kernel<EPI_GPP, 64, false>,
                                                             tcx::Cfg<64, false, true>::SMEM, tcx::THREADS, c.sms / 2);
                static const int pairs_apre =
                    tcx::resident_pairs(tcx::tc_contract_pair_apre_kernel<EPI_GPP, 64>,
                                        tcx::Cfg<64, false, true, true>::SMEM, tcx::THREADS, c.sms / 2);
                const int grid1 = 2 * std::min(p.units, p.apre ? pairs_apre : pairs);
                if (p.apre) {
                    // aqsntemp rows m0 .. split once; an even number of 128-row tiles, rows past
                    // number_bands and k-values past ncouls zero
                    const int MTa = 2 * p.MT;  // the conversion also writes the padding (zeros)
                    tcx::aimg_split3_kernel<<<dim3(ceil_div(p.kstages * (tcx::BK / 8), 128), MTa * tcx::BM), 128, 0, st>>>(
                        r.aqsn + (long)p.m0 * r.nc, M, r.nc, p.kstages, Aimg);
                    c.launches += 1;
                    t.Aimg = Aimg;
                }
                set_smem(k, smem);
                kernel_begin(c);
                k<<<grid1, tcx::THREADS, smem, st>>>(t);
                kernel_end(c);
            } else {
                auto k = tcx::tc_contract_kernel<EPI_GPP, 64, false>;
                set_smem(k, tcx::Cfg<64>::SMEM);
                kernel_begin(c);
                k<<<std::min(p.units, c.sms), tcx::THREADS, tcx::Cfg<64>::SMEM, st>>>(t);
                kernel_end(c);
            }
        } else if (p.tc64) {
            run_tc64<EPI_GPP>(c, a, p.z, zb, true);  // (the digits were queued above)
            --c.launches;
        } else {
            auto k = d64::contract_kernel<EPI_GPP>;
            set_smem(k, d64::SMEM);
            kernel_begin(c);
            k<<<grid, d64::THREADS, d64::SMEM, st>>>(a, d64::Redo{});
            kernel_end(c);
        }
        ++c.launches;
    }
    if (S) {
        ContractArgs a{};
        a.A = r.aqsn; a.lda = r.nc; a.m0 = 0; a.M = r.nb;
        a.B = r.eps; a.ldb = r.nc; a.bstride = 0; a.N = r.ng; a.K = r.nc;
        a.KS = p.KSs; a.kchunk = p.kchunks; a.batches = 1; a.batch_plane = nullptr;
        a.aqsm = r.aqsm; a.ldm = r.ldm; a.vcoul = r.vcoul; a.igp = igp; a.acol = acol; a.wscale = -0.5; a.G = 1; a.P = S;
        dim3 grid(p.MTs, p.NTs * p.KSs);
        if (p.mixed) {
            auto k = f32::contract_kernel<EPI_STAT>;
            set_smem(k, f32::SMEM);
            auto launch = [&] { k<<<grid, f32::THREADS, f32::SMEM, c.stream>>>(a); };
            if (stat) {
                stat->run(launch);
                const cudaError_t ej = stat->join();
                if (ej != cudaSuccess) return cuda_fail(c, ej, "gpp: static remainder");
            } else {
                launch();
            }
        } else if (p.tc64) {
            // not the dominant kernel of the call: outside the kernel timer
            const bool prof = c.profiling;
            const int nk = c.nk;
            c.profiling = false;
            const cudaError_t e = run_tc64<EPI_STAT>(c, a, p.zs, zb);
            c.profiling = prof;
            c.nk = nk;
            if (e != cudaSuccess) return cuda_fail(c, e, "gpp: digits");
            --c.launches;
        } else {
            auto k = d64::contract_kernel<EPI_STAT>;
            set_smem(k, d64::SMEM);
            k<<<grid, d64::THREADS, d64::SMEM, st>>>(a, d64::Redo{});
        }
        ++c.launches;
    }
    phase_mark(c, 3);
    RowsArgs ra{r.nb, r.nv, r.ng, p.KS * p.NT, P, p.KSs * p.NTs, S, p.nch, F, r.ldm, r.aqsm, r.vcoul, igp, acol, rows};
    ra.counter = counter;  // the last block also writes the totals
    ra.out = r.out;
    ra.wf = wf;
    ra.m0 = p.m0;
    ra.fsch = p.fsch;
    rows_kernel<<<rows_blocks(r.nb, r.nv), ROWS_THREADS, 0, st>>>(ra);
    ++c.launches;
    if (est) {
        // every row block of a pipelined call has landed: the contractions waited for them
        est_rows_kernel<<<r.nb, 256, 0, st>>>(r.nc, r.aqsn, estA);
        est_bands_kernel<<<r.nb, 128, 0, st>>>(r.nv, r.ng, p.nch, estE, estA, r.aqsm, r.ldm, igp, acol, r.vcoul, estB);
        est_total_kernel<<<1, 256, 0, st>>>(r.nb, estB, GPP_EST_C * 0x1p-24, c.est_dev);
        c.launches += 3;
    }
    phase_mark(c, 4);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(c, e, "gpp kernels");
    return FK_OK;
}


// ========================================================== served steps
// A served request (GppJob) keeps its plan, workspace and descriptors on the
// host; a step runs the first-step work (index map, weights, prep, and the A
// image of requests over four or more n-tiles), a range of contraction units
// and the last-step reduction of up to STEP_MAX requests with six table-driven
// kernels, replayed from one captured graph.
// A request's k-slices, partial slots and reduction order depend only on its
// own shape and plan, never on which other requests share a step.
namespace {

constexpr int STEP_MAX = tcx::TC_MAXREQ;

struct StepReq {
    int nb, nv, nc, ng, M, compact, Q, passes;
    // requests over four or more n-tiles: aqsntemp rows nvband .. split once into a
    // BF16 A image (Aimg, kst k-stages per 128-row tile) in the request's first step
    const double2* arows;
    uint8_t* Aimg;
    int MTa, kst;
    const int *inv, *indinv;
    int *igp, *acol;
    const double2* aqsm;
    long ldm;
    const double* vcoul;
    float2* W;
    PrepArgs prep;
    RowsArgs rows;
    double2* out;
};

struct StepTable {
    tcx::TcTable tc;
    StepReq req[STEP_MAX];
    int nfirst, nlast;
    int first[STEP_MAX], last[STEP_MAX];
    long setup_start[STEP_MAX + 1];  // threads: ng (index map) + M*ng (weights) per first-step request
    int prep_start[STEP_MAX + 1];    // blocks: passes*nch*ng per first-step request
    long rows_start[STEP_MAX + 1];   // rows block tasks (rows_blocks) per last-step request
    long aimg_start[STEP_MAX + 1];   // A image elements (padded) per first-step request (0 without one)
};

template <class T>
FK_DEV int find_range(const T* start, int n, T x) {  // largest i < n with start[i] <= x
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (start[mid] <= x) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__global__ void step_setup_kernel(const StepTable* T) {
    const long total = T->setup_start[T->nfirst];
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
        const int f = find_range(T->setup_start, T->nfirst, t);
        const StepReq& q = T->req[T->first[f]];
        long i = t - T->setup_start[f];
        if (i < q.ng) {
            const int g = gpp_igp_of((int)i, q.nc, q.inv, q.indinv);
            q.igp[i] = g;
            q.acol[i] = g < 0 ? -1 : (q.compact ? (int)i : g);
        } else {
            i -= q.ng;
            const int h = (int)(i / q.M), m = (int)(i % q.M);
            const int g = gpp_igp_of(h, q.nc, q.inv, q.indinv);
            float2 w = make_float2(0.f, 0.f);
            if (g >= 0) w = tcx::weight_w1(q.aqsm[(long)(q.nv + m) * q.ldm + (q.compact ? h : g)], 0.5 * q.vcoul[g]);
            q.W[(long)h * q.M + m] = w;
        }
    }
}

// First-step requests with an A image: aqsntemp rows nvband .. into the BF16
// image (the converter warps' pieces), the positions past M rows or ncouls
// k-values zero; one thread per 8 k-values of the padded extent (aimg_start
// counts those chunks).
__global__ void aimg_table_kernel(const StepTable* T) {
    const long total = T->aimg_start[T->nfirst];
    for (long t = (long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long)gridDim.x * blockDim.x) {
        const int f = find_range(T->aimg_start, T->nfirst, t);
        const StepReq& q = T->req[T->first[f]];
        const long i = t - T->aimg_start[f];
        const int CP = q.kst * (tcx::BK / 8);  // chunks per padded row
        const int m = (int)(i / CP), k0 = 8 * (int)(i % CP);
        double2 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            v[j] = (m < q.M && k0 + j < q.nc) ? q.arows[(long)m * q.nc + k0 + j] : make_double2(0.0, 0.0);
        tcx::aimg_chunk_split3(q.Aimg, q.kst, m, k0, v);
    }
}

template <int BN>
__global__ void __launch_bounds__(PREP_THREADS, 2) prep_table_kernel(const StepTable* T) {
    __shared__ double2 sm[8 * NVC * 6];
    const int total = T->prep_start[T->nfirst];
    for (int it = blockIdx.x; it < total; it += gridDim.x) {
        const int f = find_range(T->prep_start, T->nfirst, it);
        const StepReq& q = T->req[T->first[f]];
        int i = it - T->prep_start[f];
        const int per_pass = q.prep.nch * q.ng;
        const int pass = i / per_pass;
        i -= pass * per_pass;
        PrepArgs a = q.prep;
        a.n1base = pass * NVC;
        if (pass) a.D = nullptr;
        if (q.Q) prep_mixed_item<1, BN>(a, i % a.nch, i / a.nch, sm);
        else prep_mixed_item<0, BN>(a, i % a.nch, i / a.nch, sm);
        __syncthreads();  // sm is reused by the next item
    }
}

__global__ void __launch_bounds__(ROWS_THREADS) rows_table_kernel(const StepTable* T) {
    const long total = T->rows_start[T->nlast];
    for (long i = blockIdx.x; i < total; i += gridDim.x) {  // block-uniform
        const int l = find_range(T->rows_start, T->nlast, i);
        const StepReq& q = T->req[T->last[l]];
        rows_block(q.rows, (int)(i - T->rows_start[l]), threadIdx.x);
    }
}

__global__ void totals_table_kernel(const StepTable* T) {
    for (int l = blockIdx.x; l < T->nlast; l += gridDim.x) {
        const StepReq& q = T->req[T->last[l]];
        totals_block(q.nb, q.nv, q.rows.rows, q.out);
    }
}

}  // namespace

struct GppJob {
    GppDev r;
    Plan p;
    tcx::TcArgs tc;
    StepReq req;
    size_t bytes;
};

struct GppStep {
    StepTable* dev = nullptr;
    StepTable* host = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaEvent_t done = nullptr;
    bool launched = false;
};

// k-stages of a served request's unit at most.  A step hands out whole units
// within its budget (96 stages per SM by default), so the units of a large
// request, 340 stages long under the plan of a call of its own, left most SMs
// without one: 32 requests of 128-1024 bands took 40.2 ms, with units of at most
// 64, 32 and 16 stages 22.2, 19.8 and 20.1 ms.
constexpr int SERVED_UNIT = 32;

// A served request over four or more n-tiles gets an A image: without it the
// converter warps of every n-tile's units would split the same A rows again.
inline size_t job_aimg_bytes(const Plan& p) {
    return (p.mixed && p.NT >= 4) ? (size_t)p.MT * p.kstages * tcx::Cfg<64>::A_BYTES : 0;
}

size_t gpp_job_bytes(const Ctx& c, const GppDev& r, int ks) {
    const Plan p = make_plan(c, r, ks);
    return p.bytesD + p.bytesF + p.bytesP + p.bytesRows + p.bytesIgp + p.bytesW + job_aimg_bytes(p) +
           (7 + (size_t)r.nb) * sizeof(double2) + 9 * 256;
}

int gpp_job_units(const GppJob* j) { return (j->r.nb - j->r.nv) > 0 ? j->p.units : 0; }
int gpp_job_stages_per_unit(const GppJob* j) { return ceil_div(j->p.kchunk, tcx::BK); }
double2* gpp_job_out(const GppJob* j) { return j->r.out; }
int gpp_job_ks(const GppJob* j) { return j->p.KS; }
void gpp_job_destroy(GppJob* j) { delete j; }

GppJob* gpp_job_create(Ctx& c, const GppDev& r0, int ks, void* ws, size_t bytes, fk_status* st) {
    *st = FK_OK;
    if (r0.prec != FK_MIXED || (r0.flags & FK_GPP_ACHSTEMP)) {
        *st = FK_ENOTSUP;
        return nullptr;
    }
    GppJob* j = new (std::nothrow) GppJob();
    if (!j) {
        *st = FK_ENOMEM;
        return nullptr;
    }
    j->r = r0;
    j->p = make_plan(c, r0, ks);
    j->bytes = bytes;
    const Plan& p = j->p;
    Workspace w;
    w.base = ws;
    w.cap = bytes;
    int* igp = (int*)w.take(p.bytesIgp);
    int* acol = igp ? igp + r0.ng : nullptr;
    void* D = p.bytesD ? w.take(p.bytesD) : nullptr;
    double2* F = (double2*)w.take(p.bytesF);
    double2* P = p.bytesP ? (double2*)w.take(p.bytesP) : nullptr;
    double2* rows = (double2*)w.take(p.bytesRows);
    float2* W = p.bytesW ? (float2*)w.take(p.bytesW) : nullptr;
    double2* out = (double2*)w.take((7 + (size_t)r0.nb) * sizeof(double2));
    const size_t aimg_bytes = job_aimg_bytes(p);
    uint8_t* Aimg = aimg_bytes ? (uint8_t*)w.take(aimg_bytes) : nullptr;
    if (!igp || !F || !rows || !out || (p.bytesD && !D) || (p.bytesP && !P) || (p.bytesW && !W) ||
        (aimg_bytes && !Aimg)) {
        delete j;
        *st = FK_ENOMEM;
        return nullptr;
    }
    j->r.out = out;
    const GppDev& r = j->r;
    const int M = r.nb - r.nv;
    StepReq& q = j->req;
    q.nb = r.nb; q.nv = r.nv; q.nc = r.nc; q.ng = r.ng; q.M = M; q.compact = r.aqsm_compact ? 1 : 0;
    q.Q = (r.flags & FK_GPP_ROOT_QUIRKS) ? 1 : 0;
    q.passes = p.passes;
    q.inv = r.inv; q.indinv = r.indinv; q.igp = igp; q.acol = acol;
    q.aqsm = r.aqsm; q.ldm = r.ldm; q.vcoul = r.vcoul; q.W = W;
    q.prep = PrepArgs{r.nb, r.nv, r.nc, r.ng, r.aqsn, r.eps, r.wt, r.wx, igp, D, p.kstages, F, p.nch, p.tile, 0, 0};
    q.rows = RowsArgs{r.nb, r.nv, r.ng, p.KS * p.NT, P, 0, nullptr, p.nch, F, r.ldm, r.aqsm, r.vcoul, igp, acol, rows};
    q.out = out;
    q.rows.out = out;  // the band rows write acht_n1_loc
    q.arows = r.aqsn + (long)r.nv * r.nc;
    q.Aimg = M > 0 ? Aimg : nullptr;
    q.MTa = p.MT;
    q.kst = p.kstages;
    if (M > 0) {
        ContractArgs a{};
        a.A = r.aqsn; a.lda = r.nc; a.m0 = r.nv; a.M = M;
        a.B = D; a.ldb = r.nc; a.bstride = 0; a.N = 3 * r.ng; a.K = r.nc;
        a.KS = p.KS; a.kchunk = p.kchunk; a.batches = 1; a.batch_plane = nullptr;
        a.aqsm = r.aqsm; a.ldm = r.ldm; a.vcoul = r.vcoul; a.igp = igp; a.acol = acol; a.wscale = 0.5; a.G = 3; a.P = P;
        tcx::TcArgs& t = j->tc;
        t.c = a;
        t.Bimg = (const uint8_t*)D;
        t.W1 = W; t.W2 = nullptr; t.ldw = M; t.gpp_cols = GPP_COLS; t.vcol = nullptr;
        t.Aimg = q.Aimg;  // the table contraction reads a pre-split A image when the request has one
        t.kstages_total = p.kstages;
        t.MT = p.MT; t.NT = p.NT; t.units = p.units;
        t.err = c.errword;
        t.wait_limit = c.wait_limit;
        if (tcx::encode_rows_map(&t.amap, r.aqsn, r.nc, r.nc, r.nb) != cudaSuccess) {
            delete j;
            *st = FK_ECUDA;
            return nullptr;
        }
        // padding rows of the image and k >= ncouls must read as zero (the prep writes the rest)
        if (tcx::img_needs_pad(64, r.ng, GPP_COLS, r.nc))
            tcx::img_pad_kernel<64><<<dim3(p.kstages, p.NT, 1), 256, 0, c.stream>>>((uint8_t*)D, p.NT, p.kstages,
                                                                                   r.ng, GPP_COLS, r.nc);
        if (cudaGetLastError() != cudaSuccess) {
            delete j;
            *st = FK_ECUDA;
            return nullptr;
        }
    }
    return j;
}

GppStep* gpp_step_create(Ctx& c, fk_status* st) {
    *st = FK_ECUDA;
    GppStep* s = new (std::nothrow) GppStep();
    if (!s) {
        *st = FK_ENOMEM;
        return nullptr;
    }
    auto bad = [&](fk_status code) -> GppStep* {
        gpp_step_destroy(s);
        cudaGetLastError();
        *st = code;
        return nullptr;
    };
    if (cudaMalloc(&s->dev, sizeof(StepTable)) != cudaSuccess) return bad(FK_ENOMEM);
    if (cudaMallocHost(&s->host, sizeof(StepTable)) != cudaSuccess) return bad(FK_ENOMEM);
    std::memset((void*)s->host, 0, sizeof(StepTable));
    if (cudaEventCreateWithFlags(&s->done, cudaEventDisableTiming) != cudaSuccess) return bad(FK_ECUDA);
    auto tck = tcx::tc_contract_table_kernel<EPI_GPP, 64, false>;
    if (set_smem(tck, tcx::Cfg<64>::SMEM) != cudaSuccess) return bad(FK_ECUDA);
    int prep_per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&prep_per_sm, prep_table_kernel<64>, PREP_THREADS, 0) !=
            cudaSuccess ||
        prep_per_sm < 1)
        prep_per_sm = 1;
    // capture: table upload, error-word clear, the six kernels
    cudaStream_t str = c.stream;
    if (cudaStreamBeginCapture(str, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return bad(FK_ECUDA);
    cudaMemcpyAsync(s->dev, s->host, sizeof(StepTable), cudaMemcpyHostToDevice, str);
    cudaMemsetAsync(c.errword, 0, sizeof(int), str);
    step_setup_kernel<<<c.sms * 4, 256, 0, str>>>(s->dev);
    prep_table_kernel<64><<<c.sms * prep_per_sm, PREP_THREADS, 0, str>>>(s->dev);
    aimg_table_kernel<<<c.sms * 4, 256, 0, str>>>(s->dev);
    tck<<<c.sms, tcx::THREADS, tcx::Cfg<64>::SMEM, str>>>(&s->dev->tc, c.errword, c.wait_limit);
    rows_table_kernel<<<c.sms * 4, ROWS_THREADS, 0, str>>>(s->dev);
    totals_table_kernel<<<STEP_MAX, ROWS_THREADS, 0, str>>>(s->dev);
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(str, &g);
    if (e != cudaSuccess || !g) return bad(FK_ECUDA);
    e = cudaGraphInstantiate(&s->exec, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) return bad(FK_ECUDA);
    *st = FK_OK;
    return s;
}

void gpp_step_destroy(GppStep* s) {
    if (!s) return;
    if (s->launched) cudaEventSynchronize(s->done);
    if (s->exec) cudaGraphExecDestroy(s->exec);
    if (s->done) cudaEventDestroy(s->done);
    if (s->dev) cudaFree(s->dev);
    if (s->host) cudaFreeHost(s->host);
    delete s;
}

int gpp_step_capacity() { return STEP_MAX; }

fk_status gpp_step_launch(Ctx& c, GppStep* s, const GppStepItem* items, int n) {
    if (n < 0 || n > STEP_MAX) return fail(c, FK_EINVAL, "step: too many requests");
    // the previous step's table upload must be complete before the host table changes
    if (s->launched && cudaEventSynchronize(s->done) != cudaSuccess) return cuda_fail(c, cudaGetLastError(), "step");
    StepTable& T = *s->host;
    T.tc.nreq = n;
    T.nfirst = T.nlast = 0;
    int units = 0;
    T.setup_start[0] = 0;
    T.prep_start[0] = 0;
    T.rows_start[0] = 0;
    T.aimg_start[0] = 0;
    for (int i = 0; i < n; ++i) {
        const GppJob* j = items[i].job;
        T.req[i] = j->req;
        T.tc.req[i] = j->tc;
        T.tc.ustart[i] = units;
        T.tc.ulocal0[i] = items[i].u0;
        units += items[i].u1 - items[i].u0;
        if (items[i].first) {
            const int f = T.nfirst++;
            T.first[f] = i;
            T.setup_start[f + 1] = T.setup_start[f] + j->r.ng + (long)j->req.M * j->r.ng;
            T.prep_start[f + 1] = T.prep_start[f] + j->p.passes * j->p.nch * j->r.ng;
            T.aimg_start[f + 1] =
                T.aimg_start[f] + (j->req.Aimg ? (long)j->req.MTa * tcx::BM * j->req.kst * (tcx::BK / 8) : 0);
        }
        if (items[i].last) {
            const int l = T.nlast++;
            T.last[l] = i;
            T.rows_start[l + 1] = T.rows_start[l] + rows_blocks(j->r.nb, j->r.nv);
        }
    }
    T.tc.ustart[n] = units;
    T.tc.units = units;
    cudaError_t e = cudaGraphLaunch(s->exec, c.stream);
    if (e == cudaSuccess) e = cudaEventRecord(s->done, c.stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "step launch");
    s->launched = true;
    return FK_OK;
}

fk_status gpp_time_plan(Ctx& c, GppStep* s, const GppDev& r, int ks, long step_budget, void* ws, size_t bytes,
                        float* ms, int* units) {
    fk_status st = FK_OK;
    GppJob* j = gpp_job_create(c, r, ks, ws, bytes, &st);
    if (!j) return st;
    *units = gpp_job_units(j);
    const int spu = std::max(1, gpp_job_stages_per_unit(j));
    // the request alone through served steps of step_budget k-stages
    auto run = [&]() -> fk_status {
        int next = 0;
        bool first = true;
        do {
            const int k = (int)std::min<long>(*units - next, std::max(1L, step_budget / spu));
            GppStepItem it{j, next, next + k, first, next + k >= *units};
            const fk_status e = gpp_step_launch(c, s, &it, 1);
            if (e != FK_OK) return e;
            next += k;
            first = false;
        } while (next < *units);
        return FK_OK;
    };
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    st = run();  // warm
    if (st == FK_OK) {
        cudaEventRecord(e0, c.stream);
        st = run();
        cudaEventRecord(e1, c.stream);
    }
    cudaError_t e = cudaEventSynchronize(e1);
    if (st == FK_OK && e != cudaSuccess) st = cuda_fail(c, e, "tune");
    if (st == FK_OK) cudaEventElapsedTime(ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    gpp_job_destroy(j);
    return st;
}

int gpp_default_ks(const Ctx& c, const GppDev& r) { return make_plan(c, r).KS; }

int gpp_served_ks(const Ctx& c, const GppDev& r) {
    const Plan p = make_plan(c, r);
    return std::max(p.KS, ceil_div(p.kstages, SERVED_UNIT));
}


// ------------------------------------------------------------ real-valued run
namespace {
struct RealPlan {
    Plan c;         // the complex contraction over K2 pairs
    GppDev cd;      // its shape
    long K2;
    int nch, tile;
    size_t bytesDv, bytesMask, bytesF, bytesAC, bytesD64;
};

RealPlan make_real_plan(const Ctx& c, const GppRealDev& r) {
    RealPlan q{};
    q.K2 = (r.nc + 1) / 2;
    q.cd = GppDev{};
    q.cd.nb = r.nb; q.cd.nv = r.nv; q.cd.nc = (int)q.K2; q.cd.ng = r.ng; q.cd.prec = r.prec; q.cd.flags = 0; q.cd.tc64 = r.tc64;
    q.c = make_plan(c, q.cd);
    // FP64: tiles of the FP64 prep; mixed: chunks of one resident wave
    q.tile = r.prec == FK_MIXED ? ceil_div(ceil_div(r.nc, std::max(1, 4 * c.sms / r.ng)), PREP_THREADS) * PREP_THREADS
                                : PREP_TILE;
    q.nch = ceil_div(r.nc, q.tile);
    q.bytesDv = (size_t)r.ng * 3 * r.nc * sizeof(double);
    q.bytesMask = (size_t)r.ng * r.nc;
    q.bytesF = (size_t)q.nch * std::max(r.nv, 1) * r.ng * 6 * sizeof(double2);
    q.bytesAC = (size_t)r.nb * r.ng * sizeof(double2);
    return q;
}
}  // namespace

size_t gpp_real_workspace(const Ctx& c, const GppRealDev& r) {
    const RealPlan q = make_real_plan(c, r);
    return q.c.bytesD + q.c.bytesW + q.c.bytesP + q.c.bytesRows + q.c.bytesIgp + q.bytesDv + q.bytesMask + q.bytesF +
           q.bytesAC + q.c.bytesZ() + 12 * 256;
}

fk_status gpp_real_run(Ctx& c, const GppRealDev& r) {
    const RealPlan q = make_real_plan(c, r);
    const Plan& p = q.c;
    cudaStream_t st = c.stream;
    const int M = r.nb - r.nv;
    if (r.lda < 2 * q.K2 || (r.lda & 1)) return fail(c, FK_EINVAL, "gpp_real: aqsntemp rows must have an even stride");
    int* igp = (int*)c.ws.take(p.bytesIgp);
    int* acol = igp ? igp + r.ng : nullptr;
    void* D = p.bytesD ? c.ws.take(p.bytesD) : nullptr;
    double2* P = p.bytesP ? (double2*)c.ws.take(p.bytesP) : nullptr;
    double2* rows = (double2*)c.ws.take(p.bytesRows);
    float2* W = p.bytesW ? (float2*)c.ws.take(p.bytesW) : nullptr;
    double* Dv = (double*)c.ws.take(q.bytesDv);
    uint8_t* mask = (uint8_t*)c.ws.take(q.bytesMask);
    double2* F = (double2*)c.ws.take(q.bytesF);
    double2* AC = (double2*)c.ws.take(q.bytesAC);
    int* counter = (int*)c.ws.take(sizeof(int));
    if (!igp || !rows || !Dv || !mask || !F || !AC || !counter || (p.bytesD && !D) || (p.bytesP && !P) ||
        (p.bytesW && !W))
        return fail(c, FK_ENOMEM, "workspace too small for the real-valued GPP request");
    tc64::Bufs zb{};
    if (!take_tc64(c, p, zb)) return fail(c, FK_ENOMEM, "workspace too small for the real-valued GPP request");
    c.launches = 0;
    phase_mark(c, 1);
    SetupArgs sa{};
    sa.nb = r.nb; sa.nv = r.nv; sa.nc = r.nc; sa.ng = r.ng;
    sa.inv = r.inv; sa.indinv = r.indinv; sa.igp = igp; sa.acol = acol; sa.vcoul = r.vcoul;
    sa.W = p.mixed && M > 0 ? W : nullptr;
    sa.counter = counter;
    sa.err = (p.mixed || p.tc64) && D ? c.errword : nullptr;
    if (p.mixed && D && tcx::img_needs_pad(64, r.ng, GPP_COLS, (int)q.K2)) sa.img = (uint8_t*)D;
    sa.NT = p.NT; sa.kstages = p.kstages; sa.K = (int)q.K2;
    sa.aqsm_re = r.aqsm; sa.ac = AC;
    launch_setup(sa, st);
    ++c.launches;
    const int passes = std::max(1, ceil_div(r.nv, NVC));
    for (int pass = 0; pass < passes; ++pass) {
        RealPrepArgs a{r.nb, r.nv, r.nc, r.ng, r.aqsn, r.eps, r.wt, r.wx, r.lda, igp,
                       (pass == 0 && M > 0) ? Dv : nullptr, mask, F, q.nch, pass * NVC, q.tile};
        if (p.mixed) real_prep_mixed_kernel<<<dim3(q.nch, r.ng), PREP_THREADS, 0, st>>>(a);
        else real_prep_kernel<<<dim3(q.nch, r.ng), PREP_THREADS, 0, st>>>(a);
        ++c.launches;
    }
    if (M > 0) {
        RealCarryArgs ca{r.nc, r.ng, q.K2, igp, Dv, mask, (r.flags & FK_GPP_REAL_ZERO_MASKED) ? 0 : 1,
                         p.mixed ? nullptr : (double*)D, p.mixed ? (uint8_t*)D : nullptr, p.kstages};
        const long threads = (long)r.ng * r.nc;  // one per element
        const int blocks = (int)((threads + 255) / 256);
        if (p.mixed) real_carry_kernel<1><<<blocks, 256, 0, st>>>(ca);
        else real_carry_kernel<0><<<blocks, 256, 0, st>>>(ca);
        ++c.launches;
    }
    phase_mark(c, 2);
    if (M > 0) {
        ContractArgs a{};
        a.A = (const double2*)r.aqsn; a.lda = r.lda / 2; a.m0 = r.nv; a.M = M;
        a.B = D; a.ldb = q.K2; a.bstride = 0; a.N = 3 * r.ng; a.K = (int)q.K2;
        a.KS = p.KS; a.kchunk = p.kchunk; a.batches = 1; a.batch_plane = nullptr;
        a.aqsm = AC; a.ldm = r.ng; a.vcoul = r.vcoul; a.igp = igp; a.acol = acol; a.wscale = 0.5; a.G = 3; a.P = P;
        if (p.mixed) {
            tcx::TcArgs t{};
            t.c = a;
            t.Bimg = (const uint8_t*)D;
            t.W1 = W; t.W2 = nullptr; t.ldw = M; t.gpp_cols = GPP_COLS; t.Aimg = nullptr; t.vcol = nullptr;
            t.kstages_total = p.kstages;
            t.MT = p.MT; t.NT = p.NT; t.units = p.units;
            t.err = c.errword;
            t.wait_limit = c.wait_limit;
            if (tcx::encode_rows_map(&t.amap, a.A, a.lda, a.K, r.nb) != cudaSuccess)
                return fail(c, FK_ECUDA, "gpp_real: cannot describe aqsntemp as a tensor map");
            auto k = tcx::tc_contract_kernel<EPI_GPP, 64, false>;
            set_smem(k, tcx::Cfg<64>::SMEM);
            kernel_begin(c);
            k<<<std::min(p.units, c.sms), tcx::THREADS, tcx::Cfg<64>::SMEM, st>>>(t);
            kernel_end(c);
        } else if (p.tc64) {
            const cudaError_t e = run_tc64<EPI_GPP>(c, a, p.z, zb, false, true);
            if (e != cudaSuccess) return cuda_fail(c, e, "gpp_real: digits");
            --c.launches;
        } else {
            auto k = d64::contract_kernel<EPI_GPP>;
            set_smem(k, d64::SMEM);
            kernel_begin(c);
            k<<<dim3(p.MT, p.NT * p.KS), d64::THREADS, d64::SMEM, st>>>(a, d64::Redo{});
            kernel_end(c);
        }
        ++c.launches;
    }
    phase_mark(c, 3);
    RowsArgs ra{r.nb, r.nv, r.ng, P ? p.KS * p.NT : 0, P, 0, nullptr, q.nch, F, r.ng, AC, r.vcoul, igp, acol, rows};
    ra.re_only = true;
    ra.counter = counter;  // the last block also writes the totals
    ra.out_re = r.out;
    rows_kernel<<<rows_blocks(r.nb, r.nv), ROWS_THREADS, 0, st>>>(ra);
    ++c.launches;
    phase_mark(c, 4);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FK_OK : cuda_fail(c, e, "gpp_real kernels");
}

}  // namespace fk
