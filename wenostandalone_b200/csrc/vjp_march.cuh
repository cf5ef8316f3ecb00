// vjp_march.cuh -- adjoint (VJP) of the FP64 WENO5 (+MP) sweep with JS or
// TENO weights, marching along the sweep like the forward kernel of
// sweep_march_tma.cuh.
//
// A warp owns 32 columns and walks a segment of their cells (vjp_march_cut).
// At face J it recomputes the forward state from the carried window
// (March64: the beta of the new difference pair, P_k, S_L, S_R, one
// reciprocal) with the weights made explicit, then pulls the face's
// cotangents gL, gR back:
//   * MP (f90:1564-1608): the one-sided median of the forward kernel picks
//     one expression (the WENO value, v0, a neighbour, MD, UL or LC); the
//     cotangent goes to that expression's cells (and, for MD and LC, through
//     the minmod to the curvature it picked).  Faces whose median passes the
//     WENO value through -- the common case -- skip this part as a warp.
//   * weights: d out/d p_k = w_k, d out/d beta_k = -2 w_k (p_k - out)/beta_k
//     (JS); TENO weights d_k delta_k / sum d delta are constant between
//     cutoff flips, so they pull nothing back to beta; sum_k w_k = 1, so
//     d out/d v0 through the candidates is the cotangent itself;
//   * candidates and beta are linear / quadratic in the differences
//     d[k] = v[k+1] - v[k]; their gradients are summed per difference and a
//     difference is turned into its two cells once its last face is done.
// Face o (output index) is centred on cell o + 3 and reads cells o+1 .. o+5,
// so cell o + 1 is final after face o; the sums keep it one face longer
// and emit cell o after face o, so the 8 faces of a chunk starting at an
// even face emit 8 cells starting at an even index (16-byte aligned for the
// TMA unit): row tiles by a bulk tensor store from a swizzled shared tile,
// column tiles (folded y/z, lanes along x) by coalesced stores.  With
// accumulation the previous gradient arrives in the same input stage.
//
// Staging: a ring of 3 stages per warp; stage k carries the cells
// [4 + 8k, 12 + 8k) of v, the cotangents of faces [4 + 8k, 12 + 8k) and
// (accumulating) the old gradient of cells [4 + 8k, 12 + 8k), all completed
// on one mbarrier.  Waits are bounded as in the forward kernel.
//
// LDR: arrays that TMA refuses (rows that are not 16-byte multiples, 8-byte
// aligned bases) are staged by cp.async copies into the same tiles (eight
// lanes per row where the rows run along the sweep), the tiles run over the
// columns of all cross axes, and the gradient leaves by plain stores or
// (accumulating) FP64 reductions, whose one add rounds as a load and an add
// do.
//
// PF: face-dependent coefficients.  Every CTA holds the whole table of the
// sweep (27 coefficients a face) in shared memory, read at warp-uniform
// addresses; staged per chunk and warp it would not fit beside the tiles.
// us per x/y/z gradient, 97x80x65 x 5: 689 with one thread per column
// (vjp_kernel), 561 here.  Bound by latency with 8 warps an SM (issue slots
// 40%, FP64 pipe 32%, against 57% and 56% without the table and aligned):
// dependent uses, the rows' shared loads, instruction fetch, and a last round
// of the resident warps that is 11% (y) and 32% (z) full.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "sweep_march_tma.cuh"
#include "weno_adjoint.cuh"

namespace wsb {

constexpr int kVjpStages = 3;
constexpr int kVjpWarps = 8;  // one CTA per SM: 8 warps x 28 KB of shared memory, 255 registers

struct VjpMarchArgs {
    int kind;           // 0 row tiles, 1 column tiles (as MarchTmaArgs)
    int dimJ, dimU, dimW, uoff, woff;
    int odimU;          // cotangent map dimension of the lane axis (1 or 2)
    int acc;            // add to the gradient already in gv
    int vbytes;         // one v (or old-gradient) tile
    int stage_bytes;    // v (and old gradient) tiles of one stage
    int warp_bytes;     // multiple of 512
    unsigned tx_bytes;  // bytes one stage receives
    const double* gLp;  // cotangents (ns, c1, c2, V)
    const double* gRp;
    int rows;           // rows of the per-face table
    // 2 beta_coef of the squares (ucf 18, 20, 21, 23, 24, 26), exact; formed in
    // the kernel they took registers or an operation a face (832 against 802
    // us per x/y/z gradient, 128^3 x 5)
    double b2[6];
};

__device__ __forceinline__ bool finite_bits(double x) {
    return ((unsigned)__double2hiint(x) & 0x7ff00000u) != 0x7ff00000u;
}

// beta in [2^-100, 2^100): then the one-reciprocal weights, 1/beta and
// their products stay normal (an integer test on the exponent field).
__device__ __forceinline__ bool beta_ok(double b) {
    const unsigned hi = (unsigned)__double2hiint(b);
    return (hi - (923u << 20)) < (200u << 20);
}

// Gradient of one minmod (mm64) with respect to its two arguments:
// c1 = d/d(dl), c2 = d/d(dr).
__device__ __forceinline__ void mm64_grad(double dl, double dr, double& c1, double& c2) {
    const double a = fabs(dl), b = fabs(dr);
    const bool al = a < b;  // dl is the smaller
    const double m = al ? a : b, M = al ? b : a;
    const double t = fma(4.0, m, -M);
    const bool same = ((__double2hiint(dl) ^ __double2hiint(dr)) >= 0) && (t > 0.0);
    const bool pick_t = t < m;  // 4 x_small - x_large, else x_small
    const double cs = same ? (pick_t ? 4.0 : 1.0) : 0.0;
    const double cl = (same && pick_t) ? -1.0 : 0.0;
    c1 = al ? cs : cl;
    c2 = al ? cl : cs;
}

// Expression codes of the one-sided median.
enum : int { kPickW = 0, kPickV0 = 1, kPickNb = 2, kPickMD = 3, kPickUL = 4, kPickLC = 5 };

// Median of one side with the picked expression's code (same values as
// March64::face).  nb: the neighbour (vm1 left, vp1 right).
__device__ __forceinline__ double mp_pick(double x, double v0, double nb, double UL, double MD, double LC, bool pos,
                                          bool nb_first, bool ul_first, int& code) {
    // pos: P1 = max(v0, nb) else min; nb_first: P1 is nb
    const double P1 = nb_first ? nb : v0, P2 = ul_first ? UL : v0;
    const int c1 = nb_first ? kPickNb : kPickV0, c2 = ul_first ? kPickUL : kPickV0;
    const bool sA = (P1 < MD) != pos, sB = (P2 < LC) != pos;
    const double A = sA ? P1 : MD, B = sB ? P2 : LC;
    const int cA = sA ? c1 : kPickMD, cB = sB ? c2 : kPickLC;
    const bool s1 = (x < A) != !pos;
    const double T1 = s1 ? x : A;
    const int cT1 = s1 ? kPickW : cA;
    const bool s2 = (T1 < B) != !pos;
    code = s2 ? cT1 : cB;
    return s2 ? T1 : B;
}

// Whether the three ideal weights of one side suit the one-reciprocal form
// with betas in [2^-100, 2^100): each 0 or within [2^-60, 2^60], so that the
// product of both sides' sums stays within 2^(+-920), and not all 0; TENO:
// none 0, as the cutoff may keep a stencil without weight alone.  (Not so:
// negative and NaN weights, which the limiter's one-sided median does not
// take either.)
__host__ __device__ inline bool vjp_side_ok(double d0, double d1, double d2, bool teno) {
    const double lo = 0x1p-60, hi = 0x1p60;
    auto one = [&](double x) { return (x >= lo && x <= hi) || (x == 0.0 && !teno); };
    return one(d0) && one(d1) && one(d2) && d0 + d1 + d2 > 0.0;
}

// Coefficient sources of one face (Coef<5> order): the kernel parameters, or
// the face's row of the CTA's table, kVjpRow doubles with a mark at the end
// (1: ideal weights that are not vjp_side_ok; the face is redone from the
// arrays).
constexpr int kVjpRow = 28;
// Coef<5> index of the k-th square's coefficient (VjpMarchArgs::b2)
__host__ __device__ constexpr int vjp_square(int k) { return 18 + 3 * (k / 2) + 2 * (k % 2); }
struct VjpParam {
    const MarchArgs& a;
    const double* b2;
    __device__ __forceinline__ double operator()(int q) const { return a.ucf[q]; }
    __device__ __forceinline__ double twice(int k) const { return b2[k]; }
    __device__ __forceinline__ bool marked() const { return false; }
};
struct VjpRow {
    const double2* p;
    __device__ __forceinline__ explicit VjpRow(const double* row) : p(reinterpret_cast<const double2*>(row)) {}
    __device__ __forceinline__ double operator()(int q) const { return (q & 1) ? p[q >> 1].y : p[q >> 1].x; }
    __device__ __forceinline__ double twice(int k) const { return 2.0 * (*this)(vjp_square(k)); }
    __device__ __forceinline__ bool marked() const { return p[13].y != 0.0; }
};
// Beta coefficients the pair (d[J], d[J+1]) of row's face J enters, stencil r
// of face J + r (March64::push).
struct VjpPair {
    const double* row;
    __device__ __forceinline__ double b(int q) const { return row[(q / 3) * kVjpRow + 18 + q]; }
};

// Row f of the table: core face clamp(f - 3) of the arrays.  One thread per
// entry, as the sweeps' tables.
__global__ void vjp_face_table_kernel(CoefPtrs cp, long long nc, int rows, bool teno, double* __restrict__ tab) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long f = i / kVjpRow;
    const int q = (int)(i % kVjpRow);
    if (f >= rows) return;
    const long long c = table_core(f, nc);
    auto side = [&](const double* p) { return vjp_side_ok(p[5 * c], p[5 * c + 1], p[5 * c + 2], teno); };
    const bool mark = q >= 12 && (q < 18 || q == 27) && !(side(cp.dL) && side(cp.dR));
    double x;
    if (q < 6) x = cp.polyL[c + nc * (q / 2 + 5 * (q % 2))];
    else if (q < 12) x = cp.polyR[c + nc * ((q - 6) / 2 + 5 * (q % 2))];
    else if (q < 18) x = mark ? 1.0 : (q < 15 ? cp.dL[q - 12 + 5 * c] : cp.dR[q - 15 + 5 * c]);
    else if (q < 27) x = cp.beta[c + nc * ((q - 18) / 3 + 5 * (q % 3))];
    else x = mark ? 1.0 : 0.0;
    tab[i] = x;
}

struct MarchVjp {
    March64 f;                          // forward window at face J
    double gdm2, gdm1, gd0, gdp1;       // pending gradients of d[J-2] .. d[J+1]
    double gcm3, gcm2, gcm1, gc0, gcp1; // pending gradients of cells J-3 .. J+1

    __device__ __forceinline__ void init(const MarchArgs& a, double c0, double c1, double c2, double c3,
                                         double c4) {
        f.init(a, c0, c1, c2, c3, c4);
        start();
    }
    // row: the row of face J in the table
    __device__ __forceinline__ void init(const MarchArgs& a, const double* row, double c0, double c1, double c2,
                                         double c3, double c4) {
        f.init(a, VjpPair{row - 2 * kVjpRow}, VjpPair{row - kVjpRow}, VjpPair{row}, c0, c1, c2, c3, c4);
        start();
    }
    __device__ __forceinline__ void start() {
        gdm2 = gdm1 = gd0 = gdp1 = 0.0;
        gcm3 = gcm2 = gcm1 = gc0 = gcp1 = 0.0;
    }

    // Face o (centre J = o + 3): accumulate the pull-back of (gL, gR)
    // through the weights and candidates.  Straight-line code (consecutive
    // faces overlap): the limiter's choice is only recorded -- `pick` gets
    // the codes of the left and right state (0: the WENO value passed
    // through) -- and a state whose limiter returned a bound gets its
    // cotangent routed after the chunk (route_side).  `ok` is false when a
    // beta is outside [2^-100, 2^100): the face then contributes nothing
    // here and is redone after the chunk with the generic pull-back.
    // TENOW: TENO weights (f90:578-606), d_k delta_k / sum d delta with the
    // cutoff flags delta_k of the forward sequence; the flags are constant
    // between cutoff flips, so the weights pull nothing back to beta.
    // FULL (layouts and coefficients that vjp_kernel served before):
    // reciprocals within one ulp (rcp_sum); a face whose cotangents are not
    // finite is redone too, and no difference that is not finite enters the
    // sums of a face that is, so NaN and infinities reach the cells that the
    // generic pull-back sends them to and no others.
    template <bool MPF, bool TENOW, bool FULL, class C>
    __device__ __forceinline__ void face(const MarchArgs& a, const C& cf, double gLin, double gRin, int& pick, bool& ok) {
        const March64& w = f;
        ok = beta_ok(w.b0) && beta_ok(w.b1) && beta_ok(w.b2) && !cf.marked();
        if constexpr (FULL) ok = ok && finite_bits(gLin) && finite_bits(gRin);
        const double B0 = ok ? w.b0 : 1.0, B1 = ok ? w.b1 : 1.0, B2 = ok ? w.b2 : 1.0;
        double P0, P1, P2;
        if constexpr (TENOW) {
            bool k0, k1, k2;
            ok = teno5_keep<FULL>(B0, B1, B2, a.wp.teno_ct, k0, k1, k2) && ok;
            P0 = k0 ? 1.0 : 0.0;
            P1 = k1 ? 1.0 : 0.0;
            P2 = k2 ? 1.0 : 0.0;
        } else {
            const double q0 = B0 * B0, q1 = B1 * B1, q2 = B2 * B2;
            P0 = q1 * q2; P1 = q0 * q2; P2 = q0 * q1;
        }
        const double gL = ok ? gLin : 0.0, gR = ok ? gRin : 0.0;
        const bool use = !FULL || ok;
        const double dm2 = use ? w.dm2 : 0.0, dm1 = use ? w.dm1 : 0.0, d0 = use ? w.d0 : 0.0, dp1 = use ? w.dp1 : 0.0;
        const double aL0 = cf(12) * P0, aL1 = cf(13) * P1, aL2 = cf(14) * P2;
        const double aR0 = cf(15) * P0, aR1 = cf(16) * P1, aR2 = cf(17) * P2;
        const double SL = (aL0 + aL1) + aL2, SR = (aR0 + aR1) + aR2;
        const double r = rcp_sum<FULL>(SL * SR), gSL = SR * r, gSR = SL * r;
        const double wL0 = aL0 * gSL, wL1 = aL1 * gSL, wL2 = aL2 * gSL;
        const double wR0 = aR0 * gSR, wR1 = aR1 * gSR, wR2 = aR2 * gSR;
        // candidate offsets e_k = p_k - v0
        const double eL0 = fma(cf(1), d0, cf(0) * dp1), eL1 = fma(cf(3), dm1, cf(2) * d0),
                     eL2 = fma(cf(5), dm2, cf(4) * dm1);
        const double eR0 = fma(cf(7), d0, cf(6) * dp1), eR1 = fma(cf(9), dm1, cf(8) * d0),
                     eR2 = fma(cf(11), dm2, cf(10) * dm1);
        const double xL = fma(wL0, eL0, fma(wL1, eL1, wL2 * eL2));
        const double xR = fma(wR0, eR0, fma(wR1, eR1, wR2 * eR2));
        double gLw = gL, gRw = gR;
        pick = 0;
        if constexpr (MPF) {
            const double kBetaMP = 4.0 / 3.0;
            const bool up_l = sign_clear(w.dm1), up_r = sign_clear(w.d0);
            const double v0 = w.v0;
            int cl, cr;
            {
                const bool pos = sign_clear(xL);
                const double UL = fma(-2.0, w.d0, v0);
                const double MD = fma(-0.5, w.dm1 + w.mA, v0);
                const double LC = fma(kBetaMP, w.mB, fma(-0.5, w.d0, v0));
                mp_pick(v0 + xL, v0, w.vm1, UL, MD, LC, pos, pos != up_l, pos != up_r, cl);
            }
            {
                const bool pos = sign_clear(xR);
                const double UL = fma(2.0, w.dm1, v0);
                const double MD = fma(0.5, w.d0 - w.mB, v0);
                const double LC = fma(kBetaMP, w.mA, fma(0.5, w.dm1, v0));
                mp_pick(v0 + xR, v0, w.vp1, UL, MD, LC, pos, pos == up_r, pos == up_l, cr);
            }
            gLw = cl == kPickW ? gL : 0.0;
            gRw = cr == kPickW ? gR : 0.0;
            pick = ok ? (cl | (cr << 3)) : 0;
        }
        // weights and candidates
        const double gpL0 = gLw * wL0, gpL1 = gLw * wL1, gpL2 = gLw * wL2;
        const double gpR0 = gRw * wR0, gpR1 = gRw * wR1, gpR2 = gRw * wR2;
        gc0 += gLw + gRw;
        gdp1 = fma(cf(0), gpL0, fma(cf(6), gpR0, gdp1));
        gd0 = fma(cf(1), gpL0, fma(cf(7), gpR0, fma(cf(2), gpL1, fma(cf(8), gpR1, gd0))));
        gdm1 = fma(cf(3), gpL1, fma(cf(9), gpR1, fma(cf(4), gpL2, fma(cf(10), gpR2, gdm1))));
        gdm2 = fma(cf(5), gpL2, fma(cf(11), gpR2, gdm2));
        if constexpr (TENOW) return;
        // d out / d beta_k = -2 w_k (e_k - x) / beta_k
        const double t0 = fma(gpL0, eL0 - xL, gpR0 * (eR0 - xR));
        const double t1 = fma(gpL1, eL1 - xL, gpR1 * (eR1 - xR));
        const double t2 = fma(gpL2, eL2 - xL, gpR2 * (eR2 - xR));
        const double b12 = B1 * B2, b02 = B0 * B2, b01 = B0 * B1;
        const double rB = -2.0 * rcp_sum<FULL>(B0 * b12);
        const double gb0 = t0 * (rB * b12), gb1 = t1 * (rB * b02), gb2 = t2 * (rB * b01);
        // beta_0 (d0, dp1): b0 dp1^2 + b1 d0 dp1 + b2 d0^2; beta_1 (dm1, d0); beta_2 (dm2, dm1)
        gdp1 = fma(gb0, fma(cf.twice(0), dp1, cf(19) * d0), gdp1);
        gd0 = fma(gb0, fma(cf(19), dp1, cf.twice(1) * d0), gd0);
        gd0 = fma(gb1, fma(cf.twice(2), d0, cf(22) * dm1), gd0);
        gdm1 = fma(gb1, fma(cf(22), d0, cf.twice(3) * dm1), gdm1);
        gdm1 = fma(gb2, fma(cf.twice(4), dm1, cf(25) * dm2), gdm1);
        gdm2 = fma(gb2, fma(cf(25), dm1, cf.twice(5) * dm2), gdm2);
    }

    // After face o (centre J): d[J-2] is complete, so is cell J-2; returns
    // cell J-3 (= o) and advances to face o+1 with cell J+3 = n.
    __device__ __forceinline__ double advance(const MarchArgs& a, double n) {
        return advance([&](March64& w) { w.push(a, n); });
    }
    // row: the row of face o + 1 in the table
    __device__ __forceinline__ double advance(const MarchArgs& a, const double* row, double n) {
        return advance([&](March64& w) { w.push(a, VjpPair{row}, n); });
    }
    template <class Push>
    __device__ __forceinline__ double advance(const Push& push) {
        gcm1 += gdm2;
        gcm2 -= gdm2;
        const double out = gcm3;
        push(f);
        gdm2 = gdm1; gdm1 = gd0; gd0 = gdp1; gdp1 = 0.0;
        gcm3 = gcm2; gcm2 = gcm1; gcm1 = gc0; gc0 = gcp1; gcp1 = 0.0;
        return out;
    }
};

// Cotangent of one limited state routed to the picked bound expression,
// on cells c[0..4] = J-2 .. J+2 of the face (centre J), added to the
// per-cell sums acc[0..4].  left: nb = J-1, far = J+1; right mirrored.
// MD = (v0 + nb - m)/2, UL = 3 v0 - 2 far, LC = 1.5 v0 - 0.5 far + 4/3 m'
// with m, m' the two minmods; their gradients go through the curvatures
// e2[k] = (v[k+1] - v[k]) - (v[k] - v[k-1]) they picked.
__device__ __forceinline__ void route_side(bool left, int code, double g, const double* c, double* acc) {
    const double kBetaMP = 4.0 / 3.0;
    const int nb = left ? 1 : 3, far = left ? 3 : 1;
    double gmMD = 0.0, gmLC = 0.0;  // cotangents of the minmod in MD and in LC
    switch (code) {
        case kPickV0: acc[2] += g; break;
        case kPickNb: acc[nb] += g; break;
        case kPickMD:
            acc[2] += 0.5 * g;
            acc[nb] += 0.5 * g;
            gmMD = -0.5 * g;
            break;
        case kPickUL:
            acc[2] += 3.0 * g;
            acc[far] -= 2.0 * g;
            break;
        case kPickLC:
            acc[2] += 1.5 * g;
            acc[far] -= 0.5 * g;
            gmLC = kBetaMP * g;
            break;
        default: break;
    }
    // mA = minmod(e2[J-1], e2[J]), mB = minmod(e2[J], e2[J+1]); MD uses mA
    // on the left and mB on the right, LC the other one
    const double gmA = left ? gmMD : gmLC, gmB = left ? gmLC : gmMD;
    if (gmA != 0.0 || gmB != 0.0) {
        const double d0 = c[1] - c[0], d1 = c[2] - c[1], d2 = c[3] - c[2], d3 = c[4] - c[3];
        const double em = d1 - d0, ez = d2 - d1, ep = d3 - d2;
        double a1, a2, b1, b2;
        mm64_grad(em, ez, a1, a2);
        mm64_grad(ez, ep, b1, b2);
        const double ge[3] = {gmA * a1, fma(gmA, a2, gmB * b1), gmB * b2};  // e2[J-1], e2[J], e2[J+1]
        // e2[J+q] = c[q+3] - 2 c[q+2] + c[q+1]
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            acc[q + 2] += ge[q];
            acc[q + 1] -= 2.0 * ge[q];
            acc[q] += ge[q];
        }
    }
}

// SEG: columns in segments; whole columns have kernels of their own, as the
// segment's bounds cost them registers (us per x/y/z gradient of whole columns,
// 128^3 x 5: JS 802 with the bounds, 791 without, TENO 866 and 849).
// PF: coefficients from the per-face table `tab` of `rows` rows (with LDR,
// for every layout), which each CTA copies to shared memory: 28 doubles a
// face, read at warp-uniform addresses.
template <bool MPF, int KIND, bool TENOW, bool LDR, bool PF, bool SEG>
__global__ void __launch_bounds__(kVjpWarps * 32, 1)
    vjp_march_kernel(const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tgL,
                     const __grid_constant__ CUtensorMap tgR, const __grid_constant__ CUtensorMap tgo,
                     const __grid_constant__ CUtensorMap tgs, const __grid_constant__ MarchArgs a,
                     const VjpMarchArgs t, double* __restrict__ gv) {
    static_assert(LDR || !PF, "per-face table: loads by the lanes");
    constexpr int F = kTmaF, S = kVjpStages;
    // column tiles: 34 cells from one left of column 0 (TMA's 16-byte start)
    constexpr int XW = LDR ? 32 : 34, XS = LDR ? 0 : 1;
    extern __shared__ __align__(1024) unsigned char smem_vj[];
    unsigned char* base = smem_vj + ((1024u - (smem_u32(smem_vj) & 1023u)) & 1023u);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char* wbase = base + (size_t)warp * t.warp_bytes;
    // per warp: the cotangent tiles of the S stages (gL, gR: 2048 bytes each,
    // 512-aligned for the swizzle), the field (and old-gradient) tiles of
    // the S stages, then one area that holds the per-lane corrections of a
    // chunk and afterwards (row tiles) the outgoing [32 u][8 cells] tile;
    // LDR: the columns' offsets in the field and in the cotangents, and what
    // the redone first core face adds to the first chunk
    unsigned char* gring = wbase;
    unsigned char* vring = wbase + S * 4096;
    unsigned char* obuf = wbase + S * 4096 + S * t.stage_bytes;   // t.stage_bytes: v (+ old) per stage
    double* slot = (double*)obuf;  // 13 cells f0 .. f0+12 x 32 lanes
    long long* offs = (long long*)(obuf + 13 * 32 * 8);
    long long* offo = offs + 32;
    double* first = (double*)(offo + 32);
    unsigned long long* bars = (unsigned long long*)(base + (size_t)kVjpWarps * t.warp_bytes) + warp * S;
    if (lane == 0) {
        for (int s = 0; s < S; ++s) mbar_init(&bars[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    double* rows = (double*)(base + (size_t)kVjpWarps * t.warp_bytes + (size_t)kVjpWarps * S * 8);
    if constexpr (PF) {
        for (int i = threadIdx.x; i < t.rows * kVjpRow; i += kVjpWarps * 32) rows[i] = __ldg(a.ftab + i);
        __syncthreads();
    }
    __syncwarp();
    const long long nwarps = (long long)gridDim.x * kVjpWarps;
    const int ns = (int)a.ns;
    const int o_last = ns - 3;                // one past the last core face
    const long long ncell = a.ns + 6;
    unsigned n_issued = 0, n_waited = 0, n_out = 0;
    bool failed = false;
    // this lane's column: its cells, its gradient, its cotangents' offset
    const double* col = nullptr;
    double* gcol = nullptr;
    long long oo = 0;

    auto gstage = [&](unsigned k) { return gring + (size_t)(k % S) * 4096; };
    auto vstage = [&](unsigned k) { return vring + (size_t)(k % S) * t.stage_bytes; };
    auto voff = [&](int p) -> unsigned {  // position p of this lane's column in a v / old-gradient tile
        if constexpr (KIND == 0) return swz<double>((unsigned)lane, (unsigned)p);
        else return (unsigned)((p * XW + lane + XS) * 8);
    };
    auto issue = [&](unsigned k, int c, int u0, int w, int v) {
        const int J0 = 4 + F * c;
        unsigned char* sp = gstage(k);
        unsigned char* vp = vstage(k);
        if constexpr (LDR) {
            // cells and faces past the column's end are zero-filled
            auto copy8 = [&](const void* dst, const double* p, bool inb) {
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(smem_u32(dst)), "l"(p),
                             "r"(inb ? 8u : 0u)
                             : "memory");
            };
            // rows along the sweep (the cotangents, and row tiles' cells):
            // eight lanes per row, so one copy touches 4 rows, not 32
            const int pp = lane & (F - 1), o = J0 + pp;
#pragma unroll
            for (int kk = 0; kk < F; ++kk) {
                const int r = lane / F + (32 / F) * kk;
                const unsigned so = swz<double>((unsigned)r, (unsigned)pp);
                const long long co = offo[r] + (o < ns ? o : 0);
                copy8(sp + so, t.gLp + co, o < ns);
                copy8(sp + 2048 + so, t.gRp + co, o < ns);
                if constexpr (KIND == 0)
                    copy8(vp + so, (const double*)a.in + offs[r] + (o < ncell ? o : 0), o < ncell);
            }
            if constexpr (KIND == 1) {
#pragma unroll
                for (int p = 0; p < F; ++p) {
                    const bool in = J0 + p < ncell;
                    copy8(vp + voff(p), col + (in ? J0 + p : 0) * a.sJ, in);
                }
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        } else if (lane == 0) {
            unsigned long long* bar = &bars[k % S];
            const int cU = t.uoff + u0, cW = t.woff + w;
            mbar_arrive_expect_tx(bar, t.tx_bytes);
            const int o1 = t.odimU == 1 ? u0 : w, o2 = t.odimU == 2 ? u0 : w;
            tma_load_4d(sp, &tgL, bar, J0, o1, o2, v);
            tma_load_4d(sp + 2048, &tgR, bar, J0, o1, o2, v);
            const int c0 = t.dimJ == 0 ? J0 : (t.dimU == 0 ? cU : cW);
            const int c1 = t.dimJ == 1 ? J0 : (t.dimU == 1 ? cU : cW);
            const int c2 = t.dimJ == 2 ? J0 : (t.dimU == 2 ? cU : cW);
            tma_load_4d(vp, &tv, bar, c0, c1, c2, v);
            if (t.acc) tma_load_4d(vp + t.vbytes, &tgo, bar, c0, c1, c2, v);
        }
    };
    auto wait_stage = [&](unsigned k) -> bool {
        if constexpr (LDR) {
            // copy groups issued after stage k may stay in flight
            const unsigned after = n_issued - (k + 1);
            if (after >= 2) asm volatile("cp.async.wait_group 2;\n" ::: "memory");
            else if (after == 1) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncwarp();  // the rows are filled by eight lanes each
        } else {
            if (!mbar_wait(&bars[k % S], (k / S) & 1u)) return false;
        }
        n_waited = k + 1;
        return true;
    };
    auto cell = [&](unsigned k, int p) -> double { return *(const double*)(vstage(k) + voff(p)); };
    auto oldg = [&](unsigned k, int p) -> double {
        if constexpr (LDR) return 0.0;  // added by the reductions
        else return t.acc ? *(const double*)(vstage(k) + t.vbytes + voff(p)) : 0.0;
    };
    auto cot = [&](unsigned k, int arr, int i) -> double {
        return *(const double*)(gstage(k) + arr * 2048 + swz<double>((unsigned)lane, (unsigned)i));
    };
    // generic pull-back of face o on the cells c7 = J-3 .. J+3
    auto redo = [&](int o, const double* c7, double gL, double gR, double* acc7) {
        Coef<5> cf;
        if constexpr (PF) {
            cf.load(a.cp.polyL, a.cp.polyR, a.cp.dL, a.cp.dR, a.cp.beta, a.nc, table_core(o, a.nc));
        } else {
            for (int q = 0; q < 6; ++q) { cf.pL[q] = a.ucf[q]; cf.pR[q] = a.ucf[6 + q]; }
            for (int q = 0; q < 3; ++q) { cf.dL[q] = a.ucf[12 + q]; cf.dR[q] = a.ucf[15 + q]; }
            for (int q = 0; q < 9; ++q) cf.b[q] = a.ucf[18 + q];
        }
        face_vjp<5>(c7 + 3, cf, TENOW ? TENO : JS, a.wp.eps, a.wp.teno_ct, MPF, gL, gR, acc7);
    };
    // the pull-back of face o, and the step to face o + 1 with cell n
    auto face = [&](MarchVjp& m, int o, double gL, double gR, int& pk, bool& ok) {
        if constexpr (PF) m.template face<MPF, TENOW, LDR>(a, VjpRow(rows + o * kVjpRow), gL, gR, pk, ok);
        else m.template face<MPF, TENOW, LDR>(a, VjpParam{a, t.b2}, gL, gR, pk, ok);
    };
    auto advance = [&](MarchVjp& m, int o, double n) -> double {
        if constexpr (PF) return m.advance(a, rows + (o + 1) * kVjpRow, n);
        else return m.advance(a, n);
    };

    for (long long item = (long long)blockIdx.x * kVjpWarps + warp; item < a.n_items && !failed; item += nwarps) {
        const int sg = SEG ? (int)(item % a.n_seg) : 0;
        long long tt = SEG ? item / a.n_seg : item;
        int u0 = 0, wv = 0, vv = 0, c_end = 32;
        bool live;
        long long u, wl, vl;
        if constexpr (LDR) {
            const long long c0 = tt * 32;
            live = c0 + lane < a.n_cols;
            c_end = a.n_cols - c0 < 32 ? (int)(a.n_cols - c0) : 32;
            tt = live ? c0 + lane : a.n_cols - 1;  // idle lanes shadow the last column
            u = tt % a.Nu;
            tt /= a.Nu;
            wl = tt % a.Nw;
            vl = tt / a.Nw;
        } else {
            u0 = (int)(tt % a.n_ut) * 32;
            tt /= a.n_ut;
            wv = (int)(tt % a.Nw);
            vv = (int)(tt / a.Nw);
            live = u0 + lane < a.Nu;
            u = live ? u0 + lane : a.Nu - 1;
            wl = wv;
            vl = vv;
        }
        {
            const long long io = a.in_off + u * a.sU + wl * a.sW + vl * a.sV;
            col = (const double*)a.in + io;
            gcol = gv + io;
            oo = u * a.oU + wl * a.oW + vl * a.oV;
            // (the previous item's readers of the offsets synced since)
            if constexpr (LDR) {
                offs[lane] = io;
                offo[lane] = oo;
                __syncwarp();
            }
        }
        // chunks [cs, ce) are written; a segment starts one chunk early, whose
        // faces reach its first cells
        const int n_all = (ns + 1) / F + 1;     // chunks until cell ns+5 is out
        const int cs = SEG ? sg * a.seg : 0, ce = SEG && cs + a.seg < n_all ? cs + a.seg : n_all;
        const int cb = cs > 0 ? cs - 1 : 0;
        const int nch = ce - cb;
        const int ntiles = nch + 1;
        const unsigned k0 = n_issued;
        for (int k = 0; k < ntiles && k < S; ++k) {
            issue(k0 + k, cb + k, u0, wv, vv);
            ++n_issued;
        }
        if (!wait_stage(k0)) { failed = true; break; }

        // the window of the face before the first chunk, f0 - 1 (cells
        // f0 .. f0+4 = positions 0..4 of the first stage)
        // cells 0..3 receive nothing
        if (live && !t.acc && sg == 0)
            for (int q = 0; q < 4; ++q) gcol[q * a.sJ] = 0.0;
        MarchVjp m;
        const int ob = 3 + F * cb;
        if constexpr (PF)
            m.init(a, rows + ob * kVjpRow, cell(k0, 0), cell(k0, 1), cell(k0, 2), cell(k0, 3), cell(k0, 4));
        else m.init(a, cell(k0, 0), cell(k0, 1), cell(k0, 2), cell(k0, 3), cell(k0, 4));
        if constexpr (LDR) first[lane] = 0.0;
        if (cb == 0) {
            // face 3 (a later segment's reaches only cells of the
            // chunk it does not write)
            const double gL = live ? __ldg(t.gLp + oo + 3) : 0.0, gR = live ? __ldg(t.gRp + oo + 3) : 0.0;
            int pk;
            bool ok;
            face(m, 3, gL, gR, pk, ok);
            if (pk || (!ok && live)) {
                // cells 3..9 of the column = J-3 .. J+3 of face 3 (J = 6)
                double c7[7], acc7[7] = {0, 0, 0, 0, 0, 0, 0};
                for (int q = 0; q < 7; ++q) c7[q] = __ldg(col + (3 + q) * a.sJ);
                if (!ok) {
                    redo(3, c7, gL, gR, acc7);
                } else {
                    route_side(true, pk & 7, gL, c7 + 1, acc7 + 1);
                    route_side(false, pk >> 3, gR, c7 + 1, acc7 + 1);
                }
                // acc7[q] is cell J-3+q; pending: J-3 .. J+1, and J+2 through
                // d[J+1] (LDR: with the first chunk, whose cell f0 + 4 it is)
                m.gcm3 += acc7[0];
                m.gcm2 += acc7[1];
                m.gcm1 += acc7[2];
                m.gc0 += acc7[3];
                if constexpr (LDR) {
                    m.gcp1 += acc7[4];
                    first[lane] = acc7[5];
                } else {
                    m.gcp1 += acc7[4] + acc7[5];
                    m.gdp1 += acc7[5];
                }
            }
        }
        (void)advance(m, ob, cell(k0, 5));  // cell f0 - 1: not written here
        // chunk c: faces f0 .. f0+7 (f0 = 4 + 8 (cb + c)); face f0+i pushes cell
        // f0+i+6 = stage c position 6+i (i < 2) or stage c+1 position i-2,
        // and emits cell f0+i = position i of stage c's tiles
        for (int c = 0; c < nch; ++c) {
            const unsigned kc = k0 + c;
            if (!wait_stage(kc + 1)) { failed = true; break; }
            const int f0 = 4 + F * (cb + c);
            const bool emit = !SEG || cb + c >= cs;
            if constexpr (KIND == 0 && !LDR) {
                if (n_out >= 1) {
                    if (lane == 0) bulk_wait_read0();
                    __syncwarp();
                }
            }
            double outv[F];
            unsigned long long picks = 0;
            unsigned bad = 0;
#pragma unroll
            for (int i = 0; i < F; ++i) {
                const int o = f0 + i;
                const bool valid = live && o < o_last;
                const double gL = valid ? cot(kc, 0, i) : 0.0;
                const double gR = valid ? cot(kc, 1, i) : 0.0;
                int pk;
                bool ok;
                face(m, o, gL, gR, pk, ok);
                picks |= (unsigned long long)(valid ? pk : 0) << (6 * i);
                bad |= (ok || !valid) ? 0u : (1u << i);
                outv[i] = advance(m, o, (i < 2) ? cell(kc, 6 + i) : cell(kc + 1, i - 2)) + oldg(kc, i);
            }
            if (LDR && c == 0) outv[4] += first[lane];
            if (__any_sync(0xffffffffu, picks != 0ull || bad != 0u)) {
                // (the area is the row tiles' outgoing tile too; its last store
                // has been read: waited at the start of the chunk)
                // limited states and faces outside the one-reciprocal range:
                // their pull-backs go to per-lane slots of cells f0 .. f0+12
#pragma unroll
                for (int k = 0; k < 13; ++k) slot[k * 32 + lane] = 0.0;
                for (int i = 0; i < F; ++i) {
                    const int pk = (int)((picks >> (6 * i)) & 63ull);
                    const bool again = (bad >> i) & 1u;
                    if (!pk && !again) continue;
                    // cells f0+i .. f0+i+6 = J-3 .. J+3 (J = f0+i+3)
                    double c7[7], acc7[7] = {0, 0, 0, 0, 0, 0, 0};
                    for (int q = 0; q < 7; ++q) {
                        const int k = i + q;  // cell f0 + k: tile c below 8, tile c+1 from 8
                        c7[q] = k < 8 ? cell(kc, k) : cell(kc + 1, k - 8);
                    }
                    const double gL = cot(kc, 0, i), gR = cot(kc, 1, i);
                    if (again) {
                        redo(f0 + i, c7, gL, gR, acc7);
                    } else {
                        route_side(true, pk & 7, gL, c7 + 1, acc7 + 1);
                        route_side(false, pk >> 3, gR, c7 + 1, acc7 + 1);
                    }
                    for (int q = 0; q < 7; ++q)
                        if (i + q < 13) slot[(i + q) * 32 + lane] += acc7[q];
                }
                // slots 0..7 are this chunk's emitted cells, 8..12 the pending
                // cells J-3 .. J+1 of the next face
#pragma unroll
                for (int k = 0; k < F; ++k) outv[k] += slot[k * 32 + lane];
                m.gcm3 += slot[8 * 32 + lane];
                m.gcm2 += slot[9 * 32 + lane];
                m.gcm1 += slot[10 * 32 + lane];
                m.gc0 += slot[11 * 32 + lane];
                m.gcp1 += slot[12 * 32 + lane];
                // (every lane's slots are read before the outgoing tile, which
                // shares their memory, is written)
                if constexpr (KIND == 0) __syncwarp();
            }
            if (emit) {
                if constexpr (KIND == 0) {
                    unsigned char* ob = obuf;
#pragma unroll
                    for (int i = 0; i < F; ++i) *(double*)(ob + swz<double>((unsigned)lane, (unsigned)i)) = outv[i];
                    if constexpr (LDR) {
                        __syncwarp();
                        const int fi = lane & (F - 1);
                        if (f0 + fi < ncell) {
#pragma unroll 4
                            for (int cc = lane / F; cc < c_end; cc += 32 / F) {
                                double* g = gv + offs[cc] + f0 + fi;
                                const double x = *(const double*)(ob + swz<double>((unsigned)cc, (unsigned)fi));
                                if (t.acc) atomicAdd(g, x);
                                else *g = x;
                            }
                        }
                    } else {
                        fence_async_shared();
                        __syncwarp();
                        if (lane == 0) {
                            const int cU = t.uoff + u0, cW = t.woff + wv;
                            const int c0 = t.dimJ == 0 ? f0 : (t.dimU == 0 ? cU : cW);
                            const int c1 = t.dimJ == 1 ? f0 : (t.dimU == 1 ? cU : cW);
                            const int c2 = t.dimJ == 2 ? f0 : (t.dimU == 2 ? cU : cW);
                            tma_store_4d(&tgs, ob, c0, c1, c2, vv);
                            bulk_commit();
                        }
                        ++n_out;
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < F; ++i) {
                        const long long J = (long long)f0 + i;
                        if (live && J < ncell) {
                            if (LDR && t.acc) atomicAdd(gcol + J * a.sJ, outv[i]);
                            else gcol[J * a.sJ] = outv[i];
                        }
                    }
                }
            }
            __syncwarp();
            if (c + S < ntiles) {
                issue(kc + S, cb + c + S, u0, wv, vv);
                ++n_issued;
            }
        }
        if (failed) break;
    }
    if (failed) {
        for (unsigned k = n_waited; k < n_issued; ++k) mbar_wait(&bars[k % S], (k / S) & 1u);
    }
    if (LDR) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    else if (lane == 0) bulk_wait_all();
    __syncwarp();
}

// Cut the columns' chunks into segments for `warps` resident warps, as
// march_segments: a segment runs one chunk more than it writes, and takes
// about a chunk's time to start.
inline void vjp_march_cut(MarchArgs& a, long long tiles, long long warps) {
    const long long chunks = (a.ns + 1) / kTmaF + 1;
    double best = -1.0;
    for (long long n = 1; n <= chunks; ++n) {
        const long long c = (chunks + n - 1) / n;
        if (n > 1 && c == (chunks + n - 2) / (n - 1)) continue;
        const long long nseg = (chunks + c - 1) / c;
        const double exact = (double)(tiles * nseg) / (double)warps;
        const double cost = 0.5 * (exact + std::ceil(exact)) * (double)(c + 1 + (nseg > 1 ? 1 : 0));
        if (best < 0.0 || cost < best) {
            best = cost;
            a.seg = (int)c;
            a.n_seg = (int)nseg;
        }
    }
    a.n_items = tiles * a.n_seg;
}

// Rows of the per-face table (the last chunk's last face reads the pairs of
// three rows after its own), and the most for which it fits into shared
// memory beside the warps' tiles (227 KB in all: sweeps of up to 214 faces);
// longer sweeps take vjp_kernel.
constexpr int kVjpMaxSmem = 227 * 1024;
inline long long vjp_table_rows(const SweepGeom& g) { return (g.ns + 1) / kTmaF * kTmaF + 15; }
constexpr int kVjpLdrWarpBytes = (kVjpStages * (4096 + 2048) + 13 * 32 * 8 + 3 * 32 * 8 + 511) / 512 * 512;
constexpr long long kVjpMaxRows =
    (kVjpMaxSmem - 1024 - kVjpWarps * (kVjpLdrWarpBytes + kVjpStages * 8)) / (kVjpRow * 8);
// Host side: the marching adjoint for FP64 WENO5 with JS or TENO weights and
// face-independent coefficients (ucf), or with the per-face table tab built
// from cp (the lanes then load in every layout).  TMA staging when every base
// and row is a 16-byte multiple, copies by the lanes otherwise.  Returns 1003
// (unsupported) for sweeps of fewer than 8 faces or a lane axis the march
// arguments did not choose; the caller then runs vjp_kernel.  gv must already
// hold what is to be added to when acc is set.
inline int launch_vjp_march(const long long E[3], const SweepGeom& g, int dir, bool folded, bool mp, bool acc,
                            const double* v, const double* ucf, const double* tab, const CoefPtrs& cp,
                            const WenoParams& wp, const double* gL, const double* gR, double* gv, cudaStream_t st,
                            int sms) {
    const EncodeTiledFn enc = tab ? nullptr : encode_tiled_fn();
    if (g.ns < 8 || g.nc < 1) return 1003;
    MarchArgs a = make_march_args(g, v, nullptr, nullptr, wp, ucf);
    a.ftab = tab;
    a.cp = cp;
    VjpMarchArgs t{};
    const bool kind1 = folded && dir != 0;
    if (kind1 != (a.sU == 1)) return 1003;
    t.kind = kind1 ? 1 : 0;
    t.acc = acc ? 1 : 0;
    t.gLp = gL;
    t.gRp = gR;
    for (int k = 0; k < 6; ++k) t.b2[k] = ucf ? 2.0 * ucf[vjp_square(k)] : 0.0;
    cuuint64_t dims[4], strides[3];
    cuuint32_t box[4], estr[4] = {1, 1, 1, 1};
    if (!folded) {
        dims[0] = g.ns + 6; dims[1] = g.c1; dims[2] = g.c2; dims[3] = g.nv;
        t.dimJ = 0; t.dimU = 1; t.dimW = 2; t.uoff = 0; t.woff = 0;
    } else {
        dims[0] = E[0]; dims[1] = E[1]; dims[2] = E[2]; dims[3] = g.nv;
        if (dir == 0) { t.dimJ = 0; t.dimU = 1; t.dimW = 2; t.uoff = 3; t.woff = 3; }
        else if (dir == 1) { t.dimJ = 1; t.dimU = 0; t.dimW = 2; t.uoff = 2; t.woff = 3; }
        else { t.dimJ = 2; t.dimU = 0; t.dimW = 1; t.uoff = 2; t.woff = 3; }
    }
    CUtensorMapSwizzle swz;
    if (!kind1) {
        box[0] = kTmaF; box[1] = 32; box[2] = 1; box[3] = 1;
        swz = CU_TENSOR_MAP_SWIZZLE_64B;
        t.vbytes = 2048;
    } else {
        box[0] = 34; box[1] = 1; box[2] = 1; box[3] = 1;
        box[t.dimJ] = kTmaF;
        swz = CU_TENSOR_MAP_SWIZZLE_NONE;
        t.vbytes = kTmaF * 34 * 8;
    }
    strides[0] = dims[0] * 8;
    strides[1] = dims[0] * dims[1] * 8;
    strides[2] = dims[0] * dims[1] * dims[2] * 8;
    const CUtensorMapDataType dt = CU_TENSOR_MAP_DATA_TYPE_FLOAT64;
    CUtensorMap mv, mL, mR, mo, ms;
    for (CUtensorMap* m : {&mv, &mL, &mR, &mo, &ms}) std::memset(m, 0, sizeof(*m));
    auto make = [&](CUtensorMap* m, const void* p, const cuuint64_t* d, const cuuint64_t* s2, const cuuint32_t* b,
                    CUtensorMapSwizzle z) {
        return enc(m, dt, 4, (void*)p, d, s2, b, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, z,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    cuuint64_t od[4] = {(cuuint64_t)g.ns, (cuuint64_t)g.c1, (cuuint64_t)g.c2, (cuuint64_t)g.nv};
    cuuint64_t os[3] = {(cuuint64_t)g.ns * 8, (cuuint64_t)(g.ns * g.c1) * 8, (cuuint64_t)(g.ns * g.c1 * g.c2) * 8};
    cuuint32_t ob[4] = {kTmaF, 1, 1, 1};
    t.odimU = (a.oU == g.ns) ? 1 : 2;
    ob[t.odimU] = 32;
    // the store map (row tiles) ends at the last column of the sweep, so the
    // lanes past it (the last 32-column tile) write nothing
    cuuint64_t sd[4] = {dims[0], dims[1], dims[2], dims[3]};
    sd[t.dimU] = (cuuint64_t)(t.uoff + a.Nu);
    const bool tma = enc && ((((uintptr_t)v) | ((uintptr_t)gL) | ((uintptr_t)gR) | ((uintptr_t)gv)) & 15) == 0 &&
                     (g.ns & 1) == 0 && strides[0] % 16 == 0 && make(&mv, v, dims, strides, box, swz) &&
                     (!acc || make(&mo, gv, dims, strides, box, swz)) &&
                     (kind1 || make(&ms, gv, sd, strides, box, swz)) &&
                     make(&mL, gL, od, os, ob, CU_TENSOR_MAP_SWIZZLE_64B) &&
                     make(&mR, gR, od, os, ob, CU_TENSOR_MAP_SWIZZLE_64B);
    if (tma) {
        t.stage_bytes = t.vbytes * (acc ? 2 : 1);   // field (+ old gradient) tiles of one stage
        t.tx_bytes = (unsigned)(2 * 2048 + t.vbytes * (acc ? 2 : 1));
    } else {
        t.stage_bytes = 2048;
    }
    t.warp_bytes = tma ? (kVjpStages * (4096 + t.stage_bytes) + 13 * 32 * 8 + 511) / 512 * 512 : kVjpLdrWarpBytes;
    t.rows = tab ? (int)vjp_table_rows(g) : 0;
    const size_t smem = (size_t)t.rows * kVjpRow * 8 + 1024 + (size_t)kVjpWarps * t.warp_bytes + (size_t)kVjpWarps * kVjpStages * 8;
    using KFn = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, MarchArgs, VjpMarchArgs,
                         double*);
    // the occupancy is that of one CTA per SM for every kernel
    // (its registers), so the cut comes first and picks the kernel
    vjp_march_cut(a, tma ? (long long)a.n_ut * a.Nw * a.NV : (a.n_cols + 31) / 32, (long long)sms * kVjpWarps);
#define WSB_VJP_ROW(MPF, TENOW)                                                                                    \
    {{vjp_march_kernel<MPF, 0, TENOW, false, false, false>, vjp_march_kernel<MPF, 1, TENOW, false, false, false>}, \
     {vjp_march_kernel<MPF, 0, TENOW, false, false, true>, vjp_march_kernel<MPF, 1, TENOW, false, false, true>},   \
     {vjp_march_kernel<MPF, 0, TENOW, true, false, true>, vjp_march_kernel<MPF, 1, TENOW, true, false, true>},     \
     {vjp_march_kernel<MPF, 0, TENOW, true, true, true>, vjp_march_kernel<MPF, 1, TENOW, true, true, true>}}
    static const KFn table[2][2][4][2] = {{WSB_VJP_ROW(false, false), WSB_VJP_ROW(true, false)},
                                          {WSB_VJP_ROW(false, true), WSB_VJP_ROW(true, true)}};
#undef WSB_VJP_ROW
    const int form = tma ? (a.n_seg > 1 ? 1 : 0) : (tab ? 3 : 2);
    const KFn kfn = table[wp.scheme == TENO ? 1 : 0][mp ? 1 : 0][form][kind1 ? 1 : 0];
    // always the same limit: the size differs from call to call, and another
    // thread's call must not lower it between here and the launch
    int occ = 0;
    if (cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, kVjpMaxSmem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kfn, kVjpWarps * 32, smem) != cudaSuccess || occ < 1) {
        cudaGetLastError();
        return 1003;
    }
    const long long blocks = std::min((a.n_items + kVjpWarps - 1) / kVjpWarps, (long long)sms * occ);
    kfn<<<(unsigned)blocks, kVjpWarps * 32, smem, st>>>(mv, mL, mR, mo, ms, a, t, gv);
    return 0;
}

}  // namespace wsb
