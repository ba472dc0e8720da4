// Fused RK4 stage kernel.
//
// One launch computes, for every point of every scheduled tile, the Euler right-hand side
//   k = ((-dE/dxi - dF/deta) + diss_xi(alpha_u q) + diss_eta(alpha_v q)) / detJ
// (RHS_upwind, euler/src/lib.rs:571-616; RHS_trad 483-515 without the dissipation terms) and
// performs this stage's share of the RK4 update (integrate::<Rk4>,
// utils/integrate/src/lib.rs:176-222):
//   stage 0: acc  = prev + (b0 dt) k ; next = prev + (a dt) k
//   stage 1: acc += (b1 dt) k        ; next = prev + (a dt) k
//   stage 2: acc += (b2 dt) k        ; next = prev + (a dt) k
//   stage 3: new  = acc + (b3 dt) k
// which is the reference's sequence fut = prev; fut += b_j dt k_j (j = 0..3) evaluated
// incrementally, so the k_j of interior points never go to memory.  Points on a block edge
// store their k in the edge-k buffer instead; the edge kernel (sat_kernel, launched right after
// on the same stream) adds the characteristic SATs in the order north, south, east, west
// (SAT_characteristics, euler/src/lib.rs:1002-1013) and does their update.  The SAT of one
// point is a long dependent f64 chain (vortex data, roots, reciprocals); evaluated by
// a few threads of a tile it held the whole CTA at the next barrier, in a launch of its own it
// runs one thread per edge point.
//
// Work decomposition.  A persistent grid of 256-thread CTAs walks a list of (block, y0, x0)
// output tiles of TY rows x tile_tx(TY) columns (32, with 8 rows 16).  One direction at a time: the fluxes of the tile rows
// widened by the xi halo (Ehat and alpha_u q, 4 components each) go to a shared flux buffer and
// every thread forms the xi sums of its micro-tile in registers; the fluxes of the tile columns
// widened by the eta halo (Fhat, alpha_v q) then replace them in the same buffer for the eta sums.
// Holding one direction's fluxes instead of both leaves room for the tile's raw state and metric
// rows, which arrive by asynchronous copies: the next tile's copies start as soon as the eta fluxes
// are formed and run under the eta sums, the update and the other resident CTA's work.
//   What bounds it.  With direct loads and both directions' fluxes in shared memory (the form
// before this one, one output of four components per thread) a tile waited on global loads for
// most of its time: dropping every stencil sum made an Upwind9 f64 launch only 16% shorter.  Now the
// shared-memory pipe (about 11 wavefronts per point, 53% busy) and issue (42%) lead; FP64 is at 25%
// and HBM at 24%.
//   Micro-tiles.  64 threads per component, each MR rows x MC columns of it (2 x 4 on 16-row tiles):
// a xi window of MC + 2 H values serves MC outputs and an eta window of MR + 2 H rows serves MR, in
// 16-byte loads, instead of D loads per output.  The sums then pass through shared memory once, so
// the update pass reads and writes global memory with consecutive threads on consecutive columns.
//   Measured (f64, the 256 first instances of the seed-1 ensemble, one stage 1 launch): Upwind9
// (3.74 M points) 537 -> 315 us, Upwind4 (3.06 M points) 372 -> 204 us.  One bulk copy per row and
// plane instead of the per-lane copies: 490 us (188 small copies per tile hold up their issuing warp).
//
// Precision: T = double is the f64 form: the reference's terms and stencil sums, with the taps of
// an output in the reference's order as fma chains, one reciprocal of rho per point and a product
// with 1 / J in place of its divisions (compile with -fmad=false, so that every tile shape rounds
// the same way).  T = float with COMP = true runs fluxes, dissipation and
// stencils in f32 and keeps the RK4 state as a (hi, lo) f32 pair; the step's increment
// sum_j (b_j dt) k_j is accumulated in f32 and added to the pair once per step with TwoSum;
// the f32 metrics hold 1 / J (rounded from f64), so the flux divergence is scaled by a product.
// The SAT terms are computed in f64 from f64 metrics.
#pragma once

#include <type_traits>

#include "dependent_launch.cuh"
#include "euler_device.cuh"
#include "eval_program.cuh"
#include "interp.cuh"
#include "sbp_ops.cuh"

namespace sbp {

constexpr int kStageThreads = 256;
constexpr int kTileX = 32;

template <class T>
struct StageArgs {
    const BlockDev* __restrict__ blocks;
    const InstanceDev* __restrict__ inst;
    const int4* __restrict__ tiles;
    int ntiles;
    int stage;               // 0..3 (RK4), or kStageK: write k to u_out (other tableaus)
    double ctime;            // kStageK: the stage's C coefficient (SAT data at time + dt * ctime)
    const T* u_in;           // stage input state, all blocks
    const T* prev_hi;        // state at the start of the step
    const T* prev_lo;        // low part of the state (compensated precision only)
    T* acc_hi;               // RK4 accumulator (compensated form: the step's f32 increment)
    T* u_out;                // next stage input (stages 0..2)
    T* new_hi;               // new state (stage 3)
    T* new_lo;
    T* kedge;                // k of block-edge points, 4 per point (edge_index order per block)
    const double* egeo;      // edge geometry, kEdgeGeo per point (edge_geo_kernel)
    const int4* mg;          // MultiGrid segments (block, start, end, -) of all block sides
    const EvalDev* eval;     // expression programs of SBP_BC_EVAL sides
    double* evz;             // SBP_BC_EVAL data of the launch's edge points (eval_kernel), 4 per point
    const T* met;            // metric planes in T
    const T* jinv;           // f64: 1 / J planes (BlockDev::r_off)
    const float* rinf;       // compensated f32, upwind: free-stream dissipation planes (BlockDev::r_off)
    const double* xy;        // coordinates
    double gamma;
    unsigned* status;
    // fused form, stage 3 of a step: CTAs of all groups (0: the launch advances no time), their counter,
    // and the instances to advance
    int time_ctas, ninst;
    unsigned* time_done;
    const int* active;
};

// Stage index of the k-only mode: the launch computes k = RHS(u_in) (SATs included) into u_out
// and updates nothing else; explicit tableaus other than RK4 combine the k on the host side.
constexpr int kStageK = 4;

// Tiles along a line of n outputs (tile_starts in system.cu) start at multiples of T, except that
// the last tile starts at e = n - M (rounded down to even where T > M) whenever a multiple of T would fall
// in (e, n): so the first tile holds every start-closure output, the last every end-closure output,
// and no tile holds outputs of both ends (n >= 2 M).  The input region of a tile is then at most
// T + 2 H wide (interior tiles and the first one: H on each side, [0, max(T + H, N)) for the
// first; the tile before the last ends at e <= n - M, so its region stops H after it), or
// max(N, M + H + 1) for the last tile, which reads from min(e - H, n - N) to n.
constexpr int region_extent(int T, int H, int M, int N) {
    const int a = T + 2 * H, b = N > M + H + 1 ? N : M + H + 1;
    return a > b ? a : b;
}

// Output rows and columns of a tile: the tile list holds (block, y0, x0, th << 16 | tw).
__device__ __forceinline__ int tile_rows(const int4& td) { return td.w >> 16; }
__device__ __forceinline__ int tile_cols(const int4& td) { return td.w & 0xffff; }

// Characteristic SAT of one edge point (SAT_characteristic, euler/src/lib.rs:1150-1252), f64:
// k += hi tau T ((L + sign |L|) o (T^-1 (y - z))), written row by row so no 4x4 matrix is ever
// live, with five reciprocals in place of the reference's divisions and sqrt(kx^2 + ky^2) in place of
// hypot (no overflow at these magnitudes).  igm1 = 1 / (gamma - 1).
__device__ __forceinline__ void sat_point(double gamma, const double y[4], const double z[4], double hi,
                                               double sign, double tau, double detj, double detj_d_dx,
                                               double detj_d_dy, double igm1, double k[4]) {
    const double rho = y[0], rhou = y[1], rhov = y[2], e = y[3];
    const double ij = 1.0 / detj;
    const double kx_ = detj_d_dx * ij, ky_ = detj_d_dy * ij;
    const double hyp = sqrt(kx_ * kx_ + ky_ * ky_);
    const double ih = 1.0 / hyp;
    const double kx = kx_ * ih, ky = ky_ * ih;
    const double irho = 1.0 / rho;
    const double u = rhou * irho, v = rhov * irho;
    const double gm1 = gamma - 1.0;
    const double q2 = u * u + v * v;
    const double p = gm1 * (e - 0.5 * (rhou * u + rhov * v));
    const double cc = gamma * p * irho;
    const double c = sqrt(cc);
    const double icc = 1.0 / cc;
    const double theta = kx * u + ky * v;
    const double phi2 = 0.5 * gm1 * q2;
    const double alpha = 0.70710678118654752440 * rho * c * icc;  // rho / (sqrt(2) c)
    const double phi2_c2 = (phi2 + cc) * igm1;
    const double U = kx_ * u + ky_ * v;
    const double beta = 0.5 * icc;
    const double r0 = rho - z[0], r1 = rhou - z[1], r2 = rhov - z[2], r3 = e - z[3];
    const double gc = gm1 * icc;
    const double t0 = (1.0 - phi2 * icc) * r0 + gc * (u * r1 + v * r2 - r3);
    const double w = ky * u - kx * v;
    const double t1 = irho * (-w * r0 + ky * r1 - kx * r2);
    const double t2 = beta * ((phi2 - c * theta) * r0 + (kx * c - gm1 * u) * r1 + (ky * c - gm1 * v) * r2 + gm1 * r3);
    const double t3 = beta * ((phi2 + c * theta) * r0 - (kx * c + gm1 * u) * r1 - (ky * c + gm1 * v) * r2 + gm1 * r3);
    const double L2 = U + c * hyp, L3 = U - c * hyp;
    const double f0 = U + sign * fabs(U);
    const double l0 = f0 * t0, l1 = f0 * t1;
    const double l2 = (L2 + sign * fabs(L2)) * t2;
    const double l3 = (L3 + sign * fabs(L3)) * t3;
    const double a2 = alpha * l2, a3 = alpha * l3;
    const double ht = hi * tau;
    k[0] += ht * (l0 + a2 + a3);
    k[1] += ht * (u * l0 + ky * l1 + (u + kx * c) * a2 + (u - kx * c) * a3);
    k[2] += ht * (v * l0 - kx * l1 + (v + ky * c) * a2 + (v - ky * c) * a3);
    k[3] += ht * (phi2 * igm1 * l0 + rho * w * l1 + (phi2_c2 + c * theta) * a2 + (phi2_c2 - c * theta) * a3);
}

// Pointwise quantities of one point of the f64 form in one direction (fluxes,
// euler/src/lib.rs:680-735; upwind_dissipation 619-674) from its state qv and the direction's metrics
// jx, jy (each times detJ): the flux Ehat or Fhat and alpha q into shared memory at dst.  The
// reference divides nine times and takes three roots per point; here one reciprocal of rho serves
// every quotient, and c |J grad| is one root, sqrt(c^2 |J grad|^2): an f64 division or root is
// about twenty instructions, and the region of a tile holds almost two points per output.
template <bool UPW>
__device__ __forceinline__ void pointwise(const double qv[4], double jx, double jy, double gamma, double* dst,
                                          int stride, unsigned& bad) {
    const double rho = qv[0], rhou = qv[1], rhov = qv[2], e = qv[3];
    const double ri = 1.0 / rho;
    const double u = rhou * ri, v = rhov * ri;
    const double p = (gamma - 1.0) * fma_rn(-0.5, fma_rn(rhou, u, rhov * v), e);
    const double h = e + p;
    const double E[4] = {rhou, fma_rn(rhou, u, p), rhou * v, u * h};
    const double F[4] = {rhov, E[2], fma_rn(rhov, v, p), v * h};
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) dst[cc * stride] = fma_rn(jx, E[cc], jy * F[cc]);
    if constexpr (UPW) {
        if (!(rho > 0.0)) bad |= STATUS_RHO;
        if (!(p > 0.0)) bad |= STATUS_P;
        const double a = fabs(fma_rn(jx, u, jy * v)) + sqrt(gamma * p * ri * fma_rn(jx, jx, jy * jy));
        double* d = dst + 4 * stride;
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) d[cc * stride] = a * qv[cc];
    }
}

// Pointwise quantities of the compensated-f32 form, on deviations.  The state is stored as its
// deviation d = q - q_r from the instance's reference state (its free stream), and every
// quantity the stencils read is formed as its own deviation from the value at q_r:
//   Ehat' = Jxi_x (E(q) - E(q_r)) + Jxi_y (F(q) - F(q_r)),   Fhat' likewise with Jeta,
//   (alpha q)' = alpha_u q - alpha_u,r q_r = alpha_u d + (alpha_u - alpha_u,r) q_r,
// where alpha_u,r is alpha_u at q_r on the point's metrics.  Each deviation is evaluated from d
// with algebra that subtracts no two large numbers (below), so its f32 rounding error is
// relative to the deviation, not to the state: for the vortex runs that is two to three orders
// of magnitude smaller.  The parts dropped from the stencil inputs are restored exactly or
// vanish: the fluxes of q_r are constants times the metrics, whose discrete divergence is the
// metric identity d/dxi(Jxi) + d/deta(Jeta) = 0 (the metrics are built by the same operators,
// which commute), and the dissipation of alpha_r q_r is q_r times a time-independent field that
// the system computes once in f64 (BlockDev::r_off) and the stage kernels add to k.
//   rho = rho_r + d0,  u - u_r = (d1 - u_r d0) / rho,  v - v_r = (d2 - v_r d0) / rho,
//   m u - m_r u_r = m_r du + d1 u,  n v - n_r v_r = n_r dv + d2 v,  m v - m_r v_r = m_r dv + d1 v,
//   p - p_r = (gamma - 1) (d3 - (dmu + dnv) / 2),  H - H_r = d3 + dp,
//   u H - u_r H_r = du H_r + u dH,  c^2 - c_r^2 = (gamma / rho_r) (dp rho_r - p_r d0) / rho,
//   c - c_r = (c^2 - c_r^2) / (c + c_r),  |uhat| - |uhat_r| = sign(uhat_r) duhat when both have
//   one sign (else the plain difference, whose operands are then no larger than duhat).
// The reference state is the free stream of the reference's vortex (rho_r = 1, u_r = 1,
// v_r = 0, so m_r = 1 and n_r = 0; only e_r, p_r and c_r vary with the Mach number), which
// removes the terms of m_r, n_r and v_r from the algebra above.
template <bool UPW>
__device__ __forceinline__ void pointwise_dev(const float d[4], const float m[4], float gamma, const RefState& R,
                                              float* sxi, int xa, float* seta, int ya, bool want_xi, bool want_eta,
                                              unsigned& bad) {
    const float rho = 1.0f + d[0];
    const float ri = 1.0f / rho;
    const float du = (d[1] - d[0]) * ri, v = d[2] * ri;  // u - 1 and v
    const float u = 1.0f + du;
    const float dmu = du + d[1] * u;  // m u - 1
    const float dnv = d[2] * v;       // n v
    const float mv = v + d[1] * v;    // m v
    const float dp = (gamma - 1.0f) * (d[3] - 0.5f * (dmu + dnv));
    const float dh = d[3] + dp;
    float E[4], F[4];
    E[0] = d[1];
    E[1] = dmu + dp;
    E[2] = mv;
    E[3] = du * R.h + u * dh;
    F[0] = d[2];
    F[1] = mv;
    F[2] = dnv + dp;
    F[3] = v * (R.h + dh);
    float c = 0.0f, dc = 0.0f;
    if constexpr (UPW) {
        if (!(rho > 0.0f)) bad |= STATUS_RHO;
        if (!(R.p + dp > 0.0f)) bad |= STATUS_P;
        const float dc2 = gamma * (dp - R.p * d[0]) * ri;  // c^2 - c_r^2 with rho_r = 1
        c = sqrtf(R.c2 + dc2);
        dc = dc2 / (c + R.c);
    }
    auto store = [&](float jx, float jy, float* dst, int stride) {
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) dst[cc * stride] = jx * E[cc] + jy * F[cc];
        if constexpr (UPW) {
            const float dhat = jx * du + jy * v;  // uhat - uhat_r, uhat_r = jx
            const float hat = jx + dhat;
            const float dabs = hat * jx > 0.0f ? (jx > 0.0f ? dhat : -dhat) : fabsf(hat) - fabsf(jx);
            const float s = sqrtf(jx * jx + jy * jy);
            const float a = fabsf(hat) + c * s;
            const float da = dabs + dc * s;
            float* o = dst + 4 * stride;
            o[0] = a * d[0] + da;  // q_r = (1, 1, 0, e_r)
            o[stride] = a * d[1] + da;
            o[2 * stride] = a * d[2];
            o[3 * stride] = a * d[3] + da * R.q[3];
        }
    };
    if (want_xi) store(m[0], m[1], sxi, xa);
    if (want_eta) store(m[2], m[3], seta, ya);
}

// This stage's RK4 update of one component at element e (see the header comment) with its operands
// in registers: o0, o1, o2 as loaded by the update pass of stage_kernel; cb, ca this stage's B and A
// tableau entries times dt (ca unused in stage 3).  The compensated form accumulates the step's
// increment delta = sum_j (b_j dt) k_j in f32 (acc_hi) and adds it to the (hi, lo) state once, in
// stage 3, with TwoSum.
template <class T, bool COMP>
__device__ __forceinline__ void rk_update_ops(const StageArgs<T>& A, int64_t e, T cb, T ca, T k, T o0, T o1, T o2) {
    if (A.stage == kStageK) {
        A.u_out[e] = k;
    } else if (A.stage == 0) {
        A.u_out[e] = fma_rn(ca, k, o0);
        A.acc_hi[e] = COMP ? cb * k : fma_rn(cb, k, o0);
    } else if (A.stage < 3) {
        A.u_out[e] = fma_rn(ca, k, o1);
        A.acc_hi[e] = fma_rn(cb, k, o0);
    } else if constexpr (COMP) {
        float hi = o1, lo = o2;
        comp_add(hi, lo, fma_rn(cb, k, o0));
        A.new_hi[e] = hi;
        A.new_lo[e] = lo;
    } else {
        A.new_hi[e] = fma_rn(cb, k, o0);
    }
}

// Element of a block's edge opposite to side d (north -> the block's south row, ...) at position
// k along that edge: the point whose state a neighbour's side-d SAT reads.
__device__ __forceinline__ int opposite_edge_point(int d, int k, int gnx, int gny) {
    if (d == NORTH) return k;                      // south row
    if (d == SOUTH) return (gny - 1) * gnx + k;    // north row
    if (d == EAST) return k * gnx;                 // west column
    return k * gnx + (gnx - 1);                    // east column
}

// Value of component cc of a state stored in T at a point of block Gb, as the absolute state:
// the compensated-f32 form stores deviations from the instance's reference state.
template <class T>
__device__ __forceinline__ double absolute_state(const StageArgs<T>& A, const BlockDev& Gb, int cc, T v) {
    if constexpr (sizeof(T) == 4) return double(v) + A.inst[Gb.instance].qref[cc];
    else return double(v);
}

// The time-independent data of one block-edge point the SATs read: coordinates, the f64
// metrics (detJ, J dxi/dx, J dxi/dy, J deta/dx, J deta/dy).
struct EdgeGeo {
    double x, y, m[5];
};
// A schedule gathers the geometry of its block-edge points once into one contiguous 64-byte record per
// point (slot e_off + edge_index: x, y, detJ, the 4 metric terms, padding; edge_geo_kernel), which
// the SATs read instead of seven scattered sectors (the first and last columns of a block are nx
// elements apart).
constexpr int kEdgeGeo = 8;
__device__ __forceinline__ EdgeGeo edge_record(const double* p) {
    const double2* gp = reinterpret_cast<const double2*>(p);
    const double2 g0 = gp[0], g1 = gp[1], g2 = gp[2], g3 = gp[3];
    return EdgeGeo{g0.x, g0.y, {g1.x, g1.y, g2.x, g2.y, g3.x}};
}

// The sides of a block on which an edge point lies (at most two of N, S, E, W, in that order; -1: none),
// and the vortex data at the point if one of them takes those: what its SATs need beside the state.
struct SatSides {
    int d[2];
    double z[4];
};
template <class T>
__device__ __forceinline__ SatSides sat_sides(const StageArgs<T>& A, const InstanceDev& I, const BlockDev& B, int row,
                                              int col, const EdgeGeo& geo) {
    const double cst = A.stage == kStageK ? A.ctime : (A.stage == 0 ? 0.0 : (A.stage == 3 ? 1.0 : 0.5));
    const double stime = cst == 0.0 ? I.time : I.time + I.dt * cst;
    const int ns = row == B.ny - 1 ? NORTH : (row == 0 ? SOUTH : -1);
    const int ew = col == B.nx - 1 ? EAST : (col == 0 ? WEST : -1);
    SatSides s{};
    s.d[0] = ns >= 0 ? ns : ew;
    s.d[1] = ns >= 0 ? ew : -1;
    if ((s.d[0] >= 0 && B.bc_kind[s.d[0]] == BC_VORTEX) || (s.d[1] >= 0 && B.bc_kind[s.d[1]] == BC_VORTEX)) {
        if (A.gamma == 1.4 && (sizeof(T) == 4 || I.v_regular))
            vortex_point_fast(I, stime, geo.x, geo.y, s.z);
        else
            vortex_point<true>(I, A.gamma, stime, geo.x, geo.y, s.z);
    }
    return s;
}

// Sum of the SATs of one block-edge point in the reference's order N, S, E, W, added to kv.
template <class T>
__device__ __forceinline__ void sat_apply(const StageArgs<T>& A, const InstanceDev& I, const BlockDev& B, int eidx, int row,
                                          int col, const EdgeGeo& geo, const SatSides& side, const double yv[4],
                                          double kv[4]) {
    const int nx = B.nx, ny = B.ny;
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
        const int d = k == 0 ? side.d[0] : side.d[1];
        if (d < 0) continue;
        double zv[4];
        const int kind = B.bc_kind[d];
        if (kind == BC_VORTEX) {
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) zv[cc] = side.z[cc];
        } else if (kind == BC_EVAL) {
            // BoundaryCharacteristic::Eval (euler/src/lib.rs:853-863): the expressions at the stage
            // time, evaluated for this edge point by eval_kernel just before
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) zv[cc] = A.evz[4 * (int64_t)eidx + cc];
        } else if (kind == BC_INTERPOLATE || kind == BC_MULTIGRID) {
            // boundary_extract (euler/src/lib.rs:816-846): data from neighbours' opposite edges
            const bool ns_ = d == NORTH || d == SOUTH;
            const int i = ns_ ? col : row;       // position along this edge
            const int len = ns_ ? nx : ny;
            if (kind == BC_INTERPOLATE) {
                const BlockDev& Gb = A.blocks[B.bc_nb[d]];
                const T* gq = A.u_in + Gb.q_off;
                const int lg = ns_ ? Gb.nx : Gb.ny;
                const bool f2c = nx < Gb.nx;  // fine2coarse when this block's nx is smaller (:818)
                // in f64 for both state precisions (the f32 state widened), as the SAT itself
                const InterpDev<double> ip = interp_dev<double>(B.bc_aux[d], f2c);
#pragma unroll 1
                for (int cc = 0; cc < 4; ++cc) {
                    const T* plane = gq + cc * (int64_t)Gb.npad;
                    zv[cc] = interp_at<double>(ip, i, lg, len, [&](int64_t k) {
                        return absolute_state<T>(A, Gb, cc, plane[opposite_edge_point(d, (int)k, Gb.nx, Gb.ny)]);
                    });
                }
            } else {
                // Segments (g, start, end) are laid end to end, each starting on the previous
                // one's last point; the first point of every segment but the last is halved.
                const int4* sg = A.mg + B.bc_aux[d];
                const int nseg = B.bc_aux2[d];
                int p0 = 0, hit = 0, hp = 0;
                for (int k = 0; k < nseg; ++k) {
                    const int n = sg[k].z - sg[k].y;
                    if (i >= p0 && i < p0 + n) {
                        hit = k;
                        hp = p0;
                    }
                    p0 += n - 1;
                }
                const int4 seg = sg[hit];
                const BlockDev& Gb = A.blocks[seg.x];
                const T* gq = A.u_in + Gb.q_off;
                const int gp = opposite_edge_point(d, seg.y + (i - hp), Gb.nx, Gb.ny);
                const bool halve = i == hp && hit != nseg - 1;
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    const double v = absolute_state<T>(A, Gb, cc, gq[cc * (int64_t)Gb.npad + gp]);
                    zv[cc] = halve ? v / 2.0 : v;
                }
            }
        } else {
            // This: own opposite edge; Grid(g): neighbour's opposite edge
            // (boundary_extracts, euler/src/lib.rs:869-930).
            const BlockDev& Gb = kind == BC_GRID ? A.blocks[B.bc_nb[d]] : B;
            const T* gq = A.u_in + Gb.q_off;
            const int gp = opposite_edge_point(d, (d == NORTH || d == SOUTH) ? col : row, Gb.nx, Gb.ny);
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) zv[cc] = absolute_state<T>(A, Gb, cc, gq[cc * (int64_t)Gb.npad + gp]);
        }
        const bool ns = d == NORTH || d == SOUTH;
        const double sign = (d == NORTH || d == EAST) ? -1.0 : 1.0;
        const double tau = (d == NORTH || d == EAST) ? 1.0 : -1.0;
        const double hi = ns ? B.hi_eta : B.hi_xi;
        const double ddx = ns ? geo.m[3] : geo.m[1];
        const double ddy = ns ? geo.m[4] : geo.m[2];
        sat_point(A.gamma, yv, zv, hi, sign, tau, geo.m[0], ddx, ddy, I.v_igm1, kv);
    }
}

// ---- geometry of one tile ------------------------------------------------------------------
// Tiles are TY rows x tile_tx(TY) columns; 256 threads, 64 per component.  A thread's micro-tile
// is tile_mr(TY) rows x tile_mc(TY) columns, so 8 x 8 threads cover a tile of one component.
__host__ __device__ constexpr int tile_tx(int ty) { return ty == 8 ? 16 : kTileX; }
__host__ __device__ constexpr int tile_mr(int ty) { return ty / 8; }
__host__ __device__ constexpr int tile_mc(int ty) { return tile_tx(ty) / 8; }

// Local column of column x is x - x0 + xi_lead: room for the H halo columns, and for the N - M
// columns before the last M that an end-closure block reads; xi_lead - H is even, so that every
// thread's window starts at a pair.  Rows have the same without the evenness.
__host__ __device__ constexpr int lead_of(int H, int M, int N) { return H > N - M ? H : N - M; }
__host__ __device__ constexpr int xi_lead(int H, int M, int N) { return H + ((lead_of(H, M, N) - H + 1) & ~1); }
// 16-byte (f64) pairs of adjacent columns that one thread's xi window spans.
__host__ __device__ constexpr int xi_window(int ty, int H, int M, int N) {
    return (tile_mc(ty) + 2 * H + 1) / 2;
}
// Column pairs of one xi row: every region column, and every thread's window.
__host__ __device__ constexpr int xi_pairs(int ty, int H, int M, int N) {
    const int L = xi_lead(H, M, N), a = L + (tile_tx(ty) + H > N ? tile_tx(ty) + H : N);
    const int b = tile_tx(ty) - tile_mc(ty) + L - H + 2 * xi_window(ty, H, M, N);
    return ((a > b ? a : b) + 1) / 2;
}
// Pair p of a row is at slot (p & 1) * S + (p >> 1): the 8 threads of one micro-row read pairs
// of one parity, 8 consecutive 16-byte slots.  S = 4 (mod 8) puts 16 consecutive columns stored
// by phase 1 on 16 different 8-byte banks; an odd number of slots per row spreads the rows that
// the closure pass reads down a column.
__host__ __device__ constexpr int xi_split(int ty, int H, int M, int N) {
    return (xi_pairs(ty, H, M, N) + 1) / 2 <= 4 ? 4 : 12;
}
__host__ __device__ constexpr int xi_pitch(int ty, int H, int M, int N) {
    return 2 * ((xi_split(ty, H, M, N) + xi_pairs(ty, H, M, N) / 2) | 1);
}
__host__ __device__ constexpr int eta_rows(int ty, int H, int M, int N) {
    return lead_of(H, M, N) + (ty + H > N ? ty + H : N);
}
// Raw rows of a tile's region (state and xi metrics) and of its columns (eta metrics), widened to
// 16-byte boundaries; `al` elements are 16 bytes.
__host__ __device__ constexpr int raw_pitch(int w, int al) { return (w + 2 * (al - 1)) / al * al; }
__host__ __device__ constexpr int xi_region(int ty, int H, int M, int N) {
    return region_extent(tile_tx(ty), H, M, N);
}
__host__ __device__ constexpr int flux_elems(int ty, int hx, int mx, int nx, int hy, int my, int ny) {
    const int a = ty * xi_pitch(ty, hx, mx, nx), b = eta_rows(ty, hy, my, ny) * tile_tx(ty);
    return a > b ? a : b;
}
// Shared memory of a tile in bytes (elements of `ts` bytes): the raw rows and the fluxes of one
// direction.
__host__ __device__ constexpr int tile_smem(int ty, bool upw, int ts, int hx, int mx, int nx, int hy, int my, int ny) {
    const int al = 16 / ts, rp = raw_pitch(xi_region(ty, hx, mx, nx), al), ep = raw_pitch(tile_tx(ty), al);
    const int rh = eta_rows(ty, hy, my, ny);
    return ts * (4 * rh * rp + 2 * ty * rp + 2 * rh * ep + (upw ? 8 : 4) * flux_elems(ty, hx, mx, nx, hy, my, ny));
}

template <int OPX, int OPY, int TY, class T>
struct TileGeom {
    using X = OpShape<OPX>;
    using Y = OpShape<OPY>;
    static constexpr int TX = tile_tx(TY), MR = tile_mr(TY), MC = tile_mc(TY);
    static constexpr int XL = xi_lead(X::H, X::M, X::N), YL = lead_of(Y::H, Y::M, Y::N);
    static constexpr int NP = xi_window(TY, X::H, X::M, X::N);
    static constexpr int XS = xi_split(TY, X::H, X::M, X::N), XP = xi_pitch(TY, X::H, X::M, X::N);
    static constexpr int XA = TY * XP;                                    // elements of one xi array
    static constexpr int YA = eta_rows(TY, Y::H, Y::M, Y::N) * TX;        // elements of one eta array
    static constexpr int RH = eta_rows(TY, Y::H, Y::M, Y::N);
    static constexpr int RP = raw_pitch(xi_region(TY, X::H, X::M, X::N), 16 / (int)sizeof(T));
    static constexpr int EP = raw_pitch(TX, 16 / (int)sizeof(T));
    static constexpr int FL = flux_elems(TY, X::H, X::M, X::N, Y::H, Y::M, Y::N);
    static_assert(xi_pairs(TY, X::H, X::M, X::N) <= 24, "xi rows fit the split");
    // element of local column c in a xi row
    __device__ __forceinline__ static int xpos(int c) { return (((c >> 1) & 1) * XS + (c >> 2)) * 2 + (c & 1); }
    // Element of tile column c in an eta row.  Micro-tiles of 4 columns: the even column pairs
    // first, then the odd ones with their halves of 4 pairs exchanged, so both the 16-byte loads of
    // phase 2 (8 threads, one parity) and the 8-byte stores of 16 consecutive columns use every
    // bank once.  Micro-tiles of 2 columns: in order.
    __device__ __forceinline__ static int epos(int c) {
        if constexpr (MC == 2) return c;
        const int p = c >> 1;
        return (((p & 1) * (TX / 4)) + ((p >> 1) ^ ((p & 1) * 4))) * 2 + (c & 1);
    }
};

template <class T>
struct PairOf;
template <>
struct PairOf<double> {
    using type = double2;
};
template <>
struct PairOf<float> {
    using type = float2;
};

// acc += sign * (taps I .. D - 1 of one interior stencil), w[d] the input of tap d; coefficients
// are compile-time constants and zero taps cost nothing.
template <int OP, int KIND, int SIGN, int I, class T>
__device__ __forceinline__ void add_taps(const T* w, T& acc) {
    if constexpr (I < OpShape<OP>::D) {
        constexpr T c = CDiag<OP, KIND, T>::v[I];
        if constexpr (c != T(0)) acc = fma_rn(T(SIGN) * c, w[I], acc);
        add_taps<OP, KIND, SIGN, I + 1>(w, acc);
    }
}

// Xi sums of a micro-tile: acc[u][j] += sign * stencil at (row u, column j); row 0's array row at
// `row`, the first pair of the thread's window at slot `s0` of parity PAR0.
template <int OP, int KIND, int SIGN, class G, class T>
__device__ __forceinline__ void xi_sums(const T* __restrict__ row, int gx, T acc[G::MR][G::MC]) {
    using V = typename PairOf<T>::type;
    constexpr int OFF = G::XL - OpShape<OP>::H;  // local column of the first tap of tile column 0
#pragma unroll
    for (int u = 0; u < G::MR; ++u) {
        T w[2 * G::NP];
#pragma unroll
        for (int q = 0; q < G::NP; ++q) {
            // pair p = gx MC / 2 + OFF / 2 + q
            int slot;
            if constexpr (G::MC == 4) {
                constexpr int o = OFF / 2;
                slot = ((o + q) & 1) * G::XS + gx + ((o + q) >> 1);
            } else {
                const int p = gx + OFF / 2 + q;
                slot = (p & 1) * G::XS + (p >> 1);
            }
            const V v = reinterpret_cast<const V*>(row + u * G::XP)[slot];
            w[2 * q] = v.x;
            w[2 * q + 1] = v.y;
        }
#pragma unroll
        for (int j = 0; j < G::MC; ++j) add_taps<OP, KIND, SIGN, 0>(w + j, acc[u][j]);
    }
}

// Row R of the eta window applied to the MR outputs of each column, then the rows after it.
template <int OP, int KIND, int SIGN, class G, int R, int U, class T>
__device__ __forceinline__ void eta_row_taps(const T v[G::MC], T acc[G::MR][G::MC]) {
    if constexpr (U < G::MR) {
        constexpr int d = R - U;
        if constexpr (d >= 0 && d < OpShape<OP>::D) {
            constexpr T c = CDiag<OP, KIND, T>::v[d];
            if constexpr (c != T(0)) {
#pragma unroll
                for (int j = 0; j < G::MC; ++j) acc[U][j] = fma_rn(T(SIGN) * c, v[j], acc[U][j]);
            }
        }
        eta_row_taps<OP, KIND, SIGN, G, R, U + 1>(v, acc);
    }
}
template <int OP, int KIND, int SIGN, class G, int R, class T>
__device__ __forceinline__ void eta_sums(const T* __restrict__ col, int gx, T acc[G::MR][G::MC]) {
    using V = typename PairOf<T>::type;
    if constexpr (R < G::MR + OpShape<OP>::D - 1) {
        T v[G::MC];
        const V* p = reinterpret_cast<const V*>(col + R * G::TX);
        const V a = p[gx];
        v[0] = a.x;
        v[1] = a.y;
        if constexpr (G::MC == 4) {
            const V b = p[G::TX / 4 + (gx ^ 4)];
            v[2] = b.x;
            v[3] = b.y;
        }
        eta_row_taps<OP, KIND, SIGN, G, R, 0>(v, acc);
        eta_sums<OP, KIND, SIGN, G, R + 1>(col, gx, acc);
    }
}

// Closure-block coefficient (row I, input K) of one end of a line: the start block, or the end
// block (row I applies -/+ st[(M - 1 - I) N + (N - 1 - K)], DIFF negated).
template <int OP, int KIND, bool RIGHT, int I, int K, class T>
struct ClosureCoef {
    static constexpr int M = OpShape<OP>::M, N = OpShape<OP>::N;
    static constexpr T value = RIGHT ? (KIND == DIFF ? T(-1) : T(1)) * CDiag<OP, KIND, T>::st[(M - 1 - I) * N + (N - 1 - K)]
                                     : CDiag<OP, KIND, T>::st[I * N + K];
};
// Row I of the closure block: the sum over the N inputs v, first product then an fma chain.
template <int OP, int KIND, bool RIGHT, int I, int K = 1, class T>
__device__ __forceinline__ T closure_sum(const T* v, T t) {
    if constexpr (K == 1) t = v[0] * ClosureCoef<OP, KIND, RIGHT, I, 0, T>::value;
    if constexpr (K < OpShape<OP>::N) {
        constexpr T c = ClosureCoef<OP, KIND, RIGHT, I, K, T>::value;
        return closure_sum<OP, KIND, RIGHT, I, K + 1>(v, fma_rn(v[K], c, t));
    } else {
        return t;
    }
}
// st(i, diss - diff) for closure rows i = I .. I + CNT - 1.
template <int OP, bool UPW, bool RIGHT, int I, int CNT, class T, class ST>
__device__ __forceinline__ void closure_out(const T* ve, const T* va, const ST& st) {
    if constexpr (CNT > 0) {
        T d = T(0);
        if constexpr (UPW) d = closure_sum<OP, DISS, RIGHT, I>(va, T(0));
        st(I, d - closure_sum<OP, DIFF, RIGHT, I>(ve, T(0)));
        closure_out<OP, UPW, RIGHT, I + 1, CNT - 1>(ve, va, st);
    }
}

// Closure outputs part * CNT .. of one line (diss - diff) into o[CNT], for the warp-uniform run-time
// `part` of PARTS: ld(kind, k) is input k of the closure block.
template <int OP, bool UPW, bool RIGHT, int PARTS, int P, class T, class LD>
__device__ __forceinline__ void closure_part(int part, const LD& ld, T* o) {
    constexpr int M = OpShape<OP>::M, N = OpShape<OP>::N, CNT = M >= PARTS ? M / PARTS : 1;
    if constexpr (P * CNT < M && P < PARTS) {
        if (part == P) {
            T ve[N], va[N];
#pragma unroll
            for (int k = 0; k < N; ++k) {
                ve[k] = ld(DIFF, k);
                va[k] = UPW ? ld(DISS, k) : T(0);
            }
            closure_out<OP, UPW, RIGHT, P * CNT, CNT>(ve, va, [&](int i, T v) { o[i - P * CNT] = v; });
        } else {
            closure_part<OP, UPW, RIGHT, PARTS, P + 1>(part, ld, o);
        }
    }
}

// 16-byte asynchronous global -> shared copy (cp.async), and the wait for all of this thread's.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The SAT threads of the fused form: the tiles of the CTA in the order of the stencil threads, one edge
// point per thread, its SAT terms into ssat (slot: tile column on a horizontal edge, TX + tile row on a
// vertical one).  Two barriers per tile with the stencil threads: terms ready, terms used.
template <int MX, int MY, class T, int TY>
__device__ __forceinline__ void sat_tiles(const StageArgs<T>& A, double* __restrict__ ssat) {
    constexpr int TX = tile_tx(TY);
    const int lane = threadIdx.x - kStageThreads;
    bool waited = false;
    for (int t = blockIdx.x; t < A.ntiles; t += gridDim.x) {
        const int4 td = A.tiles[t];
        const BlockDev& B = A.blocks[td.x];
        const int nx = B.nx, ny = B.ny, y0 = td.y, x0 = td.z, th = tile_rows(td), tw = tile_cols(td);
        if ((x0 < MX && x0 + tw > nx - MX) || (y0 < MY && y0 + th > ny - MY)) return;  // as the stencil threads
        const bool top = y0 == 0, bot = y0 + th == ny, left = x0 == 0, right = x0 + tw == nx;
        const int nh = top || bot ? tw : 0, nv = left || right ? th : 0;
        int row = -1, col = -1;
        if (lane < nh) {
            row = top ? 0 : ny - 1;
            col = x0 + lane;
        } else if (lane < nh + nv) {
            row = y0 + lane - nh;
            col = left ? 0 : nx - 1;
            if (nh && row == (top ? 0 : ny - 1)) row = -1;  // the corner is in the row
        }
        const InstanceDev& I = A.inst[B.instance];
        EdgeGeo geo{};
        SatSides side{};
        if (row >= 0) {
            geo = edge_record(A.egeo + kEdgeGeo * (B.e_off + edge_index(row, col, nx, ny)));
            side = sat_sides(A, I, B, row, col, geo);
        }
        if (!waited) {
            dependency_wait();
            waited = true;
        }
        if (row >= 0) {
            const T* q = A.u_in + B.q_off + row * nx + col;
            double yv[4], sv[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) yv[cc] = absolute_state<T>(A, B, cc, q[cc * (int64_t)B.npad]);
            sat_apply<T>(A, I, B, 0, row, col, geo, side, yv, sv);
            const int slot = row == 0 || row == ny - 1 ? col - x0 : TX + row - y0;
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) ssat[4 * slot + cc] = sv[cc];
        }
        __syncthreads();
        __syncthreads();
    }
    if (!waited) dependency_wait();
}

// Threads of the fused form that evaluate the SATs: one per edge point of a tile, which lies on at
// most one horizontal and one vertical block edge.
__host__ __device__ constexpr int sat_threads(int ty) { return ty + tile_tx(ty) <= 32 ? 32 : 64; }

// Barrier of the kStageThreads stencil threads (all threads where there are no others).
__device__ __forceinline__ void tile_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kStageThreads) : "memory"); }

// SATF: the fused form for systems that leave SMs without work (see fused_rows in system.cu).  The
// SATs of a tile's edge points are evaluated in the same launch by threads of their own, beside the
// stencils, instead of an edge kernel after it, and the last CTA of stage 3 advances the instance
// times: a step is four launches instead of nine.
// The stage launches of a step after its first are dependent ones: what does not depend on the stage
// input -- the metric rows, the edge geometry, the vortex boundary data -- is fetched and evaluated
// before the predecessor has finished, and a kernel lets its successor start only after its own
// wait, so that such early work sees the finished step before it.
//   Measured, us per step, separate -> fused: one 64 x 64 Upwind4 block 64 -> 21 (f64), 64 -> 21
// (compensated); six Upwind9 blocks of 37,310 points 70 -> 39 and 68 -> 35.
template <int OPX, int OPY, class T, bool UPW, bool COMP, int TY, bool SATF>
__global__ void __launch_bounds__(kStageThreads + (SATF ? sat_threads(TY) : 0),
                                  SATF || (TY == 32 && sizeof(T) == 8) ? 1 : 2) stage_kernel(const StageArgs<T> A) {
    using G = TileGeom<OPX, OPY, TY, T>;
    using V = typename PairOf<T>::type;
    constexpr int TX = G::TX, MR = G::MR, MC = G::MC, XA = G::XA, YA = G::YA, RP = G::RP, EP = G::EP, RH = G::RH;
    constexpr int HY = OpShape<OPY>::H, MX = OpShape<OPX>::M, MY = OpShape<OPY>::M;
    constexpr int AL = 16 / sizeof(T);  // elements of a 16-byte copy unit
    // update pass: points and components per thread
    constexpr int PTS = TY * TX, PPT = PTS >= kStageThreads ? PTS / kStageThreads : 1;
    constexpr int CPT = PTS >= kStageThreads ? 4 : 4 * PTS / kStageThreads;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* rq = reinterpret_cast<T*>(smem_raw);  // [4][RH][RP]: raw state of the tile's region
    T* rx = rq + 4 * RH * RP;                // [2][TY][RP]: raw xi metrics of the tile rows
    T* re = rx + 2 * TY * RP;                // [2][RH][EP]: raw eta metrics of the tile columns
    T* fl = re + 2 * RH * EP;                // fluxes of one direction: [UPW ? 8 : 4] xi or eta arrays
    // SATF: the SAT terms of the tile's edge points, one row of points then one column
    double* ssat = reinterpret_cast<double*>(smem_raw + tile_smem(TY, UPW, sizeof(T), OpShape<OPX>::H, OpShape<OPX>::M,
                                                                  OpShape<OPX>::N, OpShape<OPY>::H, OpShape<OPY>::M,
                                                                  OpShape<OPY>::N));
    const T gamma = T(A.gamma);
    const int tid = threadIdx.x;
    const int comp = tid >> 6, gx = tid & 7, gy = (tid >> 3) & 7;  // stencil phases
    unsigned bad = 0;

    // Starts the asynchronous copies of one tile's raw rows: every row of the region's state planes,
    // the xi metrics of the tile rows and the eta metrics of the tile columns, a warp per row, in
    // 16-byte pieces widened to 16-byte boundaries (a plane's padding holds the overhang).
    // what: 1 = metrics, 2 = state, 3 = both.
    auto fetch = [&](const int4 td, int what) {
        const BlockDev& B = A.blocks[td.x];
        const int nx = B.nx, np = B.npad, y0 = td.y, x0 = td.z;
        const int th = tile_rows(td), tw = tile_cols(td);
        int lx0, lx1, ly0, ly1;
        region_of<OPX>(x0, x0 + tw, nx, lx0, lx1);
        region_of<OPY>(y0, y0 + th, B.ny, ly0, ly1);
        const T* q = A.u_in + B.q_off;
        const T* mt = A.met + B.m_off;
        const int warp = tid >> 5, lane = tid & 31;
        for (int r = warp; r < ly1 - ly0; r += kStageThreads / 32) {
            const int off = (ly0 + r) * nx;
            {
                const int e = ((off + lx0) & ~(AL - 1)) + lane * AL;
                if (e < off + lx1) {
                    if (what & 2) {
#pragma unroll
                        for (int pl = 0; pl < 4; ++pl) cp_async16(rq + (pl * RH + r) * RP + lane * AL, q + pl * np + e);
                    }
                    const int tr = ly0 + r - y0;
                    if ((what & 1) && tr >= 0 && tr < th) {
#pragma unroll
                        for (int pl = 0; pl < 2; ++pl)
                            cp_async16(rx + (pl * TY + tr) * RP + lane * AL, mt + (1 + pl) * np + e);
                    }
                }
            }
            const int e = ((off + x0) & ~(AL - 1)) + lane * AL;
            if ((what & 1) && e < off + x0 + tw) {
#pragma unroll
                for (int pl = 0; pl < 2; ++pl) cp_async16(re + (pl * RH + r) * EP + lane * AL, mt + (3 + pl) * np + e);
            }
        }
    };
    static_assert(RP <= 32 * AL && EP <= 32 * AL, "one 16-byte piece per lane");

    if constexpr (SATF) {
        if (tid >= kStageThreads) {
            sat_tiles<MX, MY, T, TY>(A, ssat);
            return;
        }
    }
    if (blockIdx.x < A.ntiles) {
        const int4 td = A.tiles[blockIdx.x];
        fetch(td, 1);
        dependency_wait();
        fetch(td, 2);
    } else {
        dependency_wait();
    }

    for (int t = blockIdx.x; t < A.ntiles; t += gridDim.x) {
        const int4 td = A.tiles[t];
        const BlockDev& B = A.blocks[td.x];
        const int nx = B.nx, ny = B.ny;
        const int np = B.npad;  // in-block offsets fit 32 bits (checked when the system is built)
        const int y0 = td.y, x0 = td.z;
        const int th = tile_rows(td), tw = tile_cols(td);
        const int y1 = y0 + th, x1 = x0 + tw;
        int lx0, lx1, ly0, ly1;
        region_of<OPX>(x0, x1, nx, lx0, lx1);
        region_of<OPY>(y0, y1, ny, ly0, ly1);
        // Everything later phases need from the block and instance descriptors is read here,
        // once: the global stores of the update would otherwise force the compiler to reload it.
        const int64_t qoff = B.q_off, eoff = B.e_off, roff = B.r_off;
        const InstanceDev& I = A.inst[B.instance];
        const T cb = T(A.stage < 4 ? I.cb[A.stage] : 0.0);
        const T ca = T(A.stage < 3 ? I.ca[A.stage] : 0.0);
        // the f64 sums still lack the spacing factors (the f32 metrics carry them)
        const T fx = COMP ? T(1) : T(B.idx_xi), fy = COMP ? T(1) : T(B.idx_eta);
        // The tile list gives every closure column of a block row to its first or its last tile
        // and no tile both (tile_starts), and likewise for rows.
        const bool left_cl = x0 < MX, right_cl = x1 > nx - MX;
        const bool top_cl = y0 < MY, bot_cl = y1 > ny - MY;
        if ((left_cl && right_cl) || (top_cl && bot_cl)) {  // a tile list not made by tile_starts
            if (tid == 0) atomicOr(A.status, STATUS_BAD_LAUNCH);
            return;
        }
        const bool xi_pre = left_cl || right_cl, eta_pre = top_cl || bot_cl;
        // Operands of the update pass for this thread's points (coalesced: consecutive threads take
        // consecutive columns); the fused form, which has the registers, loads them here, the other just
        // before they are used:
        // 1 / J, the free-stream plane, and up to three state arrays.
        constexpr int NOP = COMP ? 3 : 2;
        T jinv[PPT], rv[PPT], op[NOP][PPT][CPT];
        int pe[PPT];  // element of the point in a plane (-1: not in the tile)
        const int uc = PTS >= kStageThreads ? 0 : (tid / PTS) * CPT;  // first component
        const T* src[3] = {A.stage == 0 ? A.u_in + qoff : A.acc_hi + qoff, A.prev_hi + qoff, A.prev_lo + qoff};
        const int nsrc = A.stage == kStageK ? 0 : (A.stage == 0 ? 1 : (A.stage < 3 ? 2 : (COMP ? 3 : 1)));
        const T* ji = COMP ? A.met + B.m_off : A.jinv + roff;
        auto load_operands = [&]() {
#pragma unroll
            for (int i = 0; i < PPT; ++i) {
                const int p = tid % (PTS < kStageThreads ? PTS : kStageThreads) + i * kStageThreads;
                const int ur = p / TX, ux = p % TX;
                pe[i] = ur < th && ux < tw ? (y0 + ur) * nx + x0 + ux : -1;
                jinv[i] = T(1);
                rv[i] = T(0);
                if (pe[i] >= 0) {
                    jinv[i] = __ldg(ji + pe[i]);
                    if constexpr (COMP && UPW) rv[i] = __ldg(A.rinf + roff + pe[i]);
#pragma unroll
                    for (int a = 0; a < NOP; ++a)
#pragma unroll
                        for (int cc = 0; cc < CPT; ++cc)
                            op[a][i][cc] = a < nsrc ? src[a][(uc + cc) * np + pe[i]] : T(0);
                }
            }
        };
        if constexpr (SATF) load_operands();

        cp_async_wait_all();
        tile_sync();

        // ---------------- xi fluxes of the tile rows, widened by the xi halo ----------------
        {
            const int cw = lx1 - lx0;
            const unsigned inv = (65536u + cw - 1) / cw;  // exact floor(p / cw) for p * cw < 65536
            for (int p = tid; p < th * cw; p += kStageThreads) {
                const int r = (int)(((unsigned)p * inv) >> 16), c = p - r * cw;
                const int a = (((y0 + r) * nx + lx0) & (AL - 1)) + c;
                const T* s = rq + (y0 - ly0 + r) * RP + a;
                const T* m = rx + r * RP + a;
                const T qv[4] = {s[0], s[RH * RP], s[2 * RH * RP], s[3 * RH * RP]};
                T* o = fl + r * G::XP + G::xpos(lx0 + c - x0 + G::XL);
                if constexpr (COMP) {
                    const T mm[4] = {m[0], m[TY * RP], T(0), T(0)};
                    pointwise_dev<UPW>(qv, mm, gamma, I.ref, o, XA, o, XA, true, false, bad);
                } else {
                    pointwise<UPW>(qv, m[0], m[TY * RP], gamma, o, XA, bad);
                }
            }
        }
        tile_sync();

        // the next tile, its block descriptor brought near for fetch
        const int tn = t + (int)gridDim.x;
        int4 ntd = make_int4(0, 0, 0, 0);
        if (tn < A.ntiles) {
            ntd = A.tiles[tn];
            asm volatile("prefetch.global.L1 [%0];" ::"l"(A.blocks + ntd.x));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(reinterpret_cast<const char*>(A.blocks + ntd.x) + 128));
        }
        // ---------------- xi sums ----------------
        // Thread (comp, gy, gx): component comp at rows y0 + gy MR .., columns x0 + gx MC ...  In a
        // tile with closure columns every thread runs the interior path, and the closure outputs
        // (diss - diff, all threads, compile-time coefficients) then replace its result through the
        // flux buffer.
        T ax[MR][MC], ay[MR][MC];
#pragma unroll
        for (int u = 0; u < MR; ++u)
#pragma unroll
            for (int j = 0; j < MC; ++j) ax[u][j] = ay[u][j] = T(0);
        const int r0 = gy * MR, c0 = gx * MC;
        const bool active = c0 < tw && r0 < th;
        if (active) {
            const T* xr = fl + comp * XA + r0 * G::XP;
            xi_sums<OPX, DIFF, -1, G>(xr, gx, ax);
            if constexpr (UPW) xi_sums<OPX, DISS, 1, G>(xr + 4 * XA, gx, ax);
        }
        if (xi_pre) {
            constexpr int PARTS = kStageThreads / (4 * TY), CNT = MX >= PARTS ? MX / PARTS : 1;
            const int r = tid % TY, cc = (tid / TY) & 3, part = tid / (4 * TY);
            T o[CNT];
            const bool own = r < th && part * CNT < MX;
            if (own) {
                const int lc = (right_cl ? nx - OpShape<OPX>::N : 0) - x0 + G::XL;
                const T* e = fl + cc * XA + r * G::XP;
                auto ld = [&](int kind, int k) { return e[(kind == DISS ? 4 * XA : 0) + G::xpos(lc + k)]; };
                if (right_cl) closure_part<OPX, UPW, true, PARTS, 0>(part, ld, o);
                else closure_part<OPX, UPW, false, PARTS, 0>(part, ld, o);
            }
            tile_sync();
            if (own) {
#pragma unroll
                for (int i = 0; i < CNT; ++i) fl[(cc * MX + part * CNT + i) * TY + r] = o[i];
            }
            tile_sync();
            if (active) {
#pragma unroll
                for (int j = 0; j < MC; ++j) {
                    const int ci = x0 + c0 + j - (left_cl ? 0 : nx - MX);
                    if (ci >= 0 && ci < MX) {
#pragma unroll
                        for (int u = 0; u < MR; ++u) ax[u][j] = fl[(comp * MX + ci) * TY + r0 + u];
                    }
                }
            }
        }
        tile_sync();

        // ---------------- eta fluxes of the tile columns, widened by the eta halo ----------------
        for (int p = tid; p < (ly1 - ly0) * TX; p += kStageThreads) {
            const int r = p / TX, c = p % TX;
            if (c < tw) {
                const int off = (ly0 + r) * nx;
                const T* s = rq + r * RP + ((off + lx0) & (AL - 1)) + (x0 - lx0) + c;
                const T* m = re + r * EP + ((off + x0) & (AL - 1)) + c;
                const T qv[4] = {s[0], s[RH * RP], s[2 * RH * RP], s[3 * RH * RP]};
                T* o = fl + (ly0 + r - y0 + G::YL) * TX + G::epos(c);
                if constexpr (COMP) {
                    const T mm[4] = {T(0), T(0), m[0], m[RH * EP]};
                    pointwise_dev<UPW>(qv, mm, gamma, I.ref, o, YA, o, YA, false, true, bad);
                } else {
                    pointwise<UPW>(qv, m[0], m[RH * EP], gamma, o, YA, bad);
                }
            }
        }
        tile_sync();
        // the raw rows are no longer needed: the next tile's copies run from here on
        if (tn < A.ntiles) fetch(ntd, 3);

        // ---------------- eta sums ----------------
        if (active) {
            const T* ec = fl + comp * YA + (r0 + G::YL - HY) * TX;
            eta_sums<OPY, DIFF, -1, G, 0>(ec, gx, ay);
            if constexpr (UPW) eta_sums<OPY, DISS, 1, G, 0>(ec + 4 * YA, gx, ay);
        }
        if (eta_pre) {
            constexpr int PARTS = kStageThreads / (4 * TX), CNT = MY >= PARTS ? MY / PARTS : 1;
            const int col = tid % TX, cc = (tid / TX) & 3, part = tid / (4 * TX);
            T o[CNT];
            const bool own = col < tw && part * CNT < MY;
            if (own) {
                const int lr = (bot_cl ? ny - OpShape<OPY>::N : 0) - y0 + G::YL;
                const T* f = fl + cc * YA + lr * TX + G::epos(col);
                auto ld = [&](int kind, int k) { return f[(kind == DISS ? 4 * YA : 0) + k * TX]; };
                if (bot_cl) closure_part<OPY, UPW, true, PARTS, 0>(part, ld, o);
                else closure_part<OPY, UPW, false, PARTS, 0>(part, ld, o);
            }
            tile_sync();
            if (own) {
#pragma unroll
                for (int i = 0; i < CNT; ++i) fl[(cc * MY + part * CNT + i) * TX + col] = o[i];
            }
            tile_sync();
            if (active) {
#pragma unroll
                for (int u = 0; u < MR; ++u) {
                    const int ri = y0 + r0 + u - (top_cl ? 0 : ny - MY);
                    if (ri >= 0 && ri < MY) {
#pragma unroll
                        for (int j = 0; j < MC; ++j) ay[u][j] = fl[(comp * MY + ri) * TX + c0 + j];
                    }
                }
            }
        }
        tile_sync();
        // the sums through shared memory to the update pass
        if (active) {
#pragma unroll
            for (int u = 0; u < MR; ++u) {
                T s[MC];
#pragma unroll
                for (int j = 0; j < MC; ++j)
                    s[j] = COMP ? ax[u][j] + ay[u][j] : fma_rn(ax[u][j], fx, ay[u][j] * fy);
                V* o = reinterpret_cast<V*>(fl + comp * PTS + (r0 + u) * TX);
                o[gx] = {s[0], s[1]};
                if constexpr (MC == 4) o[TX / 4 + (gx ^ 4)] = {s[2], s[3]};
            }
        }
        if constexpr (!SATF) load_operands();
        if constexpr (SATF) __syncthreads();  // the SAT terms are there
        else tile_sync();

        // ---------------- update pass ----------------
        // Interior points finish; points on a block edge store k for the edge kernel.
#pragma unroll
        for (int i = 0; i < PPT; ++i) {
            if (pe[i] < 0) continue;
            const int p = tid % (PTS < kStageThreads ? PTS : kStageThreads) + i * kStageThreads;
            const int ur = p / TX, ux = p % TX;
            const int row = y0 + ur, col = x0 + ux;
            const bool edge = row == 0 || row == ny - 1 || col == 0 || col == nx - 1;
#pragma unroll
            for (int cc = 0; cc < CPT; ++cc) {
                T k = fl[(uc + cc) * PTS + ur * TX + G::epos(ux)] * jinv[i];
                if constexpr (COMP && UPW) k = fma_rn(I.ref.q[uc + cc], rv[i], k);
                const int64_t e = qoff + (uc + cc) * np + pe[i];
                if (edge) {
                    if constexpr (SATF) {
                        const int slot = row == 0 || row == ny - 1 ? ux : TX + ur;
                        k = T(double(k) + ssat[4 * slot + uc + cc]);
                    } else {
                        A.kedge[4 * (eoff + edge_index(row, col, nx, ny)) + uc + cc] = k;
                        continue;
                    }
                }
                rk_update_ops<T, COMP>(A, e, cb, ca, k, op[0][i][cc], op[1][i][cc], COMP ? op[NOP - 1][i][cc] : T(0));
            }
        }
        // Every thread is done with the flux buffer (and the SAT terms) before the next tile's.
        if constexpr (SATF) __syncthreads();
        else tile_sync();
    }
    if (bad) atomicOr(A.status, bad);
    if constexpr (SATF) {
        // stage 3: the last CTA of the step's groups advances the times of the active instances; the SAT
        // threads have read them before the last barrier
        if (A.time_ctas > 0) {
            __shared__ bool last;
            tile_sync();
            if (tid == 0) {
                __threadfence();
                last = atomicAdd(A.time_done, 1u) == (unsigned)A.time_ctas - 1u;
            }
            tile_sync();
            if (last) {
                InstanceDev* inst = const_cast<InstanceDev*>(A.inst);
                for (int i = tid; i < A.ninst; i += kStageThreads)
                    if (A.active[i]) inst[i].time = inst[i].time + inst[i].dt;
                if (tid == 0) *A.time_done = 0u;
            }
        }
    }
}

// Edge kernel: one thread per block-edge point of a stage launch's blocks (edges[i] = block,
// row, col).  Adds the SATs to the k the stage kernel stored and does the point's RK update.
constexpr int kSatThreads = 128;
template <class T, bool COMP>
__global__ void __launch_bounds__(kSatThreads, 4) sat_kernel(const StageArgs<T> A, const int4* __restrict__ edges,
                                                          int nedges) {
    const int i = blockIdx.x * kSatThreads + threadIdx.x;
    if (i >= nedges) return;
    const int4 ed = edges[i];
    const BlockDev& B = A.blocks[ed.x];
    const InstanceDev& I = A.inst[B.instance];
    const int row = ed.y, col = ed.z;
    const int nx = B.nx, ny = B.ny;
    const int64_t np = B.npad, qoff = B.q_off;
    const int64_t slot = 4 * (B.e_off + edge_index(row, col, nx, ny));
    const T cb = T(A.stage < 4 ? I.cb[A.stage] : 0.0);
    const T ca = T(A.stage < 3 ? I.ca[A.stage] : 0.0);
    const int pt = row * nx + col;
    const T* q = A.u_in + qoff;
    const EdgeGeo geo = edge_record(A.egeo + kEdgeGeo * (B.e_off + edge_index(row, col, nx, ny)));
    const SatSides side = sat_sides(A, I, B, row, col, geo);
    dependency_wait();
    double yv[4], kv[4], sv[4] = {0.0, 0.0, 0.0, 0.0};
    T qs[4];  // the stored stage input (a deviation in the compensated form)
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
        qs[cc] = q[cc * np + pt];
        yv[cc] = absolute_state<T>(A, B, cc, qs[cc]);
        kv[cc] = double(A.kedge[slot + cc]);
    }
    sat_apply<T>(A, I, B, i, row, col, geo, side, yv, sv);
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
        // the operands of the update pass of stage_kernel
        const int64_t e = qoff + cc * np + pt;
        T o0 = qs[cc], o1 = T(0), o2 = T(0);
        if (A.stage != 0 && A.stage != kStageK) {
            o0 = A.acc_hi[e];
            if (COMP || A.stage < 3) o1 = A.prev_hi[e];
            if (COMP && A.stage == 3) o2 = A.prev_lo[e];
        }
        rk_update_ops<T, COMP>(A, e, cb, ca, T(kv[cc] + sv[cc]), o0, o1, o2);
    }
}

// Expression boundary data (SBP_BC_EVAL sides) of a stage launch's edge points (edges[i] =
// block, row, col) at the stage time, into evz[4 i ..]; launched before the edge kernel only for
// systems with such sides, so the edge kernel itself stays free of the interpreter.
template <class T>
__global__ void __launch_bounds__(kSatThreads) eval_kernel(const StageArgs<T> A, const int4* __restrict__ edges,
                                                           int nedges) {
    dependency_wait();
    const int i = blockIdx.x * kSatThreads + threadIdx.x;
    if (i >= nedges) return;
    const int4 ed = edges[i];
    const BlockDev& B = A.blocks[ed.x];
    const int row = ed.y, col = ed.z;
    const bool on[4] = {row == B.ny - 1, row == 0, col == B.nx - 1, col == 0};
    bool any = false;
    for (int d = 0; d < 4; ++d) any = any || (on[d] && B.bc_kind[d] == BC_EVAL);
    if (!any) return;
    const InstanceDev& I = A.inst[B.instance];
    const double cst = A.stage == kStageK ? A.ctime : (A.stage == 0 ? 0.0 : (A.stage == 3 ? 1.0 : 0.5));
    const double stime = cst == 0.0 ? I.time : I.time + I.dt * cst;
    const int64_t pt = (int64_t)row * B.nx + col;
    const double* xy = A.xy + B.x_off;
    double z[4];
    eval_state(*A.eval, A.gamma, stime, xy[pt], xy[B.npad + pt], z);
    for (int cc = 0; cc < 4; ++cc) A.evz[4 * (int64_t)i + cc] = z[cc];
}

}  // namespace sbp
