// Systems of curvilinear blocks on one GPU: the euler::System / multigrid::System surface and
// ensembles of independent solves (instances), behind the C ABI.
//
// Per RK4 step the device runs, for each of the 4 stages, one persistent fused stage kernel per
// operator pair present (all tiles of all active blocks of that pair in one launch) and its edge
// kernel (uncoupled operator groups on their own streams, joined once per step), then one tiny
// kernel that advances the instance times.  Systems too small to fill the GPU take the fused form of
// the stage kernel, with the SATs and the times in it (fused_rows).  The whole step is captured once as a CUDA
// graph and replayed; the graph is re-captured only when the tile schedule or the set of
// active instances changes.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.h"
#include "euler_device.cuh"
#include "interp.cuh"
#include "op_apply.h"
#include "sbp_ops.cuh"
#include "stage_dispatch.h"
#include "eval_program.cuh"
#include "stage_kernel.cuh"
#include "stage_kernel_vec.cuh"
#include "system_kernels.h"

namespace sbp {
const double* op_h_weights(int op);

const void* stage_kernel_ptr(int prec, int opx, int opy, bool upw, int ty, int sc) {
    using F = const void* (*)(int, int, bool, int, int);
    static const F f64[] = {stage_ptr_f64_u4,   stage_ptr_f64_u9,   stage_ptr_f64_sbp, stage_ptr_f64_x49a,
                            stage_ptr_f64_x49b, stage_ptr_f64_xsa, stage_ptr_f64_xsb};
    static const F f32[] = {stage_ptr_f32_u4, stage_ptr_f32_u9, stage_ptr_f32_sbp, stage_ptr_f32_x49,
                            stage_ptr_f32_xs};
    const F* fs = prec == 0 ? f64 : f32;
    const size_t nf = prec == 0 ? sizeof(f64) / sizeof(F) : sizeof(f32) / sizeof(F);
    for (size_t i = 0; i < nf; ++i) {
        const void* p = fs[i](opx, opy, upw, ty, sc);
        if (p) return p;
    }
    return nullptr;
}

namespace {

void region_host(int op, int a0, int a1, int n, int& lo, int& hi) {
    switch (op) {
        case UPWIND4: region_of<UPWIND4>(a0, a1, n, lo, hi); break;
        case UPWIND4H2: region_of<UPWIND4H2>(a0, a1, n, lo, hi); break;
        case UPWIND9: region_of<UPWIND9>(a0, a1, n, lo, hi); break;
        case UPWIND9H2: region_of<UPWIND9H2>(a0, a1, n, lo, hi); break;
        case SBP4: region_of<SBP4>(a0, a1, n, lo, hi); break;
        default: region_of<SBP8>(a0, a1, n, lo, hi); break;
    }
}

int64_t pad64(int64_t n) { return (n + 63) / 64 * 64; }

// Largest block: 5 planes of pad64(points) elements stay below 2^31.
constexpr int64_t kMaxBlockPoints = (int64_t)1 << 28;

// The compensated-f32 kernel of 32-row tiles is the 2 x 2 micro-tile kernel (stage_kernel_vec).
bool vec_kernel(int prec, int ty) { return prec == 1 && ty == kVecRows; }

// Shared memory of one stage-kernel CTA (tile_smem in stage_kernel.cuh, VecGeom in
// stage_kernel_vec.cuh).
size_t stage_smem_host(int prec, int opx, int opy, bool upw, int ty) {
    OpInfo ox, oy;
    op_info(opx, ox);
    op_info(opy, oy);
    if (vec_kernel(prec, ty)) {
        const int xc = region_extent(kTileX, (ox.D - 1) / 2, ox.M, ox.N);
        const int hyp = region_extent(ty, (oy.D - 1) / 2, oy.M, oy.N);
        return sizeof(float) *
               ((size_t)(4 * 2 * ((xc + 1) / 2) * kVecPitch + 4 * hyp * kTileX) * (upw ? 2 : 1) + closure_xi_elems(ox.M) +
                closure_eta_elems(oy.M));
    }
    return (size_t)tile_smem(ty, upw, prec == 0 ? 8 : 4, (ox.D - 1) / 2, ox.M, ox.N, (oy.D - 1) / 2, oy.M, oy.N);
}

// Edge geometry of a group's edge points (edges[i] = block, row, col) at their slots.
__global__ void edge_geo_kernel(const BlockDev* __restrict__ blocks, const double* __restrict__ met64,
                                const double* __restrict__ xy, const int4* __restrict__ edges, int nedges,
                                double* __restrict__ geo) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nedges) return;
    const int4 ed = edges[i];
    const BlockDev& B = blocks[ed.x];
    const int64_t np = B.npad, pt = (int64_t)ed.y * B.nx + ed.z;
    double* o = geo + kEdgeGeo * (B.e_off + edge_index(ed.y, ed.z, B.nx, B.ny));
    o[0] = xy[B.x_off + pt];
    o[1] = xy[B.x_off + np + pt];
#pragma unroll
    for (int c = 0; c < 5; ++c) o[2 + c] = met64[B.m_off + c * np + pt];
    o[7] = 0.0;
}

struct Group {
    int opx, opy;
    bool upw;
    const void* fn[3];  // stage kernel per RK stage class (vec_stage_class); the same entry thrice
                        // for kernels that take the stage at run time
    bool fused = false; // the SATs are part of the stage kernel (its fused form)
    int4* d_tiles = nullptr;
    int ntiles = 0;
    int4* d_edges = nullptr;  // (block, row, col) of every edge point of the group's blocks
    int nedges = 0;
    double* d_evz = nullptr;  // SBP_BC_EVAL data of those edge points (systems with such sides)
    int64_t points = 0;       // grid points of the group's blocks
    int WX = 0, HY = 0;
    int ty = 16;              // tile rows
    int ctas = -1;            // persistent CTAs per SM (-1: as many as fit), 0: one CTA per tile
    size_t smem = 0;
    int grid = 0;
};

// Tile schedule chosen for one operator group (set by the autotuner): tile rows and the width
// of the stage kernel's grid.
struct TileChoice {
    int opx, opy;
    bool upw;
    int ty, ctas;
    bool fused;
};

// One chunk of sbp_system_advance_host: the blocks [b0, b1) (whole instances), their own step
// graph and time-update mask, and the stream the chunk's copies and steps run on.
struct Chunk {
    int b0 = 0, b1 = 0;
    std::vector<int> active;  // instances of the chunk
    std::vector<Group> groups;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t gexec = nullptr;
    int* d_active = nullptr;
    cudaStream_t st = nullptr;
    cudaEvent_t done = nullptr;
};

}  // namespace
}  // namespace sbp

using namespace sbp;

struct sbp_system {
    int device = 0;
    int prec = 0;
    double gamma = 1.4;
    bool force_trad = false;
    int nblocks = 0, ninst = 0;
    int num_sms = 148;
    size_t smem_optin = 0;
    std::vector<BlockDev> hb;
    std::vector<InstanceDev> hi;
    int64_t nq = 0, nm = 0, nx2 = 0, max_points = 0, dense_total = 0;
    std::vector<int64_t> dense_off;  // packed (4, ny, nx) offsets
    // device memory
    BlockDev* d_blocks = nullptr;
    InstanceDev* d_inst = nullptr;
    int* d_active = nullptr;
    void *prev_hi = nullptr, *prev_lo = nullptr, *acc_hi = nullptr, *acc_lo = nullptr, *uA = nullptr, *uB = nullptr;
    double* met64 = nullptr;
    float* met32 = nullptr;
    double* jinv64 = nullptr;  // f64: 1 / J planes (BlockDev::r_off)
    float* rinf = nullptr;  // compensated f32: free-stream dissipation planes (BlockDev::r_off)
    double* xy = nullptr;
    double* hw = nullptr;
    int64_t* d_hoff = nullptr;
    std::vector<int64_t> hoff;
    int64_t* d_poff4 = nullptr;  // packed offsets in elements for dtype f64 (4n per block)
    int64_t* d_poff8 = nullptr;  // packed offsets for dtype f32 hi+lo (8n per block)
    int64_t* d_zero = nullptr;
    void* staging = nullptr;
    size_t staging_bytes = 0;
    unsigned* status = nullptr;
    double* d_sums = nullptr;
    unsigned long long* d_speeds = nullptr;
    void* kedge = nullptr;   // k of block-edge points between the stage and the edge kernel
    double* egeo = nullptr;   // edge geometry (kEdgeGeo per point, edge_geo_kernel)
    int64_t nedge = 0;
    int4* d_mg = nullptr;    // MultiGrid segments of all block sides
    EvalDev* d_eval = nullptr;  // expression programs of SBP_BC_EVAL sides
    bool has_eval = false, eval_set = false;
    double* kbuf = nullptr;  // k of the stages of a general tableau (kMaxStages x nq, f64), on demand
    int kbuf_stages = 0;
    // schedule
    int TY = 16, threads = kStageThreads;  // threads: of the stencil
    std::vector<TileChoice> tile_choice;  // per operator group; groups not listed use (TY, -1)
    bool tiles_auto = true;               // until a caller chooses: small systems take the fused form
    bool fused = false;                   // a caller's choice: the fused form with TY rows
    int tiles_gen = 0;                    // bumped whenever the tile schedule changes
    std::vector<int> active;
    std::vector<Group> groups;
    bool sched_dirty = true;
    cudaStream_t stream = nullptr;
    cudaStream_t user_stream = nullptr;
    bool has_user_stream = false;
    std::vector<cudaStream_t> side;
    std::vector<cudaEvent_t> ev;
    cudaEvent_t ev_fork = nullptr;
    cudaGraphExec_t gexec = nullptr;
    cudaGraph_t graph = nullptr;
    // chunk schedules of sbp_system_advance_host, valid for the tile shape and form they were
    // built with
    std::vector<Chunk> chunks;
    int chunk_gen = -1, chunk_req = 0;
    bool chunk_trad = false;

    cudaStream_t st() const { return has_user_stream ? user_stream : stream; }
    size_t tsize() const { return prec == 0 ? sizeof(double) : sizeof(float); }
};

namespace {

void free_group_list(std::vector<Group>& groups, cudaGraph_t& graph, cudaGraphExec_t& gexec) {
    for (auto& g : groups) {
        cudaFree(g.d_tiles);
        cudaFree(g.d_edges);
        if (g.d_evz) cudaFree(g.d_evz);
    }
    groups.clear();
    if (gexec) cudaGraphExecDestroy(gexec);
    if (graph) cudaGraphDestroy(graph);
    gexec = nullptr;
    graph = nullptr;
}

void free_groups(sbp_system* s) { free_group_list(s->groups, s->graph, s->gexec); }

void free_chunks(sbp_system* s) {
    for (auto& c : s->chunks) {
        if (c.st) cudaStreamSynchronize(c.st);
        free_group_list(c.groups, c.graph, c.gexec);
        if (c.d_active) cudaFree(c.d_active);
        if (c.st) cudaStreamDestroy(c.st);
        if (c.done) cudaEventDestroy(c.done);
    }
    s->chunks.clear();
    s->chunk_req = 0;
}

void destroy_all(sbp_system* s) {
    if (!s) return;
    cudaSetDevice(s->device);
    if (s->stream) cudaStreamSynchronize(s->stream);
    free_chunks(s);
    free_groups(s);
    void* ptrs[] = {s->d_blocks, s->d_inst, s->d_active, s->prev_hi, s->prev_lo, s->acc_hi, s->acc_lo,
                    s->uA,       s->uB,     s->met64,    s->met32,   s->xy,      s->hw,      s->d_hoff,
                    s->d_poff4,  s->d_poff8, s->d_zero,  s->staging, s->status,  s->d_sums,  s->d_speeds,
                    s->jinv64,   s->kedge,  s->d_mg,     s->kbuf,    s->d_eval,  s->rinf,    s->egeo};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    for (auto st : s->side) cudaStreamDestroy(st);
    for (auto e : s->ev) cudaEventDestroy(e);
    if (s->ev_fork) cudaEventDestroy(s->ev_fork);
    if (s->stream) cudaStreamDestroy(s->stream);
    delete s;
}

// Free-stream dissipation planes of the compensated form for the upwind blocks of one instance
// (instance < 0: all), from the instances' reference states on the device.
sbp_status build_free_stream_dissipation(sbp_system* s, int instance) {
    if (!s->rinf) return SBP_OK;
    cudaStream_t st = s->st();
    for (int b = 0; b < s->nblocks; ++b) {
        const BlockDev& B = s->hb[b];
        if (instance >= 0 && B.instance != instance) continue;
        OpInfo ox, oy;
        op_info(B.op_xi, ox);
        op_info(B.op_eta, oy);
        if (!(ox.upwind && oy.upwind)) continue;
        SBP_TRY_CUDA(free_stream_dissipation(s->d_blocks + b, s->d_inst, s->gamma, B.op_xi, B.op_eta, B.nx, B.ny,
                                             s->met64, static_cast<double*>(s->staging), s->rinf, st));
    }
    return SBP_OK;
}

sbp_status upload_instances(sbp_system* s) {
    SBP_TRY_CUDA(cudaMemcpyAsync(s->d_inst, s->hi.data(), s->hi.size() * sizeof(InstanceDev), cudaMemcpyHostToDevice,
                                 s->st()));
    return SBP_OK;
}

// Pull device-advanced instance times into the host copy before editing it.
sbp_status sync_times(sbp_system* s) {
    std::vector<InstanceDev> tmp(s->hi.size());
    SBP_TRY_CUDA(cudaMemcpyAsync(tmp.data(), s->d_inst, tmp.size() * sizeof(InstanceDev), cudaMemcpyDeviceToHost,
                                 s->st()));
    SBP_TRY_CUDA(cudaStreamSynchronize(s->st()));
    for (size_t i = 0; i < tmp.size(); ++i) s->hi[i].time = tmp[i].time;
    return SBP_OK;
}

void set_dt_host(InstanceDev& I, double dt) {
    // Tableau entries times dt exactly as integrate() forms them (utils/integrate/src/lib.rs:30-35,
    // 193-211): a*dt for the stage states and b*dt for the final combination.
    I.dt = dt;
    I.ca[0] = 0.5 * dt;
    I.ca[1] = 0.5 * dt;
    I.ca[2] = 1.0 * dt;
    I.cb[0] = (1.0 / 6.0) * dt;
    I.cb[1] = (1.0 / 3.0) * dt;
    I.cb[2] = (1.0 / 3.0) * dt;
    I.cb[3] = (1.0 / 6.0) * dt;
}

// Reference state of an instance: the free stream of its vortex parameters (rho 1, u 1, v 0,
// p = 1 / (gamma M^2); euler/src/vortex.rs:26-40), against which compensated systems store the
// state, and its f32 constants for the stage kernels.
void set_reference(InstanceDev& I, double gamma) {
    const double p = 1.0 / (gamma * I.mach * I.mach);
    const double rho = 1.0, u = 1.0, v = 0.0;
    I.qref[0] = rho;
    I.qref[1] = rho * u;
    I.qref[2] = rho * v;
    I.qref[3] = p / (gamma - 1.0) + rho * (u * u + v * v) / 2.0;
    RefState& R = I.ref;
    for (int c = 0; c < 4; ++c) R.q[c] = float(I.qref[c]);
    R.u = float(u);
    R.v = float(v);
    R.p = float(p);
    R.h = float(I.qref[3] + p);
    R.c2 = float(gamma * p / rho);
    R.c = float(std::sqrt(gamma * p / rho));
    R.g_rho = float(gamma / rho);
    // constants of the division-free vortex boundary data (vortex_point_fast)
    const double PI = 3.14159265358979323846;
    const double m = I.mach, p_inf = 1.0 / (gamma * m * m);
    I.v_pinf = p_inf;
    I.v_igm1 = 1.0 / (gamma - 1.0);
    I.v_regular = 1;
    for (int k = 0; k < I.nvort; ++k)
        if (!(I.rstar[k] * I.rstar[k] > 0.0)) I.v_regular = 0;
    for (int k = 0; k < 5; ++k) {
        const double rs2 = I.rstar[k] * I.rstar[k];
        I.vk_f[k] = rs2 > 0.0 ? 1.0 / rs2 : 0.0;
        I.vk_b[k] = rs2 > 0.0 ? I.eps[k] * I.eps[k] * (gamma - 1.0) * m * m / (8.0 * PI * PI * p_inf * rs2) : 0.0;
        I.vk_u[k] = rs2 > 0.0 ? I.eps[k] / (2.0 * PI * std::sqrt(p_inf) * rs2) : 0.0;
    }
}

template <class T>
StageArgs<T> stage_args(sbp_system* s, int stage, const Group& g) {
    StageArgs<T> a{};
    a.blocks = s->d_blocks;
    a.inst = s->d_inst;
    a.tiles = g.d_tiles;
    a.ntiles = g.ntiles;
    a.stage = stage;
    T* prev = static_cast<T*>(s->prev_hi);
    T* uA = static_cast<T*>(s->uA);
    T* uB = static_cast<T*>(s->uB);
    const T* ins[4] = {prev, uA, uB, uA};
    T* outs[4] = {uA, uB, uA, nullptr};
    a.u_in = ins[stage];
    a.u_out = outs[stage];
    a.prev_hi = prev;
    a.prev_lo = static_cast<const T*>(s->prev_lo);
    a.acc_hi = static_cast<T*>(s->acc_hi);
    a.new_hi = prev;
    a.new_lo = static_cast<T*>(s->prev_lo);
    a.met = s->prec == 0 ? reinterpret_cast<const T*>(s->met64) : reinterpret_cast<const T*>(s->met32);
    a.jinv = s->prec == 0 ? reinterpret_cast<const T*>(s->jinv64) : nullptr;
    a.rinf = s->rinf;
    a.xy = s->xy;
    a.kedge = static_cast<T*>(s->kedge);
    a.egeo = s->egeo;
    a.mg = s->d_mg;
    a.eval = s->d_eval;
    a.evz = g.d_evz;
    a.gamma = s->gamma;
    a.status = s->status;
    return a;
}

// Advance of the instance times by the fused stage kernels of a step (StageArgs::time_ctas).
struct TimeAdvance {
    int ctas = 0;
    const int* active = nullptr;  // ninst flags, then the counter
};

template <class T>
cudaError_t launch_group_t(sbp_system* s, int stage, const Group& g, cudaStream_t st, bool edges_too, bool dependent,
                           const TimeAdvance& ta) {
    StageArgs<T> a = stage_args<T>(s, stage, g);
    if (g.fused && stage == 3 && ta.ctas > 0) {
        a.time_ctas = ta.ctas;
        a.ninst = s->ninst;
        a.active = ta.active;
        a.time_done = reinterpret_cast<unsigned*>(const_cast<int*>(ta.active) + s->ninst);
    }
    // A dependent launch may begin while the stream's previous kernel drains (dependency_wait).  Stage
    // kernels are; edge kernels are not: their early CTAs cost the separate f64 stage kernel the tail of its
    // launch (one 700 x 700 Upwind9 block 180 instead of 183 us a step, the f64 ensemble 2-3%).
    auto launch = [&](const void* fn, int grid, int threads, void** args, size_t smem, bool dep) {
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cfg.attrs = &at;
        cfg.numAttrs = dep ? 1 : 0;
        return cudaLaunchKernelExC(&cfg, fn, args);
    };
    void* args[] = {&a};
    const int threads = s->threads + (g.fused ? sat_threads(g.ty) : 0);
    cudaError_t e = launch(g.fn[vec_stage_class(stage)], g.grid, threads, args, g.smem, dependent);
    if (g.fused || !edges_too) return e;
    const int sat_grid = (g.nedges + kSatThreads - 1) / kSatThreads;
    int4* edges = g.d_edges;
    int nedges = g.nedges;
    void* sargs[] = {&a, &edges, &nedges};
    if (e == cudaSuccess && s->has_eval)
        e = launch(s->prec == 0 ? eval_ptr_f64() : eval_ptr_f32(), sat_grid, kSatThreads, sargs, 0, false);
    if (e == cudaSuccess) e = launch(s->prec == 0 ? sat_ptr_f64() : sat_ptr_f32(), sat_grid, kSatThreads, sargs, 0, false);
    return e;
}

// One stage of one group: the stage kernel and, unless its form includes the SATs, the edge kernel.
// dependent: the stream's previous operation is a kernel of this group's previous stage.
sbp_status launch_group(sbp_system* s, int stage, const Group& g, cudaStream_t st, bool edges_too = true,
                        bool dependent = false, const TimeAdvance& ta = {}) {
    if (g.ntiles == 0) return SBP_OK;
    const cudaError_t e = s->prec == 0 ? launch_group_t<double>(s, stage, g, st, edges_too, dependent, ta)
                                       : launch_group_t<float>(s, stage, g, st, edges_too, dependent, ta);
    return cuda_status(e, "stage kernel launch");
}

// Butcher tableaus of utils/integrate/src/lib.rs:30-152 (explicit; A lower triangle by rows of
// stages 2..S, then B, C and, for the embedded ones, BSTAR).  The values are the reference's
// constant expressions, evaluated in f64 as its compiler does (one rounding per operation).
struct Tableau {
    int s;
    double a[kMaxStages][kMaxStages];  // a[i][j]: stage i+1 (1-based 2..S), j < i+1
    double b[kMaxStages];
    double c[kMaxStages];
    double bstar[kMaxStages];
    bool embedded;
};

std::vector<Tableau> make_tableaus() {
    std::vector<Tableau> t(7);
    {
        const double SQRT_5 = 2.236067977499789696409173668731276235440618359611525724270897245410520925637804899414414408378782275;
        for (auto& x : t) std::memset(&x, 0, sizeof x);
        // Rk4
        t[0].s = 4;
        t[0].a[0][0] = 0.5;
        t[0].a[1][0] = 0.0, t[0].a[1][1] = 0.5;
        t[0].a[2][0] = 0.0, t[0].a[2][1] = 0.0, t[0].a[2][2] = 1.0;
        t[0].b[0] = 1.0 / 6.0, t[0].b[1] = 1.0 / 3.0, t[0].b[2] = 1.0 / 3.0, t[0].b[3] = 1.0 / 6.0;
        t[0].c[0] = 0.5, t[0].c[1] = 0.5, t[0].c[2] = 1.0;
        // Rk4_38
        t[1].s = 4;
        t[1].a[0][0] = 1.0 / 3.0;
        t[1].a[1][0] = -1.0 / 3.0, t[1].a[1][1] = 1.0;
        t[1].a[2][0] = 1.0, t[1].a[2][1] = -1.0, t[1].a[2][2] = 1.0;
        t[1].b[0] = 1.0 / 8.0, t[1].b[1] = 3.0 / 8.0, t[1].b[2] = 3.0 / 8.0, t[1].b[3] = 1.0 / 8.0;
        t[1].c[0] = 1.0 / 3.0, t[1].c[1] = 2.0 / 3.0, t[1].c[2] = 1.0;
        // EulerMethod
        t[2].s = 1;
        t[2].b[0] = 1.0;
        // MidpointMethod
        t[3].s = 2;
        t[3].a[0][0] = 0.5;
        t[3].b[0] = 0.0, t[3].b[1] = 1.0;
        t[3].c[0] = 1.0 / 2.0;
        // Rk6
        t[4].s = 7;
        t[4].a[0][0] = 4.0 / 7.0;
        t[4].a[1][0] = 115.0 / 112.0, t[4].a[1][1] = -5.0 / 16.0;
        t[4].a[2][0] = 589.0 / 630.0, t[4].a[2][1] = 5.0 / 18.0, t[4].a[2][2] = -16.0 / 45.0;
        t[4].a[3][0] = 229.0 / 1200.0 - 29.0 / 6000.0 * SQRT_5;
        t[4].a[3][1] = 119.0 / 240.0 - 187.0 / 1200.0 * SQRT_5;
        t[4].a[3][2] = -14.0 / 75.0 + 34.0 / 375.0 * SQRT_5;
        t[4].a[3][3] = -3.0 / 100.0 * SQRT_5;
        t[4].a[4][0] = 71.0 / 2400.0 - 587.0 / 12000.0 * SQRT_5;
        t[4].a[4][1] = 187.0 / 480.0 - 391.0 / 2400.0 * SQRT_5;
        t[4].a[4][2] = -38.0 / 75.0 + 26.0 / 375.0 * SQRT_5;
        t[4].a[4][3] = 27.0 / 80.0 - 3.0 / 400.0 * SQRT_5;
        t[4].a[4][4] = (1.0 + SQRT_5) / 4.0;
        t[4].a[5][0] = -49.0 / 480.0 + 43.0 / 160.0 * SQRT_5;
        t[4].a[5][1] = -425.0 / 96.0 + 51.0 / 32.0 * SQRT_5;
        t[4].a[5][2] = 52.0 / 15.0 - 4.0 / 5.0 * SQRT_5;
        t[4].a[5][3] = -27.0 / 16.0 + 3.0 / 16.0 * SQRT_5;
        t[4].a[5][4] = 5.0 / 4.0 - 3.0 / 4.0 * SQRT_5;
        t[4].a[5][5] = 5.0 / 2.0 - 1.0 / 2.0 * SQRT_5;
        t[4].b[0] = 1.0 / 12.0, t[4].b[4] = 5.0 / 12.0, t[4].b[5] = 5.0 / 12.0, t[4].b[6] = 1.0 / 12.0;
        t[4].c[0] = 4.0 / 7.0, t[4].c[1] = 5.0 / 7.0, t[4].c[2] = 6.0 / 7.0;
        t[4].c[3] = (5.0 - SQRT_5) / 10.0, t[4].c[4] = (5.0 + SQRT_5) / 10.0, t[4].c[5] = 1.0;
        // Fehlberg (C has S entries: C[i - 1] is used for stage i as in the other tableaus)
        t[5].s = 6;
        t[5].a[0][0] = 1.0 / 4.0;
        t[5].a[1][0] = 3.0 / 32.0, t[5].a[1][1] = 9.0 / 32.0;
        t[5].a[2][0] = 1932.0 / 2197.0, t[5].a[2][1] = -7200.0 / 2197.0, t[5].a[2][2] = 7296.0 / 2197.0;
        t[5].a[3][0] = 439.0 / 216.0, t[5].a[3][1] = -8.0, t[5].a[3][2] = 3680.0 / 513.0, t[5].a[3][3] = -845.0 / 4104.0;
        t[5].a[4][0] = -8.0 / 27.0, t[5].a[4][1] = 2.0, t[5].a[4][2] = -3544.0 / 2565.0, t[5].a[4][3] = 1859.0 / 4104.0;
        t[5].a[4][4] = -11.0 / 40.0;
        t[5].b[0] = 16.0 / 135.0, t[5].b[2] = 6656.0 / 12825.0, t[5].b[3] = 28561.0 / 56430.0, t[5].b[4] = -9.0 / 50.0;
        t[5].b[5] = 2.0 / 55.0;
        t[5].c[0] = 0.0, t[5].c[1] = 1.0 / 4.0, t[5].c[2] = 3.0 / 8.0, t[5].c[3] = 12.0 / 13.0, t[5].c[4] = 1.0;
        t[5].c[5] = 1.0 / 2.0;
        t[5].bstar[0] = 25.0 / 216.0, t[5].bstar[2] = 1408.0 / 2565.0, t[5].bstar[3] = 2197.0 / 4104.0;
        t[5].bstar[4] = -1.0 / 5.0;
        t[5].embedded = true;
        // BogackiShampine
        t[6].s = 4;
        t[6].a[0][0] = 1.0 / 2.0;
        t[6].a[1][0] = 0.0, t[6].a[1][1] = 3.0 / 4.0;
        t[6].a[2][0] = 2.0 / 9.0, t[6].a[2][1] = 1.0 / 3.0, t[6].a[2][2] = 4.0 / 9.0;
        t[6].b[0] = 2.0 / 9.0, t[6].b[1] = 1.0 / 3.0, t[6].b[2] = 4.0 / 9.0, t[6].b[3] = 0.0;
        t[6].c[0] = 0.0, t[6].c[1] = 1.0 / 2.0, t[6].c[2] = 3.0 / 4.0, t[6].c[3] = 1.0;
        t[6].bstar[0] = 7.0 / 24.0, t[6].bstar[1] = 1.0 / 4.0, t[6].bstar[2] = 1.0 / 3.0, t[6].bstar[3] = 1.0 / 8.0;
        t[6].embedded = true;
    }
    return t;
}

const Tableau* tableau_of(int id) {
    static const std::vector<Tableau> t = make_tableaus();  // thread-safe initialisation
    return id >= 0 && id < 7 ? &t[id] : nullptr;
}

// Build per-operator-pair tile lists for the blocks of the instances flagged in `active`, size
// shared memory and grids, and capture one RK4 step (time update with the device mask
// d_active) into a graph.
// Tile boundaries along a line of n >= 2 M outputs, tiles of up to T, for an operator with M
// closure rows: multiples of T, except that the boundaries in (e, n), e = n - M rounded down to
// even, give way to e (and a line shorter than T + M is cut at e), so the last tile holds every
// end-closure output and no tile holds outputs of both ends (region_extent in stage_kernel.cuh).
// Returns the starts followed by n.
std::vector<int> tile_starts(int n, int T, int M) {
    std::vector<int> b;
    const int e = T > M ? (n - M) & ~1 : n - M;  // (tiles of M rows hold exactly the closure)
    bool moved = false;
    for (int x = 0; x < n; x += T) {
        if (x <= e) b.push_back(x);
        else moved = true;
    }
    // a boundary was dropped, or the last tile would also hold start-closure outputs
    if ((moved || b.back() < M) && b.back() != e) b.push_back(e);
    b.push_back(n);
    return b;
}

// Whether the fused form with `ty` rows exists for every block: expression sides need their own kernel, and
// pairs of operators of two families are not instantiated.
bool fused_built(const sbp_system* s, int ty) {
    if (s->has_eval) return false;
    for (const BlockDev& B : s->hb) {
        OpInfo ox, oy;
        op_info(B.op_xi, ox);
        op_info(B.op_eta, oy);
        const bool upw = ox.upwind && oy.upwind && !s->force_trad;
        if (!stage_kernel_ptr(s->prec, B.op_xi, B.op_eta, upw, ty | kTileFused, 0)) return false;
    }
    return true;
}
// The tile rows of the fused stage kernel for a system that leaves SMs without work, 0 where the other
// forms are better.  The fused kernel evaluates the SATs beside the stencils, saves the edge and time
// launches and overlaps successive stages, but runs one CTA an SM.  Measured per step (Upwind9 f64,
// one vortex block; 8-row tiles, 16-row tiles, the separate form): 128^2 (128 tiles of 8 rows) 30,
// 37, 60 us; 160^2 (200) 41, 37, 60; 350^2 (242 tiles of 16 rows) -, 64, 76; 400^2 (325) -, 88, 101;
// 500^2 (512) -, 115, 111.  So 8 rows while their tiles fit the SMs at once, 16 rows up to three tiles
// an SM.  The line holds for the other operators and precision too; fused, separate with 16 and with 32
// rows at 288^2 (162 tiles) and 448^2 (392): Upwind9 compensated 56, 70, 70 and 78, 89, 84; Upwind4 51,
// 66, 68 and 74, 86, 99, compensated 49, 64, 64 and 70, 80, 73; SBP8 45, 60, 64 and 64, 78, 88,
// compensated 43, 58, 58 and 60, 70, 65.
// The rule goes by all blocks of the system and not by the instances or the chunk at hand, so every
// schedule of a system takes the same form.
int fused_rows(const sbp_system* s) {
    if (!s->tiles_auto) return s->fused ? s->TY : 0;
    for (int ty : {8, 16}) {
        if (!fused_built(s, ty)) return 0;
        int64_t tiles = 0;
        for (const BlockDev& B : s->hb) {
            OpInfo ox, oy;
            op_info(B.op_xi, ox);
            op_info(B.op_eta, oy);
            tiles += (int64_t)(tile_starts(B.ny, ty, oy.M).size() - 1) * (tile_starts(B.nx, tile_tx(ty), ox.M).size() - 1);
        }
        if (tiles <= (ty == 8 ? 1 : 3) * (int64_t)s->num_sms) return ty;
    }
    return 0;
}

sbp_status build_step_graph(sbp_system* s, const std::vector<int>& active, const int* d_active,
                            std::vector<Group>& groups, cudaGraph_t& graph_out, cudaGraphExec_t& gexec_out) {
    free_group_list(groups, graph_out, gexec_out);
    const int fused = fused_rows(s);
    for (int b = 0; b < s->nblocks; ++b) {
        const BlockDev& B = s->hb[b];
        if (!active[B.instance]) continue;
        OpInfo ox, oy;
        op_info(B.op_xi, ox);
        op_info(B.op_eta, oy);
        const bool upw = ox.upwind && oy.upwind && !s->force_trad;
        Group* gp = nullptr;
        for (auto& g : groups)
            if (g.opx == B.op_xi && g.opy == B.op_eta && g.upw == upw) gp = &g;
        if (!gp) {
            Group g;
            g.opx = B.op_xi;
            g.opy = B.op_eta;
            g.upw = upw;
            g.ty = fused ? fused : s->TY;
            g.fused = fused != 0;
            for (const TileChoice& c : s->tile_choice)
                if (c.opx == g.opx && c.opy == g.opy && c.upw == g.upw) {
                    g.ty = c.ty;
                    g.ctas = c.ctas;
                    g.fused = c.fused;
                }
            for (int sc = 0; sc < 3; ++sc)
                g.fn[sc] = stage_kernel_ptr(s->prec, B.op_xi, B.op_eta, upw, g.ty | (g.fused ? kTileFused : 0), sc);
            if (!g.fn[0] || !g.fn[1] || !g.fn[2]) {
                set_error("operator pair (xi %d, eta %d) is not built into the stage kernels", B.op_xi, B.op_eta);
                return SBP_ERR_UNSUPPORTED;
            }
            groups.push_back(g);
            gp = &groups.back();
        }
    }
    std::vector<std::vector<int4>> tiles(groups.size()), edges(groups.size());
    std::vector<int> group_of(s->nblocks, -1);
    for (int b = 0; b < s->nblocks; ++b) {
        const BlockDev& B = s->hb[b];
        if (!active[B.instance]) continue;
        OpInfo ox, oy;
        op_info(B.op_xi, ox);
        op_info(B.op_eta, oy);
        const bool upw = ox.upwind && oy.upwind && !s->force_trad;
        size_t gi = 0;
        for (; gi < groups.size(); ++gi)
            if (groups[gi].opx == B.op_xi && groups[gi].opy == B.op_eta && groups[gi].upw == upw) break;
        group_of[b] = (int)gi;
        Group& g = groups[gi];
        const int TY = g.ty, TX = tile_tx(TY);
        const std::vector<int> ys = tile_starts(B.ny, TY, oy.M), xs = tile_starts(B.nx, TX, ox.M);
        for (size_t iy = 0; iy + 1 < ys.size(); ++iy)
            for (size_t ix = 0; ix + 1 < xs.size(); ++ix) {
                const int y0 = ys[iy], y1 = ys[iy + 1], x0 = xs[ix], x1 = xs[ix + 1];
                int lo, hi;
                region_host(B.op_xi, x0, x1, B.nx, lo, hi);
                g.WX = std::max(g.WX, hi - lo);
                region_host(B.op_eta, y0, y1, B.ny, lo, hi);
                g.HY = std::max(g.HY, hi - lo);
                tiles[gi].push_back(make_int4(b, y0, x0, (y1 - y0) << 16 | (x1 - x0)));
            }
        g.points += (int64_t)B.nx * B.ny;
        // edge points in edge_index order: first row, last row, first column, last column
        for (int c = 0; c < B.nx; ++c) edges[gi].push_back(make_int4(b, 0, c, 0));
        for (int c = 0; c < B.nx; ++c) edges[gi].push_back(make_int4(b, B.ny - 1, c, 0));
        for (int r = 1; r < B.ny - 1; ++r) edges[gi].push_back(make_int4(b, r, 0, 0));
        for (int r = 1; r < B.ny - 1; ++r) edges[gi].push_back(make_int4(b, r, B.nx - 1, 0));
    }
    for (size_t gi = 0; gi < groups.size(); ++gi) {
        Group& g = groups[gi];
        const int TY = g.ty;
        g.ntiles = (int)tiles[gi].size();
        const int TX = tile_tx(TY);
        g.smem = stage_smem_host(s->prec, g.opx, g.opy, g.upw, TY) + (g.fused ? 4 * (TX + TY) * sizeof(double) : 0);
        const int threads = s->threads + (g.fused ? sat_threads(TY) : 0);
        {
            OpInfo ox, oy;
            op_info(g.opx, ox);
            op_info(g.opy, oy);
            // every region fits the kernel's fixed shared-memory geometry
            if (g.WX > region_extent(TX, (ox.D - 1) / 2, ox.M, ox.N) ||
                g.HY > region_extent(TY, (oy.D - 1) / 2, oy.M, oy.N)) {
                set_error("internal: tile region exceeds the shared-memory geometry");
                return SBP_ERR_INVALID_ARGUMENT;
            }
        }
        if (g.smem > s->smem_optin) {
            set_error("tile %dx%d needs %zu bytes of shared memory (limit %zu)", TY, TX, g.smem, s->smem_optin);
            return SBP_ERR_INVALID_ARGUMENT;
        }
        int per_sm = 1 << 30;
        for (int sc = 0; sc < 3; ++sc) {
            SBP_TRY_CUDA(cudaFuncSetAttribute(g.fn[sc], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)g.smem));
            int n = 0;
            SBP_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, g.fn[sc], threads, g.smem));
            per_sm = std::min(per_sm, n);
        }
        if (per_sm < 1) {
            set_error("stage kernel cannot be resident with %d threads and %zu bytes shared memory", threads, g.smem);
            return SBP_ERR_INVALID_ARGUMENT;
        }
        // persistent grid of up to `ctas` CTAs per SM, or one CTA per tile (ctas == 0)
        const int cps = g.ctas < 0 ? per_sm : std::min(g.ctas, per_sm);
        g.grid = g.ctas == 0 ? g.ntiles : std::min(g.ntiles, cps * s->num_sms);
        if (g.ntiles) {
            SBP_TRY_CUDA(cudaMalloc(&g.d_tiles, g.ntiles * sizeof(int4)));
            SBP_TRY_CUDA(cudaMemcpyAsync(g.d_tiles, tiles[gi].data(), g.ntiles * sizeof(int4),
                                         cudaMemcpyHostToDevice, s->stream));
            g.nedges = (int)edges[gi].size();
            SBP_TRY_CUDA(cudaMalloc(&g.d_edges, g.nedges * sizeof(int4)));
            SBP_TRY_CUDA(cudaMemcpyAsync(g.d_edges, edges[gi].data(), g.nedges * sizeof(int4),
                                         cudaMemcpyHostToDevice, s->stream));
            if (s->has_eval) SBP_TRY_CUDA(cudaMalloc(&g.d_evz, (size_t)g.nedges * 4 * sizeof(double)));
            // the geometry of the group's edge points for their SATs (time-independent)
            edge_geo_kernel<<<(g.nedges + 127) / 128, 128, 0, s->stream>>>(s->d_blocks, s->met64, s->xy, g.d_edges,
                                                                           g.nedges, s->egeo);
            SBP_TRY_CUDA(cudaGetLastError());
        }
    }
    SBP_TRY_CUDA(cudaStreamSynchronize(s->stream));
    while (s->side.size() < groups.size()) {
        cudaStream_t st;
        cudaEvent_t e;
        SBP_TRY_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        SBP_TRY_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        s->side.push_back(st);
        s->ev.push_back(e);
    }
    // Groups are independent when no block reads an edge of a block of another group (Grid and
    // Interpolate neighbours; MultiGrid sides are taken as coupling).  Independent groups run their
    // four stages on their own streams and join once per step, so one group's edge kernel can run
    // beside another group's stage kernel; coupled groups join after every stage.
    bool coupled = false;
    for (int b = 0; b < s->nblocks && !coupled; ++b) {
        if (group_of[b] < 0) continue;
        const BlockDev& B = s->hb[b];
        for (int d = 0; d < 4; ++d) {
            const int k = B.bc_kind[d];
            if (k == BC_MULTIGRID || ((k == BC_GRID || k == BC_INTERPOLATE) && group_of[B.bc_nb[d]] != group_of[b]))
                coupled = true;
        }
    }
    // Fused kernels advance the times themselves, if every group has one.
    TimeAdvance ta;
    ta.active = d_active;
    bool all_fused = !groups.empty();
    for (const Group& g : groups) {
        all_fused = all_fused && g.fused;
        ta.ctas += g.grid;
    }
    if (!all_fused) ta.ctas = 0;
    // Capture one RK4 step.
    SBP_TRY_CUDA(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
    sbp_status rc = SBP_OK;
    if (groups.size() > 1 && !coupled) {
        cudaEventRecord(s->ev_fork, s->stream);
        for (size_t gi = 0; gi < groups.size() && rc == SBP_OK; ++gi) {
            cudaStreamWaitEvent(s->side[gi], s->ev_fork, 0);
            for (int stage = 0; stage < 4 && rc == SBP_OK; ++stage)
                rc = launch_group(s, stage, groups[gi], s->side[gi], true, stage > 0, ta);
            cudaEventRecord(s->ev[gi], s->side[gi]);
        }
        for (size_t gi = 0; gi < groups.size(); ++gi) cudaStreamWaitEvent(s->stream, s->ev[gi], 0);
    }
    for (int stage = 0; stage < 4 && rc == SBP_OK && (groups.size() == 1 || coupled); ++stage) {
        if (groups.size() == 1) {
            rc = launch_group(s, stage, groups[0], s->stream, true, stage > 0, ta);
        } else {
            cudaEventRecord(s->ev_fork, s->stream);
            for (size_t gi = 0; gi < groups.size() && rc == SBP_OK; ++gi) {
                cudaStreamWaitEvent(s->side[gi], s->ev_fork, 0);
                rc = launch_group(s, stage, groups[gi], s->side[gi], true, false, ta);
                cudaEventRecord(s->ev[gi], s->side[gi]);
            }
            for (size_t gi = 0; gi < groups.size(); ++gi) cudaStreamWaitEvent(s->stream, s->ev[gi], 0);
        }
    }
    if (rc == SBP_OK && !all_fused) rc = cuda_status(time_update(s->d_inst, d_active, s->ninst, s->stream), "time update");
    cudaGraph_t graph = nullptr;
    cudaError_t ee = cudaStreamEndCapture(s->stream, &graph);
    if (rc != SBP_OK) {
        if (graph) cudaGraphDestroy(graph);
        return rc;
    }
    SBP_TRY_CUDA(ee);
    graph_out = graph;
    SBP_TRY_CUDA(cudaGraphInstantiate(&gexec_out, graph, 0));
    return SBP_OK;
}

// The system's own schedule: every active instance.  Steps of the previous schedule may still
// be in flight on the system's stream (a caller's stream, see sbp_system_set_stream) and read the
// time-update mask, so they finish before the mask changes.
sbp_status build_schedule(sbp_system* s) {
    SBP_TRY_CUDA(cudaStreamSynchronize(s->st()));
    SBP_TRY_CUDA(cudaStreamSynchronize(s->stream));
    free_groups(s);
    std::vector<int> act(s->active);
    act.push_back(0);  // the fused kernels' counter
    SBP_TRY_CUDA(cudaMemcpyAsync(s->d_active, act.data(), act.size() * sizeof(int), cudaMemcpyHostToDevice, s->stream));
    SBP_TRY(build_step_graph(s, s->active, s->d_active, s->groups, s->graph, s->gexec));
    s->sched_dirty = false;
    return SBP_OK;
}

sbp_status check_status(sbp_system* s) {
    unsigned hs = 0;
    SBP_TRY_CUDA(cudaMemcpyAsync(&hs, s->status, sizeof hs, cudaMemcpyDeviceToHost, s->st()));
    SBP_TRY_CUDA(cudaStreamSynchronize(s->st()));
    if (hs & STATUS_BAD_LAUNCH) {
        set_error("internal: a stage kernel was launched for another RK stage class (flags 0x%x)", hs);
        return SBP_ERR_INVALID_ARGUMENT;
    }
    if (hs) {
        set_error("non-physical state detected on device (flags 0x%x: 1 rho<=0, 2 p<=0, 4 detJ<=0)", hs);
        return SBP_ERR_NONPHYSICAL;
    }
    return SBP_OK;
}

// Sides of kind SBP_BC_EVAL read the expression programs: they must be set before any step.
sbp_status check_eval(const sbp_system* s) {
    if (s->has_eval && !s->eval_set) {
        set_error("the system has SBP_BC_EVAL sides: call sbp_system_set_eval first");
        return SBP_ERR_INVALID_ARGUMENT;
    }
    return SBP_OK;
}

sbp_status run_steps(sbp_system* s, int64_t n) {
    SBP_TRY(check_eval(s));
    if (s->sched_dirty) SBP_TRY(build_schedule(s));
    for (int64_t i = 0; i < n; ++i) SBP_TRY_CUDA(cudaGraphLaunch(s->gexec, s->st()));
    return SBP_OK;
}

bool valid_block(const sbp_system* s, int b) { return b >= 0 && b < s->nblocks; }

// k = RHS(u_in) (SATs included) into k_out for every group: the stage and edge kernels in their
// k-only mode, SAT data at time + dt * ctime.
sbp_status launch_rhs(sbp_system* s, const double* u_in, double* k_out, double ctime) {
    SBP_TRY(check_eval(s));
    cudaStream_t st = s->st();
    for (const Group& g : s->groups) {
        if (g.ntiles == 0) continue;
        StageArgs<double> a = stage_args<double>(s, 0, g);
        a.stage = kStageK;
        a.ctime = ctime;
        a.u_in = u_in;
        a.u_out = k_out;
        void* args[] = {&a};
        const int threads = s->threads + (g.fused ? sat_threads(g.ty) : 0);
        SBP_TRY_CUDA(cudaLaunchKernel(g.fn[0], dim3(g.grid), dim3(threads), args, g.smem, st));  // f64: one entry
        if (g.fused) continue;
        int4* edges = g.d_edges;
        int nedges = g.nedges;
        void* sargs[] = {&a, &edges, &nedges};
        if (s->has_eval)
            SBP_TRY_CUDA(cudaLaunchKernel(eval_ptr_f64(), dim3((g.nedges + kSatThreads - 1) / kSatThreads),
                                          dim3(kSatThreads), sargs, 0, st));
        SBP_TRY_CUDA(cudaLaunchKernel(sat_ptr_f64(), dim3((g.nedges + kSatThreads - 1) / kSatThreads),
                                      dim3(kSatThreads), sargs, 0, st));
    }
    return SBP_OK;
}

sbp_status ensure_kbuf(sbp_system* s, int stages) {
    if (s->kbuf_stages >= stages) return SBP_OK;
    if (s->kbuf) cudaFree(s->kbuf);
    s->kbuf = nullptr;
    s->kbuf_stages = 0;
    SBP_TRY_CUDA(cudaMalloc((void**)&s->kbuf, (size_t)kMaxStages * s->nq * sizeof(double)));
    s->kbuf_stages = kMaxStages;
    return SBP_OK;
}

// integrate::<Tableau> (utils/integrate/src/lib.rs:176-222) for every block: the stage inputs
// fut = prev; fut += (a dt) k_j in order, the RHS of each stage into its k, and at the end
// prev = prev + (b dt) k_j in order (in place).  dt_fixed < 0: each instance's own dt.
// Embedded tableaus also form fut2 = prev + (bstar dt) k_j into `fut2` when it is given and
// leave prev untouched, writing the B combination to `fut` instead.
sbp_status integrate_tableau(sbp_system* s, const Tableau& T, double dt_fixed, double* fut, double* fut2) {
    cudaStream_t st = s->st();
    double* prev = static_cast<double*>(s->prev_hi);
    double* stage_in = static_cast<double*>(s->uA);
    auto kk = [&](int j) { return s->kbuf + (size_t)j * s->nq; };
    for (int i = 0; i < T.s; ++i) {
        const double* in = prev;
        double ctime = 0.0;
        if (i > 0) {
            StageCombination cm{};
            for (int j = 0; j < i; ++j) {
                cm.coef[j] = T.a[i - 1][j];
                cm.k[j] = kk(j);
            }
            cm.nk = i;
            cm.dt_fixed = dt_fixed;
            SBP_TRY_CUDA(combine_stages(s->d_blocks, s->d_inst, s->nblocks, prev, stage_in, cm, s->max_points, st));
            in = stage_in;
            ctime = T.c[i - 1];
        }
        SBP_TRY(launch_rhs(s, in, kk(i), ctime));
    }
    StageCombination cm{};
    for (int j = 0; j < T.s; ++j) {
        cm.coef[j] = T.b[j];
        cm.k[j] = kk(j);
    }
    cm.nk = T.s;
    cm.dt_fixed = dt_fixed;
    SBP_TRY_CUDA(combine_stages(s->d_blocks, s->d_inst, s->nblocks, prev, fut ? fut : prev, cm, s->max_points, st));
    if (fut2) {
        for (int j = 0; j < T.s; ++j) cm.coef[j] = T.bstar[j];
        SBP_TRY_CUDA(combine_stages(s->d_blocks, s->d_inst, s->nblocks, prev, fut2, cm, s->max_points, st));
    }
    return SBP_OK;
}

}  // namespace

extern "C" {

sbp_status sbp_system_create(int device, const sbp_block_desc* blocks, int nblocks, int ninstances, int precision,
                             double gamma, sbp_system** out) {
    clear_error();
    if (!out || !blocks || nblocks <= 0 || ninstances <= 0 || nblocks > 65535) {
        set_error("bad arguments (need 1..65535 blocks and at least one instance)");
        return SBP_ERR_INVALID_ARGUMENT;
    }
    if (precision != SBP_PRECISION_F64 && precision != SBP_PRECISION_F32_COMPENSATED) {
        set_error("unknown precision %d", precision);
        return SBP_ERR_INVALID_ARGUMENT;
    }
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        set_error("no CUDA device");
        return SBP_ERR_NO_DEVICE;
    }
    if (device < 0 || device >= ndev) {
        set_error("device %d out of range", device);
        return SBP_ERR_INVALID_ARGUMENT;
    }
    // validate blocks
    for (int b = 0; b < nblocks; ++b) {
        const sbp_block_desc& D = blocks[b];
        OpInfo ox, oy;
        if (!op_info(D.op_xi, ox) || !op_info(D.op_eta, oy)) {
            set_error("block %d: unknown operator", b);
            return SBP_ERR_INVALID_ARGUMENT;
        }
        if (!D.x || !D.y) {
            set_error("block %d: null grid", b);
            return SBP_ERR_INVALID_ARGUMENT;
        }
        if (D.nx < 2 * ox.M || D.nx < ox.N || D.ny < 2 * oy.M || D.ny < oy.N) {
            set_error("block %d: %lld x %lld grid does not fit the operators (n >= max(2M, N))", b, (long long)D.ny,
                      (long long)D.nx);
            return SBP_ERR_SHAPE;
        }
        // the stage kernels address a block's 5 metric planes with 32-bit offsets
        if (D.nx * D.ny > kMaxBlockPoints) {
            set_error("block %d: %lld x %lld grid has more than %lld points", b, (long long)D.ny, (long long)D.nx,
                      (long long)kMaxBlockPoints);
            return SBP_ERR_SHAPE;
        }
        if (D.instance < 0 || D.instance >= ninstances) {
            set_error("block %d: instance %d out of range", b, D.instance);
            return SBP_ERR_INVALID_ARGUMENT;
        }
        for (int d = 0; d < 4; ++d) {
            const int k = D.bc_kind[d];
            if (k != SBP_BC_THIS && k != SBP_BC_GRID && k != SBP_BC_VORTEX && k != SBP_BC_INTERPOLATE &&
                k != SBP_BC_MULTIGRID && k != SBP_BC_EVAL) {
                set_error("block %d: unknown boundary kind %d", b, k);
                return SBP_ERR_INVALID_ARGUMENT;
            }
            const bool ns = d == SBP_NORTH || d == SBP_SOUTH;
            const int64_t mine = ns ? D.nx : D.ny;
            if (k == SBP_BC_INTERPOLATE) {
                const int g = D.bc_neighbour[d];
                const int op = D.bc_interp_op[d];
                if (g < 0 || g >= nblocks || op < 0 || op > 3) {
                    set_error("block %d: interpolation neighbour %d or operator %d out of range", b, g, op);
                    return SBP_ERR_INVALID_ARGUMENT;
                }
                if (blocks[g].instance != D.instance) {
                    set_error("block %d: neighbour %d belongs to another instance", b, g);
                    return SBP_ERR_INVALID_ARGUMENT;
                }
                const int64_t theirs = ns ? blocks[g].nx : blocks[g].ny;
                const bool f2c = D.nx < blocks[g].nx;  // euler/src/lib.rs:818
                const bool sizes = f2c ? interp_sizes_ok(op, theirs, mine) : interp_sizes_ok(op, mine, theirs);
                if (!sizes || !interp_reads_in_range(op, f2c, theirs, mine)) {
                    set_error("block %d: %s interpolation from %lld to %lld points does not fit the operator", b,
                              f2c ? "fine2coarse" : "coarse2fine", (long long)theirs, (long long)mine);
                    return SBP_ERR_SHAPE;
                }
            }
            if (k == SBP_BC_MULTIGRID) {
                const int nseg = D.bc_multigrid_count[d];
                if (nseg < 1 || !D.bc_multigrid[d]) {
                    set_error("block %d: multigrid boundary without segments", b);
                    return SBP_ERR_INVALID_ARGUMENT;
                }
                int64_t cover = 0;
                for (int q = 0; q < nseg; ++q) {
                    const int g = D.bc_multigrid[d][3 * q], st = D.bc_multigrid[d][3 * q + 1],
                              en = D.bc_multigrid[d][3 * q + 2];
                    if (g < 0 || g >= nblocks || blocks[g].instance != D.instance) {
                        set_error("block %d: multigrid segment %d: bad block %d", b, q, g);
                        return SBP_ERR_INVALID_ARGUMENT;
                    }
                    const int64_t theirs = ns ? blocks[g].nx : blocks[g].ny;
                    if (st < 0 || en > theirs || en - st < 1) {
                        set_error("block %d: multigrid segment %d [%d, %d) outside block %d's edge", b, q, st, en, g);
                        return SBP_ERR_SHAPE;
                    }
                    cover += (en - st) - (q + 1 < nseg ? 1 : 0);
                }
                if (cover != mine) {
                    // the reference asserts that the segments fill the edge (euler/src/lib.rs:840)
                    set_error("block %d: multigrid segments cover %lld of %lld edge points", b, (long long)cover,
                              (long long)mine);
                    return SBP_ERR_SHAPE;
                }
            }
            if (k == SBP_BC_GRID) {
                const int g = D.bc_neighbour[d];
                if (g < 0 || g >= nblocks) {
                    set_error("block %d: neighbour %d out of range", b, g);
                    return SBP_ERR_INVALID_ARGUMENT;
                }
                const bool ns = d == SBP_NORTH || d == SBP_SOUTH;
                const int64_t mine = ns ? D.nx : D.ny, theirs = ns ? blocks[g].nx : blocks[g].ny;
                if (mine != theirs) {
                    // SAT_characteristic asserts equal shapes (euler/src/lib.rs:1163)
                    set_error("block %d: interface with block %d has %lld vs %lld points", b, g, (long long)mine,
                              (long long)theirs);
                    return SBP_ERR_SHAPE;
                }
                if (blocks[g].instance != D.instance) {
                    set_error("block %d: neighbour %d belongs to another instance", b, g);
                    return SBP_ERR_INVALID_ARGUMENT;
                }
            }
        }
    }
    sbp_system* s = new sbp_system();
    s->device = device;
    s->prec = precision;
    s->gamma = gamma;
    s->nblocks = nblocks;
    s->ninst = ninstances;
    auto fail = [&](sbp_status st) {
        destroy_all(s);
        return st;
    };
    if (cudaSetDevice(device) != cudaSuccess) return fail(cuda_status(cudaSetDevice(device), "cudaSetDevice"));
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device);
    s->num_sms = v > 0 ? v : 148;
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    s->smem_optin = v > 0 ? (size_t)v : 48 * 1024;
    {
        cudaError_t e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
        if (e != cudaSuccess) return fail(cuda_status(e, "stream"));
        e = cudaEventCreateWithFlags(&s->ev_fork, cudaEventDisableTiming);
        if (e != cudaSuccess) return fail(cuda_status(e, "event"));
    }
    // layout
    std::vector<int4> mg_host;
    s->hb.resize(nblocks);
    s->dense_off.resize(nblocks);
    s->hoff.resize(nblocks);
    int64_t hw_total = 0;
    for (int b = 0; b < nblocks; ++b) {
        const sbp_block_desc& D = blocks[b];
        BlockDev& B = s->hb[b];
        std::memset(&B, 0, sizeof B);
        OpInfo ox, oy;
        op_info(D.op_xi, ox);
        op_info(D.op_eta, oy);
        B.nx = (int)D.nx;
        B.ny = (int)D.ny;
        const int64_t n = D.nx * D.ny;
        B.npad = (int)pad64(n);
        B.op_xi = D.op_xi;
        B.op_eta = D.op_eta;
        B.instance = D.instance;
        for (int d = 0; d < 4; ++d) {
            B.bc_kind[d] = D.bc_kind[d];
            if (D.bc_kind[d] == SBP_BC_EVAL) s->has_eval = true;
            B.bc_nb[d] = (D.bc_kind[d] == SBP_BC_GRID || D.bc_kind[d] == SBP_BC_INTERPOLATE) ? D.bc_neighbour[d] : b;
            if (D.bc_kind[d] == SBP_BC_INTERPOLATE) B.bc_aux[d] = D.bc_interp_op[d];
            if (D.bc_kind[d] == SBP_BC_MULTIGRID) {
                B.bc_aux[d] = (int)mg_host.size();
                B.bc_aux2[d] = D.bc_multigrid_count[d];
                for (int q = 0; q < D.bc_multigrid_count[d]; ++q)
                    mg_host.push_back(make_int4(D.bc_multigrid[d][3 * q], D.bc_multigrid[d][3 * q + 1],
                                                D.bc_multigrid[d][3 * q + 2], 0));
            }
        }
        B.q_off = s->nq;
        B.r_off = s->nq / 4;
        B.m_off = s->nm;
        B.x_off = s->nx2;
        B.e_off = s->nedge;
        s->nedge += edge_count(D.nx, D.ny);
        s->nq += 4 * (int64_t)B.npad;
        s->nm += 5 * (int64_t)B.npad;
        s->nx2 += 2 * (int64_t)B.npad;
        B.idx_xi = inv_spacing<double>(ox.h2, D.nx);
        B.idx_eta = inv_spacing<double>(oy.h2, D.ny);
        // SAT_north/.. penalties: (n-1)/H_0, or (n-2)/H_0 for h2 (euler/src/lib.rs:1033-1037, 1093-1097)
        B.hi_eta = (oy.h2 ? double(D.ny - 2) : double(D.ny - 1)) / op_h_weights(D.op_eta)[0];
        B.hi_xi = (ox.h2 ? double(D.nx - 2) : double(D.nx - 1)) / op_h_weights(D.op_xi)[0];
        s->max_points = std::max(s->max_points, n);
        s->dense_off[b] = s->dense_total;
        s->dense_total += 4 * n;
        s->hoff[b] = hw_total;
        hw_total += D.nx + D.ny;
    }
    s->hi.assign(ninstances, InstanceDev{});
    for (auto& I : s->hi) {
        std::memset(&I, 0, sizeof I);
        set_dt_host(I, NAN);
        I.time = 0.0;
        I.mach = 0.5;
        set_reference(I, gamma);
    }
    s->active.assign(ninstances, 1);
    // allocations
    const size_t ts = s->tsize();
    auto alloc = [&](void** p, size_t bytes) { return cudaMalloc(p, bytes < 16 ? 16 : bytes); };
    cudaError_t e = cudaSuccess;
    e = e ?: alloc((void**)&s->d_blocks, nblocks * sizeof(BlockDev));
    e = e ?: alloc((void**)&s->d_inst, ninstances * sizeof(InstanceDev));
    e = e ?: alloc((void**)&s->d_active, (ninstances + 1) * sizeof(int));
    e = e ?: alloc(&s->prev_hi, s->nq * ts);
    e = e ?: alloc(&s->acc_hi, s->nq * ts);
    e = e ?: alloc(&s->uA, s->nq * ts);
    e = e ?: alloc(&s->uB, s->nq * ts);
    if (precision == SBP_PRECISION_F32_COMPENSATED) {
        e = e ?: alloc(&s->prev_lo, s->nq * ts);
        e = e ?: alloc((void**)&s->met32, s->nm * sizeof(float));
        e = e ?: alloc((void**)&s->rinf, (s->nq / 4) * sizeof(float));
    } else {
        e = e ?: alloc((void**)&s->jinv64, (s->nq / 4) * sizeof(double));
    }
    e = e ?: alloc((void**)&s->met64, s->nm * sizeof(double));
    e = e ?: alloc((void**)&s->xy, s->nx2 * sizeof(double));
    e = e ?: alloc((void**)&s->hw, hw_total * sizeof(double));
    e = e ?: alloc((void**)&s->d_hoff, nblocks * sizeof(int64_t));
    e = e ?: alloc((void**)&s->d_poff4, nblocks * sizeof(int64_t));
    e = e ?: alloc((void**)&s->d_poff8, nblocks * sizeof(int64_t));
    e = e ?: alloc((void**)&s->d_zero, sizeof(int64_t));
    s->staging_bytes = (size_t)s->dense_total * sizeof(double);
    e = e ?: alloc(&s->staging, s->staging_bytes);
    e = e ?: alloc((void**)&s->status, sizeof(unsigned));
    // per-block norms, then kNormParts partial sums per block (error_terms / diff_terms)
    e = e ?: alloc((void**)&s->d_sums, (size_t)nblocks * (1 + kNormParts) * sizeof(double));
    e = e ?: alloc((void**)&s->d_speeds, 2 * nblocks * sizeof(unsigned long long));
    e = e ?: alloc(&s->kedge, 4 * s->nedge * ts);
    e = e ?: alloc((void**)&s->egeo, kEdgeGeo * s->nedge * sizeof(double));
    e = e ?: alloc((void**)&s->d_mg, (mg_host.size() + 1) * sizeof(int4));
    e = e ?: alloc((void**)&s->d_eval, sizeof(EvalDev));
    if (e != cudaSuccess) return fail(cuda_status(e, "device allocation"));
    cudaStream_t st = s->stream;
    e = e ?: cudaMemsetAsync(s->prev_hi, 0, s->nq * ts, st);
    e = e ?: cudaMemsetAsync(s->acc_hi, 0, s->nq * ts, st);
    e = e ?: cudaMemsetAsync(s->uA, 0, s->nq * ts, st);
    e = e ?: cudaMemsetAsync(s->uB, 0, s->nq * ts, st);
    if (s->prev_lo) e = e ?: cudaMemsetAsync(s->prev_lo, 0, s->nq * ts, st);
    e = e ?: cudaMemsetAsync(s->met64, 0, s->nm * sizeof(double), st);
    e = e ?: cudaMemsetAsync(s->status, 0, sizeof(unsigned), st);
    e = e ?: cudaMemsetAsync(s->d_zero, 0, sizeof(int64_t), st);
    e = e ?: cudaMemcpyAsync(s->d_blocks, s->hb.data(), nblocks * sizeof(BlockDev), cudaMemcpyHostToDevice, st);
    e = e ?: cudaMemcpyAsync(s->d_inst, s->hi.data(), ninstances * sizeof(InstanceDev), cudaMemcpyHostToDevice, st);
    e = e ?: cudaMemcpyAsync(s->d_hoff, s->hoff.data(), nblocks * sizeof(int64_t), cudaMemcpyHostToDevice, st);
    if (!mg_host.empty())
        e = e ?: cudaMemcpyAsync(s->d_mg, mg_host.data(), mg_host.size() * sizeof(int4), cudaMemcpyHostToDevice, st);
    {
        std::vector<int64_t> p8(nblocks);
        for (int b = 0; b < nblocks; ++b) p8[b] = 2 * s->dense_off[b];
        e = e ?: cudaMemcpyAsync(s->d_poff4, s->dense_off.data(), nblocks * sizeof(int64_t), cudaMemcpyHostToDevice,
                                 st);
        e = e ?: cudaMemcpyAsync(s->d_poff8, p8.data(), nblocks * sizeof(int64_t), cudaMemcpyHostToDevice, st);
    }
    // H-norm weights per block: hx then hy (euler/src/lib.rs:391-420)
    {
        std::vector<double> w(hw_total);
        for (int b = 0; b < nblocks; ++b) {
            const sbp_block_desc& D = blocks[b];
            double* hx = w.data() + s->hoff[b];
            double* hy = hx + D.nx;
            for (int dir = 0; dir < 2; ++dir) {
                const int op = dir == 0 ? D.op_xi : D.op_eta;
                const int64_t n = dir == 0 ? D.nx : D.ny;
                double* h = dir == 0 ? hx : hy;
                OpInfo oi;
                op_info(op, oi);
                const double* hw = op_h_weights(op);
                const double factor = oi.h2 ? 1.0 / double(n - 2) : 1.0 / double(n - 1);
                for (int64_t i = 0; i < n; ++i) h[i] = 1.0;
                for (int i = 0; i < oi.M; ++i) {
                    h[i] = hw[i];
                    h[n - 1 - i] = hw[i];
                }
                for (int64_t i = 0; i < n; ++i) h[i] = h[i] * factor;
            }
        }
        e = e ?: cudaMemcpyAsync(s->hw, w.data(), hw_total * sizeof(double), cudaMemcpyHostToDevice, st);
        e = e ?: cudaStreamSynchronize(st);
    }
    if (e != cudaSuccess) return fail(cuda_status(e, "system setup"));
    // grids and metrics (Metrics::new per block, in f64)
    double* tmp = static_cast<double*>(s->staging);  // >= 4 * max_points doubles
    for (int b = 0; b < nblocks && e == cudaSuccess; ++b) {
        const sbp_block_desc& D = blocks[b];
        const BlockDev& B = s->hb[b];
        const int64_t n = D.nx * D.ny;
        double* x = s->xy + B.x_off;
        double* y = x + B.npad;
        e = e ?: cudaMemcpyAsync(x, D.x, n * sizeof(double), cudaMemcpyHostToDevice, st);
        e = e ?: cudaMemcpyAsync(y, D.y, n * sizeof(double), cudaMemcpyHostToDevice, st);
        e = e ?: op_apply(D.op_xi, 0, 0, 0, x, tmp, D.ny, D.nx, 1, n, st);
        e = e ?: op_apply(D.op_eta, 1, 0, 0, x, tmp + n, D.ny, D.nx, 1, n, st);
        e = e ?: op_apply(D.op_xi, 0, 0, 0, y, tmp + 2 * n, D.ny, D.nx, 1, n, st);
        e = e ?: op_apply(D.op_eta, 1, 0, 0, y, tmp + 3 * n, D.ny, D.nx, 1, n, st);
        e = e ?: metrics_combine(tmp, tmp + n, tmp + 2 * n, tmp + 3 * n, n, s->met64 + B.m_off, B.npad, s->status, st);
    }
    if (e == cudaSuccess && s->met32) {
        e = narrow_f32(s->met64, s->met32, s->nm, st);
        e = e ?: jacobian_inverse_f32(s->d_blocks, nblocks, s->met64, s->met32, s->max_points, st);
    }
    if (e == cudaSuccess && s->jinv64)
        e = jacobian_inverse_f64(s->d_blocks, nblocks, s->met64, s->jinv64, s->max_points, st);
    if (e != cudaSuccess) return fail(cuda_status(e, "metrics"));
    if (s->rinf) {
        // the state starts at zero: in the compensated form a deviation of -qref
        e = cudaMemsetAsync(s->staging, 0, s->staging_bytes, st);
        e = e ?: unpack_state(s->d_blocks, s->d_inst, nblocks, s->d_poff4, s->prec, SBP_F64, s->staging, s->prev_hi,
                              s->prev_lo, s->max_points, st);
        if (e != cudaSuccess) return fail(cuda_status(e, "initial state"));
        const sbp_status rs = build_free_stream_dissipation(s, -1);
        if (rs != SBP_OK) return fail(rs);
    }
    sbp_status cs = check_status(s);
    if (cs != SBP_OK) {
        set_error("non-positive Jacobian determinant in the grid (Metrics::new asserts detj > 0)");
        return fail(cs);
    }
    // every operator pair must be available
    for (int b = 0; b < nblocks; ++b) {
        OpInfo ox, oy;
        op_info(s->hb[b].op_xi, ox);
        op_info(s->hb[b].op_eta, oy);
        if (!stage_kernel_ptr(s->prec, s->hb[b].op_xi, s->hb[b].op_eta, ox.upwind && oy.upwind, 16, 0)) {
            set_error("operator pair (xi %d, eta %d) is not built into the stage kernels", s->hb[b].op_xi,
                      s->hb[b].op_eta);
            return fail(SBP_ERR_UNSUPPORTED);
        }
    }
    *out = s;
    return SBP_OK;
}

sbp_status sbp_system_destroy(sbp_system* sys) {
    clear_error();
    destroy_all(sys);
    return SBP_OK;
}

sbp_status sbp_system_set_force_trad(sbp_system* sys, int force_trad) {
    clear_error();
    if (!sys) return SBP_ERR_INVALID_ARGUMENT;
    if (sys->force_trad != (force_trad != 0)) {
        sys->force_trad = force_trad != 0;
        sys->sched_dirty = true;
    }
    return SBP_OK;
}

sbp_status sbp_system_set_vortex(sbp_system* sys, int instance, const sbp_vortex_params* vp) {
    clear_error();
    if (!sys || !vp || instance >= sys->ninst || vp->nvortices < 0 || vp->nvortices > 5) {
        set_error("bad vortex parameters / instance");
        return SBP_ERR_INVALID_ARGUMENT;
    }
    cudaSetDevice(sys->device);
    SBP_TRY(sync_times(sys));
    cudaStream_t st = sys->st();
    // A compensated system keeps each instance's state as a deviation from the instance's
    // reference state, which follows the vortex's free stream: the state is taken out as the
    // absolute state and stored again against the new reference.
    if (sys->prec == 1)
        SBP_TRY_CUDA(pack_state(sys->d_blocks, sys->d_inst, sys->nblocks, sys->d_poff4, sys->prec, SBP_F64,
                                sys->prev_hi, sys->prev_lo, sys->staging, sys->max_points, st));
    for (int i = 0; i < sys->ninst; ++i) {
        if (instance >= 0 && i != instance) continue;
        InstanceDev& I = sys->hi[i];
        I.nvort = vp->nvortices;
        for (int k = 0; k < 5; ++k) {
            I.x0[k] = vp->x0[k];
            I.y0[k] = vp->y0[k];
            I.rstar[k] = vp->rstar[k];
            I.eps[k] = vp->eps[k];
        }
        I.mach = vp->mach;
        set_reference(I, sys->gamma);
    }
    SBP_TRY(upload_instances(sys));
    if (sys->prec == 1) {
        SBP_TRY_CUDA(unpack_state(sys->d_blocks, sys->d_inst, sys->nblocks, sys->d_poff4, sys->prec, SBP_F64,
                                  sys->staging, sys->prev_hi, sys->prev_lo, sys->max_points, st));
        SBP_TRY(build_free_stream_dissipation(sys, instance));
        SBP_TRY_CUDA(cudaStreamSynchronize(st));
    }
    return SBP_OK;
}

sbp_status sbp_system_init_vortex(sbp_system* sys, int instance, double t) {
    clear_error();
    if (!sys || instance >= sys->ninst) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    SBP_TRY_CUDA(vortex_init(sys->d_blocks, sys->d_inst, sys->nblocks, instance, sys->gamma, t, sys->xy, sys->prec,
                             sys->prev_hi, sys->prev_lo, sys->max_points, sys->st()));
    SBP_TRY_CUDA(cudaMemsetAsync(sys->status, 0, sizeof(unsigned), sys->st()));
    SBP_TRY_CUDA(cudaStreamSynchronize(sys->st()));
    return SBP_OK;
}

sbp_status sbp_system_set_state(sbp_system* sys, int block, const double* q) {
    clear_error();
    if (!sys || !q || !valid_block(sys, block)) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    const BlockDev& B = sys->hb[block];
    const int64_t n = (int64_t)B.nx * B.ny;
    cudaStream_t st = sys->st();
    if (sys->prec == 0) {
        SBP_TRY_CUDA(cudaMemcpy2DAsync(static_cast<double*>(sys->prev_hi) + B.q_off, B.npad * sizeof(double), q,
                                       n * sizeof(double), n * sizeof(double), 4, cudaMemcpyHostToDevice, st));
    } else {
        SBP_TRY_CUDA(cudaMemcpyAsync(sys->staging, q, 4 * n * sizeof(double), cudaMemcpyHostToDevice, st));
        SBP_TRY_CUDA(unpack_state(sys->d_blocks + block, sys->d_inst, 1, sys->d_zero, sys->prec, 0, sys->staging, sys->prev_hi,
                                  sys->prev_lo, n, st));
    }
    SBP_TRY_CUDA(cudaMemsetAsync(sys->status, 0, sizeof(unsigned), st));
    SBP_TRY_CUDA(cudaStreamSynchronize(st));
    return SBP_OK;
}

sbp_status sbp_system_get_state(sbp_system* sys, int block, double* q) {
    clear_error();
    if (!sys || !q || !valid_block(sys, block)) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    const BlockDev& B = sys->hb[block];
    const int64_t n = (int64_t)B.nx * B.ny;
    cudaStream_t st = sys->st();
    if (sys->prec == 0) {
        SBP_TRY_CUDA(cudaMemcpy2DAsync(q, n * sizeof(double), static_cast<double*>(sys->prev_hi) + B.q_off,
                                       B.npad * sizeof(double), n * sizeof(double), 4, cudaMemcpyDeviceToHost, st));
    } else {
        SBP_TRY_CUDA(pack_state(sys->d_blocks + block, sys->d_inst, 1, sys->d_zero, sys->prec, 0, sys->prev_hi, sys->prev_lo,
                                sys->staging, n, st));
        SBP_TRY_CUDA(cudaMemcpyAsync(q, sys->staging, 4 * n * sizeof(double), cudaMemcpyDeviceToHost, st));
    }
    SBP_TRY_CUDA(cudaStreamSynchronize(st));
    return SBP_OK;
}

int64_t sbp_system_state_count(const sbp_system* sys, int dtype) {
    if (!sys) return -1;
    return dtype == SBP_F32 ? 2 * sys->dense_total : sys->dense_total;
}

sbp_status sbp_system_set_state_all(sbp_system* sys, int dtype, const void* q) {
    clear_error();
    if (!sys || !q || (dtype != SBP_F64 && dtype != SBP_F32)) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    cudaStream_t st = sys->st();
    const size_t bytes = (size_t)sys->dense_total * (dtype == SBP_F64 ? 8 : 8);
    SBP_TRY_CUDA(cudaMemcpyAsync(sys->staging, q, bytes, cudaMemcpyHostToDevice, st));
    SBP_TRY_CUDA(unpack_state(sys->d_blocks, sys->d_inst, sys->nblocks, dtype == SBP_F64 ? sys->d_poff4 : sys->d_poff8, sys->prec,
                              dtype, sys->staging, sys->prev_hi, sys->prev_lo, sys->max_points, st));
    SBP_TRY_CUDA(cudaMemsetAsync(sys->status, 0, sizeof(unsigned), st));
    SBP_TRY_CUDA(cudaStreamSynchronize(st));
    return SBP_OK;
}

sbp_status sbp_system_get_state_all(sbp_system* sys, int dtype, void* q) {
    clear_error();
    if (!sys || !q || (dtype != SBP_F64 && dtype != SBP_F32)) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    cudaStream_t st = sys->st();
    const size_t bytes = (size_t)sys->dense_total * 8;
    SBP_TRY_CUDA(pack_state(sys->d_blocks, sys->d_inst, sys->nblocks, dtype == SBP_F64 ? sys->d_poff4 : sys->d_poff8, sys->prec,
                            dtype, sys->prev_hi, sys->prev_lo, sys->staging, sys->max_points, st));
    SBP_TRY_CUDA(cudaMemcpyAsync(q, sys->staging, bytes, cudaMemcpyDeviceToHost, st));
    SBP_TRY_CUDA(cudaStreamSynchronize(st));
    return SBP_OK;
}

sbp_status sbp_system_get_state_all_device(sbp_system* sys, int dtype, void* d_q) {
    clear_error();
    if (!sys || !d_q || (dtype != SBP_F64 && dtype != SBP_F32)) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    cudaStream_t st = sys->st();
    SBP_TRY_CUDA(pack_state(sys->d_blocks, sys->d_inst, sys->nblocks, dtype == SBP_F64 ? sys->d_poff4 : sys->d_poff8, sys->prec,
                            dtype, sys->prev_hi, sys->prev_lo, d_q, sys->max_points, st));
    SBP_TRY_CUDA(cudaStreamSynchronize(st));
    return SBP_OK;
}

sbp_status sbp_system_set_eval(sbp_system* sys, int form, const int32_t* const code[4], const int32_t len[4],
                               const double* consts, int nconsts) {
    clear_error();
    if (!sys || !code || !len || (nconsts > 0 && !consts) || nconsts < 0) return SBP_ERR_INVALID_ARGUMENT;
    if (form != EVAL_CONSERVATION && form != EVAL_PRESSURE) {
        set_error("unknown expression form %d", form);
        return SBP_ERR_INVALID_ARGUMENT;
    }
    if (nconsts > kEvalConsts) {
        set_error("%d constants (at most %d)", nconsts, kEvalConsts);
        return SBP_ERR_INVALID_ARGUMENT;
    }
    std::vector<EvalDev> h(1);
    EvalDev& E = h[0];
    std::memset(&E, 0, sizeof E);
    E.form = form;
    for (int k = 0; k < 4; ++k) {
        if (!code[k]) return SBP_ERR_INVALID_ARGUMENT;
        if (const char* why = eval_check(code[k], len[k], nconsts)) {
            set_error("expression program %d: %s", k, why);
            return SBP_ERR_INVALID_ARGUMENT;
        }
        E.len[k] = len[k];
        std::memcpy(E.code[k], code[k], len[k] * sizeof(int32_t));
    }
    if (nconsts) std::memcpy(E.consts, consts, nconsts * sizeof(double));
    cudaSetDevice(sys->device);
    SBP_TRY_CUDA(cudaMemcpyAsync(sys->d_eval, &E, sizeof E, cudaMemcpyHostToDevice, sys->st()));
    SBP_TRY_CUDA(cudaStreamSynchronize(sys->st()));
    sys->eval_set = true;
    return SBP_OK;
}

namespace {

// Plan and build the chunks of sbp_system_advance_host: at most `want` contiguous block ranges
// of whole instances with about equal points.  Instances coupled to another instance (a Grid or
// Interpolate side naming a block of another instance, or any MultiGrid side) keep everything
// in one chunk.
sbp_status build_chunks(sbp_system* s, int want) {
    free_chunks(s);
    const int nb = s->nblocks;
    bool coupled = false;
    for (int b = 0; b < nb && !coupled; ++b)
        for (int d = 0; d < 4; ++d) {
            const BlockDev& B = s->hb[b];
            if (B.bc_kind[d] == BC_MULTIGRID) coupled = true;
            if ((B.bc_kind[d] == BC_GRID || B.bc_kind[d] == BC_INTERPOLATE) &&
                s->hb[B.bc_nb[d]].instance != B.instance)
                coupled = true;
        }
    // a cut before block b is allowed when no instance has blocks on both sides of it
    std::vector<int> last(s->ninst, -1);
    for (int b = 0; b < nb; ++b) last[s->hb[b].instance] = b;
    std::vector<int> cuts = {0};
    if (!coupled && want > 1) {
        int64_t total = 0;
        for (int b = 0; b < nb; ++b) total += (int64_t)s->hb[b].nx * s->hb[b].ny;
        int reach = -1;
        int64_t acc = 0;
        for (int b = 0; b < nb; ++b) {
            if (b > 0 && reach < b && acc >= total * (int64_t)cuts.size() / want && (int)cuts.size() < want)
                cuts.push_back(b);
            reach = std::max(reach, last[s->hb[b].instance]);
            acc += (int64_t)s->hb[b].nx * s->hb[b].ny;
        }
    }
    cuts.push_back(nb);
    for (size_t c = 0; c + 1 < cuts.size(); ++c) {
        s->chunks.emplace_back();
        Chunk& ch = s->chunks.back();
        ch.b0 = cuts[c];
        ch.b1 = cuts[c + 1];
        ch.active.assign(s->ninst, 0);
        for (int b = ch.b0; b < ch.b1; ++b) ch.active[s->hb[b].instance] = 1;
        SBP_TRY_CUDA(cudaStreamCreateWithFlags(&ch.st, cudaStreamNonBlocking));
        SBP_TRY_CUDA(cudaEventCreateWithFlags(&ch.done, cudaEventDisableTiming));
        SBP_TRY_CUDA(cudaMalloc((void**)&ch.d_active, (s->ninst + 1) * sizeof(int)));
        SBP_TRY_CUDA(cudaMemcpyAsync(ch.d_active, ch.active.data(), s->ninst * sizeof(int), cudaMemcpyHostToDevice,
                                     s->stream));
        SBP_TRY_CUDA(cudaMemsetAsync(ch.d_active + s->ninst, 0, sizeof(int), s->stream));  // the fused kernels' counter
        SBP_TRY(build_step_graph(s, ch.active, ch.d_active, ch.groups, ch.graph, ch.gexec));
    }
    s->chunk_gen = s->tiles_gen;
    s->chunk_trad = s->force_trad;
    s->chunk_req = want;
    return SBP_OK;
}

}  // namespace

sbp_status sbp_system_advance_host(sbp_system* sys, int dtype, const void* q_in, void* q_out, int64_t nsteps,
                                   int nchunks) {
    clear_error();
    if (!sys || !q_in || !q_out || nsteps < 0 || (dtype != SBP_F64 && dtype != SBP_F32))
        return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    for (int i = 0; i < sys->ninst; ++i)
        if (nsteps > 0 && !(sys->hi[i].dt == sys->hi[i].dt)) {
            set_error("instance %d has no dt (call sbp_system_set_dt first)", i);
            return SBP_ERR_INVALID_ARGUMENT;
        }
    SBP_TRY(check_eval(sys));
    const int want = nchunks > 0 ? std::min(nchunks, 64) : 16;
    if (sys->chunks.empty() || sys->chunk_req != want || sys->chunk_gen != sys->tiles_gen ||
        sys->chunk_trad != sys->force_trad)
        SBP_TRY(build_chunks(sys, want));
    cudaStream_t st = sys->st();
    const int64_t* poff = dtype == SBP_F64 ? sys->d_poff4 : sys->d_poff8;
    SBP_TRY_CUDA(cudaMemsetAsync(sys->status, 0, sizeof(unsigned), st));
    SBP_TRY_CUDA(cudaEventRecord(sys->ev_fork, st));
    const char* in = static_cast<const char*>(q_in);
    char* out = static_cast<char*>(q_out);
    char* stg = static_cast<char*>(sys->staging);
    // every packed value takes 8 bytes (an f64, or an f32 hi and lo): block b starts at byte 8 dense_off[b]
    for (Chunk& c : sys->chunks) {
        const int64_t o0 = 8 * sys->dense_off[c.b0];
        const int64_t o1 = c.b1 < sys->nblocks ? 8 * sys->dense_off[c.b1] : 8 * sys->dense_total;
        SBP_TRY_CUDA(cudaStreamWaitEvent(c.st, sys->ev_fork, 0));
        SBP_TRY_CUDA(cudaMemcpyAsync(stg + o0, in + o0, o1 - o0, cudaMemcpyHostToDevice, c.st));
        SBP_TRY_CUDA(unpack_state(sys->d_blocks + c.b0, sys->d_inst, c.b1 - c.b0, poff + c.b0, sys->prec, dtype, sys->staging,
                                  sys->prev_hi, sys->prev_lo, sys->max_points, c.st));
        for (int64_t k = 0; k < nsteps; ++k) SBP_TRY_CUDA(cudaGraphLaunch(c.gexec, c.st));
        SBP_TRY_CUDA(pack_state(sys->d_blocks + c.b0, sys->d_inst, c.b1 - c.b0, poff + c.b0, sys->prec, dtype, sys->prev_hi,
                                sys->prev_lo, sys->staging, sys->max_points, c.st));
        SBP_TRY_CUDA(cudaMemcpyAsync(out + o0, stg + o0, o1 - o0, cudaMemcpyDeviceToHost, c.st));
        SBP_TRY_CUDA(cudaEventRecord(c.done, c.st));
    }
    for (Chunk& c : sys->chunks) SBP_TRY_CUDA(cudaStreamWaitEvent(st, c.done, 0));
    return check_status(sys);
}

int sbp_system_advance_host_chunks(sbp_system* sys) { return sys ? (int)sys->chunks.size() : -1; }

sbp_status sbp_system_set_dt(sbp_system* sys, int instance, double dt) {
    clear_error();
    if (!sys || instance >= sys->ninst) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    SBP_TRY(sync_times(sys));
    for (int i = 0; i < sys->ninst; ++i)
        if (instance < 0 || i == instance) set_dt_host(sys->hi[i], dt);
    SBP_TRY(upload_instances(sys));
    SBP_TRY_CUDA(cudaStreamSynchronize(sys->st()));
    return SBP_OK;
}

sbp_status sbp_system_set_time(sbp_system* sys, int instance, double t) {
    clear_error();
    if (!sys || instance >= sys->ninst) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    // written on the device, where the times are advanced: the host's copies are read back before every use
    SBP_TRY_CUDA(time_set(sys->d_inst, instance, sys->ninst, t, sys->st()));
    SBP_TRY_CUDA(cudaStreamSynchronize(sys->st()));
    return SBP_OK;
}

sbp_status sbp_system_get_time(sbp_system* sys, int instance, double* t) {
    clear_error();
    if (!sys || !t || instance < 0 || instance >= sys->ninst) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    SBP_TRY(sync_times(sys));
    *t = sys->hi[instance].time;
    return SBP_OK;
}

sbp_status sbp_system_max_dt(sbp_system* sys, int instance, double* dt) {
    clear_error();
    if (!sys || !dt || instance < 0 || instance >= sys->ninst) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    cudaStream_t st = sys->st();
    SBP_TRY_CUDA(cudaMemsetAsync(sys->d_speeds, 0, 2 * sys->nblocks * sizeof(unsigned long long), st));
    SBP_TRY_CUDA(max_speeds(sys->d_blocks, sys->d_inst, sys->nblocks, sys->prec, sys->prev_hi, sys->prev_lo, sys->met64, sys->max_points,
                            sys->d_speeds, st));
    std::vector<unsigned long long> sp(2 * sys->nblocks);
    SBP_TRY_CUDA(cudaMemcpyAsync(sp.data(), sys->d_speeds, sp.size() * sizeof(unsigned long long),
                                 cudaMemcpyDeviceToHost, st));
    SBP_TRY_CUDA(cudaStreamSynchronize(st));
    bool is_h2 = false;
    for (const auto& B : sys->hb) {
        if (B.instance != instance) continue;
        OpInfo ox, oy;
        op_info(B.op_xi, ox);
        op_info(B.op_eta, oy);
        is_h2 = is_h2 || ox.h2 || oy.h2;
    }
    const double c_max = is_h2 ? 0.5 : 1.0;
    double max_dt = INFINITY;
    for (int b = 0; b < sys->nblocks; ++b) {
        const BlockDev& B = sys->hb[b];
        if (B.instance != instance) continue;
        double mu, mv;
        std::memcpy(&mu, &sp[2 * b], 8);
        std::memcpy(&mv, &sp[2 * b + 1], 8);
        const double dx = 1.0 / double(B.nx), dy = 1.0 / double(B.ny);
        const double c_dt = std::fmax(mu / dx, mv / dy);
        max_dt = std::fmin(max_dt, c_max / c_dt);
    }
    *dt = max_dt;
    return SBP_OK;
}

sbp_status sbp_system_advance(sbp_system* sys, int64_t nsteps) {
    clear_error();
    if (!sys || nsteps < 0) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    for (int i = 0; i < sys->ninst; ++i)
        if (!(sys->hi[i].dt == sys->hi[i].dt)) {
            set_error("instance %d has no dt (call sbp_system_set_dt first)", i);
            return SBP_ERR_INVALID_ARGUMENT;
        }
    bool all = true;
    for (int a : sys->active) all = all && a;
    if (!all) {
        std::fill(sys->active.begin(), sys->active.end(), 1);
        sys->sched_dirty = true;
    }
    SBP_TRY(run_steps(sys, nsteps));
    return check_status(sys);
}

sbp_status sbp_system_advance_instances(sbp_system* sys, const int64_t* nsteps) {
    clear_error();
    if (!sys || !nsteps) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    std::vector<int64_t> left(nsteps, nsteps + sys->ninst);
    for (int i = 0; i < sys->ninst; ++i) {
        if (left[i] < 0) return SBP_ERR_INVALID_ARGUMENT;
        if (left[i] > 0 && !(sys->hi[i].dt == sys->hi[i].dt)) {
            set_error("instance %d has no dt", i);
            return SBP_ERR_INVALID_ARGUMENT;
        }
    }
    for (;;) {
        int64_t seg = INT64_MAX;
        std::vector<int> act(sys->ninst, 0);
        for (int i = 0; i < sys->ninst; ++i)
            if (left[i] > 0) {
                act[i] = 1;
                seg = std::min(seg, left[i]);
            }
        if (seg == INT64_MAX) break;
        if (act != sys->active) {
            sys->active = act;
            sys->sched_dirty = true;
        }
        SBP_TRY(run_steps(sys, seg));
        for (int i = 0; i < sys->ninst; ++i)
            if (act[i]) left[i] -= seg;
    }
    return check_status(sys);
}

sbp_status sbp_system_error(sbp_system* sys, double* per_instance) {
    clear_error();
    if (!sys || !per_instance) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    cudaStream_t st = sys->st();
    SBP_TRY_CUDA(error_terms(sys->d_blocks, sys->d_inst, sys->nblocks, sys->gamma, sys->xy, sys->prec, sys->prev_hi,
                             sys->prev_lo, sys->hw, sys->d_hoff, sys->max_points, sys->d_sums,
                             sys->d_sums + sys->nblocks, st));
    std::vector<double> sums(sys->nblocks);
    SBP_TRY_CUDA(cudaMemcpyAsync(sums.data(), sys->d_sums, sums.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
    SBP_TRY_CUDA(cudaStreamSynchronize(st));
    for (int i = 0; i < sys->ninst; ++i) per_instance[i] = 0.0;
    for (int b = 0; b < sys->nblocks; ++b) per_instance[sys->hb[b].instance] += std::sqrt(sums[b]);
    return SBP_OK;
}

sbp_status sbp_system_h2_err(sbp_system* sys, int block, const double* q, double* err) {
    clear_error();
    if (!sys || !q || !err || !valid_block(sys, block)) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    cudaStream_t st = sys->st();
    const BlockDev& B = sys->hb[block];
    const int64_t n = (int64_t)B.nx * B.ny;
    SBP_TRY_CUDA(cudaMemcpyAsync(sys->staging, q, 4 * n * sizeof(double), cudaMemcpyHostToDevice, st));
    const double* hx = sys->hw + sys->hoff[block];
    SBP_TRY_CUDA(diff_terms(sys->d_blocks + block, sys->d_inst, sys->prec, sys->prev_hi, sys->prev_lo,
                            static_cast<const double*>(sys->staging), hx, hx + B.nx, n, sys->d_sums,
                            sys->d_sums + 1, st));
    double s = 0;
    SBP_TRY_CUDA(cudaMemcpyAsync(&s, sys->d_sums, sizeof(double), cudaMemcpyDeviceToHost, st));
    SBP_TRY_CUDA(cudaStreamSynchronize(st));
    *err = std::sqrt(s);
    return SBP_OK;
}

sbp_status sbp_system_set_tiles(sbp_system* sys, int ty, int tx, int threads) {
    clear_error();
    if (!sys) return SBP_ERR_INVALID_ARGUMENT;
    const bool fused = (ty == 8 || ty == 16) && tx == tile_tx(ty) && threads == kStageThreads + sat_threads(ty);
    if (!fused && ((ty != 16 && ty != 32) || tx != kTileX || (threads != 0 && threads != kStageThreads))) {
        set_error("tiles are 16 or 32 rows x %d columns with %d threads, or those of the fused form", kTileX, kStageThreads);
        return SBP_ERR_INVALID_ARGUMENT;
    }
    if (fused && !fused_built(sys, ty)) {
        set_error("the fused form takes no expression sides and no operators of two families in a block");
        return SBP_ERR_INVALID_ARGUMENT;
    }
    sys->TY = ty;
    sys->fused = fused;
    sys->threads = kStageThreads;
    sys->tile_choice.clear();
    sys->tiles_auto = false;
    ++sys->tiles_gen;
    sys->sched_dirty = true;
    return SBP_OK;
}

sbp_status sbp_system_autotune(sbp_system* sys, int* ty, int* tx, int* threads) {
    clear_error();
    if (!sys) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    for (int i = 0; i < sys->ninst; ++i)
        if (!(sys->hi[i].dt == sys->hi[i].dt)) {
            set_error("instance %d has no dt", i);
            return SBP_ERR_INVALID_ARGUMENT;
        }
    std::fill(sys->active.begin(), sys->active.end(), 1);
    const size_t ts = sys->tsize();
    // save state and times; the copies and events are released on every return path
    struct Saved {
        void* hi = nullptr;
        void* lo = nullptr;
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        ~Saved() {
            if (hi) cudaFree(hi);
            if (lo) cudaFree(lo);
            if (e0) cudaEventDestroy(e0);
            if (e1) cudaEventDestroy(e1);
        }
    } saved;
    SBP_TRY_CUDA(cudaMalloc(&saved.hi, sys->nq * ts));
    if (sys->prev_lo) SBP_TRY_CUDA(cudaMalloc(&saved.lo, sys->nq * ts));
    SBP_TRY_CUDA(cudaEventCreate(&saved.e0));
    SBP_TRY_CUDA(cudaEventCreate(&saved.e1));
    cudaStream_t st = sys->st();
    SBP_TRY(sync_times(sys));
    std::vector<InstanceDev> save_inst = sys->hi;
    SBP_TRY_CUDA(cudaMemcpyAsync(saved.hi, sys->prev_hi, sys->nq * ts, cudaMemcpyDeviceToDevice, st));
    if (saved.lo) SBP_TRY_CUDA(cudaMemcpyAsync(saved.lo, sys->prev_lo, sys->nq * ts, cudaMemcpyDeviceToDevice, st));

    // One RK4 step of the whole schedule (every group, the groups running concurrently as in
    // production), median of a few replays after a warm-up replay; infinite if it cannot run.
    auto time_step = [&]() -> float {
        ++sys->tiles_gen;
        sys->sched_dirty = true;
        if (build_schedule(sys) != SBP_OK || run_steps(sys, 1) != SBP_OK) {
            clear_error();
            return 1e30f;
        }
        std::vector<float> t;
        for (int r = 0; r < 5; ++r) {
            cudaEventRecord(saved.e0, st);
            if (run_steps(sys, 1) != SBP_OK) {
                clear_error();
                return 1e30f;
            }
            cudaEventRecord(saved.e1, st);
            cudaEventSynchronize(saved.e1);
            float ms = 0;
            cudaEventElapsedTime(&ms, saved.e0, saved.e1);
            t.push_back(ms);
        }
        std::sort(t.begin(), t.end());
        return t[t.size() / 2];
    };
    // the operator groups of the schedule
    SBP_TRY(build_schedule(sys));
    std::vector<TileChoice> choice;
    for (const Group& g : sys->groups) choice.push_back(TileChoice{g.opx, g.opy, g.upw, g.ty, g.ctas, g.fused});
    // Candidates per group: tile rows {16, 32} x grid {as many CTAs per SM as fit, one per SM,
    // one CTA per tile}, from the current schedule (a small system's fused form is left only for
    // one that is faster); coordinate descent over the groups (each group's choice timed with the
    // others at their current choice), two sweeps.
    static const int kCand[][2] = {{16, -1}, {32, -1}, {16, 1}, {32, 1}, {16, 0}, {32, 0}};
    sys->tile_choice = choice;
    float best = time_step();
    for (int sweep = 0; sweep < 2; ++sweep) {
        bool changed = false;
        for (size_t gi = 0; gi < choice.size(); ++gi) {
            for (const auto& c : kCand) {
                if (!choice[gi].fused && choice[gi].ty == c[0] && choice[gi].ctas == c[1]) continue;
                std::vector<TileChoice> trial = choice;
                trial[gi].ty = c[0];
                trial[gi].ctas = c[1];
                trial[gi].fused = false;
                sys->tile_choice = trial;
                const float ms = time_step();
                if (ms < 0.99f * best) {  // keep a change only for a clear gain
                    best = ms;
                    choice = trial;
                    changed = true;
                }
            }
        }
        if (!changed) break;
    }
    sys->tile_choice = choice;
    ++sys->tiles_gen;
    sys->sched_dirty = true;
    // restore
    SBP_TRY_CUDA(cudaMemcpyAsync(sys->prev_hi, saved.hi, sys->nq * ts, cudaMemcpyDeviceToDevice, st));
    if (saved.lo) SBP_TRY_CUDA(cudaMemcpyAsync(sys->prev_lo, saved.lo, sys->nq * ts, cudaMemcpyDeviceToDevice, st));
    sys->hi = save_inst;
    SBP_TRY(upload_instances(sys));
    SBP_TRY_CUDA(cudaMemsetAsync(sys->status, 0, sizeof(unsigned), st));
    SBP_TRY_CUDA(cudaStreamSynchronize(st));
    clear_error();
    if (!(best < 1e29f)) {
        set_error("no tile candidate could run");
        return SBP_ERR_CUDA;
    }
    // the tiles of the group with the most points
    SBP_TRY(build_schedule(sys));
    const Group* big = &sys->groups[0];
    for (const Group& g : sys->groups)
        if (g.points > big->points) big = &g;
    if (ty) *ty = big->ty;
    if (tx) *tx = tile_tx(big->ty);
    if (threads) *threads = sys->threads + (big->fused ? sat_threads(big->ty) : 0);
    return SBP_OK;
}

int sbp_system_group_fused(sbp_system* sys, int group) {
    clear_error();
    if (!sys) return -1;
    cudaSetDevice(sys->device);
    if (sys->sched_dirty && build_schedule(sys) != SBP_OK) return -1;
    if (group < 0 || group >= (int)sys->groups.size()) return -1;
    return sys->groups[group].fused;
}

sbp_status sbp_system_group_tiles(sbp_system* sys, int group, int* ty, int* ctas_per_sm, int* grid) {
    clear_error();
    if (!sys) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    if (sys->sched_dirty) SBP_TRY(build_schedule(sys));
    if (group < 0 || group >= (int)sys->groups.size()) return SBP_ERR_INVALID_ARGUMENT;
    const Group& g = sys->groups[group];
    if (ty) *ty = g.ty;
    if (ctas_per_sm) *ctas_per_sm = g.ctas;
    if (grid) *grid = g.grid;
    return SBP_OK;
}

sbp_status sbp_system_set_stream(sbp_system* sys, void* stream) {
    clear_error();
    if (!sys) return SBP_ERR_INVALID_ARGUMENT;
    sys->user_stream = static_cast<cudaStream_t>(stream);
    sys->has_user_stream = stream != nullptr;
    return SBP_OK;
}

sbp_status sbp_system_device_state(sbp_system* sys, int block, void** d_q) {
    clear_error();
    if (!sys || !d_q || !valid_block(sys, block)) return SBP_ERR_INVALID_ARGUMENT;
    *d_q = static_cast<char*>(sys->prev_hi) + sys->hb[block].q_off * sys->tsize();
    return SBP_OK;
}

sbp_status sbp_system_advance_tableau(sbp_system* sys, int tableau, int64_t nsteps) {
    clear_error();
    const Tableau* T = tableau_of(tableau);
    if (!sys || !T || nsteps < 0) {
        set_error("bad system, tableau %d or step count", tableau);
        return SBP_ERR_INVALID_ARGUMENT;
    }
    if (sys->prec != 0) {
        set_error("tableaus other than the fused RK4 run on f64 systems only");
        return SBP_ERR_UNSUPPORTED;
    }
    cudaSetDevice(sys->device);
    for (size_t i = 0; i < sys->active.size(); ++i)
        if (!sys->active[i]) {
            sys->active[i] = 1;
            sys->sched_dirty = true;  // every instance takes part in the tableau steps
        }
    if (sys->sched_dirty) SBP_TRY(build_schedule(sys));
    SBP_TRY(ensure_kbuf(sys, T->s));
    for (int64_t n = 0; n < nsteps; ++n) {
        SBP_TRY(integrate_tableau(sys, *T, -1.0, nullptr, nullptr));
        SBP_TRY_CUDA(time_update(sys->d_inst, sys->d_active, sys->ninst, sys->st()));
    }
    return check_status(sys);
}

sbp_status sbp_system_advance_adaptive(sbp_system* sys, double dt, double* guess_dt, double maxerr) {
    clear_error();
    if (!sys || !guess_dt || !(*guess_dt > 0.0) || !(dt >= 0.0)) {
        set_error("bad system, dt or guess_dt");
        return SBP_ERR_INVALID_ARGUMENT;
    }
    if (sys->prec != 0 || sys->nblocks != 1) {
        set_error("advance_adaptive runs on single-block f64 systems (euler::System)");
        return SBP_ERR_UNSUPPORTED;
    }
    for (int d = 0; d < 4; ++d)
        if (sys->hb[0].bc_kind[d] != BC_THIS) {
            set_error("advance_adaptive uses the own opposite edges on every side (This), as the reference");
            return SBP_ERR_UNSUPPORTED;
        }
    cudaSetDevice(sys->device);
    if (sys->sched_dirty) SBP_TRY(build_schedule(sys));
    const Tableau& T = *tableau_of(6);  // BogackiShampine
    SBP_TRY(ensure_kbuf(sys, T.s));
    cudaStream_t st = sys->st();
    const BlockDev& B = sys->hb[0];
    const int64_t n = (int64_t)B.nx * B.ny;
    const double* hx = sys->hw + sys->hoff[0];
    double* fut = static_cast<double*>(sys->uB);
    double* fut2 = static_cast<double*>(sys->acc_hi);
    double time = 0.0, guess = *guess_dt;
    // euler::System::advance_adaptive (euler/src/lib.rs:149-186) as written: integrate advances
    // `time` by the step, an accepted step adds the step once more; the error compared against
    // maxerr is h2_err(prev, fut2).
    for (int64_t iter = 0; time < dt; ++iter) {
        if (iter > 100000000) {
            set_error("advance_adaptive: no progress after %lld attempts", (long long)iter);
            return SBP_ERR_NONPHYSICAL;
        }
        SBP_TRY(integrate_tableau(sys, T, guess, fut, fut2));
        time += guess;
        SBP_TRY_CUDA(pack_state(sys->d_blocks, sys->d_inst, 1, sys->d_poff4, 0, 0, fut2, nullptr, sys->staging, sys->max_points, st));
        SBP_TRY_CUDA(diff_terms(sys->d_blocks, sys->d_inst, 0, sys->prev_hi, nullptr, static_cast<const double*>(sys->staging), hx,
                                hx + B.nx, n, sys->d_sums, sys->d_sums + 1, st));
        double e2 = 0.0;
        SBP_TRY_CUDA(cudaMemcpyAsync(&e2, sys->d_sums, sizeof(double), cudaMemcpyDeviceToHost, st));
        SBP_TRY_CUDA(cudaStreamSynchronize(st));
        const double err = std::sqrt(e2);
        if (err < maxerr) {
            time += guess;
            SBP_TRY_CUDA(cudaMemcpyAsync(sys->prev_hi, fut, sys->nq * sizeof(double), cudaMemcpyDeviceToDevice, st));
            guess *= 1.05;
        } else {
            guess *= 0.8;
        }
    }
    *guess_dt = guess;
    return check_status(sys);
}

int sbp_system_group_count(sbp_system* sys) {
    clear_error();
    if (!sys) return -1;
    cudaSetDevice(sys->device);
    if (sys->sched_dirty && build_schedule(sys) != SBP_OK) return -1;
    return (int)sys->groups.size();
}

sbp_status sbp_system_group_info(sbp_system* sys, int group, int* op_xi, int* op_eta, int64_t* points) {
    clear_error();
    if (!sys) return SBP_ERR_INVALID_ARGUMENT;
    cudaSetDevice(sys->device);
    SBP_TRY(check_eval(sys));
    if (sys->sched_dirty) SBP_TRY(build_schedule(sys));
    if (group < 0 || group >= (int)sys->groups.size()) {
        set_error("group %d out of range (%d groups)", group, (int)sys->groups.size());
        return SBP_ERR_INVALID_ARGUMENT;
    }
    const Group& g = sys->groups[group];
    if (op_xi) *op_xi = g.opx;
    if (op_eta) *op_eta = g.opy;
    if (points) *points = g.points;
    return SBP_OK;
}

sbp_status sbp_system_launch_stage(sbp_system* sys, int group, int stage, int with_edges) {
    clear_error();
    if (!sys || stage < 0 || stage > 3) {
        set_error("bad system or stage %d", stage);
        return SBP_ERR_INVALID_ARGUMENT;
    }
    cudaSetDevice(sys->device);
    SBP_TRY(check_eval(sys));
    if (sys->sched_dirty) SBP_TRY(build_schedule(sys));
    if (group < 0 || group >= (int)sys->groups.size()) {
        set_error("group %d out of range (%d groups)", group, (int)sys->groups.size());
        return SBP_ERR_INVALID_ARGUMENT;
    }
    return launch_group(sys, stage, sys->groups[group], sys->st(), with_edges != 0);
}

int sbp_system_launches_per_step(const sbp_system* sys) {
    if (!sys) return -1;
    if (sys->sched_dirty) {
        // count the operator pairs present without building
        std::vector<std::pair<int, int>> pairs;
        for (const auto& B : sys->hb) {
            if (!sys->active[B.instance]) continue;
            auto p = std::make_pair(B.op_xi, B.op_eta);
            if (std::find(pairs.begin(), pairs.end(), p) == pairs.end()) pairs.push_back(p);
        }
        return fused_rows(sys) ? 4 * (int)pairs.size() : (sys->has_eval ? 12 : 8) * (int)pairs.size() + 1;
    }
    int n = 0;
    bool all_fused = !sys->groups.empty();
    for (const Group& g : sys->groups) {
        n += g.fused ? 4 : (sys->has_eval ? 12 : 8);
        all_fused = all_fused && g.fused;
    }
    return n + (all_fused ? 0 : 1);
}

}  // extern "C"
