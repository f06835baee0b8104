// pd_solver.cu -- solver sequencing of src/solvers/*.jl on the device:
// update_acc!, velocity_verlet_step!, minimize! (QSDrag), apply_bc_at0,
// and the block-level device-pointer entry point.  Compiled with
// -fmad=false (the QSDrag update below must round like the reference).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "pd_env_impl.h"
#include "pd_launch.h"

using namespace pd;

void pd_env::release_device() {
    fast_release(this);
    map.reset();
    x4.reset();
    y.reset();
    v.reset();
    f.reset();
    p.reset();
    mass.reset();
    dens.reset();
    tdens.reset();
    tinfo.reset();
    cnt.reset();
    intact0.reset();
    deformed.reset();
    sinfo.reset();
    fam.reset();
    nbr.reset();
    words[0].reset();
    words[1].reset();
    words0.reset();
    mth.reset();
    blocks_d.reset();
    pairs.reset();
    partials.reset();
    out3.reset();
    stage.reset();
    flag.reset();
    bcs.clear();
    contacts.clear();
    tmp_y.reset();
    scr_d.reset();
    scr_i.reset();
    splan_off.reset();
    splan.reset();
    spos.reset();
    tmp_f.reset();
    opt.reset();
    free_mask.reset();
    red.reset();
}

namespace {

pd_status need_final(const pd_env *env) {
    if (!env) return fail(PD_ERR_ARG, "environment handle is NULL");
    if (!env->finalized) return fail(PD_ERR_STATE, "environment is not finalized (call pd_env_finalize)");
    return PD_OK;
}

pd::BCDev bc_view(pd_env *env, size_t k) {
    const HostBC &h = env->hbc[k];
    DevBC &d = env->bcs[k];
    BCDev b;
    b.kind = h.kind;
    b.dims = h.dims;
    for (int i = 0; i < 3; ++i) b.rate[i] = h.rate[i];
    for (int i = 0; i < 3; ++i) {
        b.scale[i] = h.scale[i];
        b.fix[i] = h.fix[i];
        b.lo[i] = h.lo[i];
        b.hi[i] = h.hi[i];
    }
    b.has_limits = h.has_limits;
    b.pad = 0;
    b.n = d.n;
    b.idx = d.idx.p;
    b.last = d.last.p;
    b.sn = d.sn;
    b.sidx = d.sidx.p;
    return b;
}

// ToFroBC.jl:101-105 check!: flip when time_step > applyafter and
// time_step % freq == 0 (Int % Float64 is rem).
// ScaleFixWaitBC.jl:63-68 check!: at time_step % wait == 0 scale the
// scalebool particles about the fix point and re-read last.
void bc_check(pd_env *env) {
    for (size_t k = 0; k < env->hbc.size(); ++k) {
        auto &h = env->hbc[k];
        if (h.scales_at(env->ts)) launch_bc_scale(env->st, bc_view(env, k), env->dt, env->y.p);
        if (h.kind != PD_BC_TOFRO) continue;
        double r = std::fmod((double)env->ts, h.freq);
        if ((env->ts > h.applyafter) && (r == 0.0)) h.dir = -h.dir;
    }
}

__device__ __forceinline__ double jl_min(double x, double y) {
    if (x != x || y != y) return x + y;  // NaN propagates
    if (x < y) return x;
    if (y < x) return y;
    return signbit(x) ? x : y;
}
__device__ __forceinline__ double jl_max(double x, double y) {
    if (x != x || y != y) return x + y;
    if (x > y) return x;
    if (y > x) return y;
    return signbit(x) ? y : x;
}

__device__ __forceinline__ double nanmax(double a, double b) {
    if (a != a || b != b) return __longlong_as_double(0x7ff8000000000000LL);
    return a > b ? a : b;
}

// Fixed partial-reduction width, independent of the device's SM count so
// that the reduction order is the same on every GPU.
constexpr int kRedBlocks = 148;
// Largest number of CTAs sharing one block in the gate's partial norms
// (fixed for the same reason).
constexpr int kGateWidth = 148;

// Progress of a quasi-static minimisation on the device.
struct QsState {
    double h[2];      // max|f|, max|dy| of the last iteration
    int64_t iters;    // iterations applied
    int32_t done;     // both below their tolerances: later iterations do nothing
    uint32_t arrived;
};

// minimize.jl:149-155 apply_! and :202 y[:, mask] .+= dy, fused with the
// max|f| / max|dy| reductions of :204 and the convergence test: the last
// block to arrive combines the blocks' maxima (exact in any order).
__global__ void __launch_bounds__(256)
    k_qs_apply(int64_t N, const int32_t *freem, const double4 *f, double4 *opt, double4 *y, double lambda, double kk,
               double ss, double a, double f_tol, double x_tol, double *partial, QsState *qs) {
    __shared__ double sf[8], sy[8];
    __shared__ bool last;
    pdl_enter();
    if (*(volatile int32_t *)&qs->done) return;
    double mf = 0.0, my = 0.0;
    for (int64_t i = blockIdx.x * 256 + threadIdx.x; i < N; i += (int64_t)kRedBlocks * 256) {
        if (!freem[i]) continue;
        double4 fi = f[i], oi = opt[i], yi = y[i];
        double fo[3] = {fi.x, fi.y, fi.z}, o[3] = {oi.x, oi.y, oi.z}, yy[3] = {yi.x, yi.y, yi.z};
        for (int d = 0; d < 3; ++d) {
            double force = fo[d] - lambda * o[d] * (1.0 + kk * fabs(o[d]));
            double dy = 0.5 * force * (ss * ss) + o[d] * ss;
            o[d] = o[d] + ss * force;
            dy = jl_max(jl_min(dy, a), -a);
            yy[d] = yy[d] + dy;
            mf = nanmax(mf, fabs(fo[d]));
            my = nanmax(my, fabs(dy));
        }
        opt[i] = make_double4(o[0], o[1], o[2], 0.0);
        y[i] = make_double4(yy[0], yy[1], yy[2], yi.w);
    }
    // the block's maxima in sf[0], sy[0]: within the warps, then over them
    auto reduce = [&](double vf, double vy) {
        for (int o = 16; o; o >>= 1) {
            vf = nanmax(vf, __shfl_xor_sync(0xffffffffu, vf, o));
            vy = nanmax(vy, __shfl_xor_sync(0xffffffffu, vy, o));
        }
        const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
        if (lane == 0) {
            sf[wid] = vf;
            sy[wid] = vy;
        }
        __syncthreads();
        if (wid == 0) {
            vf = lane < 8 ? sf[lane] : 0.0;
            vy = lane < 8 ? sy[lane] : 0.0;
            for (int o = 4; o; o >>= 1) {
                vf = nanmax(vf, __shfl_xor_sync(0xffffffffu, vf, o));
                vy = nanmax(vy, __shfl_xor_sync(0xffffffffu, vy, o));
            }
            __syncwarp();
            if (lane == 0) {
                sf[0] = vf;
                sy[0] = vy;
            }
        }
        __syncthreads();
    };
    reduce(mf, my);
    if (threadIdx.x == 0) {
        partial[2 * blockIdx.x] = sf[0];
        partial[2 * blockIdx.x + 1] = sy[0];
        __threadfence();
        last = atomicAdd(&qs->arrived, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    const bool one = threadIdx.x < kRedBlocks;
    const volatile double *vp = partial;
    reduce(one ? vp[2 * threadIdx.x] : 0.0, one ? vp[2 * threadIdx.x + 1] : 0.0);
    if (threadIdx.x == 0) {
        qs->h[0] = sf[0];
        qs->h[1] = sy[0];
        qs->iters += 1;
        qs->arrived = 0;
        if (sf[0] < f_tol && sy[0] < x_tol) qs->done = 1;
    }
}

__global__ void k_set_free(int64_t N, const int32_t *__restrict__ tinfo, int32_t *__restrict__ freem) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= N) return;
    freem[i] = tinfo[i] >= 0 ? 1 : 0;
}

__global__ void k_clear_idx(int64_t n, const int32_t *__restrict__ idx, int32_t *__restrict__ freem) {
    int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= n) return;
    freem[idx[j]] = 0;
}

}  // namespace

namespace pd {

// How a block of an evaluation over S slices in all is evaluated.  A block of warps per slice
// evaluates every bond once and side by side, but an SM holds two or three of
// them, each some 4.5 us long however few its slots; a thread per particle
// evaluates every bond at both visits, one after another.  Short slot lists
// on many slices are therefore left to threads.  Steps of strained
// bond-based cubes in us, threads / slices:
//   slots         6          18           26           32          120
//     250 slices  15 / 11    28 / 12      37 / 13      42 / 13     132 / 23
//     686         17 / 18    30 / 22      40 / 23      44 / 23     147 / 47
//   1,229         20 / 25    32 / 31      41 / 34      48 / 34     153 / 71
//   2,000         21 / 37    38 / 45      50 / 48      59 / 49     198 / 108
//   8,192         52 / 117   109 / 148    149 / 161    179 / 163   641 / 394
//  65,536         364 / 1054 807 / 1290   1100 / 1390  1331 / 1395 4741 / 3231
// The dilatation evaluates a bond once in either form, so that threads win
// from some 3,500 slices on however long the lists (state-based steps, the
// force by slices where that is faster, dilatation by threads / slices:
// 32 slots 2,000 slices 76 / 74, 8,192 228 / 257; 120 slots 2,000 192 / 174,
// 3,907 309 / 319, 65,536 4768 / 5313).  The elasto-plastic force, whose two
// visits differ, has the thread form only.
SerialRun serial_run(const HostBlock &b, int64_t S, bool theta) {
    const bool ep = b.kind == PD_MAT_ELASTO_PLASTIC;
    const int64_t line = 300 + 70 * (int64_t)b.mean_slots;  // slices from which on threads are faster
    const bool by_slice = theta ? S < std::min<int64_t>(line, 3500) : !ep && (b.mean_slots > 28 || S < line);
    return SerialRun{b.first_int, b.first_int + (b.n + kSlice - 1) / kSlice * kSlice, b.slots, by_slice, ep};
}

// Runs of the environment's blocks for the force or the dilatation.
std::vector<SerialRun> serial_runs(const pd_env *env, bool theta) {
    constexpr size_t kMaxRuns = 8;
    auto takes = [&](const HostBlock &b) {
        return b.n > 0 && (!theta || b.kind == PD_MAT_ORDINARY_STATE_BASED || b.kind == PD_MAT_ELASTO_PLASTIC);
    };
    int64_t S = 0, wide = 0;
    for (const auto &b : env->hb)
        if (takes(b)) S += (b.n + kSlice - 1) / kSlice;
    std::vector<SerialRun> runs;
    for (const auto &b : env->hb) {
        if (!takes(b)) continue;
        const SerialRun r = serial_run(b, S, theta);
        if (r.by_slice) wide += (r.p1 - r.p0) / kSlice;
        if (!runs.empty() && runs.back().p1 == r.p0 && runs.back().by_slice == r.by_slice) {
            runs.back().p1 = r.p1;
            runs.back().slots = std::max(runs.back().slots, r.slots);
            runs.back().ep |= r.ep;
        } else {
            runs.push_back(r);
        }
    }
    if (runs.size() <= kMaxRuns) return runs;
    // many alternating blocks: one launch over all of them (the kernels leave
    // what they do not evaluate), in the form that suits more slices
    SerialRun all{runs.front().p0, runs.back().p1, 0, 2 * wide >= S, false};
    for (const auto &r : runs) {
        all.slots = std::max(all.slots, r.slots);
        all.ep |= r.ep;
    }
    return {all};
}

// update_acc! (solvers.jl:320-336) in serial-order FP64.
pd_status update_acc_serial(pd_env *env, bool momentum, const int32_t *stop) {
    cudaStream_t st = env->st;
    Geo g = env->geo();
    g.stop = stop;
    // force_density! gate for blocks still undeformed
    std::vector<GateItem> items;
    for (size_t b = 0; b < env->hb.size() && !env->gate_hold; ++b) {
        const HostBlock &hb = env->hb[b];
        if (hb.kind == PD_MAT_SKIP || env->deformed_h[b]) continue;
        items.push_back(GateItem{hb.first_int, hb.n, (int32_t)b, 0});
    }
    if (!items.empty()) {
        const int ni = (int)items.size();
        const int gx = std::max(1, std::min(kGateWidth, (kGateWidth * 8) / ni));
        if (env->gate_items_h.size() != items.size() ||
            std::memcmp(env->gate_items_h.data(), items.data(), items.size() * sizeof(GateItem)) != 0) {
            PD_TRY(grow(env->gate_items, (int64_t)items.size()));
            PD_TRY(grow(env->gate_part, 3 * (int64_t)ni * gx));
            CK(cudaMemcpyAsync(env->gate_items.p, items.data(), items.size() * sizeof(GateItem),
                               cudaMemcpyHostToDevice, st));
            CK(cudaStreamSynchronize(st));
            env->gate_items_h = items;
        }
        launch_gate_multi(st, env->gate_items.p, ni, gx, env->x4.p, env->y.p, env->gate_part.p, env->deformed.p);
    }
    // out_of_loop!: dilatation for state-based blocks
    bool any_lps = false, any_ep = false;
    for (const auto &hb : env->hb) {
        any_lps |= hb.kind == PD_MAT_ORDINARY_STATE_BASED || hb.kind == PD_MAT_ELASTO_PLASTIC;
        any_ep |= hb.kind == PD_MAT_ELASTO_PLASTIC;
    }
    if (any_lps)
        launch_theta_serial(st, g, env->y.p, env->words[env->cur].p, env->mth.p, env->theta_runs.data(),
                            env->theta_runs.size());
    bool idle = false;
    for (size_t b = 0; b < env->hb.size(); ++b) idle |= env->hb[b].kind != PD_MAT_SKIP && !env->deformed_h[b];
    const SerialRun *runs = env->force_runs.data();
    const size_t n_runs = env->force_runs.size();
    if (any_ep) {
        // elasto_plastic.jl:170-171: td_norm2 pass (breaks bonds), then the
        // bond loop on its flags, back into words[cur]; edp is double-buffered
        launch_td_serial(st, g, env->y.p, env->mth.p, env->words[env->cur].p, env->words[1 - env->cur].p, 0,
                         env->N);
        prof_begin(env, st);
        launch_force_serial(st, g, env->y.p, env->mth.p, env->words[1 - env->cur].p, env->words[env->cur].p,
                            env->f.p, 0, runs, n_runs, idle);
        prof_end(env, st);
        env->ecur = 1 - env->ecur;
    } else {
        // fill!(f, 0) + force_density_T! for every block
        prof_begin(env, st);
        launch_force_serial(st, g, env->y.p, env->mth.p, env->words[env->cur].p, env->words[1 - env->cur].p,
                            env->f.p, 0, runs, n_runs, idle);
        prof_end(env, st);
        env->cur = 1 - env->cur;
    }
    CK(cudaGetLastError());
    // short_range_contact!
    PD_TRY(contacts_force(env));
    // update_misc!
    if (momentum) launch_momentum(st, env->N, env->mass.p, env->v.p, env->p.p);
    CK(cudaGetLastError());
    return PD_OK;
}

pd_status refresh_deformed(pd_env *env) {
    bool all = true;
    for (size_t b = 0; b < env->hb.size(); ++b)
        if (env->hb[b].kind != PD_MAT_SKIP && !env->deformed_h[b]) all = false;
    if (all) return PD_OK;
    std::vector<int32_t> h(env->hb.size());
    CK(cudaMemcpyAsync(h.data(), env->deformed.p, h.size() * 4, cudaMemcpyDeviceToHost, env->st));
    CK(cudaStreamSynchronize(env->st));
    for (size_t b = 0; b < h.size(); ++b) env->deformed_h[b] = h[b];
    return PD_OK;
}

}  // namespace pd

extern "C" pd_status pd_env_update_acc(pd_env *env) {
    PD_TRY(need_final(env));
    CK(cudaSetDevice(env->device));
    if (env->precision != PD_PREC_FP64_SERIAL) return fast_update_acc(env);
    PD_TRY(sync_state_to_fp64(env));
    PD_TRY(update_acc_serial(env));
    PD_TRY(refresh_deformed(env));
    CK(cudaStreamSynchronize(env->st));
    return PD_OK;
}

extern "C" pd_status pd_env_apply_bc_at0(pd_env *env) {
    PD_TRY(need_final(env));
    CK(cudaSetDevice(env->device));
    PD_TRY(sync_state_to_fp64(env, false));
    for (size_t k = 0; k < env->hbc.size(); ++k)
        if (env->hbc[k].kind != PD_BC_CONTAINER)  // ContainerBC.jl:84 does nothing
            launch_bc_snapshot(env->st, bc_view(env, k), env->y.p);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(env->st));
    return PD_OK;
}

// The fused integration's view of the conditions: the directions of the
// velocity conditions as they are now, of the position conditions filled in
// by the caller.
static FusedBCs fused_bcs(pd_env *env) {
    FusedBCs b;
    std::memset(&b, 0, sizeof(b));
    b.n = (int32_t)env->hbc.size();
    b.bits = env->bc_bits.p;
    for (size_t k = 0; k < env->hbc.size(); ++k) {
        b.c[k].bc = bc_view(env, k);
        b.c[k].lo = env->bc_rank_lo[k];
        b.c[k].rank = env->bc_rank.p + env->bc_rank_off[k];
        b.c[k].dir_vel = b.c[k].dir_pos = env->hbc[k].dir;
    }
    return b;
}

// velocity_verlet.jl:57-89, nsteps times, in the serial mode, enqueued on
// the environment's stream.  With at most kMaxFusedBC conditions the second
// half of a step and the first half of the next run as one kernel.
static pd_status serial_steps(pd_env *env, int64_t nsteps) {
    const double c = env->dt / 2;
    const double dt = env->dt;
    const bool fused = env->hbc.size() <= (size_t)kMaxFusedBC;
    FusedBCs b;
    auto advance = [&](bool post, bool pre, double4 *p) {
        launch_advance(env->st, env->N, c, dt, post, pre, env->f.p, env->v.p, env->y.p, env->mass.p, p, b, env->ts);
    };
    if (fused && nsteps > 0) {
        b = fused_bcs(env);
        advance(false, true, nullptr);
    }
    for (int64_t s = 0; s < nsteps; ++s) {
        const bool last = s == nsteps - 1;
        if (!fused) {
            launch_kick_drift(env->st, env->N, c, dt, env->f.p, env->v.p, env->y.p);
            for (size_t k = 0; k < env->hbc.size(); ++k)
                launch_bc_pos(env->st, bc_view(env, k), dt, env->hbc[k].dir, env->ts, env->y.p);
        }
        PD_TRY(update_acc_serial(env, !fused));
        if (fused) {
            bool scales = false;  // ScaleFixWait's check! moves particles between the two halves
            for (const auto &h : env->hbc) scales |= h.scales_at(env->ts);
            b = fused_bcs(env);
            if (last || scales) advance(true, false, last ? env->p.p : nullptr);
            bc_check(env);
            env->ts += 1;
            for (size_t k = 0; k < env->hbc.size(); ++k) b.c[k].dir_pos = env->hbc[k].dir;
            if (!last) advance(!scales, true, nullptr);
        } else {
            launch_kick(env->st, env->N, c, env->f.p, env->v.p);
            for (size_t k = 0; k < env->hbc.size(); ++k)
                launch_bc_vel(env->st, bc_view(env, k), env->hbc[k].dir, env->y.p, env->v.p);
            bc_check(env);
            env->ts += 1;
        }
        if ((s & 63) == 63) CK(cudaGetLastError());
    }
    CK(cudaGetLastError());
    return PD_OK;
}

extern "C" pd_status pd_env_vv_steps(pd_env *env, int64_t nsteps) {
    PD_TRY(need_final(env));
    if (nsteps < 0) return fail(PD_ERR_ARG, "nsteps < 0");
    CK(cudaSetDevice(env->device));
    if (env->precision != PD_PREC_FP64_SERIAL) return fast_vv_steps(env, nsteps);
    PD_TRY(serial_steps(env, nsteps));
    PD_TRY(refresh_deformed(env));
    CK(cudaStreamSynchronize(env->st));
    return PD_OK;
}

// pd_env_vv_steps without the final wait: the steps are enqueued on the
// environment's stream.  Only an environment whose deformed flags the host
// already knows (every block deformed, or the gate held) can skip the
// read-back; others wait as pd_env_vv_steps does.
extern "C" pd_status pd_env_vv_steps_async(pd_env *env, int64_t nsteps) {
    PD_TRY(need_final(env));
    if (nsteps < 0) return fail(PD_ERR_ARG, "nsteps < 0");
    bool known = env->gate_hold;
    if (!known) {
        known = true;
        for (size_t b = 0; b < env->hb.size(); ++b)
            if (env->hb[b].kind != PD_MAT_SKIP && !env->deformed_h[b]) known = false;
    }
    if (!known) return pd_env_vv_steps(env, nsteps);
    CK(cudaSetDevice(env->device));
    if (env->precision != PD_PREC_FP64_SERIAL) return fast_vv_enqueue(env, nsteps);
    return serial_steps(env, nsteps);
}

// minimize.jl:105-231 (one QSDrag solver step).
extern "C" pd_status pd_env_qsdrag(pd_env *env, double step_size, double drag, int64_t max_iter,
                                   double x_tol, double f_tol, int64_t *iters) {
    PD_TRY(need_final(env));
    if (max_iter < 1) return fail(PD_ERR_ARG, "max_iter must be >= 1");
    CK(cudaSetDevice(env->device));
    PD_TRY(sync_state_to_fp64(env));
    cudaStream_t st = env->st;
    const int64_t N = env->N;
    // :112-115 apply BCs (position then velocity, per BC)
    for (size_t k = 0; k < env->hbc.size(); ++k) {
        launch_bc_pos(st, bc_view(env, k), env->dt, env->hbc[k].dir, env->ts, env->y.p);
        launch_bc_vel(st, bc_view(env, k), env->hbc[k].dir, env->y.p, env->v.p);
    }
    const double dt = step_size;
    const double ps = env->hb[0].particle_size;
    // :138-145 free particles: not in any BC that acts beyond the start
    if (!env->free_mask.p) PD_TRY(env->free_mask.alloc(N));
    if (!env->opt.p) PD_TRY(env->opt.alloc(N));
    if (!env->red.p) PD_TRY(env->red.alloc(2 * kRedBlocks));
    if (!env->qs_state.p) PD_TRY(env->qs_state.alloc((sizeof(QsState) + 3) / 4));
    k_set_free<<<(unsigned)((N + 255) / 256), 256, 0, st>>>(N, env->tinfo.p, env->free_mask.p); pd::note_launch();
    for (size_t k = 0; k < env->hbc.size(); ++k)
        if (!env->hbc[k].onlyatstart && env->bcs[k].n > 0)
            k_clear_idx<<<(unsigned)((env->bcs[k].n + 255) / 256), 256, 0, st>>>(env->bcs[k].n, env->bcs[k].idx.p,
                                                                                  env->free_mask.p); pd::note_launch();
    // :146 opt = zero(f[:, mask]); :147 k = lambda/10
    CK(cudaMemsetAsync(env->opt.p, 0, N * sizeof(double4), st));
    const double lambda = drag;
    const double kk = lambda / 10;
    const double a = ps / 10;
    // Iterations are enqueued in batches of up to kQsBatch between two reads
    // of the progress; an iteration after the converged one finds the done
    // flag and changes nothing (a read-back per iteration cost 10 us of 70 on
    // a 9,500-particle bar).  While a block is undeformed, or with contacts,
    // whose kernels do not look at the flag, every iteration is read; the
    // gate flags of undeformed blocks come with the same wait (one of their
    // own cost 4 % of an iteration with contacts, 30 us of a single one).
    constexpr int64_t kQsBatch = 16;
    QsState *qs = (QsState *)env->qs_state.p;
    CK(cudaMemsetAsync(qs, 0, sizeof(QsState), st));
    QsState h{};
    bool ep = false;
    for (const auto &b : env->hb) ep |= b.kind == PD_MAT_ELASTO_PLASTIC;
    std::vector<int32_t> flags(env->hb.size());
    for (int64_t batch = 2; h.iters < max_iter && !h.done; batch = std::min(2 * batch, kQsBatch)) {
        bool gated = false;
        for (size_t b = 0; b < env->hb.size() && !env->gate_hold; ++b)
            gated |= env->hb[b].kind != PD_MAT_SKIP && !env->deformed_h[b];
        const bool known = !gated && env->hc.empty() && !env->prof;  // (profiling counts the iterations that run)
        const int64_t m = known ? std::min(batch, max_iter - h.iters) : 1;
        const int64_t it0 = h.iters;
        const int cur0 = env->cur, ecur0 = env->ecur;
        for (int64_t i = 0; i < m; ++i) {
            PD_TRY(update_acc_serial(env, false, &qs->done));
            launch_dep(k_qs_apply, kRedBlocks, 256, st, (int64_t)N, (const int32_t *)env->free_mask.p,
                       (const double4 *)env->f.p, env->opt.p, env->y.p, lambda, kk, step_size, a, f_tol, x_tol,
                       env->red.p, qs);
            pd::note_launch();
        }
        CK(cudaGetLastError());
        if (gated)
            CK(cudaMemcpyAsync(flags.data(), env->deformed.p, flags.size() * 4, cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(&h, qs, sizeof(h), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        if (gated) std::copy(flags.begin(), flags.end(), env->deformed_h.begin());
        // the buffers as the iterations that ran left them
        const int odd = (int)((h.iters - it0) & 1);
        env->cur = ep ? cur0 : cur0 ^ odd;
        env->ecur = ep ? ecur0 ^ odd : ecur0;
    }
    const int64_t it = h.iters;
    launch_momentum(st, N, env->mass.p, env->v.p, env->p.p);
    (void)dt;
    bc_check(env);
    env->ts += 1;
    CK(cudaStreamSynchronize(st));
    if (iters) *iters = it;
    return PD_OK;
}

extern "C" pd_status pd_env_update_neighs(pd_env *env, int64_t max_part) {
    PD_TRY(need_final(env));
    CK(cudaSetDevice(env->device));
    PD_TRY(sync_state_to_fp64(env, false));
    PD_TRY(contacts_update_neighs(env, max_part));
    CK(cudaStreamSynchronize(env->st));
    return PD_OK;
}

// force_density_T!(f, y, limits, mat, Val{:cuda}) on caller-owned device
// arrays (3 x N_env column-major).
extern "C" pd_status pd_force_density_device(pd_env *env, int64_t block, double *f_dev,
                                             const double *y_dev, void *stream) {
    PD_TRY(need_final(env));
    if (block < 0 || block >= (int64_t)env->hb.size()) return fail(PD_ERR_ARG, "no block %lld", (long long)block);
    if (!f_dev || !y_dev) return fail(PD_ERR_ARG, "f/y device pointer is NULL");
    if (env->precision != PD_PREC_FP64_SERIAL)
        return fail(PD_ERR_UNSUPPORTED, "pd_force_density_device requires PD_PREC_FP64_SERIAL");
    CK(cudaSetDevice(env->device));
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, f_dev) != cudaSuccess || at.type != cudaMemoryTypeDevice ||
        at.device != env->device || cudaPointerGetAttributes(&at, y_dev) != cudaSuccess ||
        at.type != cudaMemoryTypeDevice || at.device != env->device) {
        cudaGetLastError();
        return fail(PD_ERR_ARG, "f/y must be device pointers on the environment's device %d", env->device);
    }
    cudaStream_t st = stream ? (cudaStream_t)stream : env->st;
    const HostBlock &hb = env->hb[block];
    if (hb.kind == PD_MAT_ELASTO_PLASTIC)
        return fail(PD_ERR_UNSUPPORTED, "the device-pointer entry point does not evaluate elasto-plastic blocks");
    if (!env->tmp_y.p) PD_TRY(env->tmp_y.alloc(env->N));
    if (!env->tmp_f.p) PD_TRY(env->tmp_f.alloc(env->N));
    const int64_t *map = env->map.p + hb.first_env;
    launch_unpack3(st, hb.n, y_dev + 3 * hb.first_env, map, env->tmp_y.p);
    launch_unpack3(st, hb.n, f_dev + 3 * hb.first_env, map, env->tmp_f.p);
    Geo g = env->geo();
    int64_t p0 = hb.first_int, p1 = hb.first_int + ((hb.n + 31) / 32) * 32;
    const SerialRun theta = serial_run(hb, (p1 - p0) / kSlice, true), force = serial_run(hb, (p1 - p0) / kSlice, false);
    if (hb.kind == PD_MAT_ORDINARY_STATE_BASED)
        launch_theta_serial(st, g, env->tmp_y.p, env->words[env->cur].p, env->mth.p, &theta, 1);
    // force_density_T! itself has no gate: compute unconditionally
    std::vector<int32_t> one(1, 1);
    CK(cudaMemcpyAsync(env->deformed.p + block, one.data(), 4, cudaMemcpyHostToDevice, st));
    launch_force_serial(st, g, env->tmp_y.p, env->mth.p, env->words[env->cur].p, env->words[1 - env->cur].p,
                        env->tmp_f.p, 1, &force, 1, false);
    int64_t w0 = env->sinfo_h[p0 / 32].word, w1 = env->sinfo_h[p1 / 32].word;
    if (w1 > w0)
        CK(cudaMemcpyAsync(env->words[env->cur].p + w0, env->words[1 - env->cur].p + w0, (w1 - w0) * 4,
                           cudaMemcpyDeviceToDevice, st));
    launch_pack3(st, hb.n, env->tmp_f.p, map, f_dev + 3 * hb.first_env);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(st));
    env->deformed_h[block] = 1;
    return PD_OK;
}
