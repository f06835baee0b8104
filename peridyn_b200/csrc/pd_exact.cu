// pd_exact.cu -- FP64 kernels whose results must be bit-identical to the
// reference's CPU path.  This translation unit is compiled with
// -fmad=false: every a*b+c below rounds twice, exactly like Julia's
// unfused Float64 arithmetic.  Division and sqrt on double are IEEE
// round-to-nearest in CUDA.
//
// Expression order follows the reference literally:
//   get_magnitude  sqrt(a1*a1 + a2*a2 + a3*a3)        const_macros.jl:116
//   get_ij         x[:, j] - x[:, i]                   const_macros.jl:153-155
//   stretch        (|Y| - |X|) / |X|                   general_material.jl:338-341
//   force          ((0.5*t/|Y|) * Y_d * V_j) / rho_i   general_material.jl:351-362
#include <atomic>
#include <climits>
#include <cstdio>

#include "pd_ieee.h"
#include "pd_internal.h"
#include "pd_launch.h"
#include "pd_slots.h"

namespace pd {

namespace {

constexpr int kThreads = 128;

inline unsigned grid_for(int64_t n, int threads = kThreads) {
    int64_t g = (n + threads - 1) / threads;
    return (unsigned)(g > 0 ? g : 1);
}

__device__ __forceinline__ double mag3(double a1, double a2, double a3) {
    return sqrt(a1 * a1 + a2 * a2 + a3 * a3);
}

// One 256-bit load of a particle's record.  The dependent kernels (pdl_enter)
// are resident while the previous kernel on the stream still writes y, f and
// mth.  They read those coherently (ld4) and behind the wait, take them
// without __restrict__, and keep ld.global.nc (ld4_nc, __ldg) to data that is
// complete since pd_env_finalize: x4, nbr.
__device__ __forceinline__ double4 ld4(const double4 *p) {
    double4 r;
    asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w) : "l"(p));
    return r;
}
__device__ __forceinline__ double4 ld4_nc(const double4 *p) {
    double4 r;
    asm("ld.global.nc.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w) : "l"(p));
    return r;
}

__device__ __forceinline__ int64_t sell_base(const int64_t *slice_ptr, int64_t p) {
    return slice_ptr[p >> 5] + (p & 31);
}
__device__ __forceinline__ int64_t word_base(const int64_t *slice_ptr, int64_t p) {
    return (slice_ptr[p >> 5] >> 5) + (p & 31);
}

// ---------------------------------------------------------------------
// Family build (peri.jl:533-576): membership is the reference's exact
// test ((a1-a2)^2 + (b1-b2)^2) + (c1-c2)^2 < h*h over the 27 cells around
// the particle's cell (cells are at least one horizon wide, so the search
// is complete); the list is then sorted descending (sort + reverse,
// peri.jl:553-556 and general_material.jl:88-90).
// ---------------------------------------------------------------------
template <bool kFill>
__global__ void k_neighbors(int64_t n, int64_t first, const double4 *__restrict__ x4,
                            const int32_t *__restrict__ cell_of,
                            const int32_t *__restrict__ cell_start,
                            const int32_t *__restrict__ cell_list, int64_t cell_base, int3 dims,
                            double horizon, int32_t *__restrict__ cnt,
                            const int64_t *__restrict__ slice_ptr, int32_t *__restrict__ nbr) {
    int64_t li = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (li >= n) return;
    int64_t i = first + li;
    double4 xi = x4[i];
    int32_t c = cell_of[li] - (int32_t)cell_base;
    int cx = c % dims.x, cy = (c / dims.x) % dims.y, cz = c / (dims.x * dims.y);
    const double h2 = horizon * horizon;
    int32_t k = 0;
    int64_t base = kFill ? sell_base(slice_ptr, i) : 0;
    for (int dz = -1; dz <= 1; ++dz) {
        int zz = cz + dz;
        if (zz < 0 || zz >= dims.z) continue;
        for (int dy = -1; dy <= 1; ++dy) {
            int yy = cy + dy;
            if (yy < 0 || yy >= dims.y) continue;
            for (int dx = -1; dx <= 1; ++dx) {
                int xx = cx + dx;
                if (xx < 0 || xx >= dims.x) continue;
                int64_t cell = cell_base + xx + (int64_t)dims.x * (yy + (int64_t)dims.y * zz);
                for (int32_t s = cell_start[cell]; s < cell_start[cell + 1]; ++s) {
                    int32_t j = cell_list[s];
                    if (j == i) continue;
                    double4 xj = x4[j];
                    double a = xi.x - xj.x, b = xi.y - xj.y, cc = xi.z - xj.z;
                    if (a * a + b * b + cc * cc < h2) {
                        if (kFill) nbr[base + 32 * (int64_t)k] = j;
                        ++k;
                    }
                }
            }
        }
    }
    if (!kFill) cnt[i] = k;
}

// Cell binning of one block for the family search (a counting sort by cell
// id on the device): the cell of particle i is floor((x - lo) / cell) per
// axis, clamped to the grid (wider domains fold into the edge cells), as
// an index into the environment's concatenated cell grids; k_cell_ids
// counts the particles of each cell, the host turns the counts into cell
// starts, k_cell_scatter fills each cell's list.  The order within a cell
// is whatever the atomics give: the search finds the same members in any
// order and sorts each list afterwards.
__global__ void k_cell_ids(int64_t n, int64_t first, const double4 *__restrict__ x4, double3 lo, double cell,
                           int3 dims, int64_t cell_base, int32_t *__restrict__ cell_of, int32_t *__restrict__ count) {
    const int64_t li = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (li >= n) return;
    const double4 x = x4[first + li];
    const double xs[3] = {x.x, x.y, x.z}, los[3] = {lo.x, lo.y, lo.z};
    const int dm[3] = {dims.x, dims.y, dims.z};
    int ijk[3];
    for (int d = 0; d < 3; ++d) {
        double q = floor((xs[d] - los[d]) / cell);
        if (!(q >= 0.0)) q = 0.0;
        if (q > dm[d] - 1) q = dm[d] - 1;
        ijk[d] = (int)q;
    }
    const int64_t c = cell_base + ijk[0] + (int64_t)dm[0] * (ijk[1] + (int64_t)dm[1] * ijk[2]);
    cell_of[li] = (int32_t)c;
    atomicAdd(count + c, 1);
}

__global__ void k_cell_scatter(int64_t n, int64_t first, const int32_t *__restrict__ cell_of,
                               int32_t *__restrict__ cursor, int32_t *__restrict__ cell_list) {
    const int64_t li = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (li >= n) return;
    cell_list[atomicAdd(cursor + cell_of[li], 1)] = (int32_t)(first + li);
}

// Insertion sort of one particle's strided list into descending order.
__global__ void k_sort_neighbors(int64_t N, const int64_t *__restrict__ slice_ptr,
                                 const int32_t *__restrict__ cnt, int32_t *__restrict__ nbr) {
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= N) return;
    int32_t n = cnt[p];
    int32_t *a = nbr + sell_base(slice_ptr, p);
    for (int32_t k = 1; k < n; ++k) {
        int32_t v = a[32 * (int64_t)k];
        int32_t j = k - 1;
        while (j >= 0 && a[32 * (int64_t)j] < v) {
            a[32 * (int64_t)(j + 1)] = a[32 * (int64_t)j];
            --j;
        }
        a[32 * (int64_t)(j + 1)] = v;
    }
}

__global__ void k_init_intact(int64_t N, const int64_t *__restrict__ slice_ptr,
                              const int32_t *__restrict__ cnt, uint32_t *__restrict__ words) {
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= N) return;
    int32_t n = cnt[p];
    int64_t wb = word_base(slice_ptr, p);
    for (int32_t w = 0; w * 32 < n; ++w) {
        int32_t rem = n - w * 32;
        words[wb + 32 * (int64_t)w] = rem >= 32 ? 0xffffffffu : ((1u << rem) - 1u);
    }
}

// ---------------------------------------------------------------------
// Runtime layout on the device (the conversion build_runtime_layout in
// pd_env.cu performs on the host; both give the same arrays).  Pass 1, one
// warp per slice: the union of the lanes' neighbour offsets q - p, merged
// from the lanes' descending lists one element at a time (the warp's
// maximum of the lanes' heads is the union's next element; lanes holding it
// advance).  A slice takes the stencil form when the union has at most
// maxc + maxc/4 + 32 entries (maxc: the slice's largest family) and every
// union offset of every lane with bonds names an in-range record.
// Outputs per slice: mode, union length (stencil) and the union itself in
// uni[s * ustride ...]; the first merge only counts, so a slice found too
// large writes nothing.
// ---------------------------------------------------------------------
__global__ void k_layout_union(int64_t S, int64_t N, const int64_t *__restrict__ slice_ptr,
                               const int32_t *__restrict__ cnt, const int32_t *__restrict__ nbr_b,
                               int32_t force_explicit, int64_t ustride, int32_t *__restrict__ mode,
                               int32_t *__restrict__ len, int32_t *__restrict__ uni) {
    const int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (s >= S) return;  // whole warps: blockDim is a multiple of 32
    const int64_t p = s * 32 + lane;
    const int32_t c = cnt[p];
    int32_t maxc = c;
    for (int o = 16; o > 0; o >>= 1) maxc = max(maxc, __shfl_xor_sync(0xffffffffu, maxc, o));
    const int32_t *lst = nbr_b + slice_ptr[s] + lane;  // lane's k-th neighbour at lst[32 k]
    const int64_t limit = (int64_t)maxc + maxc / 4 + 32;
    bool stencil = !force_explicit && maxc > 0;
    int64_t ulen = 0;
    int32_t umax = 0, umin = 0;
    if (stencil) {
        for (int pass = 0; pass < 2 && stencil; ++pass) {
            int32_t k = 0;
            int32_t head = k < c ? lst[0] - (int32_t)p : INT_MIN;
            int64_t pos = 0;
            for (;;) {
                const int32_t m = __reduce_max_sync(0xffffffffu, head);
                if (m == INT_MIN) break;
                if (pass == 0) {
                    if (pos == 0) umax = m;
                    umin = m;
                    if (pos + 1 > limit) {
                        stencil = false;
                        break;
                    }
                } else if (lane == 0) {
                    uni[s * ustride + pos] = m;
                }
                if (head == m) {
                    ++k;
                    head = k < c ? lst[32 * (int64_t)k] - (int32_t)p : INT_MIN;
                }
                ++pos;
            }
            ulen = pos;
            if (pass == 0 && stencil) {
                // every slot a lane scans must name an in-range record
                const bool ok = c == 0 || (p + umax < N && p + umin >= 0);
                stencil = __all_sync(0xffffffffu, ok);
            }
        }
    }
    if (lane == 0) {
        mode[s] = stencil ? kStencil : kExplicit;
        len[s] = stencil ? (int32_t)ulen : maxc;
    }
}

// Pass 2, one thread per particle (a warp per slice): the runtime arrays.
// Stencil slices: the union offsets into nbr, and each bond's slot found by
// a binary search of its offset in the (descending) union; explicit slices:
// the build layout's indices copied.  Intact and family-member bits go to
// the lane's own words; cnt_rt = last occupied slot + 1.
__global__ void k_layout_fill(int64_t N, const int64_t *__restrict__ slice_ptr, const int32_t *__restrict__ cnt,
                              const int32_t *__restrict__ nbr_b, const uint32_t *__restrict__ w_b,
                              const SliceInfo *__restrict__ si, const int32_t *__restrict__ ulen, int64_t ustride,
                              const int32_t *__restrict__ uni, int32_t *__restrict__ nbr, uint32_t *__restrict__ words,
                              uint32_t *__restrict__ fam, int32_t *__restrict__ cnt_rt) {
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= N) return;
    const int64_t s = p >> 5;
    const int lane = (int)(p & 31);
    const SliceInfo d = si[s];
    const int32_t c = cnt[p];
    const int64_t base = slice_ptr[s] + lane, wb = slice_ptr[s] / 32 + lane, ow = d.word + lane;
    const int32_t *u = uni + s * ustride;
    const int32_t ul = d.mode == kStencil ? ulen[s] : 0;
    if (d.mode == kStencil) {
        for (int32_t j = lane; j < ul; j += 32) nbr[d.nbr + j] = u[j];
    } else {
        for (int32_t k = 0; k < d.len; ++k) nbr[d.nbr + 32 * (int64_t)k + lane] = nbr_b[base + 32 * (int64_t)k];
    }
    int32_t last = -1;
    for (int32_t k = 0; k < c; ++k) {
        int32_t slot = k;
        if (d.mode == kStencil) {
            const int32_t o = nbr_b[base + 32 * (int64_t)k] - (int32_t)p;
            int32_t lo = 0, hi = ul - 1;  // u descends: find u[slot] == o
            while (lo < hi) {
                const int32_t mid = (lo + hi) >> 1;
                if (u[mid] > o) lo = mid + 1;
                else hi = mid;
            }
            slot = lo;
        }
        const uint32_t bit = 1u << (slot & 31);
        fam[ow + 32 * (int64_t)(slot >> 5)] |= bit;
        if ((w_b[wb + 32 * (int64_t)(k >> 5)] >> (k & 31)) & 1u) words[ow + 32 * (int64_t)(slot >> 5)] |= bit;
        last = slot;
    }
    cnt_rt[p] = last + 1;
}

__global__ void k_popcount(int64_t N, const SliceInfo *__restrict__ si,
                           const int32_t *__restrict__ cnt, const uint32_t *__restrict__ words,
                           int32_t *__restrict__ out) {
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= N) return;
    int32_t n = cnt[p], c = 0;
    const uint32_t *wp = words + si[p >> 5].word + (p & 31);
    for (int32_t w = 0; w * 32 < n; ++w) c += __popc(wp[32 * (int64_t)w]);
    out[p] = c;
}

// peri.jl:342-354 weighted_volume: m_i = sum_j ((1/|X|) * (|X|*|X|)) * 1 * V_j
// over the family (every member, intact or not) in stored (descending) order.
__global__ void k_weighted_volume(Geo g, double2 *__restrict__ mth) {
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= g.N) return;
    if (g.tinfo[p] < 0) return;
    double4 xp = g.x4[p];
    int32_t n = g.cnt[p];
    const BondRef br = bond_ref(g.si, g.nbr, g.fam, p);
    double acc = 0.0;
    for (int32_t k = 0; k < n; ++k) {
        if (!((*br.word(k) >> (k & 31)) & 1u)) continue;
        int32_t q = br.q(k);
        double4 xq = g.x4[q];
        double mg = mag3(xq.x - xp.x, xq.y - xp.y, xq.z - xp.z);
        double w = 1.0 / mg;
        acc = acc + w * (mg * mg) * 1.0 * xq.w;
    }
    mth[p].x = acc;
}

// ---------------------------------------------------------------------
// peri.jl:155-172 dilatation!: theta_i = sum over intact bonds, in family
// order, of (((3/m_i) * w) * |X|) * e * V_j  (horizon correction == 1).
// ---------------------------------------------------------------------
// The operators' evaluation of a term the branch-free one does not cover.
__device__ __noinline__ double theta_term_general(double4 xp, double4 yp, double4 xq, double4 yq, double c_i) {
    const double xij = mag3(xq.x - xp.x, xq.y - xp.y, xq.z - xp.z);
    const double yij = mag3(yq.x - yp.x, yq.y - yp.y, yq.z - yp.z);
    const double e = yij - xij;
    const double wi = 1.0 / xij;
    return c_i * wi * xij * e * xq.w;
}
// The branch-free evaluation; returns whether it is exact.
__device__ __forceinline__ bool theta_slot(const double4 &xp, const double4 &yp, const double4 &xq, const double4 &yq,
                                           double c_i, double &t) {
    const double X1 = xq.x - xp.x, X2 = xq.y - xp.y, X3 = xq.z - xp.z;
    const double Y1 = yq.x - yp.x, Y2 = yq.y - yp.y, Y3 = yq.z - yp.z;
    double xij, yij, rx, ry;
    bool fast = sqrt_rcp_rn(X1 * X1 + X2 * X2 + X3 * X3, xij, rx);
    fast = sqrt_rcp_rn(Y1 * Y1 + Y2 * Y2 + Y3 * Y3, yij, ry) && fast;
    t = c_i * rx * xij * (yij - xij) * xq.w;
    return fast;
}

// A thread per particle, one term after another: short slot lists on many
// slices (serial_runs).  Bound by the latency of a term's roots.
__global__ void __launch_bounds__(kThreads)
    k_theta_serial(Geo g, const double4 *y, const uint32_t *win, double2 *mth, int64_t p0, int64_t p1) {
    const int64_t p = p0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= p1 || (g.stop && *g.stop)) return;
    const int32_t ti = g.tinfo[p];
    if (ti < 0) return;
    const int kind = g.blocks[ti >> 8].kind;
    if (kind != PD_MAT_ORDINARY_STATE_BASED && kind != PD_MAT_ELASTO_PLASTIC) return;
    const double4 xp = g.x4[p], yp = y[p];
    const double c_i = 3.0 / mth[p].x;
    const int32_t n = g.cnt[p];
    const BondRef br = bond_ref(g.si, g.nbr, win, p);
    double th = 0.0;
    uint32_t w = 0;
    for (int32_t k = 0; k < n; ++k) {
        if ((k & 31) == 0) w = *br.word(k);
        if (!((w >> (k & 31)) & 1u)) continue;
        const int32_t q = br.q(k);
        const double4 xq = ld4_nc(g.x4 + q), yq = ld4(y + q);
        double t;
        if (!theta_slot(xp, yp, xq, yq, c_i, t)) t = theta_term_general(xp, yp, xq, yq, c_i);
        th = th + t;
    }
    mth[p].y = th;
}

// One block per slice: the warps evaluate the terms of the slice's slots
// side by side (tiles of kThetaTile slots in shared memory, a contiguous run
// of a tile's slots per warp, two slots at a time), then one warp adds them
// in family order.  Slots without an intact bond hold zero (the sum starts
// at +0.0 and so is never -0.0).  A thread per particle, one term after
// another, took 102 us on the 40,000-particle bar, this kernel 29 us.
constexpr int32_t kThetaTile = 128;
template <int NW>
__global__ void __launch_bounds__(32 * NW, NW == 8 ? 3 : 1)
    k_theta_slice(Geo g, const double4 *y, const uint32_t *win, double2 *mth, int64_t s0) {
    __shared__ double term[kThetaTile][32];
    const int64_t s = s0 + blockIdx.x;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t p = 32 * s + lane;
    const int32_t ti = g.tinfo[p];
    const int32_t tb = __reduce_max_sync(0xffffffffu, ti);
    const int kind = tb >= 0 ? g.blocks[tb >> 8].kind : PD_MAT_SKIP;
    const int32_t n = g.cnt[p];
    const int32_t own = lane_record((int32_t)p, ti);
    const double4 xp = ld4_nc(g.x4 + own);
    pdl_enter();  // before any return: the next kernel may wait for this one only
    if ((kind != PD_MAT_ORDINARY_STATE_BASED && kind != PD_MAT_ELASTO_PLASTIC) || (g.stop && *g.stop)) return;
    const double4 yp = ld4(y + own);
    const double c_i = ti >= 0 ? 3.0 / mth[p].x : 0.0;
    const int32_t L = (int32_t)__reduce_max_sync(0xffffffffu, (unsigned)n);
    const SliceInfo d = g.si[s];
    const bool st = d.mode == kStencil;
    const int32_t *nb = g.nbr + d.nbr + (st ? 0 : lane);
    const uint32_t *wi = win + d.word + lane;
    auto entry = [&](int32_t k) { return __ldg(nb + (st ? k : 32 * k)); };  // (a slice stores all its slots)
    double th = 0.0;
    for (int32_t base = 0; base < L; base += kThetaTile) {
        const int32_t m = min(kThetaTile, L - base);
        const int32_t per = (m + NW - 1) / NW, j0 = min(w * per, m), j1 = min(j0 + per, m);
        if (base) __syncthreads();
        for (int32_t j = j0; j < j1; j += 2) {
            const int32_t ka = base + j, kb = base + min(j + 1, j1 - 1);
            const int32_t na = entry(ka), nb2 = entry(kb);
            const bool la = ka < n && ((wi[32 * (ka >> 5)] >> (ka & 31)) & 1u);
            const bool lb = kb < n && ((wi[32 * (kb >> 5)] >> (kb & 31)) & 1u);
            const int32_t qa = slot_record(st, own, na, la), qb = slot_record(st, own, nb2, lb);
            const double4 xa = ld4_nc(g.x4 + qa), ya = ld4(y + qa), xb = ld4_nc(g.x4 + qb), yb = ld4(y + qb);
            double ta, tb2;
            const bool ea = theta_slot(xp, yp, xa, ya, c_i, ta), eb = theta_slot(xp, yp, xb, yb, c_i, tb2);
            if (la && !ea) ta = theta_term_general(xp, yp, xa, ya, c_i);
            if (lb && !eb) tb2 = theta_term_general(xp, yp, xb, yb, c_i);
            term[j][lane] = la ? ta : 0.0;
            if (j + 1 < j1) term[j + 1][lane] = lb ? tb2 : 0.0;
        }
        __syncthreads();
        if (w == 0) {
#pragma unroll 8
            for (int32_t j = 0; j < m; ++j) th = th + term[j][lane];
        }
    }
    if (w == 0 && ti >= 0) mth[p].y = th;
}

// One bond term seen from particle p: returns true when the bond is
// stretched below critical (s < cs) and writes the acceleration term
// ((xx*Y_d)*V_q)/rho_p.  The reference adds exactly this value to f_p in
// p's own loop, and subtracts its exact negation in q's loop
// (general_material.jl:357-362), so the same function serves both.
template <int KIND>
__device__ __forceinline__ bool bond_term(const Geo &g, const DevBlock &B, int tp,
                                          double4 xp, double4 yp, double2 mp, double rho_p,
                                          int32_t q, const double4 *y,
                                          const double2 *mth, double &t0,
                                          double &t1, double &t2) {
    double4 xq = g.x4[q], yq = y[q];
    double X1 = xq.x - xp.x, X2 = xq.y - xp.y, X3 = xq.z - xp.z;
    double Y1 = yq.x - yp.x, Y2 = yq.y - yp.y, Y3 = yq.z - yp.z;
    double yij = mag3(Y1, Y2, Y3);
    double xij = mag3(X1, X2, X3);
    double ext = yij - xij;
    double s = ext / xij;
    int tq = B.nt > 1 ? (g.tinfo[q] & 255) : 0;
    const PairParam &pp = g.pairs[B.pair_base + tp + tq * B.nt];
    if (!(s < pp.cs)) return false;
    double t;
    if (KIND == PD_MAT_BOND_BASED) {
        t = s * B.c11;  // bond_based.jl:195-197
    } else {
        // ordinary_state_based.jl:176-187 (w_ij == w_ji == 1/|X|)
        double2 mq = mth[q];
        double wij = 1.0 / xij;
        double a = wij / mp.x, b = wij / mq.x;
        t = pp.k35 * (mp.y * xij * a + mq.y * xij * b) + pp.g15 * ext * (a + b);
    }
    double xx = 0.5 * t / yij;
    t0 = xx * Y1 * xq.w / rho_p;
    t1 = xx * Y2 * xq.w / rho_p;
    t2 = xx * Y3 * xq.w / rho_p;
    return true;
}

// The same in branch-free arithmetic (pd_ieee.h).
// What a particle's terms share.
struct OwnTerm {
    double4 x, y;
    double2 m;
    double rho, rrho, rm;  // rrho = 1 / rho, rm = 1 / m.x
    bool ok;               // rho, m.x and c11 are within div_ok's range
};
// What a slot's evaluation needs of its neighbour.
struct SlotIn {
    double4 x, y;
    double2 m;
    int32_t q;
};

template <int KIND>
__device__ __forceinline__ OwnTerm own_term(double4 x, double4 y, double2 m, double rho, double c11) {
    constexpr bool PMB = KIND == PD_MAT_BOND_BASED;
    return OwnTerm{x, y, m, rho, rcp_rn(rho), PMB ? 0.0 : rcp_rn(m.x),
                   div_ok(rho) && (PMB ? div_ok(fabs(c11)) : div_ok(m.x))};
}

// The slot's term (zero unless live and within the critical stretch);
// returns whether the evaluation is exact.  The numerators: ext is zero
// or at least 2^-54 of the lengths, and so is s, at most 2^200; PMB: c in
// [2^-100, 2^100) then keeps 0.5 t in range, LPS checks it; V < 2^100
// bounds the last three from above.
template <int KIND>
__device__ __forceinline__ bool slot_term(const OwnTerm &o, double c11, const SlotIn &r, const PairParam &pp, bool live,
                                          double &o0, double &o1, double &o2, bool &within) {
    constexpr bool PMB = KIND == PD_MAT_BOND_BASED;
    const double Y1 = r.y.x - o.y.x, Y2 = r.y.y - o.y.y, Y3 = r.y.z - o.y.z;
    const double X1 = r.x.x - o.x.x, X2 = r.x.y - o.x.y, X3 = r.x.z - o.x.z;
    double xij, yij, rx, ry;
    bool fast = sqrt_rcp_rn(X1 * X1 + X2 * X2 + X3 * X3, xij, rx) && o.ok;
    fast = sqrt_rcp_rn(Y1 * Y1 + Y2 * Y2 + Y3 * Y3, yij, ry) && fast;
    fast = (uint32_t)hi_word(r.x.w) < ((1023u + 100u) << 20) && fast;
    const double ext = yij - xij;
    const double s = div_rn(ext, xij, rx);
    within = s < pp.cs;
    double t;
    if (PMB) {
        t = s * c11;
    } else {
        fast = fast && div_ok(r.m.x);
        const double a = div_rn(rx, o.m.x, o.rm), b = div_rn(rx, r.m.x, rcp_rn(r.m.x));
        t = pp.k35 * (o.m.y * xij * a + r.m.y * xij * b) + pp.g15 * ext * (a + b);
    }
    const double ht = 0.5 * t;
    if (!PMB) fast = fast && magnitude(ht) >= kMagLo && (2u * (uint32_t)hi_word(ht)) < kMagHi;
    double xx = div_rn(ht, yij, ry);
    xx = live && within ? xx : 0.0;
    o0 = xx * Y1 * r.x.w;
    o1 = xx * Y2 * r.x.w;
    o2 = xx * Y3 * r.x.w;
    fast = fast && min(min(magnitude(o0), magnitude(o1)), magnitude(o2)) >= kMagLo;
    o0 = div_rn(o0, o.rho, o.rrho);
    o1 = div_rn(o1, o.rho, o.rrho);
    o2 = div_rn(o2, o.rho, o.rrho);
    return fast;
}

// A bond the branch-free evaluation does not cover, with the operators.
template <int KIND>
__device__ __noinline__ bool bond_term_general(const Geo &g, const DevBlock &B, int64_t p, int tp, int32_t q,
                                               const double4 *y, const double2 *mth, double *t) {
    return bond_term<KIND>(g, B, tp, g.x4[p], y[p], KIND != PD_MAT_BOND_BASED ? mth[p] : make_double2(0.0, 0.0),
                           g.tdens[B.type_base + tp], q, y, mth, t[0], t[1], t[2]);
}

// bond_term by the branch-free evaluation where it is exact.
template <int KIND>
__device__ __forceinline__ bool bond_term_fast(const Geo &g, const DevBlock &B, int64_t p, int tp, const OwnTerm &o,
                                               int32_t q, const double4 *y, const double2 *mth, double &t0, double &t1,
                                               double &t2) {
    SlotIn r;
    r.x = ld4_nc(g.x4 + q);
    r.y = ld4(y + q);
    r.m = KIND == PD_MAT_BOND_BASED ? make_double2(0.0, 0.0) : mth[q];
    r.q = q;
    const int tq = B.nt > 1 ? (g.tinfo[q] & 255) : 0;
    bool within;
    if (slot_term<KIND>(o, B.c11, r, g.pairs[B.pair_base + tp + tq * B.nt], true, t0, t1, t2, within)) return within;
    double t[3] = {0.0, 0.0, 0.0};
    within = bond_term_general<KIND>(g, B, p, tp, q, y, mth, t);
    t0 = t[0];
    t1 = t[1];
    t2 = t[2];
    return within;
}

// ---------------------------------------------------------------------
// Elasto-plastic solid (elasto_plastic.jl).  Unlike the PMB and LPS laws,
// the bond term depends on which end visits the bond: particle i's visit
// to bond slot k uses td_norm2[i] and edp[k, i] and updates edp[k, i].
// ---------------------------------------------------------------------
// Slot of neighbour p in q's family.
__device__ __forceinline__ int32_t find_slot(const Geo &g, int64_t q, int32_t p) {
    return slot_of(g.si, g.nbr, g.cnt, q, p);
}

// force_density_t_ij (elasto_plastic.jl:215-242) for the visit of i to j;
// mi, mj = (m, theta); the plastic update of edp[k, i] goes to *edp_new.
__device__ __forceinline__ double ep_t(const PairParam &pp, double xij, double ext, double2 mi, double2 mj,
                                       double td2_i, double edp_old, double *edp_new) {
    const double wij = 1.0 / xij;  // influence_function(X) == influence_function(-X)
    const double C = sqrt(pp.psi2 / td2_i);
    const double a = wij / mi.x, b = wij / mj.x;
    const double tw = mi.y * a + mj.y * b;
    const double theta_ij = tw / (a + b);
    const double ed = ext - theta_ij * xij / 3;
    const double ede = ed - edp_old;
    const double td_trial = pp.g15 * (a + b) * ede;
    double td;
    if (C > 1) {
        td = td_trial;
    } else {
        td = C * td_trial;
        if (edp_new) *edp_new = edp_old + ede * (1 - C);
    }
    const double tn = pp.k35 * xij * tw;
    return tn + td;
}

// The elasto-plastic term seen by p for the bond to q: from p's own visit
// (own, slot k of p) or from q's visit to p.
__device__ __forceinline__ bool bond_term_ep(const Geo &g, const DevBlock &B, int tp, int64_t p, double4 xp,
                                             double4 yp, double2 mp, double rho_p, int32_t q, int32_t k, bool own,
                                             const double4 *y, const double2 *mth,
                                             double &t0, double &t1, double &t2) {
    double4 xq = g.x4[q], yq = y[q];
    double X1 = xq.x - xp.x, X2 = xq.y - xp.y, X3 = xq.z - xp.z;
    double Y1 = yq.x - yp.x, Y2 = yq.y - yp.y, Y3 = yq.z - yp.z;
    double yij = mag3(Y1, Y2, Y3);
    double xij = mag3(X1, X2, X3);
    double ext = yij - xij;
    double s = ext / xij;
    int tq = B.nt > 1 ? (g.tinfo[q] & 255) : 0;
    const PairParam &pp = g.pairs[B.pair_base + tp + tq * B.nt];
    if (!(s < pp.cs)) return false;
    const double2 mq = mth[q];
    double t;
    if (own) {
        const int64_t e = slot_index(g.si, p, k);
        t = ep_t(pp, xij, ext, mp, mq, g.td2[p], g.edp_in[e], g.edp_out + e);
    } else {
        const int64_t e = slot_index(g.si, q, find_slot(g, q, (int32_t)p));
        t = ep_t(pp, xij, ext, mq, mp, g.td2[q], g.edp_in[e], nullptr);
    }
    double xx = 0.5 * t / yij;
    t0 = xx * Y1 * xq.w / rho_p;
    t1 = xx * Y2 * xq.w / rho_p;
    t2 = xx * Y3 * xq.w / rho_p;
    return true;
}

// peri.jl:411-445 loop_over_neighs! with td_norm2_ij! (elasto_plastic.jl:
// 274-288): td_norm2[p] over p's family in stored order; bonds at or beyond
// the critical stretch are cleared (that loop breaks them too).  Particles
// of other blocks only copy their flags.
__global__ void __launch_bounds__(kThreads)
    k_td_serial(Geo g, const double4 *__restrict__ y, const double2 *__restrict__ mth,
                const uint32_t *__restrict__ win, uint32_t *__restrict__ wout, int64_t p0, int64_t p1) {
    int64_t p = p0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= p1 || (g.stop && *g.stop)) return;
    const int32_t ti = g.tinfo[p];
    const int32_t n = g.cnt[p];
    const int64_t wb = g.si[p >> 5].word + (p & 31);
    const bool active = ti >= 0 && g.blocks[ti >> 8].kind == PD_MAT_ELASTO_PLASTIC && g.deformed[ti >> 8] != 0;
    if (!active) {
        for (int32_t w = 0; w * 32 < n; ++w) wout[wb + 32 * (int64_t)w] = win[wb + 32 * (int64_t)w];
        return;
    }
    const DevBlock &B = g.blocks[ti >> 8];
    const int tp = ti & 255;
    const double4 xp = g.x4[p], yp = y[p];
    const double2 mp = mth[p];
    const BondRef br = bond_ref(g.si, g.nbr, win, p);
    uint32_t *wo = wout + wb;
    double acc = 0.0;
    uint32_t w = 0;
    for (int32_t k = 0; k < n; ++k) {
        if ((k & 31) == 0) {
            if (k > 0) wo[32 * (int64_t)((k >> 5) - 1)] = w;
            w = *br.word(k);
        }
        if (!((w >> (k & 31)) & 1u)) continue;
        const int32_t q = br.q(k);
        const double4 xq = g.x4[q], yq = y[q];
        const double X1 = xq.x - xp.x, X2 = xq.y - xp.y, X3 = xq.z - xp.z;
        const double Y1 = yq.x - yp.x, Y2 = yq.y - yp.y, Y3 = yq.z - yp.z;
        const double yij = mag3(Y1, Y2, Y3);
        const double xij = mag3(X1, X2, X3);
        const double ext = yij - xij;
        const double s = ext / xij;
        const int tq = B.nt > 1 ? (g.tinfo[q] & 255) : 0;
        const PairParam &pp = g.pairs[B.pair_base + tp + tq * B.nt];
        if (s < pp.cs) {
            const double2 mq = mth[q];
            const double wij = 1.0 / xij;
            const double a = wij / mp.x, b = wij / mq.x;
            const double w_m = a + b;
            const double tw = mp.y * a + mq.y * b;
            const double theta_ij = tw / w_m;
            const double ed = ext - theta_ij * xij / 3;
            const double td = pp.g15 * (ed - g.edp_in[slot_index(g.si, p, k)]) * w_m;
            acc = acc + td * td * xq.w;
        } else {
            w &= ~(1u << (k & 31));
        }
    }
    if (n > 0) wo[32 * (int64_t)((n - 1) >> 5)] = w;
    g.td2[p] = acc;
}

// ---------------------------------------------------------------------
// general_material.jl:296-369 in the serial loop's summation order.
// The reference visits i = 1..N and, for each i, its family in stored
// (descending) order, adding the term to f_i and subtracting it from f_j.
// Particle p therefore receives, in order:
//   A. terms of neighbours q < p, ascending q   (from q's loop)
//   B. terms of all neighbours, descending q    (p's own loop)
//   C. terms of neighbours q > p, ascending q   (from q's loop)
// Bond flags are symmetric (both ends break in the same step because the
// stretch is the same number from both sides), so p's own flags stand in
// for q's.  Bonds with s >= cs are cleared in wout.
// ---------------------------------------------------------------------
template <int KIND>
__device__ void force_serial_particle(const Geo &g, int64_t p, int32_t ti,
                                      const double4 *y,
                                      const double2 *mth,
                                      const uint32_t *win,
                                      uint32_t *wout, double4 *f,
                                      int accumulate) {
    const DevBlock &B = g.blocks[ti >> 8];
    int tp = ti & 255;
    double4 xp = g.x4[p], yp = y[p];
    double2 mp = KIND != PD_MAT_BOND_BASED ? mth[p] : make_double2(0.0, 0.0);
    constexpr bool EP = KIND == PD_MAT_ELASTO_PLASTIC;
    double rho_p = g.tdens[B.type_base + tp];
    const OwnTerm o = own_term<EP ? PD_MAT_BOND_BASED : KIND>(xp, yp, mp, rho_p, B.c11);
    int32_t n = g.cnt[p];
    const BondRef br = bond_ref(g.si, g.nbr, win, p);
    uint32_t *wo = wout + g.si[p >> 5].word + (p & 31);
    double fx = 0.0, fy = 0.0, fz = 0.0;
    if (accumulate) {
        double4 f0 = f[p];
        fx = f0.x;
        fy = f0.y;
        fz = f0.z;
    }
    double t0, t1, t2;
    // Pass A: q < p, ascending (walk the descending list from the end).
    int32_t k = n - 1;
    for (; k >= 0; --k) {
        int32_t q = br.q(k);
        if (q > p) break;
        uint32_t w = *br.word(k);
        if (!((w >> (k & 31)) & 1u)) continue;
        if (EP ? bond_term_ep(g, B, tp, p, xp, yp, mp, rho_p, q, k, false, y, mth, t0, t1, t2)
               : bond_term_fast<EP ? PD_MAT_BOND_BASED : KIND>(g, B, p, tp, o, q, y, mth, t0, t1, t2)) {
            fx = fx + t0;
            fy = fy + t1;
            fz = fz + t2;
        }
    }
    const int32_t kc = k;
    // Pass B: p's own loop, descending q; breaks bonds.
    uint32_t w = 0;
    for (k = 0; k < n; ++k) {
        if ((k & 31) == 0) {
            if (k > 0) wo[32 * (int64_t)((k >> 5) - 1)] = w;
            w = *br.word(k);
        }
        if (EP) {  // edp carries over unless this visit yields
            const int64_t e = slot_index(g.si, p, k);
            g.edp_out[e] = g.edp_in[e];
        }
        if (!((w >> (k & 31)) & 1u)) continue;
        int32_t q = br.q(k);
        if (EP ? bond_term_ep(g, B, tp, p, xp, yp, mp, rho_p, q, k, true, y, mth, t0, t1, t2)
               : bond_term_fast<EP ? PD_MAT_BOND_BASED : KIND>(g, B, p, tp, o, q, y, mth, t0, t1, t2)) {
            fx = fx + t0;
            fy = fy + t1;
            fz = fz + t2;
        } else {
            w &= ~(1u << (k & 31));
        }
    }
    if (n > 0) wo[32 * (int64_t)((n - 1) >> 5)] = w;
    // Pass C: q > p, ascending.
    for (k = kc; k >= 0; --k) {
        int32_t q = br.q(k);
        uint32_t ww = *br.word(k);
        if (!((ww >> (k & 31)) & 1u)) continue;
        if (EP ? bond_term_ep(g, B, tp, p, xp, yp, mp, rho_p, q, k, false, y, mth, t0, t1, t2)
               : bond_term_fast<EP ? PD_MAT_BOND_BASED : KIND>(g, B, p, tp, o, q, y, mth, t0, t1, t2)) {
            fx = fx + t0;
            fy = fy + t1;
            fz = fz + t2;
        }
    }
    f[p] = make_double4(fx, fy, fz, 0.0);
}

// The slots a 32-particle slice walks: the largest slot count of its lanes.
__device__ __forceinline__ int32_t slice_slots(int32_t n) { return (int32_t)__reduce_max_sync(0xffffffffu, (unsigned)n); }

// One thread per particle, every bond evaluated from both visits: short slot
// lists on many slices (serial_runs; cap < 0: all of the range), and of the
// rest the elasto-plastic blocks (whose two visits differ) and slices with
// more than cap slots.  The other slices belong to k_force_slice.  Bound by
// the latency of a bond's roots and quotients, which it meets twice per slot
// in a row; branch-free as in k_force_slice (8,000 particles with 304 slots:
// 338 us per evaluation, 454 with the operators; 262,144 with 18 slots, most
// of them undisturbed: 108 against 249 us per step).
__global__ void __launch_bounds__(kThreads)
    k_force_serial(Geo g, const double4 *__restrict__ y, const double2 *__restrict__ mth,
                   const uint32_t *__restrict__ win, uint32_t *__restrict__ wout,
                   double4 *__restrict__ f, int accumulate, int32_t cap, int64_t p0, int64_t p1) {
    int64_t p = p0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= p1 || (g.stop && *g.stop)) return;  // whole warps: p0 and p1 are multiples of 32
    int32_t ti = g.tinfo[p];
    int32_t n = g.cnt[p];
    const int64_t wb = g.si[p >> 5].word + (p & 31);
    bool active = false;
    int kind = PD_MAT_SKIP;
    if (ti >= 0) {
        const DevBlock &B = g.blocks[ti >> 8];
        kind = B.kind;
        active = kind != PD_MAT_SKIP && g.deformed[ti >> 8] != 0;
    }
    if (!__any_sync(0xffffffffu, kind == PD_MAT_ELASTO_PLASTIC) && slice_slots(n) <= cap) return;
    if (!active) {
        for (int32_t w = 0; w * 32 < n; ++w) wout[wb + 32 * (int64_t)w] = win[wb + 32 * (int64_t)w];
        if (kind == PD_MAT_ELASTO_PLASTIC && g.edp_out)
            for (int32_t k = 0; k < n; ++k) g.edp_out[slot_index(g.si, p, k)] = g.edp_in[slot_index(g.si, p, k)];
        if (!accumulate) f[p] = make_double4(0.0, 0.0, 0.0, 0.0);
        return;
    }
    if (kind == PD_MAT_BOND_BASED)
        force_serial_particle<PD_MAT_BOND_BASED>(g, p, ti, y, mth, win, wout, f, accumulate);
    else if (kind == PD_MAT_ELASTO_PLASTIC)
        force_serial_particle<PD_MAT_ELASTO_PLASTIC>(g, p, ti, y, mth, win, wout, f, accumulate);
    else
        force_serial_particle<PD_MAT_ORDINARY_STATE_BASED>(g, p, ti, y, mth, win, wout, f,
                                                            accumulate);
}

// ---------------------------------------------------------------------
// The same sums with every bond evaluated once, one block per slice.  The
// PMB and LPS terms are the same number from either visit, so only the
// order of the additions is serial: the block's warps evaluate the slice's
// slots side by side (warp w takes the w-th run of slots) into shared
// memory, 24 bytes per slot and lane, and then one warp per component adds
// them in the order A, B, C above.  A slot without a term holds a zero,
// which changes no partial sum: x + 0 == x unless x is -0.0, and a sum of
// at least one nonnegative-zero start is never -0.0 (slices whose caller
// passes -0.0 in f take the particle loop).
//
// What bounds it: the two blocks an SM holds (94 KB of terms for 122 slots)
// alternate between evaluation, a chain of some 600 cycles per pair of
// slots, and the sums, 244 dependent additions of 17 cycles.  FP64 pipe 36 %,
// issue 50 % busy (48^3 PMB cube; state-based 40 and 51 %).  Against a thread per particle
// that evaluates a bond at each of its two visits: force pass of a
// 990-particle cube 15 against 198 us, of a 40,000-particle state-based bar
// 84 against 484 us.  16 warps of 128 registers on an SM; 24 warps of 80
// (spills) were slower, 592 against 474 us per step of a 64^3 cube.
// ---------------------------------------------------------------------
// Largest family evaluated in shared memory: 288 slots of 768 bytes and
// their broken bits, within the 227 KB a block may take.
constexpr int32_t kForceSlots = 288;
inline size_t force_slice_bytes(int32_t cap) { return 768 * (size_t)cap + 128 * (size_t)((cap + 31) / 32); }

// A particle of a slice the block evaluation does not cover (accumulating).
__device__ __noinline__ void force_particle_general(const Geo &g, int64_t p, int32_t ti, int kind,
                                                    const double4 *y, const double2 *mth,
                                                    const uint32_t *win, uint32_t *wout,
                                                    double4 *f) {
    if (kind == PD_MAT_BOND_BASED) force_serial_particle<PD_MAT_BOND_BASED>(g, p, ti, y, mth, win, wout, f, 1);
    else force_serial_particle<PD_MAT_ORDINARY_STATE_BASED>(g, p, ti, y, mth, win, wout, f, 1);
}

template <int KIND, bool MULTI, bool ST, int NW>
__device__ __forceinline__ void evaluate_slice(const Geo &g, const DevBlock &B, const SliceInfo &d, int64_t p,
                                               int32_t ti, int32_t n, int32_t L, int w, int lane,
                                               const double4 *y, const double2 *mth,
                                               const uint32_t *win, double *term, uint32_t *brk) {
    constexpr bool PMB = KIND == PD_MAT_BOND_BASED;
    const int tp = ti >= 0 ? ti & 255 : 0;
    const int32_t own = lane_record((int32_t)p, ti);
    const PairParam pp0 = g.pairs[B.pair_base + tp + tp * B.nt];
    const double c11 = B.c11;
    const OwnTerm o = own_term<KIND>(ld4_nc(g.x4 + own), ld4(y + own), PMB ? make_double2(0.0, 0.0) : mth[own],
                                     g.tdens[B.type_base + tp], c11);
    const int32_t *nb = g.nbr + d.nbr + (ST ? 0 : lane);
    const uint32_t *wi = win + d.word + lane;
    // warp w evaluates the contiguous slots [k0, k1)
    const int32_t per = (L + NW - 1) / NW, k0 = min(w * per, L), k1 = min(k0 + per, L);
    if (k0 >= k1) return;
    auto entry = [&](int32_t k) { return __ldg(nb + (ST ? k : 32 * k)); };  // (a slice stores all its slots)
    auto load = [&](int32_t q) {
        SlotIn r;
        r.x = ld4_nc(g.x4 + q);
        r.y = ld4(y + q);
        r.m = PMB ? make_double2(0.0, 0.0) : mth[q];
        r.q = q;
        return r;
    };
    auto pair = [&](const SlotIn &r, bool live) {
        return MULTI ? g.pairs[slot_pair(B.pair_base, B.nt, tp, g.tinfo[r.q], live)] : pp0;
    };
    uint32_t bits = 0, gone = 0;
    auto finish = [&](int32_t k, int32_t q, bool live, bool exact, bool within, double o0, double o1, double o2) {
        if (live && !exact) {
            double out[3] = {0.0, 0.0, 0.0};
            within = bond_term_general<KIND>(g, B, p, tp, q, y, mth, out);
            o0 = out[0];
            o1 = out[1];
            o2 = out[2];
        }
        if (live && !within) gone |= 1u << (k & 31);
        double *t = term + 96 * k + lane;
        t[0] = live ? o0 : 0.0;
        t[32] = live ? o1 : 0.0;
        t[64] = live ? o2 : 0.0;
    };
    // two slots at a time, their chains side by side (a chain is some 35
    // dependent FP64 operations of 16 cycles, and 16 warps fit an SM)
    int32_t na = entry(k0), nb2 = entry(min(k0 + 1, k1 - 1));
    for (int32_t k = k0; k < k1;) {
        const int32_t word = k >> 5, kw = min(k1, (word + 1) << 5);  // slots of one intact word
        bits = 32 * word < n ? wi[32 * word] : 0u;
        gone = 0;
        for (; k < kw; k += 2) {
            const bool two = k + 1 < kw;
            const uint32_t b2 = bits >> (k & 31);
            const bool la = (b2 & 1u) != 0u, lb = two && (b2 & 2u) != 0u;
            const SlotIn ra = load(slot_record(ST, own, na, la)), rb = load(slot_record(ST, own, nb2, lb));
            const int32_t next = two ? k + 2 : k + 1;
            na = entry(min(next, k1 - 1));
            nb2 = entry(min(next + 1, k1 - 1));
            double a0, a1, a2, b0, b1, bz;
            bool wa, wb;
            const bool ea = slot_term<KIND>(o, c11, ra, pair(ra, la), la, a0, a1, a2, wa);
            const bool eb = slot_term<KIND>(o, c11, rb, pair(rb, lb), lb, b0, b1, bz, wb);
            finish(k, ra.q, la, ea, wa, a0, a1, a2);
            if (two) finish(k + 1, rb.q, lb, eb, wb, b0, b1, bz);
        }
        k = kw;
        if (gone) atomicOr(brk + 32 * word + lane, gone);  // two warps may own parts of one word
    }
}

template <int KIND, int NW>
__device__ __forceinline__ void evaluate_kind(const Geo &g, const DevBlock &B, const SliceInfo &d, int64_t p,
                                              int32_t ti, int32_t n, int32_t L, int w, int lane,
                                              const double4 *y, const double2 *mth,
                                              const uint32_t *win, double *term, uint32_t *brk) {
    if (d.mode == kStencil) {
        if (B.nt > 1) evaluate_slice<KIND, true, true, NW>(g, B, d, p, ti, n, L, w, lane, y, mth, win, term, brk);
        else evaluate_slice<KIND, false, true, NW>(g, B, d, p, ti, n, L, w, lane, y, mth, win, term, brk);
    } else {
        if (B.nt > 1) evaluate_slice<KIND, true, false, NW>(g, B, d, p, ti, n, L, w, lane, y, mth, win, term, brk);
        else evaluate_slice<KIND, false, false, NW>(g, B, d, p, ti, n, L, w, lane, y, mth, win, term, brk);
    }
}

// What a block needs of the slice it evaluates.
struct SliceLane {
    int64_t p;
    int32_t ti, n, L, tb, kind;
};
__device__ __forceinline__ SliceLane slice_lane(const Geo &g, int64_t s, int lane) {
    SliceLane v;
    v.p = 32 * s + lane;
    v.ti = g.tinfo[v.p];
    v.n = g.cnt[v.p];
    v.L = slice_slots(v.n);
    // every particle of a slice belongs to one block (padding: -1)
    v.tb = __reduce_max_sync(0xffffffffu, v.ti);
    v.kind = v.tb >= 0 ? g.blocks[v.tb >> 8].kind : PD_MAT_SKIP;
    return v;
}
// Behind the wait: the slice's block takes part (has left the undeformed state).
__device__ __forceinline__ bool slice_active(const Geo &g, const SliceLane &v) {
    return v.kind != PD_MAT_SKIP && g.deformed[v.tb >> 8] != 0;
}
// A slice that does not, by the warps w, w + step, ...: its flags carry over.
__device__ __forceinline__ void carry_slice(const SliceLane &v, const SliceInfo &d, int w, int step, int lane,
                                            const uint32_t *win, uint32_t *wout, double4 *f, int accumulate) {
    const uint32_t *wi = win + d.word + lane;
    uint32_t *wo = wout + d.word + lane;
    for (int32_t c0 = w; 32 * c0 < v.L; c0 += 4 * step) {
        uint32_t word[4];  // (all loads before the stores, which may alias them for all the compiler knows)
#pragma unroll
        for (int i = 0; i < 4; ++i) word[i] = 32 * (c0 + i * step) < v.n ? wi[32 * (c0 + i * step)] : 0u;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (32 * (c0 + i * step) < v.n) wo[32 * (c0 + i * step)] = word[i];
    }
    if (w == 0 && !accumulate) f[v.p] = make_double4(0.0, 0.0, 0.0, 0.0);
}

// The slice's forces, by the whole block.
template <int NW>
__device__ __forceinline__ void force_slice(const Geo &g, const double4 *y, const double2 *mth, const uint32_t *win,
                                            uint32_t *wout, double4 *f, int accumulate, int32_t cap,
                                            const SliceLane &v, const SliceInfo &d, int w, int lane, double *term) {
    const int64_t p = v.p;
    const int32_t ti = v.ti, n = v.n, L = v.L, tb = v.tb;
    const int kind = v.kind;
    const int32_t words = (L + 31) >> 5;
    uint32_t *brk = reinterpret_cast<uint32_t *>(term + 96 * (int64_t)cap);
    const uint32_t *wi = win + d.word + lane;
    uint32_t *wo = wout + d.word + lane;
    if (accumulate) {
        const double4 f0 = f[lane_record((int32_t)p, ti)];
        const uint64_t nz = 0x8000000000000000ull;
        const bool neg = (uint64_t)__double_as_longlong(f0.x) == nz || (uint64_t)__double_as_longlong(f0.y) == nz ||
                         (uint64_t)__double_as_longlong(f0.z) == nz;
        __syncthreads();  // every warp has read f before one writes it
        if (__any_sync(0xffffffffu, neg)) {  // the same lanes in every warp
            if (w == 0 && ti >= 0) force_particle_general(g, p, ti, kind, y, mth, win, wout, f);
            return;
        }
    }
    for (int32_t c = w; c < words; c += NW) brk[32 * c + lane] = 0u;
    __syncthreads();
    const DevBlock &B = g.blocks[tb >> 8];
    if (kind == PD_MAT_BOND_BASED)
        evaluate_kind<PD_MAT_BOND_BASED, NW>(g, B, d, p, ti, n, L, w, lane, y, mth, win, term, brk);
    else
        evaluate_kind<PD_MAT_ORDINARY_STATE_BASED, NW>(g, B, d, p, ti, n, L, w, lane, y, mth, win, term, brk);
    __syncthreads();
    if (w >= 3) {
        for (int32_t c = w - 3; c < words; c += NW - 3)
            if (32 * c < n) wo[32 * c] = wi[32 * c] & ~brk[32 * c + lane];
        return;
    }
    // kp: slots with q > p (a prefix: slots descend in q)
    int32_t lo = 0, hi = n;
    {
        const bool st = d.mode == kStencil;
        const int32_t *nb = g.nbr + d.nbr + (st ? 0 : lane);
        const int32_t own = st ? 0 : (int32_t)p;
        while (lo < hi) {
            const int32_t mid = (lo + hi) >> 1;
            if ((st ? nb[mid] : nb[32 * mid]) > own) lo = mid + 1;
            else hi = mid;
        }
    }
    const int32_t kp = lo;
    const int32_t kmin = (int32_t)__reduce_min_sync(0xffffffffu, (unsigned)(n > 0 ? kp : L));
    const int32_t kmax = (int32_t)__reduce_max_sync(0xffffffffu, (unsigned)kp);
    const double *T = term + 32 * w + lane;
    double *fo = reinterpret_cast<double *>(f + p);
    double a = accumulate && ti >= 0 ? fo[w] : 0.0;
#pragma unroll 8
    for (int32_t k = L - 1; k >= kmin; --k) {
        const double t = T[96 * k];
        a = a + (k >= kp ? t : 0.0);
    }
#pragma unroll 8
    for (int32_t k = 0; k < L; ++k) a = a + T[96 * k];
#pragma unroll 8
    for (int32_t k = kmax - 1; k >= 0; --k) {
        const double t = T[96 * k];
        a = a + (k < kp ? t : 0.0);
    }
    if (ti >= 0) {
        fo[w] = a;
        if (w == 0) fo[3] = 0.0;
    } else if (!accumulate) {
        fo[w] = 0.0;
        if (w == 0) fo[3] = 0.0;
    }
}

// SCAN: the S slices from s0 are dealt out to the blocks, whose warps look at
// a few slices each and carry those over whose body is undeformed; the block
// then evaluates the others.  (One block per slice, of which an SM holds two, is
// slow where nothing is to be done: the first steps of a 2.1-million-particle
// body, undeformed, took 580 us each against 236 with a thread per particle.)
template <int NW, bool SCAN>
__global__ void __launch_bounds__(32 * NW, NW == 8 ? 2 : 1)
    k_force_slice(Geo g, const double4 *y, const double2 *mth, const uint32_t *win, uint32_t *wout, double4 *f,
                  int accumulate, int32_t cap, int64_t s0, int64_t S) {
    extern __shared__ double term[];  // [slot][component][lane], then the broken bits [word][lane]
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if constexpr (!SCAN) {
        const int64_t s = s0 + blockIdx.x;
        const SliceLane v = slice_lane(g, s, lane);
        const SliceInfo d = g.si[s];
        pdl_enter();  // before any return: the next kernel may wait for this one only
        if (v.kind == PD_MAT_ELASTO_PLASTIC || v.L > cap || (g.stop && *g.stop)) return;
        if (slice_active(g, v)) force_slice<NW>(g, y, mth, win, wout, f, accumulate, cap, v, d, w, lane, term);
        else carry_slice(v, d, w, NW, lane, win, wout, f, accumulate);
    } else {
        constexpr int K = 4;  // slices a warp looks at together
        __shared__ bool todo[NW * K];
        pdl_enter();
        if (g.stop && *g.stop) return;
        const int64_t stride = gridDim.x;
        for (int64_t i0 = blockIdx.x; i0 < S; i0 += NW * K * stride) {
            SliceLane v[K];
            bool mine[K], run[K];
#pragma unroll
            for (int j = 0; j < K; ++j) {  // (past the end: the last slice again)
                v[j] = slice_lane(g, s0 + min(i0 + (w * K + j) * stride, S - 1), lane);
                mine[j] = i0 + (w * K + j) * stride < S && v[j].kind != PD_MAT_ELASTO_PLASTIC && v[j].L <= cap;
                run[j] = mine[j] && slice_active(g, v[j]);
            }
            for (int j = 0; j < K; ++j) {
                if (mine[j] && !run[j])
                    carry_slice(v[j], g.si[v[j].p >> 5], 0, 1, lane, win, wout, f, accumulate);
                if (lane == 0) todo[w * K + j] = run[j];
            }
            __syncthreads();
            for (int j = 0; j < NW * K; ++j) {
                if (!todo[j]) continue;  // the same for the whole block
                const int64_t s = s0 + i0 + j * stride;
                force_slice<NW>(g, y, mth, win, wout, f, accumulate, cap, slice_lane(g, s, lane), g.si[s], w, lane,
                                term);
                __syncthreads();  // the terms are reused
            }
            __syncthreads();  // todo is
        }
    }
}

// ---------------------------------------------------------------------
// velocity_verlet.jl:62-75: v .+= (dt/2) .* f ; y .+= dt .* v
// ---------------------------------------------------------------------
__global__ void k_kick_drift(int64_t N, double c, double dt, const double4 *__restrict__ f,
                             double4 *__restrict__ v, double4 *__restrict__ y) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= N) return;
    double4 fi = f[i], vi = v[i], yi = y[i];
    vi.x = vi.x + c * fi.x;
    vi.y = vi.y + c * fi.y;
    vi.z = vi.z + c * fi.z;
    yi.x = yi.x + dt * vi.x;
    yi.y = yi.y + dt * vi.y;
    yi.z = yi.z + dt * vi.z;
    v[i] = vi;
    y[i] = yi;
}

__global__ void k_kick(int64_t N, double c, const double4 *__restrict__ f,
                       double4 *__restrict__ v) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= N) return;
    double4 fi = f[i], vi = v[i];
    vi.x = vi.x + c * fi.x;
    vi.y = vi.y + c * fi.y;
    vi.z = vi.z + c * fi.z;
    v[i] = vi;
}

__device__ __forceinline__ double &comp(double4 &a, int d) {
    return d == 0 ? a.x : (d == 1 ? a.y : a.z);
}

// boundary_conditions.jl:107-111 with FixBC.jl:213 / ToFroBC.jl:286-289:
// position of one constrained particle, j its place in the condition's list
__device__ __forceinline__ void bc_pos_one(const BCDev &bc, int64_t j, double dt, int dir, int64_t ts, double4 &yi) {
    double4 last = bc.last[j];
    double step = dt * (double)dir;
    for (int d = 0; d < 3; ++d) {
        if (!((bc.dims >> d) & 1)) continue;
        if (bc.kind == PD_BC_FIX || bc.kind == PD_BC_SCALE_FIX_WAIT) {
            // FixBC.jl:213, ScaleFixWaitBC.jl:59 xF = (last, last)
            comp(yi, d) = comp(last, d);
        } else if (bc.kind == PD_BC_DELTA_SCALE) {
            // DeltaScaleBC.jl:52-55: (last - fix) * (1 + scale*dt*time_step) + fix
            const double g = 1.0 + (bc.scale[d] * dt) * (double)ts;
            comp(yi, d) = (comp(last, d) - bc.fix[d]) * g + bc.fix[d];
        } else {
            double nl = comp(last, d) + step * bc.rate[d];
            comp(yi, d) = nl;
            comp(last, d) = nl;
        }
    }
    if (bc.kind == PD_BC_TOFRO) bc.last[j] = last;
}

__global__ void k_bc_pos(BCDev bc, double dt, int dir, int64_t ts, double4 *__restrict__ y) {
    int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= bc.n) return;
    int32_t i = bc.idx[j];
    double4 yi = y[i];
    bc_pos_one(bc, j, dt, dir, ts, yi);
    y[i] = yi;
}

// boundary_conditions.jl:122-126 with FixBC.jl:214 / ToFroBC.jl:290
__device__ __forceinline__ void bc_vel_one(const BCDev &bc, int dir, double4 yi, double4 &vi) {
    if (bc.kind == PD_BC_CONTAINER) {
        // ContainerBC.jl:63-68: v[dims] = 0 where y left the limits
        if (!bc.has_limits) return;
        bool out = false;
        for (int d = 0; d < 3; ++d)
            if ((bc.dims >> d) & 1) out |= (comp(yi, d) < bc.lo[d]) || (comp(yi, d) > bc.hi[d]);
        if (!out) return;
        for (int d = 0; d < 3; ++d)
            if ((bc.dims >> d) & 1) comp(vi, d) = 0.0;
        return;
    }
    for (int d = 0; d < 3; ++d) {
        if (!((bc.dims >> d) & 1)) continue;
        comp(vi, d) = bc.kind == PD_BC_TOFRO ? (double)dir * bc.rate[d] : 0.0;
    }
}

__global__ void k_bc_vel(BCDev bc, int dir, const double4 *__restrict__ y, double4 *__restrict__ v) {
    int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= bc.n) return;
    int32_t i = bc.idx[j];
    double4 vi = v[i];
    bc_vel_one(bc, dir, y[i], vi);
    v[i] = vi;
}

// The elementwise part between two force evaluations in one pass (momentum
// of the last step, half kick, velocity conditions; half kick, drift,
// position conditions): the operations of the single kernels on each
// particle, in their order.  Bound by launch latency at the sizes the serial
// mode runs: a 990-particle cube took 28 us per step with the single kernels
// and 19 with this one, a 40,000-particle bar with two conditions 143 and 120.
template <bool POST, bool PRE>
__global__ void __launch_bounds__(256)
    k_advance(int64_t N, double c, double dt, const double4 *f, double4 *v,
              double4 *y, const double *__restrict__ mass, double4 *p,
              const __grid_constant__ FusedBCs b, int64_t ts) {
    const int64_t i = blockIdx.x * (int64_t)256 + threadIdx.x;
    pdl_enter();
    if (i >= N) return;
    const double4 fi = f[i];
    double4 vi = v[i], yi = y[i];
    const uint32_t bits = b.n ? b.bits[i] : 0u;
    if (POST) {
        if (p) {
            const double m = mass[i];
            p[i] = make_double4(m * vi.x, m * vi.y, m * vi.z, 0.0);
        }
        vi.x = vi.x + c * fi.x;
        vi.y = vi.y + c * fi.y;
        vi.z = vi.z + c * fi.z;
        for (int k = 0; k < b.n; ++k)
            if ((bits >> k) & 1u) bc_vel_one(b.c[k].bc, b.c[k].dir_vel, yi, vi);
    }
    if (PRE) {
        vi.x = vi.x + c * fi.x;
        vi.y = vi.y + c * fi.y;
        vi.z = vi.z + c * fi.z;
        yi.x = yi.x + dt * vi.x;
        yi.y = yi.y + dt * vi.y;
        yi.z = yi.z + dt * vi.z;
        for (int k = 0; k < b.n; ++k)
            if (((bits >> k) & 1u) && b.c[k].bc.kind != PD_BC_CONTAINER)  // (moves no particle)
                bc_pos_one(b.c[k].bc, b.c[k].rank[i - b.c[k].lo], dt, b.c[k].dir_pos, ts, yi);
        y[i] = yi;
    }
    v[i] = vi;
}

// ScaleFixWaitBC.jl:63-68 (check!): y[dims, scalebool] = (y - fix) * sqrt(1 + 2*scale*dt) + fix
__global__ void k_bc_scale(BCDev bc, double dt, double4 *__restrict__ y) {
    int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= bc.sn) return;
    const int32_t i = bc.sidx[j];
    double4 yi = y[i];
    for (int d = 0; d < 3; ++d) {
        if (!((bc.dims >> d) & 1)) continue;
        const double g = sqrt(1.0 + (2.0 * bc.scale[d]) * dt);
        comp(yi, d) = (comp(yi, d) - bc.fix[d]) * g + bc.fix[d];
    }
    y[i] = yi;
}

// FixBC.jl:63 / ToFroBC.jl:94: BC.last .= y[dims, bool]
__global__ void k_bc_snapshot(BCDev bc, const double4 *__restrict__ y) {
    int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= bc.n) return;
    double4 yi = y[bc.idx[j]], last = bc.last[j];
    for (int d = 0; d < 3; ++d)
        if ((bc.dims >> d) & 1) comp(last, d) = comp(yi, d);
    bc.last[j] = last;
}

// solvers.jl:280-285 update_misc!: p = mass .* v
__global__ void k_momentum(int64_t N, const double *__restrict__ mass,
                           const double4 *__restrict__ v, double4 *__restrict__ p) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= N) return;
    double m = mass[i];
    double4 vi = v[i];
    p[i] = make_double4(m * vi.x, m * vi.y, m * vi.z, 0.0);
}

__global__ void k_zero4(int64_t N, double4 *__restrict__ a) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= N) return;
    a[i] = make_double4(0.0, 0.0, 0.0, 0.0);
}

// ---------------------------------------------------------------------
// Deformed gate: isapprox(y .- y[:,1] .+ x[:,1], x) with rtol = sqrt(eps)
// (general_material.jl:249).  Deterministic two-stage reduction.
// ---------------------------------------------------------------------
constexpr int kGateThreads = 256;

__global__ void __launch_bounds__(kGateThreads)
    k_gate_partial(const GateItem *__restrict__ items, int gx, const double4 *__restrict__ x4,
                   const double4 *__restrict__ y, double *__restrict__ part,
                   const int32_t *__restrict__ deformed) {
    const GateItem it = items[blockIdx.y];
    double *partials = part + 3 * ((int64_t)blockIdx.y * gx);
    if (deformed[it.block]) return;
    const int64_t first = it.first, n = it.n;
    __shared__ double sh[3][kGateThreads];
    double4 y1 = y[first], x1 = x4[first];
    double sd = 0.0, sa = 0.0, sx = 0.0;
    for (int64_t l = blockIdx.x * (int64_t)kGateThreads + threadIdx.x; l < n;
         l += (int64_t)gx * kGateThreads) {
        double4 yi = y[first + l], xi = x4[first + l];
        double a0 = (yi.x - y1.x) + x1.x, a1 = (yi.y - y1.y) + x1.y, a2 = (yi.z - y1.z) + x1.z;
        double d0 = a0 - xi.x, d1 = a1 - xi.y, d2 = a2 - xi.z;
        sd = sd + d0 * d0 + d1 * d1 + d2 * d2;
        sa = sa + a0 * a0 + a1 * a1 + a2 * a2;
        sx = sx + xi.x * xi.x + xi.y * xi.y + xi.z * xi.z;
    }
    sh[0][threadIdx.x] = sd;
    sh[1][threadIdx.x] = sa;
    sh[2][threadIdx.x] = sx;
    __syncthreads();
    for (int s = kGateThreads / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s)
            for (int c = 0; c < 3; ++c) sh[c][threadIdx.x] = sh[c][threadIdx.x] + sh[c][threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int c = 0; c < 3; ++c) partials[3 * blockIdx.x + c] = sh[c][0];
}

__global__ void k_gate_final(const GateItem *__restrict__ items, int nitems, int gx,
                             const double *__restrict__ part, int32_t *__restrict__ deformed) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nitems) return;
    int32_t *flag = deformed + items[i].block;
    if (*flag) return;
    const double *partials = part + 3 * ((int64_t)i * gx);
    double sd = 0.0, sa = 0.0, sx = 0.0;
    for (int b = 0; b < gx; ++b) {
        sd = sd + partials[3 * b];
        sa = sa + partials[3 * b + 1];
        sx = sx + partials[3 * b + 2];
    }
    double d = sqrt(sd);
    const double rtol = 0x1p-26;  // sqrt(eps(Float64))
    bool approx = isfinite(d) && d <= fmax(0.0, rtol * fmax(sqrt(sa), sqrt(sx)));
    if (!approx) *flag = 1;
}

// peri.jl:587-594 cal_damage: 1 - sum(intact) / intact0
// In environment order (map), or in internal order without a map.
__global__ void k_damage(int64_t n_out, const int64_t *__restrict__ map, const SliceInfo *__restrict__ si,
                         const int32_t *__restrict__ cnt, const uint32_t *__restrict__ words,
                         const int32_t *__restrict__ intact0, const int32_t *__restrict__ tinfo,
                         double *__restrict__ damage) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= n_out) return;
    const int64_t p = map ? map[e] : e;
    if (tinfo[p] < 0) {
        damage[e] = 0.0;
        return;
    }
    int32_t n = cnt[p], c = 0;
    const int64_t wb = si[p >> 5].word + (p & 31);
    for (int32_t w = 0; w * 32 < n; ++w) c += __popc(words[wb + 32 * (int64_t)w]);
    damage[e] = 1.0 - (double)c / (double)intact0[p];
}

// Fixed partial-reduction width, independent of the device's SM count so
// that the summation order (and the rounding of the gate norms) is the same
// on every GPU.
constexpr int kSumBlocks = 148;
__global__ void __launch_bounds__(256)
    k_sum4_partial(int64_t N, const double4 *__restrict__ a, double *__restrict__ partials) {
    __shared__ double sh[3][256];
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int64_t i = blockIdx.x * 256 + threadIdx.x; i < N; i += (int64_t)kSumBlocks * 256) {
        double4 v = a[i];
        s0 = s0 + v.x;
        s1 = s1 + v.y;
        s2 = s2 + v.z;
    }
    sh[0][threadIdx.x] = s0;
    sh[1][threadIdx.x] = s1;
    sh[2][threadIdx.x] = s2;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s)
            for (int c = 0; c < 3; ++c) sh[c][threadIdx.x] = sh[c][threadIdx.x] + sh[c][threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int c = 0; c < 3; ++c) partials[3 * blockIdx.x + c] = sh[c][0];
}

__global__ void k_sum4_final(const double *__restrict__ partials, double *__restrict__ out3) {
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int b = 0; b < kSumBlocks; ++b) {
        s0 = s0 + partials[3 * b];
        s1 = s1 + partials[3 * b + 1];
        s2 = s2 + partials[3 * b + 2];
    }
    out3[0] = s0;
    out3[1] = s1;
    out3[2] = s2;
}

__global__ void k_unpack3(int64_t n, const double *__restrict__ src3,
                          const int64_t *__restrict__ map, double4 *__restrict__ dst) {
    int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= n) return;
    dst[map[e]] = make_double4(src3[3 * e], src3[3 * e + 1], src3[3 * e + 2], 0.0);
}

__global__ void k_pack3(int64_t n, const double4 *__restrict__ src,
                        const int64_t *__restrict__ map, double *__restrict__ dst3) {
    int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= n) return;
    double4 v = src[map[e]];
    dst3[3 * e] = v.x;
    dst3[3 * e + 1] = v.y;
    dst3[3 * e + 2] = v.z;
}

__global__ void k_nonfinite(int64_t N, const double4 *__restrict__ a, int32_t *__restrict__ flag) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= N) return;
    double4 v = a[i];
    if (!isfinite(v.x) || !isfinite(v.y) || !isfinite(v.z)) *flag = 1;
}

}  // namespace

// ---------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------
void launch_count_neighbors(cudaStream_t st, int64_t n, int64_t first, const double4 *x4,
                            const int32_t *cell_of, const int32_t *cell_start,
                            const int32_t *cell_list, int64_t cell_base, int3 dims,
                            double horizon, int32_t *cnt) {
    if (n <= 0) return;
    k_neighbors<false><<<grid_for(n), kThreads, 0, st>>>(n, first, x4, cell_of, cell_start,
                                                         cell_list, cell_base, dims, horizon, cnt,
                                                         nullptr, nullptr); pd::note_launch();
}

void launch_fill_neighbors(cudaStream_t st, int64_t n, int64_t first, const double4 *x4,
                           const int32_t *cell_of, const int32_t *cell_start,
                           const int32_t *cell_list, int64_t cell_base, int3 dims,
                           double horizon, const int64_t *slice_ptr, int32_t *nbr) {
    if (n <= 0) return;
    k_neighbors<true><<<grid_for(n), kThreads, 0, st>>>(n, first, x4, cell_of, cell_start,
                                                        cell_list, cell_base, dims, horizon,
                                                        nullptr, slice_ptr, nbr); pd::note_launch();
}

void launch_cell_ids(cudaStream_t st, int64_t n, int64_t first, const double4 *x4, double3 lo, double cell,
                     int3 dims, int64_t cell_base, int32_t *cell_of, int32_t *count) {
    if (n <= 0) return;
    k_cell_ids<<<grid_for(n), kThreads, 0, st>>>(n, first, x4, lo, cell, dims, cell_base, cell_of, count);
    pd::note_launch();
}

void launch_cell_scatter(cudaStream_t st, int64_t n, int64_t first, const int32_t *cell_of, int32_t *cursor,
                         int32_t *cell_list) {
    if (n <= 0) return;
    k_cell_scatter<<<grid_for(n), kThreads, 0, st>>>(n, first, cell_of, cursor, cell_list);
    pd::note_launch();
}

void launch_sort_neighbors(cudaStream_t st, int64_t N, const int64_t *slice_ptr,
                           const int32_t *cnt, int32_t *nbr) {
    k_sort_neighbors<<<grid_for(N), kThreads, 0, st>>>(N, slice_ptr, cnt, nbr); pd::note_launch();
}

void launch_init_intact(cudaStream_t st, int64_t N, const int64_t *slice_ptr,
                        const int32_t *cnt, uint32_t *words) {
    k_init_intact<<<grid_for(N), kThreads, 0, st>>>(N, slice_ptr, cnt, words); pd::note_launch();
}

void launch_layout_union(cudaStream_t st, int64_t S, int64_t N, const int64_t *slice_ptr, const int32_t *cnt,
                         const int32_t *nbr_b, int32_t force_explicit, int64_t ustride, int32_t *mode, int32_t *len,
                         int32_t *uni) {
    if (S <= 0) return;
    const int64_t threads = S * 32;
    k_layout_union<<<(unsigned)((threads + kThreads - 1) / kThreads), kThreads, 0, st>>>(
        S, N, slice_ptr, cnt, nbr_b, force_explicit, ustride, mode, len, uni);
    pd::note_launch();
}

void launch_layout_fill(cudaStream_t st, int64_t N, const int64_t *slice_ptr, const int32_t *cnt,
                        const int32_t *nbr_b, const uint32_t *w_b, const SliceInfo *si, const int32_t *ulen,
                        int64_t ustride, const int32_t *uni, int32_t *nbr, uint32_t *words, uint32_t *fam,
                        int32_t *cnt_rt) {
    if (N <= 0) return;
    k_layout_fill<<<grid_for(N), kThreads, 0, st>>>(N, slice_ptr, cnt, nbr_b, w_b, si, ulen, ustride, uni, nbr,
                                                      words, fam, cnt_rt);
    pd::note_launch();
}

void launch_popcount(cudaStream_t st, int64_t N, const SliceInfo *si, const int32_t *cnt,
                     const uint32_t *words, int32_t *out) {
    k_popcount<<<grid_for(N), kThreads, 0, st>>>(N, si, cnt, words, out); pd::note_launch();
}

void launch_weighted_volume(cudaStream_t st, const Geo &g, double2 *mth) {
    k_weighted_volume<<<grid_for(g.N), kThreads, 0, st>>>(g, mth); pd::note_launch();
}

// Sixteen warps per slice when every slice has an SM to itself, else eight:
// a 990-particle cube 26.9 against 28.3 us per step with eight, a
// 40,000-particle bar (two blocks of eight on an SM, one of sixteen) 177
// against 144 us.
static bool wide_slices(const Geo &g, int64_t slices) { return slices <= g.sms; }

void launch_theta_serial(cudaStream_t st, const Geo &g, const double4 *y, const uint32_t *win,
                         double2 *mth, const SerialRun *runs, size_t n_runs) {
    for (const SerialRun *r = runs; r < runs + n_runs; ++r) {
        const int64_t S = (r->p1 - r->p0) / 32;
        if (!r->by_slice) k_theta_serial<<<grid_for(r->p1 - r->p0), kThreads, 0, st>>>(g, y, win, mth, r->p0, r->p1);
        else if (wide_slices(g, S)) launch_dep(k_theta_slice<16>, (unsigned)S, 512, st, g, y, win, mth, r->p0 / 32);
        else launch_dep(k_theta_slice<8>, (unsigned)S, 256, st, g, y, win, mth, r->p0 / 32);
        pd::note_launch();
    }
}

void launch_td_serial(cudaStream_t st, const Geo &g, const double4 *y, const double2 *mth,
                      const uint32_t *win, uint32_t *wout, int64_t p0, int64_t p1) {
    if (p1 <= p0) return;
    k_td_serial<<<grid_for(p1 - p0), kThreads, 0, st>>>(g, y, mth, win, wout, p0, p1);
    pd::note_launch();
}

// k_force_slice may use more than the default 48 KB of shared memory; the
// limit is a setting per kernel and device, made once (with the device
// current).
static void force_slice_attrs() {
    static std::atomic<bool> done[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || done[dev].load()) return;
    const int bytes = (int)force_slice_bytes(kForceSlots);
    bool ok = true;
    for (auto kern : {k_force_slice<8, false>, k_force_slice<16, false>, k_force_slice<8, true>})
        ok &= cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
    if (ok) done[dev].store(true);
}

void launch_force_serial(cudaStream_t st, const Geo &g, const double4 *y, const double2 *mth,
                         const uint32_t *win, uint32_t *wout, double4 *f, int accumulate,
                         const SerialRun *runs, size_t n_runs, bool idle) {
    for (const SerialRun *r = runs; r < runs + n_runs; ++r) {
        const int32_t cap = !r->by_slice ? -1 : r->slots < kForceSlots ? r->slots : kForceSlots;
        const int64_t S = (r->p1 - r->p0) / 32;
        if (r->by_slice) {
            const size_t sm = force_slice_bytes(cap);
            force_slice_attrs();
            // (a few waves of blocks cost little -- 2,000 undeformed slices 46
            // against 44 us per step -- and the scanning kernel is the slower
            // one for a body that moves: 1,250 slices 95 against 85 us)
            const bool scan = idle && S > 16 * g.sms;
            const bool wide = wide_slices(g, S);
            launch_dep_smem(wide   ? k_force_slice<16, false>
                            : scan ? k_force_slice<8, true>
                                   : k_force_slice<8, false>,
                            (unsigned)(scan ? 2 * g.sms : S), wide ? 512 : 256, sm, st, g, y, mth, win, wout, f,
                            accumulate, cap, r->p0 / 32, S);
            pd::note_launch();
        }
        if (r->ep || r->slots > cap) {
            k_force_serial<<<grid_for(r->p1 - r->p0), kThreads, 0, st>>>(g, y, mth, win, wout, f, accumulate, cap,
                                                                         r->p0, r->p1);
            pd::note_launch();
        }
    }
}

void launch_advance(cudaStream_t st, int64_t N, double c, double dt, bool post, bool pre, const double4 *f,
                    double4 *v, double4 *y, const double *mass, double4 *p, const FusedBCs &bcs, int64_t ts) {
    const unsigned g = grid_for(N, 256);
    auto kern = post && pre ? k_advance<true, true> : post ? k_advance<true, false> : k_advance<false, true>;
    launch_dep(kern, g, 256, st, N, c, dt, f, v, y, mass, p, bcs, ts);
    pd::note_launch();
}

void launch_kick_drift(cudaStream_t st, int64_t N, double c, double dt, const double4 *f,
                       double4 *v, double4 *y) {
    k_kick_drift<<<grid_for(N, 256), 256, 0, st>>>(N, c, dt, f, v, y); pd::note_launch();
}

void launch_kick(cudaStream_t st, int64_t N, double c, const double4 *f, double4 *v) {
    k_kick<<<grid_for(N, 256), 256, 0, st>>>(N, c, f, v); pd::note_launch();
}

void launch_bc_pos(cudaStream_t st, const BCDev &bc, double dt, int dir, int64_t ts, double4 *y) {
    if (bc.n <= 0 || bc.kind == PD_BC_CONTAINER) return;  // ContainerBC.jl:58-61 keeps y
    k_bc_pos<<<grid_for(bc.n, 256), 256, 0, st>>>(bc, dt, dir, ts, y); pd::note_launch();
}

void launch_bc_vel(cudaStream_t st, const BCDev &bc, int dir, const double4 *y, double4 *v) {
    if (bc.n <= 0 || (bc.kind == PD_BC_CONTAINER && !bc.has_limits)) return;
    k_bc_vel<<<grid_for(bc.n, 256), 256, 0, st>>>(bc, dir, y, v); pd::note_launch();
}

void launch_bc_scale(cudaStream_t st, const BCDev &bc, double dt, double4 *y) {
    if (bc.sn > 0) {
        k_bc_scale<<<grid_for(bc.sn, 256), 256, 0, st>>>(bc, dt, y);
        pd::note_launch();
    }
    launch_bc_snapshot(st, bc, y);
}

void launch_bc_snapshot(cudaStream_t st, const BCDev &bc, const double4 *y) {
    if (bc.n <= 0) return;
    k_bc_snapshot<<<grid_for(bc.n, 256), 256, 0, st>>>(bc, y); pd::note_launch();
}

void launch_momentum(cudaStream_t st, int64_t N, const double *mass, const double4 *v,
                     double4 *p) {
    k_momentum<<<grid_for(N, 256), 256, 0, st>>>(N, mass, v, p); pd::note_launch();
}

void launch_zero4(cudaStream_t st, int64_t N, double4 *a) {
    k_zero4<<<grid_for(N, 256), 256, 0, st>>>(N, a); pd::note_launch();
}

void launch_gate_multi(cudaStream_t st, const GateItem *items, int nitems, int gx, const double4 *x4,
                       const double4 *y, double *partials, int32_t *deformed) {
    if (nitems <= 0) return;
    k_gate_partial<<<dim3(gx, nitems), kGateThreads, 0, st>>>(items, gx, x4, y, partials, deformed);
    pd::note_launch();
    k_gate_final<<<(nitems + 127) / 128, 128, 0, st>>>(items, nitems, gx, partials, deformed);
    pd::note_launch();
}

void launch_damage(cudaStream_t st, int64_t n_out, const int64_t *map, const SliceInfo *si, const int32_t *cnt,
                   const uint32_t *words, const int32_t *intact0, const int32_t *tinfo,
                   double *damage) {
    k_damage<<<grid_for(n_out), kThreads, 0, st>>>(n_out, map, si, cnt, words, intact0, tinfo, damage);
    pd::note_launch();
}

void launch_sum4(cudaStream_t st, int64_t N, const double4 *a, double *partials, double *out3) {
    k_sum4_partial<<<kSumBlocks, 256, 0, st>>>(N, a, partials); pd::note_launch();
    k_sum4_final<<<1, 1, 0, st>>>(partials, out3); pd::note_launch();
}

void launch_unpack3(cudaStream_t st, int64_t n, const double *src3, const int64_t *map,
                    double4 *dst) {
    if (n <= 0) return;
    k_unpack3<<<grid_for(n, 256), 256, 0, st>>>(n, src3, map, dst); pd::note_launch();
}

void launch_pack3(cudaStream_t st, int64_t n, const double4 *src, const int64_t *map,
                  double *dst3) {
    if (n <= 0) return;
    k_pack3<<<grid_for(n, 256), 256, 0, st>>>(n, src, map, dst3); pd::note_launch();
}

void launch_nonfinite(cudaStream_t st, int64_t N, const double4 *a, int32_t *flag) {
    k_nonfinite<<<grid_for(N, 256), 256, 0, st>>>(N, a, flag); pd::note_launch();
}

}  // namespace pd
