// Particle-interaction kernels of the MPS step (src/mps.cpp:165-667).
//
// Every kernel works on the cell-sorted slots of the current StateBuf; the
// neighbour sweep visits candidates in the reference's order so that the
// FP64 sums (viscosity, number densities, matrix diagonal, gradient) round
// exactly like the reference's.  Roofline of this family: FP64 issue on
// GB300 (~0.5 T DFMA/s, ~52 G div or sqrt/s per GPU) for the exact sweeps,
// HBM for the list-driven ones.
#include "devutil.cuh"
#include "engine.cuh"

namespace mpsg {

namespace {

constexpr int kThreads = 256;
// Up to kRowSplit particles the sweeps run with one warp per slot range of a
// particle's 27 (9) cells: one warp for all of them leaves a scene of 17,000
// particles fewer warps than SM quarters, each bound by one particle's serial
// chain.  All of a step but the solve, one thread per particle and split: 3-D box of
// 17,343 particles 0.92 and 0.48 ms; dam of 2,162 0.19 and 0.14 (mixed), 0.23 and 0.15
// (FP64); planar tanks, mixed / FP64, of 9,190 particles 194 and 148 / 225 and 166 us,
// 16,606: 214 and 173 / 246 and 196, 20,272: 203 and 180 / 243 and 206, 23,988: 212 and
// 189 / 250 and 217, 32,173: 218 and 213 / 265 and 252, 47,688: 258 and 274 / 319 and
// 318, 93,872 mixed 348 and 396.  The gain is gone between 32,000 and 48,000; from 20,000
// on it is below 3 % of a mixed step and 1 % of an FP64 one.
constexpr int kRowSplit = 20000;
template <bool PLANAR>
constexpr int kRows = PLANAR ? 3 : 9;
// Survivors of one range that a thread keeps: at 3.1 particle distances up to 4 x 4
// columns of 6 in the middle row of a 3-D box, 4 x 6 planar.
template <bool PLANAR>
constexpr int kRowNear = PLANAR ? 64 : 128;
constexpr int kListWarps = 8;  // warps per 32 particles of the split gradient
constexpr int kCollBlocks = 304;  // blocks of the parallel collision pass (two per SM)


__device__ __forceinline__ void raise_status(DevStats* ds, int32_t bit) { atomicOr(&ds->status, bit); }

__device__ __forceinline__ bool outside_domain(const Consts& c, double x, double y, double z) {
    // MPS::checkBoundaryViolation: src/mps.cpp:643-667
    return x < c.dmin[0] || c.dmax[0] < x || y < c.dmin[1] || c.dmax[1] < y || z < c.dmin[2] ||
           c.dmax[2] < z;
}

// Visits, in sweep order, the candidates of particle k that survive the FP32
// pre-filter at `bound`: pass 1 collects them in a local list, pass 2 calls
// f(j), where f runs the exact FP64 test and the work.  Splitting the sweep
// keeps the FP64 work on compact lists, with nearly all lanes of a warp busy.
// More survivors than the list holds: f(j) for every candidate (f's exact
// test then selects the same neighbours in the same order).
template <bool PLANAR, class F>
__device__ __forceinline__ void for_each_near(const Consts& c, const StateBuf& s,
                                              const int32_t* __restrict__ cs, int32_t key, int k,
                                              float bound, F&& f) {
    constexpr int kNear = PLANAR ? 64 : 256;  // ~28 and ~120 neighbours at 3.1 particle distances
    int cand[kNear];
    int ns = 0;
    for_each_survivor<PLANAR>(c, s, cs, key, k, bound, [&](int j) {
        if (ns < kNear) cand[ns] = j;
        ns++;
    });
    if (ns <= kNear) {
        for (int q = 0; q < ns; q++) f(cand[q]);
    } else {
        for_each_candidate<PLANAR>(c, cs, key, [&](int j) {
            if (j != k) f(j);
        });
    }
}

// Number density at re_p over a particle's current neighbours (d < re_max),
// in sweep order: the value a later setNumberDensity reads from the stale
// list of a particle that has just become a ghost (src/mps.cpp:590-593).
template <bool PLANAR>
__device__ double sweep_number_density_p(const Consts& c, const StateBuf& s, const int32_t* cs,
                                         int32_t key, int k) {
    double xi = s.x[k], yi = s.y[k], zi = PLANAR ? 0.0 : s.z[k];
    double nd = 0.0;
    for_each_survivor<PLANAR>(c, s, cs, key, k, c.ft_max, [&](int j) {
        double d2 = dist2<PLANAR>(s, k, j, xi, yi, zi);
        if (lt_cut(d2, c.t_max) && lt_cut(d2, c.t_p)) nd = dadd(nd, weight(dsqrt(d2), c.re_p));
    });
    return nd;
}

// ---------------------------------------------------------------------------
// calcGravity + calcViscosity + moveParticles (+ checkBoundaryViolation),
// src/mps.cpp:165-215 and 643-667, fused with the first neighbour sweep.
// Reads `in`, writes the moved state to `out` (same slot order).  SPLIT: warp y of
// a block of 32 particles pre-filters slot range y, the warps share the survivors'
// terms, and the sums run in sweep order (the same bits).
template <bool PLANAR, bool MIXED, bool SPLIT>
__global__ void __launch_bounds__(SPLIT ? 32 * kRows<PLANAR> : kThreads) k_explicit(Consts c, StateBuf in, StateBuf out,
                                                       const int32_t* __restrict__ skey,
                                                       const int32_t* __restrict__ cs,
                                                       int32_t* __restrict__ nkey, int32_t* __restrict__ nrank,
                                                       int32_t* __restrict__ ncount, DevStats* ds) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (!SPLIT && k >= c.n) return;
    if (SPLIT) k = min(k, c.n - 1);
    int8_t t = in.type[k];
    double x = in.x[k], y = in.y[k], vx = in.vx[k], vy = in.vy[k];
    double z = PLANAR ? c.z0 : in.z[k], vz = PLANAR ? 0.0 : in.vz[k];
    double nd_last = in.nd_last[k];
    const bool fluid = t == T_FLUID;
    const int32_t key = fluid ? skey[k] : 0;
    // Mixed: FP32 weights and FP32 accumulation over the exact FP64 neighbour set.
    // The term of candidate j: velocity differences and weight (0 outside the radius).
    // Planar: the FP32 squared distance of the coordinate pairs decides outside the
    // band [fv_in, fv_out] around the threshold (its error is far inside the band),
    // the exact FP64 test inside it.
    const float2 hk = PLANAR && MIXED ? in.xyf[k] : float2{}, lk = PLANAR && MIXED ? in.xylo[k] : float2{},
                 vk = PLANAR && MIXED ? in.vf[k] : float2{};
    const float fvx = f32(vx), fvy = f32(vy), fvz = f32(vz);
    auto term = [&](int j) {
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        if constexpr (PLANAR) {
            const float2 hj = in.xyf[j], lj = in.xylo[j];
            const float dx = (hj.x - hk.x) + (lj.x - lk.x);
            const float dy = (hj.y - hk.y) + (lj.y - lk.y);
            const float d2f = dx * dx + dy * dy;
            bool inside = d2f < c.fv_in;
            if (!inside && !(d2f > c.fv_out)) {
                const double d2 = dist2<PLANAR>(in, k, j, x, y, z);
                inside = lt_cut(d2, c.t_max) && lt_cut(d2, c.t_v);
            }
            if (inside) {
                const float2 vj = in.vf[j];
                r = make_float4(vj.x - vk.x, vj.y - vk.y, 0.f, c.fre_v * rsqrtf(d2f) - 1.f);
            }
        } else {
            const double d2 = dist2<PLANAR>(in, k, j, x, y, z);
            if (lt_cut(d2, c.t_max) && lt_cut(d2, c.t_v))
                r = make_float4(f32(in.vx[j]) - fvx, f32(in.vy[j]) - fvy, f32(in.vz[j]) - fvz,
                                c.fre_v * rsqrtf(f32(d2)) - 1.f);
        }
        return r;
    };
    // FP64: the products themselves, rounded as the reference's
    auto term64 = [&](int j, double (&r)[3]) {
        r[0] = r[1] = r[2] = 0.0;
        const double d2 = dist2<PLANAR>(in, k, j, x, y, z);
        if (!(lt_cut(d2, c.t_max) && lt_cut(d2, c.t_v))) return;
        const double w = weight(dsqrt(d2), c.re_v);
        r[0] = dmul(dsub(in.vx[j], vx), w);
        r[1] = dmul(dsub(in.vy[j], vy), w);
        if (!PLANAR) r[2] = dmul(dsub(in.vz[j], vz), w);
    };
    float tx = 0.f, ty = 0.f, tz = 0.f;
    double sx = 0.0, sy = 0.0, sz = 0.0;
    auto add64 = [&](int j) {
        double r[3];
        term64(j, r);
        sx = dadd(sx, r[0]);
        sy = dadd(sy, r[1]);
        if (!PLANAR) sz = dadd(sz, r[2]);
    };
    if constexpr (SPLIT) {
        constexpr int R = kRows<PLANAR>, kShared = PLANAR ? 64 : 232;  // (48 KB in all)
        __shared__ int s_list[kShared][32], s_cnt[R][32];
        constexpr int kChunk = MIXED ? 32 : 16, D = PLANAR ? 2 : 3;
        __shared__ float4 s_term[MIXED ? kChunk : 1][32];
        __shared__ double s_term64[MIXED ? 1 : kChunk][D][32];
        __shared__ float s_sum[3][32];
        __shared__ double s_sum64[3][32];
        const int lane = threadIdx.x, row = threadIdx.y;
        int cand[kRowNear<PLANAR>], ns = 0;
        if (fluid) {
            const float2 fk = in.xyf[k];
            int b, e;
            row_range<PLANAR>(c, cs, key, row, b, e);
            survivors_of_range<PLANAR>(in, b, e, k, fk.x, fk.y, PLANAR ? 0.f : in.zf[k], c.ft_v, [&](int j) {
                if (ns < kRowNear<PLANAR>) cand[ns] = j;
                ns++;
            });
        }
        s_cnt[row][lane] = ns;
        __syncthreads();
        int at = 0, m = 0;
        for (int r = 0; r < R; r++) {
            if (r == row) at = m;
            m += s_cnt[r][lane];
        }
        if (__syncthreads_or(ns > kRowNear<PLANAR> || m > kShared)) {
            // more survivors than the lists hold: one warp, every candidate
            if (row == 0 && fluid)
                for_each_candidate<PLANAR>(c, cs, key, [&](int j) {
                    if (j == k) return;
                    if constexpr (MIXED) {
                        const float4 q = term(j);
                        tx = fmaf(q.x, q.w, tx);
                        ty = fmaf(q.y, q.w, ty);
                        tz = fmaf(q.z, q.w, tz);
                    } else {
                        add64(j);
                    }
                });
        } else {
            for (int q = 0; q < ns; q++) s_list[at + q][lane] = cand[q];
            __syncthreads();
            // a chunk of survivors at a time: the warps share the terms, then one warp
            // per component adds them in sweep order (zeros add nothing)
            const int wmax = __reduce_max_sync(0xffffffffu, m);
            float sum = 0.f;
            double sum64 = 0.0;
            for (int q0 = 0; q0 < wmax; q0 += kChunk) {
                for (int q = row; q < kChunk; q += R) {
                    const bool used = q0 + q < m;
                    if constexpr (MIXED) {
                        s_term[q][lane] = used ? term(s_list[q0 + q][lane]) : make_float4(0.f, 0.f, 0.f, 0.f);
                    } else {
                        double r[3] = {0.0, 0.0, 0.0};
                        if (used) term64(s_list[q0 + q][lane], r);
                        for (int d = 0; d < D; d++) s_term64[q][d][lane] = r[d];
                    }
                }
                __syncthreads();
                if (row < D) {
#pragma unroll 8
                    for (int q = 0; q < kChunk; q++) {
                        if constexpr (MIXED) {
                            const float* p = reinterpret_cast<const float*>(&s_term[q][lane]);
                            sum = fmaf(p[row], p[3], sum);
                        } else {
                            sum64 = dadd(sum64, s_term64[q][row][lane]);
                        }
                    }
                }
                __syncthreads();
            }
            if (MIXED && row < 3) s_sum[row][lane] = sum;
            if (!MIXED && row < 3) s_sum64[row][lane] = sum64;
            __syncthreads();
            if (MIXED) {
                tx = s_sum[0][lane];
                ty = s_sum[1][lane];
                tz = PLANAR ? 0.f : s_sum[2][lane];
            } else {
                sx = s_sum64[0][lane];
                sy = s_sum64[1][lane];
                sz = s_sum64[2][lane];
            }
        }
        if (row != 0 || blockIdx.x * blockDim.x + threadIdx.x >= c.n) return;
    } else if (MIXED && fluid) {
        for_each_near<PLANAR>(c, in, cs, key, k, c.ft_v, [&](int j) {
            const float4 q = term(j);
            tx = fmaf(q.x, q.w, tx);
            ty = fmaf(q.y, q.w, ty);
            if (!PLANAR) tz = fmaf(q.z, q.w, tz);
        });
    } else if (fluid) {
        for_each_near<PLANAR>(c, in, cs, key, k, c.ft_v, add64);
    }
    if (fluid) {
        double ax, ay, az;
        if (!MIXED) {
            ax = dadd(c.g[0], dmul(sx, c.visc_a));
            ay = dadd(c.g[1], dmul(sy, c.visc_a));
            az = PLANAR ? 0.0 : dadd(c.g[2], dmul(sz, c.visc_a));
        } else {
            ax = c.g[0] + (double)(tx * c.fvisc_a);
            ay = c.g[1] + (double)(ty * c.fvisc_a);
            az = PLANAR ? 0.0 : c.g[2] + (double)(tz * c.fvisc_a);
        }
        vx = dadd(vx, dmul(ax, c.dt));
        vy = dadd(vy, dmul(ay, c.dt));
        double nx = dadd(x, dmul(vx, c.dt));
        double ny = dadd(y, dmul(vy, c.dt));
        double nz = z;
        if (!PLANAR) {
            vz = dadd(vz, dmul(az, c.dt));
            nz = dadd(z, dmul(vz, c.dt));
        }
        if (outside_domain(c, nx, ny, nz)) {
            t = T_GHOST;
            atomicAdd(&ds->n_new_ghosts, 1);
            nd_last = sweep_number_density_p<PLANAR>(c, in, cs, key, k);
        }
        x = nx;
        y = ny;
        z = nz;
    }
    out.x[k] = x;
    out.y[k] = y;
    out.vx[k] = vx;
    out.vy[k] = vy;
    if (!PLANAR) {
        out.z[k] = z;
        out.vz[k] = vz;
    }
    count_cell(c, k, x, y, PLANAR ? 0.0 : z, t, nkey, nrank, ncount, ds);  // for the next build
    out.type[k] = t;
    out.nd_last[k] = nd_last;
    out.p[k] = in.p[k];
    out.minp[k] = in.minp[k];
    out.ndr[k] = in.ndr[k];
    out.id[k] = in.id[k];
    out.bc[k] = in.bc[k];
    out.dir[k] = in.dir[k];
}

// ---------------------------------------------------------------------------
// MPS::collision (src/mps.cpp:217-250).  The candidate pairs — fluid i,
// neighbour j with the stale distance < cd, skipping fluid j with id >= id_i
// — are found in parallel and laid out in the reference's order (ascending
// id_i, sweep order).  Their effect is order dependent (Gauss-Seidel, in
// place): pair t reads and writes the state of i and, for a fluid j, of j
// (a wall j is read but never changed: its inverse density is 0).  Pair t
// therefore depends exactly on the earlier pairs that touch i_t or a fluid
// j_t, and applying every pair after those (in any order otherwise) gives
// the serial loop's result bit for bit.  Each pair counts the earlier pairs
// touching each of its particles: for i_t its position in i_t's own run of
// pairs (no earlier pair has i_t as j: that needs id_i' > id_i_t); for j_t
// the pairs of j_t's own run (all earlier) plus the earlier pairs with the
// same j (from a short per-particle list).  A pair waits until the
// particles' counters of applied pairs reach those numbers, applies itself
// and increments them; chunks of pairs are taken in order from a ticket
// counter, so every pair waited on belongs to a running or finished block.
// More than kCollJList pairs with one j fall back to the serial pass.
template <bool PLANAR>
__device__ __forceinline__ int for_each_collision(const Consts& c, const StateBuf& s,
                                                  const int32_t* cs, int32_t key, int k,
                                                  CollPair* out, int row = -1) {
    double xi = s.x[k], yi = s.y[k], zi = PLANAR ? 0.0 : s.z[k];
    int32_t idi = s.id[k];
    int m = 0;
    auto pair = [&](int j) {
        double d2 = dist2<PLANAR>(s, k, j, xi, yi, zi);
        if (!(lt_cut(d2, c.t_max) && lt_cut(d2, c.t_cd))) return;
        if (s.type[j] == T_FLUID && s.id[j] >= idi) return;
        if (out) out[m] = CollPair{k, j, idi, s.id[j], dsqrt(d2)};
        m++;
    };
    if (row < 0) {
        for_each_survivor<PLANAR>(c, s, cs, key, k, c.ft_cd, pair);
    } else {
        const float2 fk = s.xyf[k];
        int b, e;
        row_range<PLANAR>(c, cs, key, row, b, e);
        survivors_of_range<PLANAR>(s, b, e, k, fk.x, fk.y, PLANAR ? 0.f : s.zf[k], c.ft_cd, pair);
    }
    return m;
}

template <bool PLANAR, bool SPLIT>
__global__ void __launch_bounds__(SPLIT ? 32 * kRows<PLANAR> : kThreads) k_coll_count(Consts c, StateBuf s,
                                                         const int32_t* __restrict__ skey,
                                                         const int32_t* __restrict__ cs,
                                                         int32_t* __restrict__ cnt_by_id, CollWork cw) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    int m = 0;
    if (SPLIT) {  // one warp per slot range, as k_explicit
        __shared__ int part[kRows<PLANAR>][32];
        const int lane = threadIdx.x & 31;
        if (k < c.n && s.type[k] == T_FLUID)
            m = for_each_collision<PLANAR>(c, s, cs, skey[k], k, nullptr, threadIdx.y);
        part[threadIdx.y][lane] = m;
        __syncthreads();
        if (threadIdx.y != 0) return;
        for (int r = 1; r < kRows<PLANAR>; r++) m += part[r][lane];
    }
    if (k >= c.n) return;
    if (!SPLIT && s.type[k] == T_FLUID) m = for_each_collision<PLANAR>(c, s, cs, skey[k], k, nullptr);
    // also resets the parallel pass's counters (every id once)
    const int id = s.id[k];
    cw.jn[id] = 0;
    cw.ver[id] = 0;
    if (k < 3) cw.ctl[k] = 0;
    cnt_by_id[id] = m;
}

template <bool PLANAR>
__global__ void __launch_bounds__(kThreads) k_coll_write(Consts c, StateBuf s,
                                                         const int32_t* __restrict__ skey,
                                                         const int32_t* __restrict__ cs,
                                                         const int32_t* __restrict__ cnt_by_id,
                                                         const int32_t* __restrict__ base_by_id,
                                                         CollPair* pairs, int32_t cap, CollWork cw,
                                                         DevStats* ds) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.n || s.type[k] != T_FLUID) return;
    int32_t id = s.id[k];
    if (cnt_by_id[id] == 0) return;
    int32_t b = base_by_id[id];
    if (b + cnt_by_id[id] > cap) {
        raise_status(ds, ST_CAPACITY);
        return;
    }
    const int m = for_each_collision<PLANAR>(c, s, cs, skey[k], k, pairs + b);
    if (cw.serial) return;
    // each pair with a fluid partner j: its index in j's short list
    for (int t = b; t < b + m; t++) {
        const CollPair q = pairs[t];
        if (s.type[q.sj] != T_FLUID) continue;
        const int p = atomicAdd(cw.jn + q.ij, 1);
        if (p < kCollJList)
            cw.jl[(size_t)q.ij * kCollJList + p] = t;
        else
            atomicOr(cw.ctl + 1, 1);
    }
}

// One pair of the collision loop (the body of src/mps.cpp:222-247), with
// loads and stores through L2 (other threads apply the neighbouring pairs).
// A wall or dummy j has inverse density 0: its update adds +-0, which leaves
// it unchanged unless it holds -0 (turned into +0); the parallel pass
// (WRITE_WALL false) skips that store, so that pairs sharing a wall do not
// race; walls hold no -0 (their velocities start at +0 and only such
// updates touch them), so both passes give the same state.
template <bool PLANAR, bool WRITE_WALL>
__device__ __forceinline__ void coll_apply_pair(const Consts& c, const StateBuf& s, const CollPair& q,
                                                double inv_rho) {
    const int i = q.si, j = q.sj;
    const double inv_i = inv_rho;  // i is fluid; Particle::inverseDensity, src/particle.cpp:19-29
    const bool jfluid = s.type[j] == T_FLUID;
    const bool wj = WRITE_WALL || jfluid;
    const double inv_j = jfluid ? inv_rho : 0.0;
    const double reduced = ddiv(1.0, dadd(inv_i, inv_j));
    const double xi = __ldcg(s.x + i), yi = __ldcg(s.y + i), xj = __ldcg(s.x + j), yj = __ldcg(s.y + j);
    const double dx = dsub(xj, xi), dy = dsub(yj, yi);
    double zi = 0.0, zj = 0.0;
    if (!PLANAR) {
        zi = __ldcg(s.z + i);
        zj = __ldcg(s.z + j);
    }
    const double dz = PLANAR ? 0.0 : dsub(zj, zi);
    const double z2 = dadd(dadd(dmul(dx, dx), dmul(dy, dy)), dmul(dz, dz));
    double nx = dx, ny = dy, nz = dz;
    if (z2 > 0.0) {
        const double r = dsqrt(z2);
        nx = ddiv(dx, r);
        ny = ddiv(dy, r);
        nz = ddiv(dz, r);
    }
    const double vxi = __ldcg(s.vx + i), vyi = __ldcg(s.vy + i), vxj = __ldcg(s.vx + j), vyj = __ldcg(s.vy + j);
    double vzi = 0.0, vzj = 0.0;
    if (!PLANAR) {
        vzi = __ldcg(s.vz + i);
        vzj = __ldcg(s.vz + j);
    }
    const double ux = dsub(vxj, vxi), uy = dsub(vyj, vyi);
    const double uz = PLANAR ? 0.0 : dsub(vzj, vzi);
    const double rel = dadd(dadd(dmul(ux, nx), dmul(uy, ny)), dmul(uz, nz));
    if (rel < 0.0) {
        const double impulse = dmul(dmul(-dadd(1.0, c.e), rel), reduced);
        const double ci = dmul(impulse, inv_i), cj = dmul(impulse, inv_j);
        __stcg(s.vx + i, dsub(vxi, dmul(ci, nx)));
        __stcg(s.vy + i, dsub(vyi, dmul(ci, ny)));
        if (wj) {
            __stcg(s.vx + j, dadd(vxj, dmul(cj, nx)));
            __stcg(s.vy + j, dadd(vyj, dmul(cj, ny)));
        }
        const double pimp = dmul(dsub(c.cd, q.dist), reduced);
        const double pi_ = dmul(pimp, inv_i), pj_ = dmul(pimp, inv_j);
        __stcg(s.x + i, dsub(xi, dmul(pi_, nx)));
        __stcg(s.y + i, dsub(yi, dmul(pi_, ny)));
        if (wj) {
            __stcg(s.x + j, dadd(xj, dmul(pj_, nx)));
            __stcg(s.y + j, dadd(yj, dmul(pj_, ny)));
        }
        if (!PLANAR) {
            __stcg(s.vz + i, dsub(vzi, dmul(ci, nz)));
            __stcg(s.z + i, dsub(zi, dmul(pi_, nz)));
            if (wj) {
                __stcg(s.vz + j, dadd(vzj, dmul(cj, nz)));
                __stcg(s.z + j, dadd(zj, dmul(pj_, nz)));
            }
        }
    }
}

__device__ __forceinline__ int ld_acquire_i32(const int32_t* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Polls before a pair gives up waiting (~0.3 us each: ~2.5 s in all); a pair
// that gives up raises ST_TIMEOUT and the abort flag, on which every waiting
// pair gives up at once.
constexpr int kCollSpinLimit = 1 << 23;

template <bool PLANAR>
__global__ void __launch_bounds__(kThreads) k_coll_wave(Consts c, StateBuf s, const CollPair* __restrict__ pairs,
                                                        const int32_t* __restrict__ total_p, int32_t cap,
                                                        const int32_t* __restrict__ cnt_by_id,
                                                        const int32_t* __restrict__ base_by_id, CollWork cw,
                                                        DevStats* ds) {
    const int32_t total = *total_p;
    if (blockIdx.x == 0 && threadIdx.x == 0) ds->n_cand = total;
    // more pairs than the table holds: those of the first particle that did not fit are
    // not set, and the step reports the overflow (k_coll_write)
    if (total == 0 || total > cap) return;
    const double inv_rho = ddiv(1.0, c.rho);
    if (cw.serial || *(volatile int32_t*)(cw.ctl + 1)) {
        // the serial pass: every pair in order by one thread (verification mode, or
        // when a particle is the partner of more than kCollJList pairs)
        if (blockIdx.x == 0 && threadIdx.x == 0)
            for (int32_t t = 0; t < total; t++) coll_apply_pair<PLANAR, true>(c, s, pairs[t], inv_rho);
        return;
    }
    __shared__ int s_chunk;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_chunk = atomicAdd(cw.ctl, 1);
        __syncthreads();
        const int t0 = s_chunk * (int)blockDim.x;
        if (t0 >= total) return;
        const int t = t0 + (int)threadIdx.x;
        if (t >= total) continue;
        const CollPair q = pairs[t];
        const bool jf = s.type[q.sj] == T_FLUID;
        const int ri = t - base_by_id[q.ii];
        int rj = 0;
        if (jf) {
            rj = cnt_by_id[q.ij];
            const int m = min(cw.jn[q.ij], kCollJList);
            for (int u = 0; u < m; u++) rj += cw.jl[(size_t)q.ij * kCollJList + u] < t;
        }
        bool go = true;
        for (int it = 0; ld_acquire_i32(cw.ver + q.ii) != ri || (jf && ld_acquire_i32(cw.ver + q.ij) != rj);
             it++) {
            if (*(volatile int32_t*)(cw.ctl + 2)) {
                go = false;
                break;
            }
            if (it > kCollSpinLimit) {
                atomicOr(&ds->status, ST_TIMEOUT);
                atomicExch(cw.ctl + 2, 1);
                go = false;
                break;
            }
            __nanosleep(64);
        }
        if (!go) continue;
        coll_apply_pair<PLANAR, false>(c, s, q, inv_rho);
        __threadfence();
        atomicAdd(cw.ver + q.ii, 1);
        if (jf) atomicAdd(cw.ver + q.ij, 1);
    }
}

// ---------------------------------------------------------------------------
// MPS::setNeighbors (src/mps.cpp:585-619): the neighbour list of the build
// that the pressure part uses, stored column-major (slot, FP64 distance,
// FP64 weight at re_p), plus the number density at re_p (kept per particle
// as the value a stale-list read returns once it becomes a ghost).  With BC
// (the pressure part's build) the same pass also runs setBoundaryCondition
// and the classic setSourceTerm (src/mps.cpp:262-320): the surface number
// density summed over the list entries within re_s, in list order (the
// order in which the reference's getNumberDensity reads the stored list).
template <bool PLANAR, bool BC>
__device__ __forceinline__ void list_serial(const Consts& c, const StateBuf& s, const int32_t* __restrict__ skey,
                                            const int32_t* __restrict__ cs, const NbList& nb, int k, int& m,
                                            double& nd, double& nsurf) {
    const int np = nb.n_pad;
    const double xi = s.x[k], yi = s.y[k], zi = PLANAR ? 0.0 : s.z[k];
    // Pass 1: the candidates that survive the FP32 pre-filter, in sweep
    // order.  Pass 2 then runs the exact FP64 test, square root and
    // division on these compact per-particle lists, with nearly all lanes
    // of a warp busy (a candidate survives for only part of a warp).
    int ns = 0;
    for_each_survivor<PLANAR>(c, s, cs, skey[k], k, c.ft_max, [&](int j) {
        if (ns < c.K) nb.slot[(size_t)ns * np + k] = j;
        ns++;
    });
    if (ns <= c.K) {
        // exact test, compacting in place (order kept): src/mps.cpp:585-619
        for (int q = 0; q < ns; q++) {
            const int j = nb.slot[(size_t)q * np + k];
            const double d2 = dist2<PLANAR>(s, k, j, xi, yi, zi);
            if (!lt_cut(d2, c.t_max)) continue;
            const double dist = dsqrt(d2);
            const double w = weight(dist, c.re_p);
            if (lt_cut(dist, c.re_p)) nd = dadd(nd, w);  // src/mps.cpp:573-583
            if (BC && lt_cut(dist, c.re_s)) nsurf = dadd(nsurf, weight(dist, c.re_s));
            const size_t e = (size_t)m * np + k;
            nb.slot[e] = j;
            nb.dist[e] = dist;
            nb.wp[e] = w;
            m++;
        }
    } else {
        // more survivors than the list holds: the exact one-pass sweep
        for_each_candidate<PLANAR>(c, cs, skey[k], [&](int j) {
            if (j == k) return;
            const double d2 = dist2<PLANAR>(s, k, j, xi, yi, zi);
            if (!lt_cut(d2, c.t_max)) return;
            const double dist = dsqrt(d2);
            const double w = weight(dist, c.re_p);
            if (lt_cut(dist, c.re_p)) nd = dadd(nd, w);
            if (m < c.K) {
                if (BC && lt_cut(dist, c.re_s)) nsurf = dadd(nsurf, weight(dist, c.re_s));
                const size_t e = (size_t)m * np + k;
                nb.slot[e] = j;
                nb.dist[e] = dist;
                nb.wp[e] = w;
            }
            m++;
        });
    }
}

// What follows a particle's list and sums: called by whole warps, one particle per lane.
template <bool BC>
__device__ __forceinline__ void list_finish(const Consts& c, const StateBuf& s, const NbList& nb, const Ppe& A,
                                            DevStats* ds, int k, bool valid, int m, double nd, double nsurf) {
    if (valid) s.nd_last[k] = nd;
    if (k < c.n) nb.cnt[k] = m < c.K ? m : c.K;
    if (m > c.K) raise_status(ds, ST_CAPACITY);
    if (BC) {
        int8_t bc = BC_IGNORED;
        if (k < c.n) {
            const int8_t t = s.type[k];
            if (t != T_GHOST && t != T_DUMMY) bc = nsurf < c.beta_n0s ? BC_SURFACE : BC_INNER;
            s.bc[k] = bc;
            double b = 0.0;
            if (bc == BC_INNER && !c.ho_on) b = ddiv(dmul(c.src_g1, dsub(nd, c.n0_p)), c.n0_p);
            A.src[k] = b;
        }
        const unsigned in_mask = __ballot_sync(0xffffffffu, k < c.n && bc == BC_INNER);
        const unsigned sf_mask = __ballot_sync(0xffffffffu, k < c.n && bc == BC_SURFACE);
        if ((threadIdx.x & 31) == 0) {
            if (in_mask) atomicAdd(&ds->n_inner, __popc(in_mask));
            if (sf_mask) atomicAdd(&ds->n_surface, __popc(sf_mask));
        }
    }
    // one atomic per warp for the largest neighbour count
    const int wmax = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0 && wmax > 0) atomicMax(&ds->max_neighbors, wmax);
}

template <bool PLANAR, bool BC>
__global__ void __launch_bounds__(kThreads) k_build_list(Consts c, StateBuf s,
                                                         const int32_t* __restrict__ skey,
                                                         const int32_t* __restrict__ cs, NbList nb,
                                                         Ppe A, DevStats* ds) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = k < c.n && s.type[k] != T_GHOST;
    int m = 0;
    double nd = 0.0, nsurf = 0.0;  // number densities at re_p and (BC) re_s
    if (valid) list_serial<PLANAR, BC>(c, s, skey, cs, nb, k, m, nd, nsurf);
    list_finish<BC>(c, s, nb, A, ds, k, valid, m, nd, nsurf);
}

// The same list with one warp per slot range (32 particles per block) for the
// pre-filter; then the block's warps share the survivors, each entry at the place
// that counts the survivors before it.  The few particles with a survivor that the
// exact test rejects close the gap afterwards.  A range with more survivors than a
// thread keeps, or a list longer than the table, sends the block through the serial
// form.
template <bool PLANAR, bool BC>
__global__ void __launch_bounds__(32 * kRows<PLANAR>) k_build_rows(Consts c, StateBuf s,
                                                                   const int32_t* __restrict__ skey,
                                                                   const int32_t* __restrict__ cs, NbList nb,
                                                                   Ppe A, DevStats* ds) {
    constexpr int R = kRows<PLANAR>;
    __shared__ int s_cnt[R][32], s_gap[32];
    __shared__ double s_term[2][1 + BC][32][32], s_surf[32];
    const int lane = threadIdx.x, row = threadIdx.y;
    const int k = blockIdx.x * 32 + lane;
    const bool valid = k < c.n && s.type[k] != T_GHOST;
    const int np = nb.n_pad;
    int cand[kRowNear<PLANAR>];
    int ns = 0;
    if (valid) {
        const float2 fk = s.xyf[k];
        int b, e;
        row_range<PLANAR>(c, cs, skey[k], row, b, e);
        survivors_of_range<PLANAR>(s, b, e, k, fk.x, fk.y, PLANAR ? 0.f : s.zf[k], c.ft_max, [&](int j) {
            if (ns < kRowNear<PLANAR>) cand[ns] = j;
            ns++;
        });
    }
    s_cnt[row][lane] = ns;
    if (row == 0) s_gap[lane] = 0;
    __syncthreads();
    int at = 0, m = 0;
    for (int r = 0; r < R; r++) {
        if (r == row) at = m;
        m += s_cnt[r][lane];
    }
    double nd = 0.0, nsurf = 0.0;
    if (__syncthreads_or(ns > kRowNear<PLANAR> || m > c.K)) {
        if (row != 0) return;
        m = 0;
        if (valid) list_serial<PLANAR, BC>(c, s, skey, cs, nb, k, m, nd, nsurf);
        list_finish<BC>(c, s, nb, A, ds, k, valid, m, nd, nsurf);
        return;
    }
    for (int q = 0; q < ns; q++) nb.slot[(size_t)(at + q) * np + k] = cand[q];
    __syncthreads();
    // 32 entries at a time: the warps share them, four per pass and warp, then one
    // warp per sum adds the terms in list order (src/mps.cpp:573-583; 0 outside the
    // radius, which adds nothing) while the others go on
    const int wmax = __reduce_max_sync(0xffffffffu, m);  // (the same in every warp)
    const double xi = valid ? s.x[k] : 0.0, yi = valid ? s.y[k] : 0.0, zi = PLANAR || !valid ? 0.0 : s.z[k];
    double sum = 0.0;
    bool gap = false;
    for (int q0 = 0, par = 0; q0 < wmax; q0 += 32, par ^= 1) {
        for (int b = row; b < 32; b += 4 * R) {
            int j[4];
            double dist[4], w[4], ws[4];
            bool in[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const int q = q0 + b + t * R;
                in[t] = b + t * R < 32 && q < m;
                j[t] = in[t] ? nb.slot[(size_t)q * np + k] : min(k, c.n - 1);
            }
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const double d2 = in[t] ? dist2<PLANAR>(s, k, j[t], xi, yi, zi) : 1.0;
                if (in[t] && !lt_cut(d2, c.t_max)) j[t] = -1;
                dist[t] = dsqrt(d2);
                w[t] = weight(dist[t], c.re_p);
                ws[t] = !BC ? 0.0 : (c.re_s == c.re_p ? w[t] : weight(dist[t], c.re_s));
            }
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const int q = b + t * R;
                if (q >= 32) break;
                const bool used = in[t] && j[t] >= 0;
                s_term[par][0][q][lane] = used && lt_cut(dist[t], c.re_p) ? w[t] : 0.0;
                if (BC) s_term[par][BC][q][lane] = used && lt_cut(dist[t], c.re_s) ? ws[t] : 0.0;
                if (!in[t]) continue;
                const size_t e = (size_t)(q0 + q) * np + k;
                if (!used) nb.slot[e] = -1;
                gap = gap || !used;
                nb.dist[e] = dist[t];
                nb.wp[e] = w[t];
            }
        }
        __syncthreads();
        if (row < 1 + BC) {
#pragma unroll 8
            for (int q = 0; q < 32; q++) sum = dadd(sum, s_term[par][row][q][lane]);
        }
    }
    if (gap) s_gap[lane] = 1;
    if (BC && row == 1) s_surf[lane] = sum;
    __syncthreads();
    if (row != 0) return;
    if (s_gap[lane]) {
        const int all = m;
        m = 0;
        for (int q = 0; q < all; q++) {
            const size_t e = (size_t)q * np + k, o = (size_t)m * np + k;
            if (nb.slot[e] < 0) continue;
            if (o != e) {
                nb.slot[o] = nb.slot[e];
                nb.dist[o] = nb.dist[e];
                nb.wp[o] = nb.wp[e];
            }
            m++;
        }
    }
    list_finish<BC>(c, s, nb, A, ds, k, valid, m, sum, BC ? s_surf[lane] : 0.0);
}

// Higher-order source term (src/mps.cpp:288-306), needs every neighbour's BC.
template <bool PLANAR>
__global__ void __launch_bounds__(kThreads) k_source_ho(Consts c, StateBuf s, NbList nb, Ppe A) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.n || s.bc[k] != BC_INNER) return;
    double b = dmul(c.ho_g1, dsub(s.ndr[k], 1.0));
    const double xi = s.x[k], yi = s.y[k], zi = PLANAR ? 0.0 : s.z[k];
    const double ui = s.vx[k], vi = s.vy[k], wi = PLANAR ? 0.0 : s.vz[k];
    const double cre = dmul(c.ho_c, c.re_p);
    const int np = nb.n_pad, m = nb.cnt[k];
    for (int q = 0; q < m; q++) {
        int j = nb.slot[(size_t)q * np + k];
        if (s.bc[j] == BC_IGNORED) continue;
        double dist = nb.dist[(size_t)q * np + k];
        if (!lt_cut(dist, c.re_p)) continue;
        double rx = dsub(s.x[j], xi), ry = dsub(s.y[j], yi);
        double ux = dsub(s.vx[j], ui), uy = dsub(s.vy[j], vi);
        double dot = dadd(dmul(rx, ux), dmul(ry, uy));
        if (!PLANAR) dot = dadd(dot, dmul(dsub(s.z[j], zi), dsub(s.vz[j], wi)));
        b = dsub(b, ddiv(dmul(cre, dot), dmul(dmul(dist, dist), dist)));
    }
    A.src[k] = b;
}

// MPS::setMatrix (src/mps.cpp:322-360): one SELL-32 row per Inner slot.  With
// FP also the matrix's symmetry fingerprint, from the entries as they are made
// (a pass of its own read them all again: 22 us at 2,000 particles).
template <bool FP>
__global__ void __launch_bounds__(kThreads) k_assemble(Consts c, StateBuf s, NbList nb, Ppe A,
                                                       int32_t* __restrict__ parent,
                                                       int8_t* __restrict__ has_surface, DevStats* ds) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    int off = 0;
    unsigned long long fp = 0;
    if (k < c.n) {
        parent[k] = k;  // the union-find's start (ensureDirichletBoundaryConnection)
        has_surface[k] = 0;
        double diag = 0.0;
        double rsum = 0.0;  // diag + the off-diagonals: the terms of neighbours without an unknown
        if (s.bc[k] == BC_INNER) {
            const int np = nb.n_pad, m = nb.cnt[k];
            const size_t sbase = (size_t)(k >> 5) * c.K * 32 + (k & 31);
            // four neighbours' loads and divisions at a time, sums in order
            for (int q0 = 0; q0 < m; q0 += 4) {
                int j[4];
                int8_t bj[4];
                double a[4];
                bool in[4];
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const size_t e = (size_t)min(q0 + t, m - 1) * np + k;
                    j[t] = nb.slot[e];
                    a[t] = nb.wp[e];
                    in[t] = q0 + t < m && lt_cut(nb.dist[e], c.re_p);
                }
#pragma unroll
                for (int t = 0; t < 4; t++) bj[t] = s.bc[j[t]];
#pragma unroll
                for (int t = 0; t < 4; t++) a[t] = ddiv(dmul(c.mat_c, a[t]), c.rho);
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    if (!in[t] || bj[t] == BC_IGNORED) continue;
                    diag = dadd(diag, a[t]);
                    if (bj[t] == BC_INNER) {
                        A.col[sbase + (size_t)off * 32] = j[t];
                        A.val[sbase + (size_t)off * 32] = -a[t];
                        if (FP) fp += entry_term(k, j[t], -a[t]);
                        off++;
                    } else {
                        rsum = dadd(rsum, a[t]);
                    }
                }
            }
            if (c.qc_on) {
                diag = dadd(diag, c.qc_term);
                rsum = dadd(rsum, c.qc_term);
            }
        }
        A.diag[k] = diag;
        A.rsum[k] = rsum;
        A.offcnt[k] = off;
    }
    int w = __reduce_max_sync(0xffffffffu, off);
    unsigned tot = __reduce_add_sync(0xffffffffu, (unsigned)off);
    // pad the row to the slice width with (own slot, 0) so that SpMV loops
    // need no per-entry predicate
    if (k < c.n) {
        const size_t sbase = (size_t)(k >> 5) * c.K * 32 + (k & 31);
        for (int m = off; m < w; m++) {
            A.col[sbase + (size_t)m * 32] = k;
            A.val[sbase + (size_t)m * 32] = 0.0;
        }
    }
    if ((threadIdx.x & 31) == 0 && (k >> 5) < (c.n + 31) / 32) {
        A.slice_w[k >> 5] = w;
    }
    if (FP) {
        fp = warp_sum64(fp);
        if ((threadIdx.x & 31) == 0 && fp) atomicAdd(&ds->sym_fp, fp);
    }
    if ((threadIdx.x & 31) == 0 && (k >> 5) < (c.n + 31) / 32) {
        if (tot) atomicAdd(&ds->nnz_off, (unsigned long long)tot);
    }
}

// ---------------------------------------------------------------------------
// MPS::ensureDirichletBoundaryConnection (src/mps.cpp:362-415).  The BFS
// from every Surface particle over edges with dist < re_p marks exactly the
// connected components that contain a Surface particle, so it is computed as
// a lock-free union-find over those edges.
constexpr int kUfLimit = 1 << 22;

__device__ int uf_find(int* par, int x, DevStats* ds) {
    volatile int* vp = par;
    for (int it = 0; it < kUfLimit; it++) {
        int p = vp[x];
        if (p == x) return x;
        int gp = vp[p];
        if (gp != p) vp[x] = gp;  // path halving; any ancestor is a valid parent
        x = p;
    }
    raise_status(ds, ST_TIMEOUT);
    return x;
}

__device__ void uf_union(int* par, int a, int b, DevStats* ds) {
    for (int it = 0; it < kUfLimit; it++) {
        a = uf_find(par, a, ds);
        b = uf_find(par, b, ds);
        if (a == b) return;
        if (a < b) {
            int t = a;
            a = b;
            b = t;
        }
        if (atomicCAS(par + a, a, b) == a) return;
    }
    raise_status(ds, ST_TIMEOUT);
}

// Sampled linking (the Afforest scheme of Sutton et al., 2018): almost every
// particle of a scene belongs to one large component, and its edges need not
// all be processed.  Pass 1 joins each particle to the components of its first
// kCcLinks neighbours within re_p; after full compression, the most frequent
// root of a fixed sample of particles names the large component; pass 2 runs
// every edge of each particle outside it.  Every edge with an endpoint outside
// the large component is then processed from that endpoint (the pressure
// phase's lists are symmetric and hold no ghost: ghosts are in no cell), so
// the components, and every flag derived from them, are those of processing
// all edges.
constexpr int kCcLinks = 2;
constexpr int kCcSamples = 256;  // (a wrong guess costs time only; 1,024 took 18 us to count)

__global__ void __launch_bounds__(kThreads) k_cc_link(Consts c, StateBuf s, NbList nb, int* par,
                                                      DevStats* ds) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.n || s.type[k] == T_GHOST) return;
    const int np = nb.n_pad, m = nb.cnt[k];
    int links = 0;
    for (int q = 0; q < m && links < kCcLinks; q++) {
        const size_t o = (size_t)q * np + k;
        if (lt_cut(nb.dist[o], c.re_p)) {
            uf_union(par, k, nb.slot[o], ds);
            links++;
        }
    }
}

// No unions run here, so every find returns the final root.
__global__ void k_cc_compress(int n, int* par, DevStats* ds) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) par[k] = uf_find(par, k, ds);
}

// One block: the most frequent root among kCcSamples evenly spaced
// particles (ties: the smaller root).
__global__ void k_cc_giant(int n, const int* __restrict__ par, int* giant) {
    __shared__ int roots[kCcSamples];
    __shared__ unsigned long long best;
    const int tid = threadIdx.x;
    if (tid == 0) best = 0ull;
    for (int i = tid; i < kCcSamples; i += blockDim.x)
        roots[i] = par[(int)(((long long)i * n) / kCcSamples)];
    __syncthreads();
    for (int i = tid; i < kCcSamples; i += blockDim.x) {
        int cnt = 0;
        for (int j = 0; j < kCcSamples; j++) cnt += roots[j] == roots[i];
        // larger count first, then smaller root
        const unsigned long long key =
            ((unsigned long long)cnt << 32) | (unsigned int)(0x7fffffff - roots[i]);
        atomicMax(&best, key);
    }
    __syncthreads();
    if (tid == 0) *giant = 0x7fffffff - (int)(unsigned int)(best & 0xffffffffull);
}

__global__ void __launch_bounds__(kThreads) k_cc_hook(Consts c, StateBuf s, NbList nb, int* par,
                                                      const int* giant, DevStats* ds) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.n || s.type[k] == T_GHOST) return;
    // after compression par[k] is k's root, unless a find moved it higher since
    if (((volatile int*)par)[k] == *giant) return;
    const int np = nb.n_pad, m = nb.cnt[k];
    for (int q = 0; q < m; q++) {
        const size_t o = (size_t)q * np + k;
        if (lt_cut(nb.dist[o], c.re_p)) uf_union(par, k, nb.slot[o], ds);
    }
}

__global__ void k_cc_mark(Consts c, StateBuf s, int* par, int8_t* has_surface, DevStats* ds) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.n) return;
    int r = uf_find(par, k, ds);
    if (s.bc[k] == BC_SURFACE) has_surface[r] = 1;
}

__global__ void k_cc_apply(Consts c, StateBuf s, const int* __restrict__ par,
                           const int8_t* __restrict__ has_surface, Ppe A, DevStats* ds) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.n) return;
    int r = k;
    for (int it = 0; it < kUfLimit && par[r] != r; it++) r = par[r];  // roots are final here
    int8_t conn = (s.type[k] != T_GHOST && has_surface[r]) ? 1 : 0;
    s.dir[k] = conn;
    if (!conn && s.bc[k] == BC_INNER) {
        A.rsum[k] = dadd(A.rsum[k], A.diag[k]);  // the row sum grows by the old diagonal
        A.diag[k] = dmul(A.diag[k], 2.0);
        atomicAdd(&ds->n_unconnected, 1);
    }
}

// ---------------------------------------------------------------------------
// solvePoissonEquation's scatter + removeNegativePressure (src/mps.cpp:466-479)
__global__ void k_pressure_out(int n, const double* __restrict__ x, double* __restrict__ p,
                               float2* __restrict__ pf, const int32_t* __restrict__ id,
                               double* __restrict__ x_prev, DevStats* ds) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    double v = x[k];
    if (!isfinite(v)) atomicOr(&ds->status, ST_NONFINITE);
    const double pv = v < 0.0 ? 0.0 : v;
    p[k] = pv;
    const float ph = f32(pv);
    pf[k] = make_float2(ph, f32(pv - (double)ph));  // pv - ph is exact
    if (x_prev) x_prev[id[k]] = v;
}

// MPS::setMinimumPressure (src/mps.cpp:481-503) for every particle that is
// not Ignored, then MPS::calcPressureGradient (src/mps.cpp:505-533) for the
// fluid ones, which use their own minimum: one kernel, two passes over the
// particle's list (the second mostly from cache).
template <bool PLANAR, bool MIXED, bool SPLIT>
__global__ void __launch_bounds__(kThreads) k_gradient(Consts c, StateBuf s, NbList nb, double* ax,
                                                       double* ay, double* az) {
    const int kk = blockIdx.x * blockDim.x + threadIdx.x;
    const bool on = kk < c.n && s.bc[kk] != BC_IGNORED;
    if (!SPLIT && !on) return;
    const int k = SPLIT ? min(kk, c.n - 1) : kk;
    // SPLIT: warp y takes every kListWarps-th group of four entries; the terms of 32
    // entries meet in shared memory, where one warp per component adds them in list
    // order (the same bits)
    constexpr int D = PLANAR ? 2 : 3;
    __shared__ double s_min[SPLIT ? kListWarps : 1][32];
    __shared__ float4 s_term[SPLIT && MIXED ? 4 * kListWarps : 1][32];
    __shared__ double s_term64[SPLIT && !MIXED ? 4 * kListWarps : 1][D][32];
    __shared__ float s_sum[SPLIT ? 3 : 1][32];
    __shared__ double s_sum64[SPLIT ? 3 : 1][32];
    const int lane = threadIdx.x & 31;
    const int q_first = SPLIT ? 4 * threadIdx.y : 0, q_step = SPLIT ? 4 * kListWarps : 4;
    const int np = nb.n_pad, m = on ? nb.cnt[k] : 0;
    // four neighbours' loads at a time (the columns of the list are one trip to
    // memory, the neighbours' fields a second), minima and sums in list order
    double pmin = s.p[k];
    for (int q0 = q_first; q0 < m; q0 += q_step) {
        int j[4];
        bool in[4];
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const size_t e = (size_t)min(q0 + t, m - 1) * np + k;
            j[t] = nb.slot[e];
            in[t] = q0 + t < m && lt_cut(nb.dist[e], c.re_p);
        }
        double pj[4];
#pragma unroll
        for (int t = 0; t < 4; t++) {
            pj[t] = s.p[j[t]];
            in[t] = in[t] && s.type[j[t]] != T_DUMMY;
        }
#pragma unroll
        for (int t = 0; t < 4; t++)
            if (in[t] && pmin > pj[t]) pmin = pj[t];
    }
    if (SPLIT) {
        s_min[threadIdx.y][lane] = pmin;
        __syncthreads();
        for (int r = 0; r < kListWarps; r++)
            if (pmin > s_min[r][lane]) pmin = s_min[r][lane];
    }
    if (on && (!SPLIT || threadIdx.y == 0)) s.minp[k] = pmin;
    // a fluid particle is never Ignored (only dummies and ghosts are)
    const bool fluid = on && s.type[k] == T_FLUID;
    if (!SPLIT && !fluid) return;
    // The FP32 sums of the particle's list; terms(q0, r): the coordinate differences
    // and coefficients of entries q0 .. q0 + 3 (0 for those that do not count).
    // false: another thread writes the result.
    auto sums = [&](float (&g)[3], auto&& terms) {
        float4 r[4];
        if constexpr (!SPLIT) {
            for (int q0 = 0; q0 < m; q0 += 4) {
                terms(q0, r);
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    g[0] = fmaf(r[t].x, r[t].w, g[0]);
                    g[1] = fmaf(r[t].y, r[t].w, g[1]);
                    if (!PLANAR) g[2] = fmaf(r[t].z, r[t].w, g[2]);
                }
            }
            return true;
        }
        const int mine = fluid ? m : 0, wmax = __reduce_max_sync(0xffffffffu, mine);
        const int row = threadIdx.y;
        float sum = 0.f;
        for (int q0 = 0; q0 < wmax; q0 += 4 * kListWarps) {
#pragma unroll
            for (int t = 0; t < 4; t++) r[t] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (q0 + q_first < mine) terms(q0 + q_first, r);
#pragma unroll
            for (int t = 0; t < 4; t++) s_term[q_first + t][lane] = r[t];
            __syncthreads();
            if (row < (PLANAR ? 2 : 3)) {
#pragma unroll 8
                for (int q = 0; q < 4 * kListWarps; q++) {
                    const float* p = reinterpret_cast<const float*>(&s_term[q][lane]);
                    sum = fmaf(p[row], p[3], sum);
                }
            }
            __syncthreads();
        }
        if (row < 3) s_sum[row][lane] = sum;
        __syncthreads();
        if (row != 0 || !fluid) return false;
        for (int d = 0; d < 3; d++) g[d] = s_sum[d][lane];
        return true;
    };
    const double xi = s.x[k], yi = s.y[k], zi = PLANAR ? 0.0 : s.z[k];
    if (!MIXED) {
        double gx = 0.0, gy = 0.0, gz = 0.0;
        auto terms = [&](int q0, double (&tx)[4], double (&ty)[4], double (&tz)[4]) {
            int j[4];
            double dist[4], w[4], dp[4];
            bool in[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const size_t e = (size_t)min(q0 + t, m - 1) * np + k;
                j[t] = nb.slot[e];
                dist[t] = nb.dist[e];
                w[t] = nb.wp[e];
            }
#pragma unroll
            for (int t = 0; t < 4; t++) {
                in[t] = q0 + t < m && lt_cut(dist[t], c.re_p) && s.type[j[t]] != T_DUMMY;
                dp[t] = s.p[j[t]];
                tx[t] = s.x[j[t]];
                ty[t] = s.y[j[t]];
                tz[t] = PLANAR ? 0.0 : s.z[j[t]];
            }
#pragma unroll
            for (int t = 0; t < 4; t++) {
                dp[t] = dsub(dp[t], pmin);
                const double d2 = dmul(dist[t], dist[t]);
                tx[t] = ddiv(dmul(dmul(dsub(tx[t], xi), dp[t]), w[t]), d2);
                ty[t] = ddiv(dmul(dmul(dsub(ty[t], yi), dp[t]), w[t]), d2);
                if (!PLANAR) tz[t] = ddiv(dmul(dmul(dsub(tz[t], zi), dp[t]), w[t]), d2);
            }
#pragma unroll
            for (int t = 0; t < 4; t++)
                if (!in[t]) tx[t] = ty[t] = tz[t] = 0.0;  // adds nothing
        };
        double tx[4], ty[4], tz[4];
        if constexpr (!SPLIT) {
            for (int q0 = 0; q0 < m; q0 += 4) {
                terms(q0, tx, ty, tz);
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    gx = dadd(gx, tx[t]);
                    gy = dadd(gy, ty[t]);
                    if (!PLANAR) gz = dadd(gz, tz[t]);
                }
            }
        } else {
            const int mine = fluid ? m : 0, wmax = __reduce_max_sync(0xffffffffu, mine), row = threadIdx.y;
            double sum = 0.0;
            for (int q0 = 0; q0 < wmax; q0 += 4 * kListWarps) {
#pragma unroll
                for (int t = 0; t < 4; t++) tx[t] = ty[t] = tz[t] = 0.0;
                if (q0 + q_first < mine) terms(q0 + q_first, tx, ty, tz);
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    s_term64[q_first + t][0][lane] = tx[t];
                    s_term64[q_first + t][1][lane] = ty[t];
                    if (!PLANAR) s_term64[q_first + t][D - 1][lane] = tz[t];
                }
                __syncthreads();
                if (row < D) {
#pragma unroll 8
                    for (int q = 0; q < 4 * kListWarps; q++) sum = dadd(sum, s_term64[q][row][lane]);
                }
                __syncthreads();
            }
            if (row < 3) s_sum64[row][lane] = sum;
            __syncthreads();
            if (row != 0 || !fluid) return;
            gx = s_sum64[0][lane];
            gy = s_sum64[1][lane];
            gz = s_sum64[2][lane];
        }
        gx = dmul(gx, c.grad_scale);
        gy = dmul(gy, c.grad_scale);
        ax[k] = ddiv(dmul(-1.0, gx), c.rho);
        ay[k] = ddiv(dmul(-1.0, gy), c.rho);
        if (!PLANAR) az[k] = ddiv(dmul(-1.0, dmul(gz, c.grad_scale)), c.rho);
    } else if (PLANAR) {
        // FP32 throughout: the coordinate and pressure differences from the
        // FP32 pairs (hi, lo), each within FP32 rounding of the exact
        // difference (the FP64 subtractions they replace were most of this
        // kernel's FP64 pipe time)
        float g[3] = {0.f, 0.f, 0.f};
        const float2 hk = s.xyf[k], lk = s.xylo[k];
        const float pmh = f32(pmin), pml = f32(pmin - (double)pmh);
        const bool writes = sums(g, [&](int q0, float4 (&r)[4]) {
            int j[4];
            double dist[4];
            float2 hj[4], lj[4], pj[4];
            bool in[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const size_t e = (size_t)min(q0 + t, m - 1) * np + k;
                j[t] = nb.slot[e];
                dist[t] = nb.dist[e];
            }
#pragma unroll
            for (int t = 0; t < 4; t++) {
                in[t] = q0 + t < m && lt_cut(dist[t], c.re_p) && s.type[j[t]] != T_DUMMY;
                hj[t] = s.xyf[j[t]];
                lj[t] = s.xylo[j[t]];
                pj[t] = s.pf[j[t]];
            }
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const float fd = f32(dist[t]);
                const float dp = (pj[t].x - pmh) + (pj[t].y - pml);
                const float coef = dp * (c.fre_p / fd - 1.f) / (fd * fd);
                r[t] = in[t] ? make_float4((hj[t].x - hk.x) + (lj[t].x - lk.x), (hj[t].y - hk.y) + (lj[t].y - lk.y),
                                           0.f, coef)
                             : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        });
        if (!writes) return;
        const float sc = -c.fgrad_scale / f32(c.rho);
        ax[k] = (double)(g[0] * sc);
        ay[k] = (double)(g[1] * sc);
    } else {
        float g[3] = {0.f, 0.f, 0.f};
        const bool writes = sums(g, [&](int q0, float4 (&r)[4]) {
            int j[4];
            double dist[4], dp[4], tx[4], ty[4], tz[4];
            bool in[4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const size_t e = (size_t)min(q0 + t, m - 1) * np + k;
                j[t] = nb.slot[e];
                dist[t] = nb.dist[e];
            }
#pragma unroll
            for (int t = 0; t < 4; t++) {
                in[t] = q0 + t < m && lt_cut(dist[t], c.re_p) && s.type[j[t]] != T_DUMMY;
                dp[t] = s.p[j[t]];
                tx[t] = s.x[j[t]];
                ty[t] = s.y[j[t]];
                tz[t] = s.z[j[t]];
            }
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const float fd = f32(dist[t]);
                const float coef = f32(dp[t] - pmin) * (c.fre_p / fd - 1.f) / (fd * fd);
                r[t] = in[t] ? make_float4(f32(tx[t] - xi), f32(ty[t] - yi), f32(tz[t] - zi), coef)
                             : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        });
        if (!writes) return;
        const float sc = -c.fgrad_scale / f32(c.rho);
        ax[k] = (double)(g[0] * sc);
        ay[k] = (double)(g[1] * sc);
        if (!PLANAR) az[k] = (double)(g[2] * sc);
    }
}

// moveParticlesWithPressureGradient + checkBoundaryViolation + the Courant
// number (src/mps.cpp:535-571).
template <bool PLANAR>
__global__ void __launch_bounds__(kThreads) k_move2(Consts c, StateBuf s, const double* __restrict__ ax,
                                                    const double* __restrict__ ay,
                                                    const double* __restrict__ az, DevStats* ds) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    double cour = 0.0;  // Courant numbers are >= 0: 0 is neutral for the max
    if (k < c.n && s.type[k] == T_FLUID) {
        double a0 = ax[k], a1 = ay[k];
        double vx = dadd(s.vx[k], dmul(a0, c.dt));
        double vy = dadd(s.vy[k], dmul(a1, c.dt));
        double x = dadd(s.x[k], dmul(dmul(a0, c.dt), c.dt));
        double y = dadd(s.y[k], dmul(dmul(a1, c.dt), c.dt));
        double vz = 0.0, z = c.z0;
        if (!PLANAR) {
            double a2 = az[k];
            vz = dadd(s.vz[k], dmul(a2, c.dt));
            z = dadd(s.z[k], dmul(dmul(a2, c.dt), c.dt));
            s.vz[k] = vz;
            s.z[k] = z;
        }
        s.vx[k] = vx;
        s.vy[k] = vy;
        s.x[k] = x;
        s.y[k] = y;
        if (outside_domain(c, x, y, z)) {
            s.type[k] = T_GHOST;
            atomicAdd(&ds->n_new_ghosts, 1);
        } else {
            double sp = dadd(dadd(dmul(vx, vx), dmul(vy, vy)), dmul(vz, vz));
            cour = ddiv(dmul(dsqrt(sp), c.dt), c.l0);
        }
    }
    // one atomic per warp instead of one per particle
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cour = fmax(cour, __shfl_xor_sync(0xffffffffu, cour, o));
    if ((threadIdx.x & 31) == 0 && cour > 0.0) atomic_max_nonneg_double(&ds->courant_bits, cour);
}

// MPS::setNumberDensity's ratio (src/mps.cpp:627-641)
__global__ void k_number_density(Consts c, StateBuf s) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.n) return;
    s.ndr[k] = s.bc[k] == BC_SURFACE ? 0.0 : ddiv(s.nd_last[k], c.n0_p);
}

}  // namespace

// ------------------------------------------------------------------ launchers

void launch_explicit(const Consts& c, const StateBuf& in, const StateBuf& out,
                     const SortScratch& sc, int mixed, DevStats* ds, cudaStream_t st) {
    const bool split = c.n <= kRowSplit;
    auto launch = [&](auto kernel, int rows) {
        const dim3 block = split ? dim3(32, rows) : dim3(block_threads(c.n));
        kernel<<<split ? (c.n + 31) / 32 : block_count(c.n), block, 0, st>>>(c, in, out, sc.skey, sc.cell_start, sc.key,
                                                                           sc.rank, sc.cell_count, ds);
        ++g_launches;
    };
    if (c.planar)
        launch(mixed ? (split ? k_explicit<true, true, true> : k_explicit<true, true, false>)
                     : (split ? k_explicit<true, false, true> : k_explicit<true, false, false>),
               kRows<true>);
    else
        launch(mixed ? (split ? k_explicit<false, true, true> : k_explicit<false, true, false>)
                     : (split ? k_explicit<false, false, true> : k_explicit<false, false, false>),
               kRows<false>);
}

void launch_collision(const Consts& c, const StateBuf& s, const SortScratch& sc,
                      int32_t* cand_cnt, int32_t* cand_base, const CollWork& cw, CollPair* pairs,
                      int32_t pair_cap, int32_t* scan_tmp, DevStats* ds, cudaStream_t st) {
    int nb = block_count(c.n);
    const bool split = c.n <= kRowSplit;
    auto count = [&](auto kernel, int rows) {
        const dim3 block = split ? dim3(32, rows) : dim3(block_threads(c.n));
        kernel<<<split ? (c.n + 31) / 32 : nb, block, 0, st>>>(c, s, sc.skey, sc.cell_start, cand_cnt, cw);
        ++g_launches;
    };
    if (c.planar)
        count(split ? k_coll_count<true, true> : k_coll_count<true, false>, kRows<true>);
    else
        count(split ? k_coll_count<false, true> : k_coll_count<false, false>, kRows<false>);
    launch_exclusive_scan(cand_cnt, cand_base, c.n, scan_tmp, false, st);
    const int32_t* total = cand_base + c.n;
    const int T = block_threads(c.n);
    if (c.planar) {
        k_coll_write<true><<<nb, T, 0, st>>>(c, s, sc.skey, sc.cell_start, cand_cnt, cand_base, pairs, pair_cap, cw, ds);
        k_coll_wave<true><<<kCollBlocks, kThreads, 0, st>>>(c, s, pairs, total, pair_cap, cand_cnt, cand_base, cw, ds);
    } else {
        k_coll_write<false><<<nb, T, 0, st>>>(c, s, sc.skey, sc.cell_start, cand_cnt, cand_base, pairs, pair_cap, cw,
                                              ds);
        k_coll_wave<false><<<kCollBlocks, kThreads, 0, st>>>(c, s, pairs, total, pair_cap, cand_cnt, cand_base, cw, ds);
    }
    g_launches += 2;
}

template <bool PLANAR, bool BC>
static void build_list(const Consts& c, const StateBuf& s, const SortScratch& sc, const NbList& nb, const Ppe& A,
                       DevStats* ds, cudaStream_t st) {
    if (c.n <= kRowSplit)
        k_build_rows<PLANAR, BC><<<(c.n + 31) / 32, dim3(32, kRows<PLANAR>), 0, st>>>(c, s, sc.skey, sc.cell_start, nb, A,
                                                                                   ds);
    else
        k_build_list<PLANAR, BC><<<block_count(c.n), block_threads(c.n), 0, st>>>(c, s, sc.skey, sc.cell_start, nb, A, ds);
    ++g_launches;
}

void launch_build_list(const Consts& c, const StateBuf& s, const SortScratch& sc,
                       const NbList& nb, DevStats* ds, cudaStream_t st) {
    const Ppe none{};
    if (c.planar)
        build_list<true, false>(c, s, sc, nb, none, ds, st);
    else
        build_list<false, false>(c, s, sc, nb, none, ds, st);
}

void launch_build_list_bc_source(const Consts& c, const StateBuf& s, const SortScratch& sc,
                                 const NbList& nb, const Ppe& A, DevStats* ds, cudaStream_t st) {
    if (c.planar)
        build_list<true, true>(c, s, sc, nb, A, ds, st);
    else
        build_list<false, true>(c, s, sc, nb, A, ds, st);
    if (c.ho_on) {
        const int g = block_count(c.n), T = block_threads(c.n);
        if (c.planar)
            k_source_ho<true><<<g, T, 0, st>>>(c, s, nb, A);
        else
            k_source_ho<false><<<g, T, 0, st>>>(c, s, nb, A);
        ++g_launches;
    }
}

void launch_assemble(const Consts& c, const StateBuf& s, const NbList& nb, const Ppe& A, int32_t* parent,
                     int8_t* has_surface, bool fingerprint, DevStats* ds, cudaStream_t st) {
    const int g = block_count(c.n), T = block_threads(c.n);
    if (fingerprint)
        k_assemble<true><<<g, T, 0, st>>>(c, s, nb, A, parent, has_surface, ds);
    else
        k_assemble<false><<<g, T, 0, st>>>(c, s, nb, A, parent, has_surface, ds);
    ++g_launches;
}

void launch_dirichlet(const Consts& c, const StateBuf& s, const NbList& nb, const Ppe& A,
                      int32_t* parent, int8_t* has_surface, DevStats* ds, cudaStream_t st) {
    int g = block_count(c.n);
    int* giant = parent + c.n;  // the parent array has one spare element
    k_cc_link<<<g, block_threads(c.n), 0, st>>>(c, s, nb, parent, ds);
    ++g_launches;
    k_cc_compress<<<g, block_threads(c.n), 0, st>>>(c.n, parent, ds);
    ++g_launches;
    k_cc_giant<<<1, kCcSamples, 0, st>>>(c.n, parent, giant);
    ++g_launches;
    k_cc_hook<<<g, block_threads(c.n), 0, st>>>(c, s, nb, parent, giant, ds);
    ++g_launches;
    k_cc_mark<<<g, block_threads(c.n), 0, st>>>(c, s, parent, has_surface, ds);
    ++g_launches;
    k_cc_apply<<<g, block_threads(c.n), 0, st>>>(c, s, parent, has_surface, A, ds);
    ++g_launches;
}

void launch_pressure_post(const Consts& c, const StateBuf& s, const NbList& nb, const double* x,
                          double* x_prev, double* ax, double* ay, double* az, int mixed,
                          DevStats* ds, cudaStream_t st) {
    int g = block_count(c.n);
    k_pressure_out<<<g, block_threads(c.n), 0, st>>>(c.n, x, s.p, s.pf, s.id, x_prev, ds);
    ++g_launches;
    const bool split = c.n <= kRowSplit;
    auto gradient = [&](auto kernel) {
        const dim3 block = split ? dim3(32, kListWarps) : dim3(block_threads(c.n));
        kernel<<<split ? (c.n + 31) / 32 : g, block, 0, st>>>(c, s, nb, ax, ay, az);
        ++g_launches;
    };
    if (c.planar) {
        gradient(mixed ? (split ? k_gradient<true, true, true> : k_gradient<true, true, false>)
                       : (split ? k_gradient<true, false, true> : k_gradient<true, false, false>));
        k_move2<true><<<g, block_threads(c.n), 0, st>>>(c, s, ax, ay, az, ds);
    } else {
        gradient(mixed ? (split ? k_gradient<false, true, true> : k_gradient<false, true, false>)
                       : (split ? k_gradient<false, false, true> : k_gradient<false, false, false>));
        k_move2<false><<<g, block_threads(c.n), 0, st>>>(c, s, ax, ay, az, ds);
    }
    ++g_launches;
}

void launch_number_density(const Consts& c, const StateBuf& s, const NbList& /*nb*/,
                           cudaStream_t st) {
    k_number_density<<<block_count(c.n), block_threads(c.n), 0, st>>>(c, s);
    ++g_launches;
}

void launch_initial_number_density(const Consts& c, const StateBuf& s, const SortScratch& sc,
                                   const NbList& nb, DevStats* ds, cudaStream_t st) {
    launch_build_list(c, s, sc, nb, ds, st);
    launch_number_density(c, s, nb, st);
}

}  // namespace mpsg
