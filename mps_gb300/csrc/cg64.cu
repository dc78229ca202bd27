// The FP64 pressure solve (src/mps.cpp:452-460): the Jacobi-preconditioned CG
// that Eigen's ConjugateGradient runs with its defaults (zero start, stop when
// ||r||^2 < max(tol^2 ||b||^2, DBL_MIN) on the recursive residual), over the
// SELL-32 FP64 matrix, as one persistent cooperative kernel.
//
// What bounds it.  This part issues FP64 at 1/64 of the FP32 rate: one FP64
// warp instruction holds its SM quarter for 64 cycles, so a row's ~37
// multiply-adds cost as much as its bytes at full HBM rate, and every
// reduction step counts.  Below ~100,000 rows neither bytes nor operations
// matter so much as the two exchanges between the blocks that an iteration
// cannot avoid.  Hence:
//  * rows are dealt in contiguous, equal runs of 32-row slices to as many
//    blocks as there are slices (up to one per SM), so that every SM quarter
//    issues its share of the FP64 work even for a few thousand rows;
//  * each block keeps the search direction p of its rows AND of the rows they
//    couple to (its window: the 32-row slices that its columns name) in shared
//    memory and advances all of it by itself, p = z + beta p, from the
//    published z.  Every copy of an entry has the same bits, the gathers hit
//    shared memory, and p needs neither a global array nor a grid barrier of
//    its own: two exchanges per iteration instead of three;
//  * entries address the window with 16-bit indices made once per solve (10
//    bytes per entry and iteration instead of 12); a block whose rows, matrix
//    and vectors fit shared memory beside the window keeps all of it there;
//  * an exchange is one tagged store per block and value and one polling warp
//    per value in every block (no counter, no second trip for the sums);
//    divisions run once per block, in that warp, on the integer pipe.
// Scenes of up to 4,000 rows run on one cluster of 16 blocks, whose exchange is a
// hardware barrier and stores into the other blocks' shared memory.
// A window that does not fit shared memory (very wide scenes) makes the whole
// grid gather p from global memory, with a third exchange per iteration.
#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "devutil.cuh"
#include "engine.cuh"

namespace mpsg {

namespace {

constexpr int kMaxBlocks = 160;   // blocks of an exchange: 5 slots per polling lane
constexpr int kPolls = kMaxBlocks / 32;
constexpr int kWinSlices = 1024;  // slices of a window at most (16-bit indices reach 2048)
constexpr int kListBytes = kWinSlices * 4;
constexpr int kStateWords = 9;    // FP64 words of a resident row: diagonal, its inverse, x, r, four sums, z
// Polls before an exchange gives up (~0.3 us each: ~2.4 s, far above any
// legitimate wait).
constexpr long long kSpinLimit64 = 1ll << 23;

struct Cg64Args {
    int32_t n, nslices, K;
    int32_t smem;       // dynamic shared memory of a block
    double tol;
    int64_t max_iter;
    uint16_t* lidx;     // window indices of streamed rows, quad layout (qsell_index)
};

// Exchange of M per-thread sums between all blocks.  Every block reduces its
// threads in a fixed order, stores each sum as two 8-byte words (one half of
// the value and the exchange's number in each, so a reader needs no flag and
// no order between words), and one warp per value polls the slots of all
// blocks and adds them in a fixed order: every block holds bitwise the same
// totals.  Two slot buffers in turn: a block writes a buffer again only after
// every block has published the exchange in between, which it does after it
// has read this one.  RELEASE: what the blocks stored to global memory before
// the exchange is visible after it (without it the exchange orders only the
// sums).  post(m, total) runs in value m's warp; its result reaches every
// thread in aux[m].
struct Exchange {
    unsigned long long* slots;
    unsigned int number;
    int rank, size;
    long long limit = kSpinLimit64;  // polls before an exchange gives up
};

__device__ __forceinline__ void st_slot(unsigned long long* p, unsigned long long a, unsigned long long b) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void ld_slot(const unsigned long long* p, unsigned long long& a,
                                        unsigned long long& b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}

// Sum of a (lane 0) and, with M = 2, of b (lane 16) over the warp: five FP64
// instructions for one value or two.
__device__ __forceinline__ double warp_add(double a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}
__device__ __forceinline__ double warp_add2(double a, double b, int lane) {
    const bool low = lane < 16;
    double v = low ? a : b;
    v += __shfl_xor_sync(0xffffffffu, low ? b : a, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// In a cluster (CL) the sums go straight into the other blocks' shared memory
// and its hardware barrier is both the wait and the release; the blocks of a
// cluster are always co-resident, so it needs no limit.
constexpr int kCluster64 = 16;

__device__ __forceinline__ void st_remote64(const double* local, int rank, double v) {
    unsigned a = (unsigned)__cvta_generic_to_shared(local), r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r), "d"(v) : "memory");
}
__device__ __forceinline__ double ld_remote64(const double* local, int rank) {
    unsigned a = (unsigned)__cvta_generic_to_shared(local), r;
    double v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(r) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_barrier64() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

template <int M, bool RELEASE, int BS, bool CL, class Post>
__device__ __forceinline__ bool exchange(Exchange& ex, const double (&v)[M], bool warp_has_rows,
                                         double (&tot)[M], double (&aux)[M], DevStats* ds, Post&& post) {
    constexpr int kW = BS / 32;
    static_assert(kW <= 32 && M <= 4, "one warp reduces the warps' sums; a slot holds four values");
    __shared__ double sh[M][kW];
    __shared__ double s_tot[M], s_aux[M];
    __shared__ int s_bad[M];
    __shared__ double slots[CL ? 2 : 1][M][kCluster64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if constexpr (M == 2) {
        double s = 0.0;
        if (warp_has_rows) s = warp_add2(v[0], v[1], lane);
        if ((lane & 15) == 0) sh[lane >> 4][warp] = s;
    } else {
#pragma unroll
        for (int m = 0; m < M; m++) {
            double s = 0.0;
            if (warp_has_rows) s = warp_add(v[m]);
            if (lane == 0) sh[m][warp] = s;
        }
    }
    __syncthreads();
    ex.number++;
    if constexpr (CL) {
        const int par = ex.number & 1;
        if (warp < M) {
            double s = lane < kW ? sh[warp][lane] : 0.0;
#pragma unroll
            for (int o = kW / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            // kW lanes hold the sum, at least as many as the cluster has blocks
            if (lane < ex.size) st_remote64(&slots[par][warp][ex.rank], lane, s);
        }
        cluster_barrier64();
        if (warp < M) {
            double t = lane < ex.size ? slots[par][warp][lane] : 0.0;
#pragma unroll
            for (int o = kCluster64 / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            // the same total in every lane: one that divided by a partial 0 would send
            // the warp through the FP64 division (1.3 us)
            t = __shfl_sync(0xffffffffu, t, 0);
            const double x = post((int)warp, t);
            if (lane == 0) {
                s_tot[warp] = t;
                s_aux[warp] = x;
            }
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < M; m++) {
            tot[m] = s_tot[m];
            aux[m] = s_aux[m];
        }
        return true;
    }
    if (warp < M) {
        double s = lane < kW ? sh[warp][lane] : 0.0;
#pragma unroll
        for (int o = kW / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const unsigned long long tag = (unsigned long long)ex.number << 32;
        unsigned long long* buf = ex.slots + (size_t)(ex.number & 1) * ex.size * 8 + 2 * warp;
        if (RELEASE) __threadfence();
        if (lane == 0) {
            const unsigned long long bits = (unsigned long long)__double_as_longlong(s);
            st_slot(buf + (size_t)ex.rank * 8, tag | (bits >> 32), tag | (bits & 0xffffffffull));
        }
        double part[kPolls];
        unsigned todo = 0;
#pragma unroll
        for (int u = 0; u < kPolls; u++) {
            part[u] = 0.0;
            if (lane + 32 * u < ex.size) todo |= 1u << u;
        }
        bool bad = false;
        for (long long it = 0; __any_sync(0xffffffffu, todo != 0); it++) {
            if (it > 256) {
                __nanosleep(16);
                bool stop = it > ex.limit;
                if (stop) atomicOr(&ds->status, ST_TIMEOUT);
                if ((it & 1023) == 0 && (*(volatile int*)&ds->status & ST_TIMEOUT)) stop = true;
                if (__any_sync(0xffffffffu, stop)) {
                    bad = true;
                    break;
                }
            }
            unsigned long long h[kPolls], l[kPolls];
#pragma unroll
            for (int u = 0; u < kPolls; u++)
                if (todo >> u & 1) ld_slot(buf + (size_t)(lane + 32 * u) * 8, h[u], l[u]);
#pragma unroll
            for (int u = 0; u < kPolls; u++)
                if ((todo >> u & 1) && (h[u] >> 32) == ex.number && (l[u] >> 32) == ex.number) {
                    part[u] = __longlong_as_double((long long)((h[u] << 32) | (l[u] & 0xffffffffull)));
                    todo &= ~(1u << u);
                }
        }
        if (RELEASE) __threadfence();
        double t = part[0];
#pragma unroll
        for (int u = 1; u < kPolls; u++)
            if (32 * u < ex.size) t += part[u];
        t = warp_add(t);
        const double x = post((int)warp, t);
        if (lane == 0) {
            s_tot[warp] = t;
            s_aux[warp] = x;
            s_bad[warp] = bad;
        }
    }
    __syncthreads();
    bool ok = true;
#pragma unroll
    for (int m = 0; m < M; m++) {
        tot[m] = s_tot[m];
        aux[m] = s_aux[m];
        ok = ok && !s_bad[m];
    }
    return ok;
}

// Off-diagonal sum of a streamed row over the window: two running sums, even
// and odd entries of the groups of four, the rest of the row on the first.
__device__ __forceinline__ double row_window(const double* __restrict__ vp, const ushort4* __restrict__ ip,
                                             int w, const double* __restrict__ pwin) {
    double s0 = 0.0, s1 = 0.0;
    int m = 0;
    for (; m + 8 <= w; m += 8) {
        const ushort4 a = __ldg(ip + (m >> 2) * 32), b = __ldg(ip + ((m >> 2) + 1) * 32);
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; q++) v[q] = __ldg(vp + (m + q) * 32);
        s0 = fma(v[0], pwin[a.x], s0);
        s1 = fma(v[1], pwin[a.y], s1);
        s0 = fma(v[2], pwin[a.z], s0);
        s1 = fma(v[3], pwin[a.w], s1);
        s0 = fma(v[4], pwin[b.x], s0);
        s1 = fma(v[5], pwin[b.y], s1);
        s0 = fma(v[6], pwin[b.z], s0);
        s1 = fma(v[7], pwin[b.w], s1);
    }
    if (m + 4 <= w) {
        const ushort4 a = __ldg(ip + (m >> 2) * 32);
        double v[4];
#pragma unroll
        for (int q = 0; q < 4; q++) v[q] = __ldg(vp + (m + q) * 32);
        s0 = fma(v[0], pwin[a.x], s0);
        s1 = fma(v[1], pwin[a.y], s1);
        s0 = fma(v[2], pwin[a.z], s0);
        s1 = fma(v[3], pwin[a.w], s1);
        m += 4;
    }
    if (m < w) {
        const ushort4 a = __ldg(ip + (m >> 2) * 32);
        s0 = fma(__ldg(vp + m * 32), pwin[a.x], s0);
        if (m + 1 < w) s0 = fma(__ldg(vp + (m + 1) * 32), pwin[a.y], s0);
        if (m + 2 < w) s0 = fma(__ldg(vp + (m + 2) * 32), pwin[a.z], s0);
    }
    return s0 + s1;
}

// The same sum gathered from global memory (no window).
__device__ __forceinline__ double row_gather(const double* __restrict__ vp, const int32_t* __restrict__ cp,
                                             int w, const double* x) {
    double s0 = 0.0, s1 = 0.0;
    int m = 0;
    for (; m + 4 <= w; m += 4) {
        double v[4], g[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            v[q] = __ldg(vp + (m + q) * 32);
            g[q] = __ldcg(x + __ldg(cp + (m + q) * 32));
        }
        s0 = fma(v[0], g[0], s0);
        s1 = fma(v[1], g[1], s1);
        s0 = fma(v[2], g[2], s0);
        s1 = fma(v[3], g[3], s1);
    }
    for (; m < w; m++) s0 = fma(__ldg(vp + m * 32), __ldcg(x + __ldg(cp + m * 32)), s0);
    return s0 + s1;
}

template <int BS, bool CL>
__global__ void __launch_bounds__(BS, 1) k_cg64(Ppe A, Krylov kv, Cg64Args a, DevStats* ds) {
    extern __shared__ __align__(16) unsigned char smem[];
    if (*(volatile int32_t*)&ds->status & ST_ASYMMETRIC) {  // the reference exits here
        if (threadIdx.x == 0 && blockIdx.x == 0) {
            ds->cg_iterations = 0;
            ds->refinements = 0;
            ds->cg_rel_residual = -1.0;
        }
        return;
    }
    if (CL) cluster_barrier64();  // every block runs before any stores into its shared memory
    constexpr int kW = BS / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    Exchange ex{reinterpret_cast<unsigned long long*>(kv.partials), 0u, (int)blockIdx.x, (int)gridDim.x};
    // this block's slices
    const int sl0 = (int)((int64_t)a.nslices * blockIdx.x / gridDim.x);
    const int S = (int)((int64_t)a.nslices * (blockIdx.x + 1) / gridDim.x) - sl0;
    const bool has_rows = warp < S;
    auto row_of = [&](int s) { return (sl0 + s) * 32 + lane; };

    // ---- the window: bits = the slices that this block's rows couple to (its
    // own among them), before = their running count per word of bits
    int* wl = reinterpret_cast<int*>(smem);
    double* pwin = reinterpret_cast<double*>(smem + kListBytes);
    const int nwords = (a.nslices + 31) >> 5;
    const bool room = kListBytes + (size_t)nwords * 8 <= (size_t)a.smem;
    unsigned* bits = reinterpret_cast<unsigned*>(smem + a.smem) - nwords;
    int* before = reinterpret_cast<int*>(bits) - nwords;
    __shared__ int s_count, s_wmax;
    if (tid == 0) {
        s_count = kWinSlices + 1;
        s_wmax = 0;
    }
    if (room)
        for (int k = tid; k < nwords; k += BS) bits[k] = 0u;
    __syncthreads();
    if (room) {
        int wm = 0;
        for (int s = warp; s < S; s += kW) {
            const int w = __ldg(A.slice_w + sl0 + s), i = row_of(s);
            wm = max(wm, w);
            if (lane == 0) atomicOr(bits + ((sl0 + s) >> 5), 1u << ((sl0 + s) & 31));
            const int32_t* cp = A.col + (size_t)(sl0 + s) * a.K * 32 + lane;
            for (int m = 0; m < w && i < a.n; m++) {
                const int c = __ldg(cp + m * 32) >> 5;
                const unsigned b = 1u << (c & 31);
                if (!(*(volatile unsigned*)(bits + (c >> 5)) & b)) atomicOr(bits + (c >> 5), b);
            }
        }
        if (lane == 0 && wm > 0) atomicMax(&s_wmax, wm);
        __syncthreads();
        if (warp == 0) {
            int carry = 0;
            for (int k0 = 0; k0 < nwords; k0 += 32) {
                const int c = k0 + lane < nwords ? __popc(bits[k0 + lane]) : 0;
                int x = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                if (k0 + lane < nwords) before[k0 + lane] = carry + x - c;
                carry += __shfl_sync(0xffffffffu, x, 31);
            }
            if (lane == 0) s_count = carry;
        }
        __syncthreads();
    }
    const int cnt = s_count;
    const bool over = cnt > kWinSlices || kListBytes + cnt * 256 > a.smem;
    auto slot_of = [&](int slice) {
        return before[slice >> 5] + __popc(bits[slice >> 5] & ((1u << (slice & 31)) - 1u));
    };
    // resident: matrix and vectors of the rows behind the window, below bits
    const int wq = (s_wmax + 3) & ~3;
    double* state = pwin + cnt * 32;
    double* rval = state + S * 32 * kStateWords;
    uint16_t* ridx = reinterpret_cast<uint16_t*>(rval + (size_t)S * 32 * wq);
    const bool resident = !over && (size_t)kListBytes + (size_t)cnt * 256 + (size_t)S * 32 * (kStateWords * 8 + wq * 10) +
                                           (size_t)nwords * 8 <= (size_t)a.smem;
    double *sd = state, *si = sd + S * 32, *sx = si + S * 32, *sr = sx + S * 32, *s_sum = sr + S * 32,
           *sz = s_sum + 4 * S * 32;
    // A cluster whose blocks are all resident publishes z in its blocks' shared
    // memory: the window reads the owner's copy, and the exchange's barrier has no
    // global stores to wait for.  src = where a block's z array lies (its offset
    // depends on the block's window), one word per block.
    __shared__ int s_src[kCluster64];
    bool zshared = false;
    if constexpr (CL) {
        const int mine = resident ? (int)(reinterpret_cast<unsigned char*>(sz) - smem) : -1;
        if (warp == 0 && lane < ex.size) {
            unsigned d = (unsigned)__cvta_generic_to_shared(&s_src[ex.rank]), r;
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(d), "r"(lane));
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(r), "r"(mine) : "memory");
        }
        cluster_barrier64();
        zshared = true;
        for (int q = 0; q < ex.size; q++) zshared = zshared && s_src[q] >= 0;
    }
    int own = 0;  // window index of this block's first row (its slices follow one another)
    if (!over) {
        own = slot_of(sl0) * 32;
        for (int s = warp; s < S; s += kW) {
            const int w = __ldg(A.slice_w + sl0 + s), i = row_of(s);
            const size_t e0 = (size_t)(sl0 + s) * a.K * 32 + lane;
            for (int m0 = 0; m0 < w; m0 += 4) {
                ushort4 q4 = make_ushort4(0, 0, 0, 0);
                uint16_t q[4] = {0, 0, 0, 0};
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const int m = m0 + t;
                    if (m >= w || i >= a.n) continue;
                    const int c = __ldg(A.col + e0 + (size_t)m * 32);
                    q[t] = (uint16_t)(slot_of(c >> 5) * 32 + (c & 31));
                    if (resident) rval[(s * wq + m) * 32 + lane] = __ldg(A.val + e0 + (size_t)m * 32);
                }
                q4 = make_ushort4(q[0], q[1], q[2], q[3]);
                if (resident)
                    reinterpret_cast<ushort4*>(ridx)[(s * (wq >> 2) + (m0 >> 2)) * 32 + lane] = q4;
                else
                    reinterpret_cast<ushort4*>(a.lidx)[qsell_index((sl0 + s) * 32 + lane, m0, a.K) >> 2] = q4;
            }
        }
        for (int k = tid; k < nwords; k += BS) {
            unsigned b = bits[k];
            for (int pos = before[k]; b; b &= b - 1, pos++) {
                const int slice = k * 32 + __ffs(b) - 1;
                if (CL && zshared) {  // owner and first byte of the slice's z there
                    const int q = (int)(((int64_t)(slice + 1) * gridDim.x - 1) / a.nslices);
                    const int first = (int)((int64_t)a.nslices * q / gridDim.x);
                    wl[pos] = q << 20 | (s_src[q] + (slice - first) * 256);
                } else {
                    wl[pos] = slice;
                }
            }
        }
    }
    __syncthreads();  // bits and before are free: a streamed block's window may cover them
    if (!over)
        for (int k = tid; k < cnt * 32; k += BS) pwin[k] = 0.0;

    const int parts = 4 * S <= kW ? 4 : 2;  // warps per slice of a resident block's products

    // ---- x = 0, r = b, z = D^-1 r (published, rows past n as 0)
    double acc[3] = {0.0, 0.0, over ? 1.0 : 0.0}, tot[3], aux[3];
    for (int s = warp; s < S; s += kW) {
        const int i = row_of(s), l = s * 32 + lane;
        double d = 0.0, b = 0.0;
        if (i < a.n) {
            d = A.diag[i];
            b = A.src[i];
        }
        const double inv = d != 0.0 ? ddiv(1.0, d) : 1.0;
        const double z = inv * b;
        if (CL && zshared)
            sz[l] = z;
        else
            __stcg(kv.z + i, z);
        kv.inv_diag[i] = inv;
        kv.x[i] = 0.0;
        kv.r[i] = b;
        __stcg(kv.p + i, 0.0);
        if (resident) {
            sd[l] = d;
            si[l] = inv;
            sx[l] = 0.0;
            sr[l] = b;
        }
        acc[0] = fma(b, b, acc[0]);
        acc[1] = fma(b, z, acc[1]);
    }
    // no rows: the block still tells whether its (empty) window fits
    auto none = [](int, double) { return 0.0; };
    if (!exchange<3, true, BS, CL>(ex, acc, has_rows, tot, aux, ds, none)) return;
    const double rhs2 = tot[0];
    const bool gather = tot[2] > 0.0;
    double rn2 = rhs2, rz = tot[1], beta = 0.0;
    const double thr = fmax(a.tol * a.tol * rhs2, DBL_MIN);
    int64_t it = 0;
    bool conv = rhs2 > 0.0 ? rn2 < thr : true;
    while (!conv && it < a.max_iter) {
        // ---- p = z + beta p on the window, q = A p and p.q on the own rows
        double pq[1] = {0.0}, t1[1], x1[1];
        if (!gather) {
            if (CL && zshared) {
                for (int k = tid; k < cnt * 32; k += BS) {
                    const int w = wl[k >> 5];
                    const double* z = reinterpret_cast<const double*>(smem + (w & 0xfffff)) + (k & 31);
                    pwin[k] = fma(beta, pwin[k], ld_remote64(z, w >> 20));
                }
            } else {
                for (int k = tid; k < cnt * 32; k += BS)
                    pwin[k] = fma(beta, pwin[k], __ldcg(kv.z + wl[k >> 5] * 32 + (k & 31)));
            }
            __syncthreads();
            if (resident) {
                // two or four warps per slice, each every second or fourth entry: a
                // shorter chain of dependent multiply-adds (~120 cycles each), as long
                // as every part has a warp of its own (22,000 rows, 5 slices per block:
                // 8.4 us per iteration in halves, 8.8 in quarters; 6,000 rows: 8.3, 8.0)
                for (int t = warp; t < parts * S; t += kW) {
                    const int s = t / parts, part = t & (parts - 1);
                    const int w = __ldg(A.slice_w + sl0 + s), i = row_of(s);
                    const double* vp = rval + (size_t)s * wq * 32 + lane;
                    const uint16_t* ip = ridx + ((size_t)s * wq * 32 + lane * 4);
                    double sum = 0.0;
                    if (i < a.n) {
#pragma unroll 4
                        for (int m = part; m < w; m += parts)
                            sum = fma(vp[m * 32], pwin[ip[(m & ~3) * 32 + (m & 3)]], sum);
                    }
                    s_sum[(part * S + s) * 32 + lane] = sum;
                }
                __syncthreads();
                for (int s = warp; s < S; s += kW) {
                    const int l = s * 32 + lane;
                    const double p = pwin[own + l];
                    double o = s_sum[l] + s_sum[S * 32 + l];
                    if (parts == 4) o += s_sum[2 * S * 32 + l] + s_sum[3 * S * 32 + l];
                    const double q = fma(sd[l], p, o);
                    s_sum[l] = q;
                    pq[0] = fma(p, q, pq[0]);
                }
            } else {
                for (int s = warp; s < S; s += kW) {
                    const int i = row_of(s);
                    if (i >= a.n) continue;
                    const int w = __ldg(A.slice_w + sl0 + s);
                    const double p = pwin[own + s * 32 + lane];
                    const double q = fma(__ldg(A.diag + i), p,
                                         row_window(A.val + (size_t)(sl0 + s) * a.K * 32 + lane,
                                                    reinterpret_cast<const ushort4*>(a.lidx) +
                                                        (qsell_index(i, 0, a.K) >> 2),
                                                    w, pwin));
                    kv.q[i] = q;
                    pq[0] = fma(p, q, pq[0]);
                }
            }
        } else {
            for (int s = warp; s < S; s += kW) {
                const int i = row_of(s);
                if (i < a.n) __stcg(kv.p + i, fma(beta, __ldcg(kv.p + i), __ldcg(kv.z + i)));
            }
            double none1[1] = {0.0};
            if (!exchange<1, true, BS, CL>(ex, none1, false, t1, x1, ds, none)) return;
            for (int s = warp; s < S; s += kW) {
                const int i = row_of(s);
                if (i >= a.n) continue;
                const int w = __ldg(A.slice_w + sl0 + s);
                const double p = __ldcg(kv.p + i);
                const size_t e0 = (size_t)(sl0 + s) * a.K * 32 + lane;
                const double q = fma(__ldg(A.diag + i), p, row_gather(A.val + e0, A.col + e0, w, kv.p));
                kv.q[i] = q;
                pq[0] = fma(p, q, pq[0]);
            }
        }
        if (!exchange<1, false, BS, CL>(ex, pq, has_rows, t1, x1, ds,
                                    [&](int, double t) { return ddiv(rz, t); }))
            return;
        const double alpha = x1[0];
        // ---- x += alpha p, r -= alpha q, z = D^-1 r
        double a2[2] = {0.0, 0.0}, t2[2], x2[2];
        if (!gather && resident) {
            for (int s = warp; s < S; s += kW) {
                const int l = s * 32 + lane;
                const double r = fma(-alpha, s_sum[l], sr[l]);
                const double z = si[l] * r;
                if (CL && zshared)
                    sz[l] = z;
                else
                    __stcg(kv.z + row_of(s), z);
                sr[l] = r;
                sx[l] = fma(alpha, pwin[own + l], sx[l]);
                a2[0] = fma(r, r, a2[0]);
                a2[1] = fma(r, z, a2[1]);
            }
        } else {
            for (int s = warp; s < S; s += kW) {
                const int i = row_of(s);
                if (i >= a.n) continue;
                const double p = gather ? __ldcg(kv.p + i) : pwin[own + s * 32 + lane];
                const double q = kv.q[i], x = kv.x[i], r0 = kv.r[i], inv = kv.inv_diag[i];
                kv.x[i] = fma(alpha, p, x);
                const double r = fma(-alpha, q, r0);
                kv.r[i] = r;
                const double z = inv * r;
                __stcg(kv.z + i, z);
                a2[0] = fma(r, r, a2[0]);
                a2[1] = fma(r, z, a2[1]);
            }
        }
        if (!exchange<2, true, BS, CL>(ex, a2, has_rows, t2, x2, ds, [&](int m, double t) {
                return m == 0 ? (t < thr ? 1.0 : 0.0) : ddiv(t, rz);
            }))
            return;
        rn2 = t2[0];
        if (__double_as_longlong(x2[0]) != 0) {
            conv = true;
            break;
        }
        beta = x2[1];
        rz = t2[1];
        it++;
    }
    if (resident && !gather)  // (where the grid gathers, every block works on the global arrays)
        for (int s = warp; s < S; s += kW)
            if (row_of(s) < a.n) kv.x[row_of(s)] = sx[s * 32 + lane];
    if (CL) cluster_barrier64();  // no block leaves while another may still store into its slots
    if (blockIdx.x == 0 && tid == 0) {
        ds->cg_iterations = it;
        ds->refinements = 0;
        ds->cg_rel_residual = rhs2 > 0.0 ? sqrt(rn2 / rhs2) : 0.0;
        if (!conv) atomicOr(&ds->status, ST_NOT_CONVERGED);
    }
}

// One exchange in a group that counts a block more than the launch has.
__global__ void __launch_bounds__(512) k_selftest_exchange(unsigned long long* slots, unsigned int* gave_up,
                                                          DevStats* ds) {
    Exchange ex{slots, 0u, (int)blockIdx.x, (int)gridDim.x + 1, 1ll << 16};
    double tot[2], aux[2];
    const double v[2] = {1.0, 2.0};
    const bool ok = exchange<2, true, 512, false>(ex, v, true, tot, aux, ds, [](int, double) { return 0.0; });
    if (threadIdx.x == 0 && !ok) atomicAdd(gave_up, 1u);
}

// Dynamic shared memory of a block: all of an SM's but the static arrays above.
constexpr int kSmem64 = 224 * 1024;
// More slices per block than this: 1024 threads (their loads are in flight
// together); fewer: 512 (cheaper block barriers).
constexpr int kWideSlices = 32;

// Largest scene of the one-cluster form (16 SMs issue all the FP64 work), per iteration
// against one block per SM: 5.5 and 7.5 us at 2,006 rows, 6.4 and 7.6 at 3,172, 6.9 and
// 7.7 at 4,078, 8.0 and 7.9 at 4,805, 8.5 and 8.1 at 5,902, 10.2 and 8.0 at 8,068.
constexpr int kClusterRows64 = 4000;

template <int BS>
int grid64(int device) {
    const void* fn = (const void*)k_cg64<BS, false>;
    int sms = 0, per = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem64) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, BS, kSmem64) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return std::min(sms * std::min(per, 1), kMaxBlocks);
}

}  // namespace

void launch_selftest_exchange(int blocks, unsigned long long* slots, unsigned int* gave_up, DevStats* ds) {
    k_selftest_exchange<<<blocks, 512>>>(slots, gave_up, ds);
}

int cg64_grid(int device) { return std::min(grid64<512>(device), grid64<1024>(device)); }

namespace {
void cluster_launch64(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& at, int blocks, cudaStream_t st) {
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(512);
    cfg.dynamicSmemBytes = kSmem64;
    cfg.stream = st;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = blocks;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
}
}  // namespace

int cg64_cluster() {
    const void* fn = (const void*)k_cg64<512, true>;
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem64);
    cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    for (int blocks = kCluster64; blocks >= 8; blocks /= 2) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[1];
        cluster_launch64(cfg, at[0], blocks, nullptr);
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, fn, &cfg) == cudaSuccess && fit > 0) return blocks;
        cudaGetLastError();
    }
    return 0;
}

void launch_solve_fp64(const Consts& c, const Ppe& A, const Krylov& k, double tol, int64_t max_iter,
                       DevStats* ds, cudaStream_t st) {
    Cg64Args a;
    a.n = c.n;
    a.nslices = (c.n + 31) / 32;
    a.K = c.K;
    a.smem = kSmem64;
    a.tol = tol;
    a.max_iter = max_iter;
    a.lidx = reinterpret_cast<uint16_t*>(A.val32);  // the mixed solver's values: not used by this one
    Ppe AA = A;
    Krylov kk = k;
    void* args[] = {&AA, &kk, &a, &ds};
    ++g_launches;
    if (k.cluster64 > 0 && c.n <= kClusterRows64) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[1];
        int blocks = k.cluster64;  // a power of two, no more than there are slices
        while (blocks > a.nslices) blocks /= 2;
        cluster_launch64(cfg, at[0], blocks, st);
        cudaLaunchKernelExC(&cfg, (const void*)k_cg64<512, true>, args);
        return;
    }
    const int grid = std::min(k.grid, a.nslices);
    cudaMemsetAsync(k.partials, 0, sizeof(unsigned long long) * 16 * grid, st);
    const bool wide = a.nslices > kWideSlices * grid;
    const void* fn = wide ? (const void*)k_cg64<1024, false> : (const void*)k_cg64<512, false>;
    cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(wide ? 1024 : 512), args, kSmem64, st);
}

}  // namespace mpsg
