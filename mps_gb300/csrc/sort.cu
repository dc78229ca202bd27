// Bucket neighbour-search rebuild: the GB300 form of Bucket::storeParticles
// (src/bucket.cpp:24-51).
//
// The reference threads particles into per-cell linked lists in ascending id
// order.  Here each build is a counting sort of the particle slots by cell
// key (x-major: key = (ix * numY + iy) * numZ + iz) and a gather of every
// state array into the second buffer, in which each particle's place in its
// cell is the number of smaller ids there (the reference's in-cell order).  Ghost particles get
// the sentinel key nkeys and collect after all cells.  Roofline: HBM; per
// particle and build the gather moves ~2 x 80 B.
#include "devutil.cuh"
#include "engine.cuh"

namespace mpsg {

thread_local int32_t g_launches = 0;

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

__global__ void k_keys(Consts c, StateBuf s, int32_t* __restrict__ key, int32_t* __restrict__ rank,
                       int32_t* __restrict__ count, DevStats* ds) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= c.n) return;
    int8_t t = s.type[k];
    const int8_t t0 = t;
    count_cell(c, k, s.x[k], s.y[k], c.planar ? 0.0 : s.z[k], t, key, rank, count, ds);
    if (t != t0) s.type[k] = t;
}

__global__ void k_scatter(int n, const int32_t* __restrict__ key, const int32_t* __restrict__ rank,
                          const int32_t* __restrict__ start, const int32_t* __restrict__ id,
                          int32_t* __restrict__ perm, int32_t* __restrict__ pid) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int p = start[key[k]] + rank[k];
    perm[p] = k;
    pid[p] = id[k];
}

// Moves particle perm[p] to its place: the particles of one cell are
// perm[start .. end) in the order of their atomics; a particle counts the
// smaller ids among them (about 10 words in a row, 30 in 3-D) and goes to that
// place.  Sorting each cell by one thread instead was a kernel of its own and a
// serial chain: 6 us per build at 2,000 particles, 24 us at 1M, 71 us on a
// 17,000-particle 3-D tank.  Ghosts (after all cells) stay where they are.
__global__ void k_gather(int n, int nkeys, const int32_t* __restrict__ perm, const int32_t* __restrict__ pid,
                         const int32_t* __restrict__ start, const int32_t* __restrict__ key,
                         int32_t* __restrict__ skey, StateBuf in, StateBuf out, int planar) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int o = perm[p];
    const int32_t kk = key[o], me = pid[p];
    // the particle's fields, in flight while its place is found
    const double x = in.x[o], y = in.y[o], vx = in.vx[o], vy = in.vy[o];
    const double z = planar ? 0.0 : in.z[o], vz = planar ? 0.0 : in.vz[o];
    const double pr = in.p[o], minp = in.minp[o], ndr = in.ndr[o], nd_last = in.nd_last[o];
    const int8_t type = in.type[o], bc = in.bc[o], dir = in.dir[o];
    int k = p;
    if (kk < nkeys) {
        const int b = start[kk], e = start[kk + 1];
        k = b;
#pragma unroll 4
        for (int t = b; t < e; t++) k += pid[t] < me;
    }
    skey[k] = kk;
    out.x[k] = x;
    out.y[k] = y;
    const float xh = f32(x), yh = f32(y);
    out.xyf[k] = make_float2(xh, yh);
    // x - xh is exact in FP64 (xh is x rounded to 24 bits)
    out.xylo[k] = make_float2(f32(x - (double)xh), f32(y - (double)yh));
    out.vx[k] = vx;
    out.vy[k] = vy;
    out.vf[k] = make_float2(f32(vx), f32(vy));
    if (!planar) {
        out.z[k] = z;
        out.zf[k] = f32(z);
        out.vz[k] = vz;
    }
    out.p[k] = pr;
    out.minp[k] = minp;
    out.ndr[k] = ndr;
    out.nd_last[k] = nd_last;
    out.id[k] = me;
    out.type[k] = type;
    out.bc[k] = bc;
    out.dir[k] = dir;
}

// ---- exclusive scan (one block, or three passes: tile sums, scan of sums, tile scan) ----

__device__ __forceinline__ int block_exclusive_scan(int v, int* sh, int* total) {
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        int nw = blockDim.x >> 5;
        int t = lane < nw ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < nw) sh[lane] = t;
    }
    __syncthreads();
    int pre = (w > 0 ? sh[w - 1] : 0) + x - v;
    *total = sh[(blockDim.x >> 5) - 1];
    __syncthreads();
    return pre;
}

__global__ void k_scan_reduce(const int32_t* __restrict__ in, int n, int32_t* __restrict__ sums) {
    __shared__ int sh[32];
    int base = blockIdx.x * kScanTile;
    int s = 0;
#pragma unroll
    for (int t = 0; t < kScanItems; t++) {
        int i = base + t * kScanThreads + threadIdx.x;
        if (i < n) s += in[i];
    }
    int tot;
    block_exclusive_scan(s, sh, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

__global__ void k_scan_top(int32_t* sums, int nb) {
    __shared__ int sh[32];
    int carry = 0;
    for (int b0 = 0; b0 < nb; b0 += blockDim.x) {
        int i = b0 + threadIdx.x;
        int v = i < nb ? sums[i] : 0;
        int tot;
        int pre = block_exclusive_scan(v, sh, &tot);
        if (i < nb) sums[i] = carry + pre;
        carry += tot;
    }
}

__global__ void k_scan_apply(int32_t* in, int n, const int32_t* __restrict__ sums, int32_t* out,
                             bool clear) {
    __shared__ int sh[32];
    int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    int v[kScanItems];
    int s = 0;
#pragma unroll
    for (int t = 0; t < kScanItems; t++) {
        int i = base + t;
        v[t] = i < n ? in[i] : 0;
        s += v[t];
    }
    int tot;
    int pre = block_exclusive_scan(s, sh, &tot) + sums[blockIdx.x];
#pragma unroll
    for (int t = 0; t < kScanItems; t++) {
        int i = base + t;
        if (i < n) {
            if (clear) in[i] = 0;
            out[i] = pre;
        }
        pre += v[t];
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) out[n] = pre;
}

// One block, tiles of four items per thread in turn.
constexpr int kScanOne = 1024;
__global__ void __launch_bounds__(kScanOne) k_scan_one(int32_t* in, int n, int32_t* out, bool clear) {
    __shared__ int sh[32];
    int carry = 0;
    for (int base = 0; base < n; base += 4 * kScanOne) {
        const int i0 = base + 4 * (int)threadIdx.x;
        int v[4], s = 0;
#pragma unroll
        for (int t = 0; t < 4; t++) {
            v[t] = i0 + t < n ? in[i0 + t] : 0;
            s += v[t];
        }
        int tot;
        int pre = carry + block_exclusive_scan(s, sh, &tot);
#pragma unroll
        for (int t = 0; t < 4; t++) {
            if (i0 + t < n) {
                if (clear) in[i0 + t] = 0;
                out[i0 + t] = pre;
            }
            pre += v[t];
        }
        carry += tot;
    }
    if (threadIdx.x == 0) out[n] = carry;
}

}  // namespace

size_t scan_tmp_ints(int32_t n) { return (size_t)(n + kScanTile - 1) / kScanTile + 32; }

void launch_exclusive_scan(int32_t* in, int32_t* out, int32_t n, int32_t* tmp, bool clear,
                           cudaStream_t st) {
    // up to four tiles one block is faster than three dependent launches (9 us)
    if (n <= 16 * kScanOne) {
        k_scan_one<<<1, kScanOne, 0, st>>>(in, n, out, clear);
        ++g_launches;
        return;
    }
    int nb = (n + kScanTile - 1) / kScanTile;
    k_scan_reduce<<<nb, kScanThreads, 0, st>>>(in, n, tmp);
    ++g_launches;
    k_scan_top<<<1, 1024, 0, st>>>(tmp, nb);
    ++g_launches;
    k_scan_apply<<<nb, kScanThreads, 0, st>>>(in, n, tmp, out, clear);
    ++g_launches;
}

void launch_rebuild(const Consts& c, const StateBuf& in, const StateBuf& out, SortScratch& s,
                    DevStats* ds, cudaStream_t st, bool counted) {
    const int T = block_threads(c.n), nb = block_count(c.n);
    if (!counted) {
        k_keys<<<nb, T, 0, st>>>(c, in, s.key, s.rank, s.cell_count, ds);
        ++g_launches;
    }
    // (the scan clears the counts for the next build)
    launch_exclusive_scan(s.cell_count, s.cell_start, c.nkeys + 1, s.scan_tmp, true, st);
    k_scatter<<<nb, T, 0, st>>>(c.n, s.key, s.rank, s.cell_start, in.id, s.perm, s.pid);
    ++g_launches;
    k_gather<<<nb, T, 0, st>>>(c.n, c.nkeys, s.perm, s.pid, s.cell_start, s.key, s.skey, in, out, c.planar);
    ++g_launches;
}

}  // namespace mpsg
