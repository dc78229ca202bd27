// Setup of the aggregation multigrid preconditioner used by the mixed
// pressure solver (the V-cycle itself runs inside the mixed solves, solver.cu).
//
// Level 1: one unknown per bucket cell (numX x numY, cell index
// cx * numY + cy, the planar cell key).  Its operator is the Galerkin
// product P^T A P of the FP32 particle matrix with piecewise-constant P over
// the Inner particles of each cell; since a particle couples only to the
// 3x3 cells around its own, the result is a 9-point stencil.  Level l+1
// aggregates 2x2 cells of level l, again a 9-point stencil.  Every coarse
// entry is summed by one thread in a fixed order, so the hierarchy is
// deterministic.  The coarsest level gets an explicit inverse (Gauss-Jordan
// without pivoting: the Galerkin operator of an SPD matrix is SPD).
#include "devutil.cuh"
#include "engine.cuh"

namespace mpsg {

namespace {

// Adds v to stencil entry d, the nine entries kept in registers (an
// indexed local array would live in local memory); the other entries add
// +0, which leaves them unchanged, so the sums equal one indexed add.
__device__ __forceinline__ void add_tap(float (&st)[9], int d, float v) {
#pragma unroll
    for (int q = 0; q < 9; q++) st[q] += q == d ? v : 0.f;
}

// Appends cell I to the level's list of cells with unknowns: one atomic per
// warp, the warp's cells in ascending order.
// Returns the entry's position (-1 for a cell that is not listed).
__device__ __forceinline__ int list_active(bool act, int I, int32_t* list, int32_t* count) {
    const unsigned am = __activemask();
    const unsigned m = __ballot_sync(am, act);
    if (!m) return -1;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(m) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(count, __popc(m));
    base = __shfl_sync(am, base, leader);
    const int pos = base + __popc(m & ((1u << lane) - 1u));
    if (act) list[pos] = I;
    return act ? pos : -1;
}

// Level 1's 9-point stencil of cell I: the sum over the cell's rows of
// their row-to-cell sums B (k_mg_rowcell), which is P1^T A P1 (rows that are
// not unknowns have B = 0).  Nine coalesced loads per row instead of a walk
// over the rows' entries.
__global__ void k_mg_level1(Consts c, MgLevel L, const float* __restrict__ B, size_t np, const int32_t* cs,
                            int32_t* nact, int2* act_rng) {
    const int I = blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= L.nx * L.ny) return;
    float st[9];
#pragma unroll
    for (int d = 0; d < 9; d++) st[d] = 0.f;
    const int b = cs[I], e = cs[I + 1];
    for (int k = b; k < e; k++) {
#pragma unroll
        for (int d = 0; d < 9; d++) st[d] += __ldg(B + (size_t)d * np + k);
    }
    const int n = L.nx * L.ny;
#pragma unroll
    for (int d = 0; d < 9; d++) L.st[(size_t)d * n + I] = st[d];
    L.invd[I] = st[4] > 0.f ? 1.f / st[4] : 0.f;
    const int pos = list_active(st[4] > 0.f, I, L.act, nact + 1);
    if (pos >= 0) act_rng[pos] = make_int2(b, e - b);  // the cell's slots, beside its list entry
}

// Smoothed transfer: B = A P1 per slot (the row's sums over the 3x3 cells
// around its own, diagonal included), in the entry order of k_mg_level1.
// Slots that are not unknowns get 0.
//
// Also, for the cycle: every cell's r, e and t to 0 on the levels the grid-wide
// phases visit by list (levels 1 .. ngrid + 1), and the list lengths to 0.
__global__ void k_mg_rowcell(Consts c, Ppe A, MatFree mf, Mg mg) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    const size_t np = (size_t)mg.n_pad;
    float* __restrict__ B = mg.rowcell;
    if (i < kMgMaxLevels) mg.nact[i] = 0;
    for (int l = 1; l <= mg.ngrid + 1 && l <= mg.nlev; l++) {
        const MgLevel& L = mg.lev[l];
        for (int I = i; I < L.nx * L.ny; I += nt) {
            L.r[I] = 0.f;
            L.e[I] = 0.f;
            L.t[I] = 0.f;
        }
    }
    if (i >= c.n) return;
    float st[9];
#pragma unroll
    for (int d = 0; d < 9; d++) st[d] = 0.f;
    const float dg = A.diag32[i];
    if (dg > 0.f) {
        st[4] = dg;
        // an unknown is Inner, so its cell is an interior cell of the grid
        const int key = mf.skey[i];
        const int cx = key / c.numY, cy = key - cx * c.numY;
        const int cnt = A.offcnt[i];
        if (mf.enabled && !mf.sell_row[i]) {
            int rs[3][4];
            for (int r = 0; r < 3; r++) {
                const int kk = (cx - 1 + r) * c.numY + cy - 1;
                for (int q = 0; q < 4; q++) rs[r][q] = mf.cs[kk + q];
            }
            const size_t q0 = qsell_index(i, 0, c.K) >> 2;
            const float4* vp = reinterpret_cast<const float4*>(A.val32) + q0;
            const uint32_t* ip = reinterpret_cast<const uint32_t*>(mf.idx8) + q0;
            const int ng = (cnt + 3) >> 2;
            for (int g0 = 0; g0 < ng; g0 += 4) {
                float4 v[4];
                uint32_t b4[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int gi = min(g0 + q, ng - 1);
                    v[q] = __ldg(vp + gi * 32);
                    b4[q] = __ldg(ip + gi * 32);
                }
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float vv[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        if ((g0 + q) * 4 + t >= cnt) break;
                        const int bt = (b4[q] >> (8 * t)) & 255;
                        const int r = bt >> 6;
                        const int j = rs[r][0] + (bt & 63);
                        const int dy = (j >= rs[r][1]) + (j >= rs[r][2]) - 1;
                        add_tap(st, r * 3 + (dy + 1), vv[t]);
                    }
                }
            }
        } else {
            const size_t base = (size_t)(i >> 5) * c.K * 32 + (i & 31);
            for (int m = 0; m < cnt; m++) {
                const float v = A.val32[qsell_index(i, m, c.K)];
                const int j = A.col[base + (size_t)m * 32];
                const int kj = mf.skey[j];
                const int jx = kj / c.numY, jy = kj - jx * c.numY;
                add_tap(st, (jx - cx + 1) * 3 + (jy - cy + 1), v);
            }
        }
    }
#pragma unroll
    for (int d = 0; d < 9; d++) B[(size_t)d * np + i] = st[d];
}

// Coarse level C from fine level F: the Galerkin 9-point stencil and C's
// restriction weights (MgLevel::rw).  The residual that the V-cycle hands
// from F to C is, for each child c of a coarse cell, r_c - sum_d st_d(c)
// omega invd_j r_j (one Jacobi step from zero on F, then its residual);
// summed over the 2x2 children it is a fixed 4x4 stencil on r_F, whose
// weights depend only on the operator and omega.
__device__ __forceinline__ void coarsen_cell(const MgLevel& F, const MgLevel& C, float omega, int32_t* nact_c, int I) {
    const int nc = C.nx * C.ny;
    const int X = I / C.ny, Y = I - X * C.ny;
    const int nf = F.nx * F.ny;
    float st[9], w[16];
#pragma unroll
    for (int d = 0; d < 9; d++) st[d] = 0.f;
#pragma unroll
    for (int k = 0; k < 16; k++) w[k] = 0.f;
    // unrolled, so that st and w stay in registers and a child's 18 loads are in
    // flight together (indexed arrays in local memory: 9 us per level)
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
        for (int bb = 0; bb < 2; bb++) {
            const int x = 2 * X + a, y = 2 * Y + bb;
            if (x >= F.nx || y >= F.ny) continue;
            const int cf = x * F.ny + y;
            w[(a + 1) * 4 + (bb + 1)] += 1.f;
            float s[9], iv[9];
#pragma unroll
            for (int d = 0; d < 9; d++) {
                const int nx = x + d / 3 - 1, ny = y + d % 3 - 1;
                const bool in = nx >= 0 && ny >= 0 && nx < F.nx && ny < F.ny;
                s[d] = in ? F.st[(size_t)d * nf + cf] : 0.f;
                iv[d] = in ? F.invd[nx * F.ny + ny] : 0.f;
            }
#pragma unroll
            for (int d = 0; d < 9; d++) {
                const int dx = a + d / 3 - 1, dy = bb + d % 3 - 1;  // the tap from the patch's child (0, 0)
                const int DX = dx < 0 ? -1 : (dx > 1 ? 1 : 0), DY = dy < 0 ? -1 : (dy > 1 ? 1 : 0);
                st[(DX + 1) * 3 + (DY + 1)] += s[d];
                // tap (nx, ny) sits at (nx - 2X + 1, ny - 2Y + 1) of the 4x4 patch
                w[(dx + 1) * 4 + (dy + 1)] -= omega * iv[d] * s[d];
            }
        }
#pragma unroll
    for (int d = 0; d < 9; d++) C.st[(size_t)d * nc + I] = st[d];
    C.invd[I] = st[4] > 0.f ? 1.f / st[4] : 0.f;
    list_active(st[4] > 0.f, I, C.act, nact_c);
#pragma unroll
    for (int k = 0; k < 16; k++) C.rw[(size_t)k * nc + I] = w[k];
}

__global__ void k_mg_coarsen(MgLevel F, MgLevel C, float omega, int32_t* nact_c) {
    const int I = blockIdx.x * blockDim.x + threadIdx.x;
    if (I < C.nx * C.ny) coarsen_cell(F, C, omega, nact_c, I);
}

// Dense inverse of the coarsest operator by Gauss-Jordan; cells without unknowns
// keep an identity row and column (their residual is 0), so their pivots are
// skipped.  32 x 32 threads hold up to 3 x 3 entries each; per pivot its row and
// column go through shared memory, in turn through two buffers: one barrier.  With
// the matrix in shared memory, two barriers per pivot and every pivot, k_mg_tail took
// 37, 66 and 55 us at 2,162, 109,202 and 1,024,618 particles; 34, 54 and 41 us so.
__device__ __forceinline__ void dense_inverse(const MgLevel& L, float* out) {
    static_assert(kMgMaxCoarsest <= 96, "three rows and columns per thread");
    __shared__ float s_row[2][96], s_col[2][96];
    __shared__ bool s_act[96];
    const int n = L.nx * L.ny;
    for (int t = threadIdx.x; t < n; t += blockDim.x) s_act[t] = L.invd[t] > 0.f;
    __syncthreads();
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    float v[3][3];
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++) {
            const int i = ty + 32 * a, j = tx + 32 * b;
            v[a][b] = i == j ? 1.f : 0.f;
            if (i >= n || j >= n || !s_act[i]) continue;
            v[a][b] = 0.f;
            if (!s_act[j]) continue;
            const int dx = j / L.ny - i / L.ny, dy = j % L.ny - i % L.ny;
            if (dx >= -1 && dx <= 1 && dy >= -1 && dy <= 1) v[a][b] = L.st[(size_t)((dx + 1) * 3 + (dy + 1)) * n + i];
        }
    int par = 0;
    for (int k = 0; k < n; k++) {
        if (!s_act[k]) continue;
        if (ty == (k & 31)) {
#pragma unroll
            for (int a = 0; a < 3; a++)
                if (a == k >> 5)
#pragma unroll
                    for (int b = 0; b < 3; b++) s_row[par][tx + 32 * b] = v[a][b];
        }
        if (tx == (k & 31)) {
#pragma unroll
            for (int b = 0; b < 3; b++)
                if (b == k >> 5)
#pragma unroll
                    for (int a = 0; a < 3; a++) s_col[par][ty + 32 * a] = v[a][b];
        }
        __syncthreads();
        const float piv = 1.f / s_row[par][k];
        float row[3], col[3];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            row[q] = (tx + 32 * q == k ? 1.f : s_row[par][tx + 32 * q]) * piv;
            col[q] = s_col[par][ty + 32 * q];
        }
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 3; b++) {
                const int i = ty + 32 * a, j = tx + 32 * b;
                if (i == k)
                    v[a][b] = row[b];
                else if (j == k)
                    v[a][b] = -col[a] * row[b];
                else
                    v[a][b] -= col[a] * row[b];
            }
        par ^= 1;
    }
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int b = 0; b < 3; b++)
            if (ty + 32 * a < n && tx + 32 * b < n) out[(ty + 32 * a) * n + tx + 32 * b] = v[a][b];
}

// The levels after `first`, one after another, and the coarsest one's inverse: a
// few thousand cells, for which a launch each costs more than one block's time
// (and a batch makes all of them once per scene).
constexpr int kTailThreads = 1024;  // (dense_inverse's 32 x 32)
constexpr int kTailCells = 2048;
__global__ void __launch_bounds__(kTailThreads) k_mg_tail(__grid_constant__ const Mg mg, int first) {
    for (int l = first; l < mg.nlev; l++) {
        const MgLevel &F = mg.lev[l], &C = mg.lev[l + 1];
        for (int I = threadIdx.x; I < C.nx * C.ny; I += kTailThreads)
            coarsen_cell(F, C, mg.omega, mg.nact + l + 1, I);
        __syncthreads();
    }
    dense_inverse(mg.lev[mg.nlev], mg.dense);
}

}  // namespace

void launch_mg_setup(const Consts& c, const Ppe& A, const MatFree& mf, const Mg& mg,
                     cudaStream_t st) {
    if (!mg.enabled) return;
    // the rows' 3x3-cell sums: the operator of modes 1 and 3, and level 1's stencil
    k_mg_rowcell<<<block_count(c.n), block_threads(c.n), 0, st>>>(c, A, mf, mg);
    const MgLevel& L1 = mg.lev[1];
    k_mg_level1<<<block_count(L1.nx * L1.ny), block_threads(L1.nx * L1.ny), 0, st>>>(
        c, L1, mg.rowcell, (size_t)mg.n_pad, mf.cs, mg.nact, mg.act1_rng);
    int l = 1;
    for (; l < mg.nlev; l++) {
        const MgLevel& C = mg.lev[l + 1];
        const int nc = C.nx * C.ny;
        if (nc <= kTailCells) break;
        k_mg_coarsen<<<block_count(nc), block_threads(nc), 0, st>>>(mg.lev[l], C, mg.omega, mg.nact + l + 1);
        ++g_launches;
    }
    k_mg_tail<<<1, kTailThreads, 0, st>>>(mg, l);
    g_launches += 3;
}

}  // namespace mpsg
