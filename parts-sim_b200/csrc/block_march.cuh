// The finest level's operator of the multi-right-hand-side (block) solve by reflection modes, marched along z.
// Included by solver.cu only; the modes and their algebra are march_kernels.cuh's.
//
// A CTA takes 8 right-hand sides (one 32-byte sector of a DOF's RB values, 64 bytes in 64 bits) of a tile of 8 x 8 voxel
// columns (64-bit: 8 x 6): a thread is one voxel column and one right-hand side, a warp 4 columns side by side x 8. Planes
// of the tile's 9 x 9 nodes come into a ring in shared memory by 16-byte asynchronous copies (zeros at inactive nodes),
// two planes ahead; each thread turns the four corners it reads into its face's modes, adds its layer of voxels and hands
// the finished shares of its three other corners to the threads that own those nodes, through shared memory. The thread
// of voxel column (a, b) owns node (a, b) for a, b >= 1: 7 x 7 (7 x 5) output nodes a tile, where the epilogue runs with r, d, 1/diag
// and the results accessed directly. The groups of 8 of one tile are neighbouring CTAs and share the DOFs' 128-byte lines in L2.
//
// What bounds it: issue and latency at 16 (12) warps an SM; the gather it replaces read each of the 27
// neighbours of a node from L2 for every node (2.4 GB for 233 k nodes x 32 right-hand sides, SIMP 96x48x48): smoothing
// step 425 us, FP64 product 677 us; 160 and 247 us here.
#pragma once

#include "march_kernels.cuh"

namespace psfea {
namespace dev {

constexpr int BM_G = 8;                                                    // right-hand sides of a CTA
constexpr int BM_VX = 8, BM_NX = BM_VX - 1;                                // voxel columns along x; output nodes
constexpr int BM_PREFETCH = 2, BM_STAGES = 8;                              // (a power of two > PREFETCH + 2)
constexpr int BM_NODE = 3 * BM_G;                                          // values of a node
template <class T> __host__ __device__ constexpr int bmVY() { return sizeof(T) == 4 ? 8 : 6; }  // voxel columns along y
template <class T> __host__ __device__ constexpr int bmNY() { return bmVY<T>() - 1; }
template <class T> __host__ __device__ constexpr int bmThreads() { return BM_VX * bmVY<T>() * BM_G; }
template <class T> __host__ __device__ constexpr int bmNodes() { return (BM_VX + 1) * (bmVY<T>() + 1); }  // staged nodes of a plane
// the ring of x planes, the shares of two planes (three corners of every voxel column)
template <class T> __host__ __device__ constexpr size_t bmSmemBytes() {
    return sizeof(T) * BM_NODE * (size_t(BM_STAGES) * bmNodes<T>() + 2 * 3 * BM_VX * bmVY<T>());
}

// 16 bytes asynchronously, or zeros (the source is then not read)
__device__ __forceinline__ void cpAsync16Or0(void* dst, const void* src, bool take) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smemAddr(dst)), "l"(src), "r"(take ? 16 : 0) : "memory");
}

// One pass over the tiles of y = K x for every right-hand side with kb_op's epilogues (BOP_*); tiles: nTiles of them,
// CTA b takes the right-hand sides 8 (b % G) .. of tile b / G, G = RB / 8. Nodes without an active voxel are not written.
template <class T, int MODE, int RB>
__global__ void __launch_bounds__(bmThreads<T>(), 1)
    kb_march(LevelView L, ModeCoefs<T> K, const MarchTile* __restrict__ tiles, int nTiles, const T* __restrict__ x, T* __restrict__ y,
             const float* __restrict__ r, float* __restrict__ d, float c1, float c2, int raw, BlockState* bs, double* partials, unsigned* ticket,
             Ctl ctl) {
    if (skipped(ctl)) return;
    constexpr int G = RB / BM_G, VY = bmVY<T>(), COLS = BM_VX * VY, THREADS = bmThreads<T>(), NODES = bmNodes<T>();
    constexpr int PLANE = NODES * BM_NODE, SHARES = COLS * BM_NODE;
    constexpr int PER = 16 / int(sizeof(T)), PIECES = PLANE / PER, MINE = (PIECES + THREADS - 1) / THREADS;  // 16-byte pieces of a plane; a thread's
    extern __shared__ __align__(16) unsigned char bmSmem[];
    T* ring = reinterpret_cast<T*>(bmSmem);    // [STAGES][node][component][8]
    T* shares = ring + BM_STAGES * PLANE;      // [2][corner 10, 01, 11][column][component][8]
    const MarchTile tile = tiles[blockIdx.x / G];
    const int q = threadIdx.x & (BM_G - 1), col = threadIdx.x / BM_G, vx = col & (BM_VX - 1), vy = col / BM_VX;
    const int rhs = int(blockIdx.x % G) * BM_G;
    const int k0 = tile.k0, k1 = tile.k1, iBase = BM_NX * int(tile.tx) - 1, jBase = bmNY<T>() * int(tile.ty) - 1;
    const int i = iBase + vx, j = jBase + vy;  // the thread's voxel and node
    const long long PXY = (long long)L.PX * L.NY, WXY = (long long)L.px * L.ny;
    const bool voxIn = i >= 0 && i < L.nx && j >= 0 && j < L.ny;
    const bool own = vx > 0 && vy > 0 && i < L.NX && j < L.NY;
    const int nodeAt = i + L.PX * j, wordAt = i + L.px * j;
    // the pieces of a plane the thread stages: their node, and where in it
    int pNode[MINE];
    bool pIn[MINE];
#pragma unroll
    for (int m = 0; m < MINE; m++) {
        const int e = (int(threadIdx.x) + m * THREADS) * PER, n = e / BM_NODE, a = iBase + n % (BM_VX + 1), b = jBase + n / (BM_VX + 1);
        pIn[m] = n < NODES && a >= 0 && a < L.NX && b >= 0 && b < L.NY;
        pNode[m] = a + L.PX * b;
    }
    auto maskAt = [&](bool in, int at, int k) -> unsigned {  // of a node of plane k, 0 outside the grid
        const uint8_t* m = L.nmask + k * PXY;
        return (in && unsigned(k) < unsigned(L.NZ)) ? unsigned(__ldg(m + at)) : 0u;
    };
    auto stage = [&](int k, const unsigned (&mk)[MINE]) {
        T* dst = ring + ((k + 1) & (BM_STAGES - 1)) * PLANE;
#pragma unroll
        for (int m = 0; m < MINE; m++) {
            const int e = (int(threadIdx.x) + m * THREADS) * PER;
            if (e < PLANE) {
                const int w = e % BM_NODE, c = w / BM_G;
                cpAsync16Or0(dst + e, x + (3 * (k * PXY + pNode[m]) + c) * RB + rhs + (w - c * BM_G), mk[m] & NM_ACTIVE);
            }
        }
        cpAsyncCommit();
    };

    T F[3][4] = {}, mine[3] = {};
    float er[3], ed[3], ei[3];  // epilogue operands of the plane being completed, loaded a step ahead
    unsigned mkNext[MINE], hold = 0, holdNext = 0;
    uint32_t wNext = 0;  // the voxel word above the plane, a step ahead; used as loaded only then
    double dot[1] = {0.0};

    // the finished sums of plane k at the thread's own node (hold: its mask there) through the epilogue
    auto finish = [&](int k) {
        if (!own || !(hold & NM_ACTIVE)) return;
        const T* sh = shares + (k & 1) * 3 * SHARES + col * BM_NODE + q;
        const T* xo = ring + ((k + 1) & (BM_STAGES - 1)) * PLANE + (vy * (BM_VX + 1) + vx) * BM_NODE + q;
        const long long n = k * PXY + nodeAt;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const long long id = (3 * n + c) * RB + rhs + q;
            const bool fx = fixedDof(uint8_t(hold), c);
            T kx = mine[c] + sh[c * BM_G - BM_NODE] + sh[SHARES + c * BM_G - BM_VX * BM_NODE] + sh[2 * SHARES + c * BM_G - (BM_VX + 1) * BM_NODE];
            const T xv = xo[c * BM_G];
            if (L.dadd) kx += (sizeof(T) == 8 ? T(L.dadd[3 * n + c]) : T(L.dadd32[3 * n + c])) * xv;
            if constexpr (MODE == BOP_APPLY) {
                y[id] = (!raw && fx) ? T(0) : kx;
            } else if constexpr (MODE == BOP_DOT) {
                const T yv = fx ? T(0) : kx;
                y[id] = yv;
                dot[0] += double(xv) * double(yv);
            } else if constexpr (MODE == BOP_RESID) {
                y[id] = fx ? T(0) : T(er[c]) - kx;
            } else {
                const float dn = fx ? 0.f : c1 * ed[c] + c2 * ei[c] * (er[c] - float(kx));
                d[id] = dn;
                y[id] = fx ? T(0) : xv + T(dn);
            }
        }
    };

#pragma unroll
    for (int p = 0; p < BM_PREFETCH; p++) {
        unsigned mk[MINE];
#pragma unroll
        for (int m = 0; m < MINE; m++) mk[m] = maskAt(pIn[m], pNode[m], k0 - 1 + p);
        stage(k0 - 1 + p, mk);
    }
#pragma unroll
    for (int m = 0; m < MINE; m++) mkNext[m] = maskAt(pIn[m], pNode[m], k0 - 1 + BM_PREFETCH);
    FaceModes<T> P{}, Q;  // the modes of planes k - 1 and k
    // (the turns at both ends run the whole body too, as in k_march: hold is 0 outside [k0, k1))
    for (int k = k0 - 1; k <= k1; k++) {
        cpAsyncWait<BM_PREFETCH - 1>();
        __syncthreads();
        finish(k - 2);
        stage(k + BM_PREFETCH, mkNext);  // into a slot whose plane's last readers were done before the barrier
#pragma unroll
        for (int m = 0; m < MINE; m++) mkNext[m] = maskAt(pIn[m] && k + BM_PREFETCH < k1, pNode[m], k + BM_PREFETCH + 1);
        hold = holdNext;  // of plane k - 1
        if (MODE == BOP_CHEB || MODE == BOP_RESID) {
            if (own && (hold & NM_ACTIVE)) {
                const long long n = (k - 1) * PXY + nodeAt, id = 3 * n * RB + rhs + q;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    er[c] = __ldg(r + id + c * RB);
                    if (MODE == BOP_CHEB) {
                        ed[c] = d[id + c * RB];
                        ei[c] = __ldg(L.invD + 3 * n + c);
                    }
                }
            }
        }
        holdNext = maskAt(own && k >= k0 && k < k1, nodeAt, k);
        const T s = T(fmaxf(__uint_as_float(wNext), 0.f));  // of the layer below
        wNext = (voxIn && unsigned(k) < unsigned(L.nz)) ? __ldg(L.word + k * WXY + wordAt) : 0u;
        const T* pl = ring + ((k + 1) & (BM_STAGES - 1)) * PLANE + (vy * (BM_VX + 1) + vx) * BM_NODE + q;
#pragma unroll
        for (int c = 0; c < 3; c++)
            Q.make(c, pl[c * BM_G], pl[BM_NODE + c * BM_G], pl[(BM_VX + 1) * BM_NODE + c * BM_G], pl[(BM_VX + 2) * BM_NODE + c * BM_G]);
        T H[3][4];
        marchLayer<T>(K, s, P, Q, F, H);
        // plane k - 1: the share of the thread's own node stays, those of its face's other corners go to their owners
        T* sh = shares + ((k - 1) & 1) * 3 * SHARES + col * BM_NODE + q;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const T s0 = H[c][0] - H[c][2], s1 = H[c][0] + H[c][2], t0 = H[c][1] - H[c][3], t1 = H[c][1] + H[c][3];
            mine[c] = s0 - t0;
            sh[c * BM_G] = s0 + t0;
            sh[SHARES + c * BM_G] = s1 - t1;
            sh[2 * SHARES + c * BM_G] = s1 + t1;
        }
        P = Q;
    }
    cpAsyncWait<0>();
    __syncthreads();
    finish(k1 - 1);

    if constexpr (MODE == BOP_DOT) {
        // each right-hand side's x . y: the CTA's 8, then (last CTA) over the tiles in order
        constexpr int NW = THREADS / 32;
        __shared__ double red[NW * BM_G];
        __shared__ bool last;
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
        for (int o = BM_G; o < 32; o <<= 1) dot[0] += __shfl_xor_sync(0xffffffffu, dot[0], o);
        if (lane < BM_G) red[wid * BM_G + lane] = dot[0];
        __syncthreads();
        if (threadIdx.x < BM_G) {
            double a = 0;
            for (int w = 0; w < NW; w++) a += red[w * BM_G + threadIdx.x];
            partials[(size_t)(blockIdx.x / G) * RB + rhs + threadIdx.x] = a;
            __threadfence();
        }
        __syncthreads();
        if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
        __syncthreads();
        if (!last) return;
        __threadfence();
        constexpr int NC = THREADS / RB;
        __shared__ double tot[NC * RB];
        if (threadIdx.x < NC * RB) {
            const int qq = threadIdx.x % RB, chunk = threadIdx.x / RB;
            double a = 0;
            for (int t = chunk; t < nTiles; t += NC) a += __ldcg(partials + (size_t)t * RB + qq);
            tot[chunk * RB + qq] = a;
        }
        __syncthreads();
        const int qq = threadIdx.x;
        if (qq < RB) {
            double pq = 0;
            for (int ch = 0; ch < NC; ch++) pq += tot[ch * RB + qq];
            bs->pq[qq] = pq;
            if (!rhsRunning(bs, qq)) {
                bs->alpha[qq] = 0;
            } else if (!(pq > 0)) {
                bs->alpha[qq] = 0;
                bs->status[qq] = ST_BREAKDOWN;
                bs->done[qq] = 1;
                bs->it[qq] = bs->iter;
            } else {
                bs->alpha[qq] = bs->rz[qq] / pq;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            *ticket = 0;
            blockAllDone(bs);
        }
    }
}

}  // namespace dev
}  // namespace psfea
