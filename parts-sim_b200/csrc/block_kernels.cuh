// Device code of the multi-right-hand-side (block) solve. Included by solver.cu only.
//
// A block holds RB right-hand sides (RB = 8, 16 or 32) in the RHS-minor layout: value of DOF
// 3 n + d of right-hand side q at [(3 n + d) RB + q], over the level's pitched nodes n. One warp
// takes 32 / RB nodes, one lane per (node, right-hand side): the lanes of a node share its mask,
// coordinates, voxel words and element matrices (broadcast loads, read once for the whole block)
// and read their values as one contiguous RB-wide access per DOF. Kernels walk the level's list
// of active nodes, so empty regions cost nothing.
//
// Every right-hand side runs its own flexible CG (the reference's recurrence,
// native/src/fea/voxel_fea.cpp:863-927): the scalars rz, alpha, beta, the residual, the V-cycle's
// input scale and the stop decision are per right-hand side (BlockState). A finished right-hand
// side keeps its iterate: its step length is 0 and its V-cycle input is 0. Reductions are
// deterministic (lane-wise partial sums per block, folded in block order by the last block).
#pragma once

#include "kernels.cuh"

namespace psfea {
namespace dev {

constexpr int RBMAX = 32;
constexpr int BLOCK_THREADS = 256;

// per right-hand side control of a block solve
struct BlockState {
    double bnorm[RBMAX], rel[RBMAX], rz[RBMAX], alpha[RBMAX], beta[RBMAX], rmax[RBMAX], scale[RBMAX], vscale[RBMAX], pq[RBMAX];
    int it[RBMAX], done[RBMAX], status[RBMAX];
    double tol;
    int iter, maxIter, first, allDone, nrhs;
};

// Lane-wise grid reduction: lane l holds K values of right-hand side l % RB. Returns true in the
// last block to finish, where thread t < RB holds in out[] the totals of right-hand side t (sums,
// or maxima for the bits of maxMask). partials: gridDim.x * RB * K doubles; ticket starts at 0 and
// is left at 0. Sums run in a fixed order (warp lanes, warps, blocks), so results are reproducible.
template <int K, int RB>
__device__ bool laneGridReduce(double (&v)[K], unsigned maxMask, double* partials, unsigned* ticket, double (&out)[K]) {
    constexpr int NW = BLOCK_THREADS / 32;
    __shared__ double sh[NW * RBMAX * K];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = RB; o < 32; o <<= 1)
#pragma unroll
        for (int c = 0; c < K; c++) {
            const double w = __shfl_xor_sync(0xffffffffu, v[c], o);
            v[c] = ((maxMask >> c) & 1) ? fmax(v[c], w) : v[c] + w;
        }
    if (lane < RB)
#pragma unroll
        for (int c = 0; c < K; c++) sh[(wid * RB + lane) * K + c] = v[c];
    __syncthreads();
    if (threadIdx.x < RB) {
        double a[K];
#pragma unroll
        for (int c = 0; c < K; c++) a[c] = 0;
        for (int w = 0; w < NW; w++)
#pragma unroll
            for (int c = 0; c < K; c++) {
                const double p = sh[(w * RB + threadIdx.x) * K + c];
                a[c] = ((maxMask >> c) & 1) ? fmax(a[c], p) : a[c] + p;
            }
#pragma unroll
        for (int c = 0; c < K; c++) partials[((size_t)blockIdx.x * RB + threadIdx.x) * K + c] = a[c];
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return false;
    __threadfence();
    // the last block: thread t sums right-hand side t % RB over the blocks b = t / RB (mod NC)
    constexpr int NC = BLOCK_THREADS / RB;
    const int q = threadIdx.x % RB, chunk = threadIdx.x / RB;
    double a[K];
#pragma unroll
    for (int c = 0; c < K; c++) a[c] = 0;
    for (unsigned b = chunk; b < gridDim.x; b += NC)
#pragma unroll
        for (int c = 0; c < K; c++) {
            const double p = __ldcg(partials + ((size_t)b * RB + q) * K + c);
            a[c] = ((maxMask >> c) & 1) ? fmax(a[c], p) : a[c] + p;
        }
    __syncthreads();  // sh is reused
#pragma unroll
    for (int c = 0; c < K; c++) sh[(chunk * RB + q) * K + c] = a[c];
    __syncthreads();
    if (threadIdx.x < RB) {
#pragma unroll
        for (int c = 0; c < K; c++) out[c] = 0;
        for (int ch = 0; ch < NC; ch++)
#pragma unroll
            for (int c = 0; c < K; c++) {
                const double p = sh[(ch * RB + threadIdx.x) * K + c];
                out[c] = ((maxMask >> c) & 1) ? fmax(out[c], p) : out[c] + p;
            }
    }
    if (threadIdx.x == 0) *ticket = 0;
    return true;
}

// the running state of a right-hand side
__device__ __forceinline__ bool rhsRunning(const BlockState* bs, int q) { return q < bs->nrhs && !bs->done[q]; }

// after a per-right-hand-side stop decision: the whole block is done when every one is (thread 0
// of the last block, after the threads t < RB have written their decisions)
__device__ __forceinline__ void blockAllDone(BlockState* bs) {
    int all = 1;
    for (int q = 0; q < bs->nrhs; q++) all &= bs->done[q] != 0;
    bs->allDone = all;
}

enum { BOP_APPLY = 0, BOP_CHEB = 1, BOP_RESID = 2, BOP_DOT = 3 };

// (K x) at node (i, j, k) of a block vector (stride S, x at the lane's right-hand side) with each of
// the node's 27 neighbours read once, two z-planes of 9 nodes in registers at a time (planes -1 and
// 0 for the voxels below the node, 0 and +1 for those above): the same sums in the same order as
// applyAt (so bitwise the same), with 81 loads instead of up to 192 on nodes that take the per-voxel
// gather. Neighbours outside the grid read 0; they only ever meet empty voxels.
// V: the storage type of x (T, or __half for the FP16 coarse-level vectors; converted on load).
template <class T, bool OWN16, int S, bool SMEM = false, class V = T>
__device__ __forceinline__ void applyNbr(const LevelView& L, const Coefs<T>& C, const V* x, int i, int j, int k, long long n,
                                         uint8_t mask, T acc[3]) {
    acc[0] = acc[1] = acc[2] = T(0);
    if (!(mask & NM_ACTIVE)) return;
    const long long NX = L.PX, NXY = (long long)L.PX * L.NY;
    auto plane = [&](int oz, T (&P)[9][3]) {
#pragma unroll
        for (int b = 0; b < 9; b++) {
            const int ox = b % 3 - 1, oy = b / 3 - 1;
            const bool in = i + ox >= 0 && j + oy >= 0 && k + oz >= 0 && i + ox < L.NX && j + oy < L.NY && k + oz < L.NZ;
            const V* xp = x + 3 * S * (n + ox + oy * NX + oz * NXY);
            P[b][0] = in ? ldv<T>(xp) : T(0);
            P[b][1] = in ? ldv<T>(xp + S) : T(0);
            P[b][2] = in ? ldv<T>(xp + 2 * S) : T(0);
        }
    };
    T A[9][3], B[9][3];  // A: planes -1 then +1; B: plane 0
    plane(-1, A);
    plane(0, B);
    const T own[3] = {B[4][0], B[4][1], B[4][2]};
    if (mask & NM_UNIFORM) {
        const float s = __uint_as_float(__ldg(L.word + L.wi(i - 1, j - 1, k - 1)));
        T a0 = 0, a1 = 0, a2 = 0;
        auto sweep = [&](int oz, const T (&P)[9][3]) {
#pragma unroll
            for (int b = 0; b < 9; b++) {
                const int ox = b % 3 - 1, oy = b / 3 - 1, m = b + 9 * (oz + 1);
                const T x0 = P[b][0], x1 = P[b][1], x2 = P[b][2];
                a0 += C.S[m * 9 + 0] * x0;
                a1 += C.S[m * 9 + 4] * x1;
                a2 += C.S[m * 9 + 8] * x2;
                if (ox && oy) { a0 += C.S[m * 9 + 1] * x1; a1 += C.S[m * 9 + 3] * x0; }
                if (ox && oz) { a0 += C.S[m * 9 + 2] * x2; a2 += C.S[m * 9 + 6] * x0; }
                if (oy && oz) { a1 += C.S[m * 9 + 5] * x2; a2 += C.S[m * 9 + 7] * x1; }
            }
        };
        sweep(-1, A);
        sweep(0, B);
        plane(1, A);
        sweep(1, A);
        acc[0] = T(s) * a0;
        acc[1] = T(s) * a1;
        acc[2] = T(s) * a2;
    } else {
        // voxel vv = di + 2 dj + 4 dk at offset (di - 1, dj - 1, dk - 1); its corner b sits in plane
        // dk + bz - 1: lo = the plane below (dk - 1), hi = the plane above (dk)
        auto voxel = [&](int vv, const T (&lo)[9][3], const T (&hi)[9][3]) {
            const int di = vv & 1, dj = (vv >> 1) & 1, dk = vv >> 2;
            const int ei = i - 1 + di, ej = j - 1 + dj, ek = k - 1 + dk;
            if (ei < 0 || ej < 0 || ek < 0 || ei >= L.nx || ej >= L.ny || ek >= L.nz) return;
            const uint32_t w = __ldg(L.word + L.wi(ei, ej, ek));
            if (w == 0) return;
            const int a = cornerOf(1 - di, 1 - dj, 1 - dk);
            T xe[24];
#pragma unroll
            for (int b = 0; b < 8; b++) {
                const int bx = (b == 1 || b == 2 || b == 5 || b == 6), by = (b == 2 || b == 3 || b == 6 || b == 7), bz = b >> 2;
                const int b9 = (di + bx) + 3 * (dj + by);
                const T* src = bz ? hi[b9] : lo[b9];
                xe[3 * b] = src[0];
                xe[3 * b + 1] = src[1];
                xe[3 * b + 2] = src[2];
            }
            if (!(w & OWN_BIT)) {
                T t[3];
                kbRows<T>(C.Kb, a, xe, t);
                const T sc = T(__uint_as_float(w));
                acc[0] += sc * t[0];
                acc[1] += sc * t[1];
                acc[2] += sc * t[2];
            } else if (OWN16) {
                T t[3];
                own16Rows<T, SMEM>(L.own16 + (long long)(w & ~OWN_BIT) * 576 + 72 * a, xe, t);
                acc[0] += T(L.hs) * t[0];
                acc[1] += T(L.hs) * t[1];
                acc[2] += T(L.hs) * t[2];
            } else {
                const float4* K4 = reinterpret_cast<const float4*>(L.own + (long long)(w & ~OWN_BIT) * 576 + 72 * a);
#pragma unroll
                for (int d = 0; d < 3; d++)
#pragma unroll
                    for (int q = 0; q < 6; q++) {
                        const float4 kv = SMEM ? K4[d * 6 + q] : __ldg(K4 + d * 6 + q);
                        acc[d] += T(kv.x) * xe[4 * q] + T(kv.y) * xe[4 * q + 1] + T(kv.z) * xe[4 * q + 2] + T(kv.w) * xe[4 * q + 3];
                    }
            }
        };
#pragma unroll
        for (int vv = 0; vv < 4; vv++) voxel(vv, A, B);
        plane(1, A);
#pragma unroll
        for (int vv = 4; vv < 8; vv++) voxel(vv, B, A);
    }
    if (L.dadd) {
#pragma unroll
        for (int d = 0; d < 3; d++) acc[d] += (sizeof(T) == 8 ? T(L.dadd[3 * n + d]) : T(L.dadd32[3 * n + d])) * own[d];
    }
}

// One pass over the level's active nodes of y = K x for every right-hand side, with a per-DOF epilogue:
//   BOP_APPLY  y = K x (held DOFs 0 unless raw)
//   BOP_CHEB   d = c1 d + c2 D^-1 (r - K x); y = x + d        (Chebyshev / Jacobi step, 32-bit)
//   BOP_RESID  y = r - K x
//   BOP_DOT    y = K x (held 0) and each right-hand side's CG step alpha = rz / (x . y); x . y <= 0
//              ends that right-hand side as a breakdown (voxel_fea.cpp:902-905); finest level only
// On the finest level block_march.cuh makes these passes; kb_op makes the first three below it.
// The product is the single-vector one (applyAt, voxel_fea.cpp:422-486) with the block's stride.
// The block path's assembled stencils are node-major: node t's row at t * STN_ROW holds its 27 3x3
// blocks with the neighbours taken in pairs (m, m + 1) = (2 P, 2 P + 1), P = 0..13 (m = (ox + 1) +
// 3 (oy + 1) + 9 (oz + 1); the 28th slot is 0): entry (p, q) of the pair's two blocks side by side
// at 18 P + 2 (3 p + q) + (m & 1). A warp copies its nodes' rows into shared memory with 16-byte
// loads (512 contiguous bytes per instruction) and every lane of a node reads them as broadcasts;
// one paired FMA then advances both neighbours of a pair: 126 paired FMAs per node and right-hand
// side where the per-voxel gather takes 288 (576 multiply-adds), the coefficients read from HBM
// once per node for the whole block.
constexpr int STN_ROW = 252;
__host__ __device__ constexpr int stnPairAt(int m, int p, int q) { return 18 * (m >> 1) + 2 * (3 * p + q) + (m & 1); }
__host__ __device__ constexpr size_t stnBlockSmem(int npw) { return size_t(BLOCK_THREADS / 32) * npw * STN_ROW * sizeof(float); }

template <int S>
__device__ __forceinline__ void stnBlock(const LevelView& L, const float* __restrict__ row, const float* __restrict__ x, long long n, int i,
                                         int j, int k, float acc[3]) {
    const long long NX = L.PX, NXY = (long long)L.PX * L.NY;
    auto xOf = [&](int m, float (&v)[3]) {
        const int ox = m % 3 - 1, oy = (m / 3) % 3 - 1, oz = m / 9 - 1;
        const bool in = m < 27 && i + ox >= 0 && j + oy >= 0 && k + oz >= 0 && i + ox < L.NX && j + oy < L.NY && k + oz < L.NZ;
        const float* xp = x + 3 * S * (n + ox + oy * NX + oz * NXY);
        v[0] = in ? __ldg(xp) : 0.f;
        v[1] = in ? __ldg(xp + S) : 0.f;
        v[2] = in ? __ldg(xp + 2 * S) : 0.f;
    };
    const float4* R = reinterpret_cast<const float4*>(row);
    float2 a2[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    float4 cf = make_float4(0.f, 0.f, 0.f, 0.f);
    int have = -1;
#pragma unroll
    for (int P = 0; P < 14; P++) {
        float u[3], w[3];
        xOf(2 * P, u);
        xOf(2 * P + 1, w);
#pragma unroll
        for (int e = 0; e < 9; e++) {
            const int f = 18 * P + 2 * e;  // the pair's entry (p, q) = (e / 3, e % 3): floats f, f + 1
            if (f / 4 != have) {
                have = f / 4;
                cf = R[have];
            }
            const float2 b = (f % 4 == 0) ? make_float2(cf.x, cf.y) : make_float2(cf.z, cf.w);
            a2[e / 3] = __ffma2_rn(b, make_float2(u[e % 3], w[e % 3]), a2[e / 3]);
        }
    }
    acc[0] = a2[0].x + a2[0].y;
    acc[1] = a2[1].x + a2[1].y;
    acc[2] = a2[2].x + a2[2].y;
}

// STN: the product from the level's assembled stencils (stn, over act) instead of the gather; latency-bound on neighbour values
// from L2, so at four CTAs an SM (load groups SIMP 96x48x48 x 32: 167.6 ms at two, 165.6 at three, 162.0 at four).
template <int MODE, bool OWN16, int RB, bool STN = false>
__global__ void __launch_bounds__(BLOCK_THREADS, STN ? 4 : 2) kb_op(LevelView L, Coefs<float> C, const int* __restrict__ act, int nAct,
                                                       const float* __restrict__ stn, const float* __restrict__ x, float* __restrict__ y,
                                                       const float* __restrict__ r, float* __restrict__ d, float c1, float c2, int raw,
                                                       Ctl ctl) {
    if (skipped(ctl)) return;
    constexpr int NPW = 32 / RB;
    const int lane = threadIdx.x & 31, q = lane % RB, sub = lane / RB;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((long long)gridDim.x * blockDim.x) >> 5;
    extern __shared__ __align__(16) unsigned char kbRaw[];
    float* rows = reinterpret_cast<float*>(kbRaw) + (threadIdx.x >> 5) * NPW * STN_ROW;  // this warp's NPW stencil rows
    // warp-uniform sweep (the stencil rows are shared within the warp); lanes past the list idle
    for (long long tb = warp * NPW; tb < nAct; tb += nw * NPW) {
        const long long t = tb + sub;
        if constexpr (STN) {
            constexpr int VP = 4, PIECES = STN_ROW / VP;  // 16-byte pieces of a row
            for (int e = lane; e < NPW * PIECES; e += 32) {
                const int u = e / PIECES, g = e - u * PIECES;
                if (tb + u < nAct) {
                    const uint4 v = __ldcs(reinterpret_cast<const uint4*>(stn + (tb + u) * STN_ROW) + g);
                    reinterpret_cast<uint4*>(rows + u * STN_ROW)[g] = v;
                }
            }
            __syncwarp();
        }
        if (t < nAct) {
            const long long n = act[t];
            const uint8_t mask = __ldg(L.nmask + n);
            int i, j, k;
            nodeCoords(L, n, i, j, k);
            float acc[3];
            if constexpr (STN) stnBlock<RB>(L, rows + sub * STN_ROW, x + q, n, i, j, k, acc);
            else applyNbr<float, OWN16, RB>(L, C, x + q, i, j, k, n, mask, acc);
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const long long id = (3 * n + c) * RB + q;
                const bool fx = fixedDof(mask, c);
                if constexpr (MODE == BOP_APPLY) {
                    y[id] = (!raw && fx) ? 0.f : acc[c];
                } else if constexpr (MODE == BOP_RESID) {
                    y[id] = fx ? 0.f : r[id] - acc[c];
                } else {
                    if (fx) {
                        d[id] = 0.f;
                        y[id] = 0.f;
                    } else {
                        const float dn = c1 * d[id] + c2 * __ldg(L.invD + 3 * n + c) * (r[id] - acc[c]);
                        d[id] = dn;
                        y[id] = x[id] + dn;
                    }
                }
            }
        }
        if constexpr (STN) __syncwarp();  // the rows are refilled next
    }
}

// z = d = c0 D^-1 r (the first Chebyshev step from zero) at the active nodes
template <int RB>
__global__ void kb_cheb_first(const int* __restrict__ act, int nAct, const float* __restrict__ invD, const float* __restrict__ r,
                              float* __restrict__ d, float* __restrict__ z, float c0, Ctl ctl) {
    if (skipped(ctl)) return;
    const long long total = (long long)nAct * 3 * RB;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
        const long long t = e / (3 * RB);
        const int rem = int(e - t * 3 * RB), c = rem / RB, q = rem - c * RB;
        const long long dof = 3 * (long long)act[t] + c, id = dof * RB + q;
        const float v = c0 * __ldg(invD + dof) * r[id];
        d[id] = v;
        z[id] = v;
    }
}

// rc = P^T rf at the coarse level's active nodes (fine 2I weight 1, 2I +- 1 weight 1/2 per axis),
// held coarse DOFs 0; with dc, the coarse level's first smoothing step d = z = c0 D^-1 rc
template <int RB>
__global__ void kb_restrict(LevelView F, LevelView C, const int* __restrict__ cAct, int nCAct, const float* __restrict__ rf,
                            float* __restrict__ rc, float* __restrict__ dc, float* __restrict__ zc, float c0, Ctl ctl) {
    if (skipped(ctl)) return;
    constexpr int NPW = 32 / RB;
    const int lane = threadIdx.x & 31, q = lane % RB, sub = lane / RB;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long t = warp * NPW + sub; t < nCAct; t += nw * NPW) {
        const long long cn = cAct[t];
        const uint8_t mask = C.nmask[cn];
        int I, J, K;
        nodeCoords(C, cn, I, J, K);
        Values<3> sv = restrictAt<RB, 3>(F, rf + q, I, J, K);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const long long id = (3 * cn + c) * RB + q;
            const float v = fixedDof(mask, c) ? 0.f : sv[c];
            rc[id] = v;
            if (dc) {
                const float dv = c0 * __ldg(C.invD + 3 * cn + c) * v;
                dc[id] = dv;
                zc[id] = dv;
            }
        }
    }
}

// zf += P zc at the free DOFs of the fine level's active nodes (trilinear)
template <int RB>
__global__ void kb_prolong(LevelView F, int CPX, int CNY, const int* __restrict__ fAct, int nFAct, const float* __restrict__ zc,
                           float* __restrict__ zf, Ctl ctl) {
    if (skipped(ctl)) return;
    constexpr int NPW = 32 / RB;
    const int lane = threadIdx.x & 31, q = lane % RB, sub = lane / RB;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((long long)gridDim.x * blockDim.x) >> 5;
    const long long CNX = CPX, CNXY = (long long)CPX * CNY;
    for (long long t = warp * NPW + sub; t < nFAct; t += nw * NPW) {
        const long long fn = fAct[t];
        const uint8_t mask = F.nmask[fn];
        if ((mask & 7) == 7) continue;
        int i, j, k;
        nodeCoords(F, fn, i, j, k);
        float* o = zf + 3 * RB * fn + q;
        const float z0 = o[0], z1 = o[RB], z2 = o[2 * RB];
        float s[3];
        prolongAt<RB>(CNX, CNXY, zc + q, i, j, k, s);
        if (!fixedDof(mask, 0)) o[0] = z0 + s[0];
        if (!fixedDof(mask, 1)) o[RB] = z1 + s[1];
        if (!fixedDof(mask, 2)) o[2 * RB] = z2 + s[2];
    }
}

// coarsest level: z = A^-1 r over the m free DOFs for every right-hand side (FP64 dense inverse). A block takes KBC_ROWS
// rows, its warps every 8th group of NPW columns each (the lane groups of a warp a column of their own), the partial sums
// meet in shared memory in a fixed order. (One lane group over a whole row, column after column, was a chain of m / 2
// dependent loads: 96 us at m = 312.)
constexpr int KBC_ROWS = 2;
template <class TI, class TO, int RB>
__global__ void __launch_bounds__(BLOCK_THREADS) kb_coarse(int m, const int* __restrict__ dof, const double* __restrict__ Ainv,
                                                           const TI* __restrict__ r, TO* __restrict__ z, Ctl ctl) {
    if (skipped(ctl)) return;
    constexpr int NPW = 32 / RB, NW = BLOCK_THREADS / 32, U = 4;
    __shared__ double sh[KBC_ROWS][NW][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, q = lane % RB, sub = lane / RB;
    const int row = blockIdx.x * KBC_ROWS;
    double s[KBC_ROWS] = {};
    for (int c0 = wid * NPW + sub; c0 < m; c0 += NW * NPW * U) {
        double rv[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int c = c0 + u * NW * NPW;
            rv[u] = c < m ? double(__ldg(r + (long long)__ldg(dof + c) * RB + q)) : 0.0;
        }
#pragma unroll
        for (int e = 0; e < KBC_ROWS; e++)
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int c = c0 + u * NW * NPW;
                if (c < m && row + e < m) s[e] += __ldg(Ainv + (size_t)(row + e) * m + c) * rv[u];
            }
    }
#pragma unroll
    for (int e = 0; e < KBC_ROWS; e++) sh[e][wid][lane] = s[e];
    __syncthreads();
    if (threadIdx.x < KBC_ROWS * RB) {
        const int e = threadIdx.x / RB, qq = threadIdx.x % RB;
        double t = 0;
        for (int w = 0; w < NW; w++)
#pragma unroll
            for (int u = 0; u < NPW; u++) t += sh[e][w][u * RB + qq];
        if (row + e < m) z[(long long)__ldg(dof + row + e) * RB + qq] = TO(t);
    }
}

// ---------------------------------------------------------------- block CG vector kernels (FP64)

// r = f - K x at free DOFs; bnorm = ||f_free||, rel = ||r|| / bnorm, rmax = max |r_free| per
// right-hand side (voxel_fea.cpp:876-886); a zero load ends its right-hand side with u = 0
template <int RB>
__global__ void kb_cg_init(const int* __restrict__ act, int nAct, const uint8_t* __restrict__ nmask, const double* __restrict__ f,
                           const double* __restrict__ kx, double* __restrict__ r, BlockState* bs, double* partials, unsigned* ticket) {
    constexpr int NPW = 32 / RB;
    const int lane = threadIdx.x & 31, q = lane % RB, sub = lane / RB;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((long long)gridDim.x * blockDim.x) >> 5;
    double v[3] = {0, 0, 0};
    for (long long t = warp * NPW + sub; t < nAct; t += nw * NPW) {
        const long long n = act[t];
        const uint8_t mask = nmask[n];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const long long id = (3 * n + c) * RB + q;
            double rv = 0;
            if (!fixedDof(mask, c)) {
                const double fv = f[id];
                rv = fv - kx[id];
                v[0] += fv * fv;
                v[1] += rv * rv;
                v[2] = fmax(v[2], fabs(rv));
            }
            r[id] = rv;
        }
    }
    double tot[3];
    if (laneGridReduce<3, RB>(v, 4u, partials, ticket, tot)) {
        const int qq = threadIdx.x;
        if (qq < RB) {
            bs->bnorm[qq] = sqrt(tot[0]);
            bs->rmax[qq] = tot[2];
            bs->scale[qq] = tot[2] > 0 ? 1.0 / tot[2] : 1.0;
            bs->it[qq] = 0;
            bs->status[qq] = ST_RUNNING;
            bs->alpha[qq] = 0;
            if (qq >= bs->nrhs) {
                bs->rel[qq] = 0;
                bs->done[qq] = 1;
            } else if (bs->bnorm[qq] == 0) {
                bs->rel[qq] = 0;
                bs->status[qq] = ST_CONVERGED;
                bs->done[qq] = 2;  // zero load: the solution is zero
            } else {
                bs->rel[qq] = sqrt(tot[1]) / bs->bnorm[qq];
                bs->done[qq] = 0;
                if (bs->rel[qq] <= bs->tol) {
                    bs->status[qq] = ST_CONVERGED;
                    bs->done[qq] = 1;
                } else if (bs->maxIter <= 0) {
                    bs->status[qq] = ST_MAXITER;
                    bs->done[qq] = 1;
                }
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) blockAllDone(bs);
    }
}

// x += alpha p, r -= alpha q at free DOFs of running right-hand sides; rel, rmax per right-hand
// side; stop on rel <= tol or the cap. Fused: the V-cycle input r32 = r * scale (0 for finished
// right-hand sides) and the finest level's first Chebyshev step d = z = c0 D^-1 r32.
template <int RB>
__global__ void kb_cg_update(const int* __restrict__ act, int nAct, const uint8_t* __restrict__ nmask, double* __restrict__ x,
                             double* __restrict__ r, const double* __restrict__ p, const double* __restrict__ kp, float* __restrict__ r32,
                             const float* __restrict__ invD, float* __restrict__ d, float* __restrict__ z, float c0, BlockState* bs,
                             double* partials, unsigned* ticket, Ctl ctl) {
    if (skipped(ctl)) return;
    constexpr int NPW = 32 / RB;
    const int lane = threadIdx.x & 31, q = lane % RB, sub = lane / RB;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((long long)gridDim.x * blockDim.x) >> 5;
    const bool run = rhsRunning(bs, q);
    const double alpha = bs->alpha[q], s = bs->scale[q];
    double v[2] = {0, 0};
    for (long long t = warp * NPW + sub; t < nAct; t += nw * NPW) {
        const long long n = act[t];
        const uint8_t mask = nmask[n];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            if (fixedDof(mask, c)) continue;
            const long long id = (3 * n + c) * RB + q;
            float rs = 0.f;
            if (run) {
                x[id] += alpha * p[id];
                const double rv = r[id] - alpha * kp[id];
                r[id] = rv;
                v[0] += rv * rv;
                v[1] = fmax(v[1], fabs(rv));
                rs = float(rv * s);
            }
            r32[id] = rs;
            const float dv = c0 * __ldg(invD + 3 * n + c) * rs;
            d[id] = dv;
            z[id] = dv;
        }
    }
    double tot[2];
    if (laneGridReduce<2, RB>(v, 2u, partials, ticket, tot)) {
        const int qq = threadIdx.x;
        if (qq < RB && rhsRunning(bs, qq)) {
            bs->rel[qq] = sqrt(tot[0]) / bs->bnorm[qq];
            bs->vscale[qq] = bs->scale[qq];
            bs->rmax[qq] = tot[1];
            bs->scale[qq] = tot[1] > 0 ? 1.0 / tot[1] : 1.0;
            bs->it[qq] = bs->iter + 1;
            if (bs->rel[qq] <= bs->tol) {
                bs->status[qq] = ST_CONVERGED;
                bs->done[qq] = 1;
            } else if (bs->iter + 1 >= bs->maxIter) {
                bs->status[qq] = ST_MAXITER;
                bs->done[qq] = 1;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            bs->iter += 1;
            blockAllDone(bs);
        }
    }
}

// the V-cycle input of every running right-hand side, r32 = float(r / max|r_free|) (voxel_fea.cpp:
// 856-857), and the first Chebyshev step d = z = c0 D^-1 r32; 0 for finished ones
template <int RB>
__global__ void kb_vc_load(const int* __restrict__ act, int nAct, const uint8_t* __restrict__ nmask, const double* __restrict__ r,
                           float* __restrict__ r32, const float* __restrict__ invD, float* __restrict__ d, float* __restrict__ z, float c0,
                           BlockState* bs, Ctl ctl) {
    if (skipped(ctl)) return;
    constexpr int NPW = 32 / RB;
    const int lane = threadIdx.x & 31, q = lane % RB, sub = lane / RB;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((long long)gridDim.x * blockDim.x) >> 5;
    const bool run = rhsRunning(bs, q);
    const double s = bs->scale[q];
    for (long long t = warp * NPW + sub; t < nAct; t += nw * NPW) {
        const long long n = act[t];
        const uint8_t mask = nmask[n];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            if (fixedDof(mask, c)) continue;
            const long long id = (3 * n + c) * RB + q;
            const float rs = run ? float(r[id] * s) : 0.f;
            r32[id] = rs;
            const float dv = c0 * __ldg(invD + 3 * n + c) * rs;
            d[id] = dv;
            z[id] = dv;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x < RB) bs->vscale[threadIdx.x] = bs->scale[threadIdx.x];
}

// z = z32 / vscale; rzNew = r.z, zq = z.(K p) per running right-hand side; beta = max(0, -alpha
// zq / rz) (voxel_fea.cpp:913-917), 0 on the first pass
template <int RB>
__global__ void kb_cg_dots(const int* __restrict__ act, int nAct, const uint8_t* __restrict__ nmask, const double* __restrict__ r,
                           const float* __restrict__ z32, const double* __restrict__ z64, const double* __restrict__ kp, BlockState* bs,
                           double* partials, unsigned* ticket, Ctl ctl) {
    if (skipped(ctl)) return;
    constexpr int NPW = 32 / RB;
    const int lane = threadIdx.x & 31, q = lane % RB, sub = lane / RB;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((long long)gridDim.x * blockDim.x) >> 5;
    const bool run = rhsRunning(bs, q), first = bs->first;
    const double inv = 1.0 / bs->vscale[q];
    double v[2] = {0, 0};
    if (run)
        for (long long t = warp * NPW + sub; t < nAct; t += nw * NPW) {
            const long long n = act[t];
            const uint8_t mask = nmask[n];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                if (fixedDof(mask, c)) continue;
                const long long id = (3 * n + c) * RB + q;
                const double zv = z64 ? z64[id] : double(z32[id]) * inv;
                v[0] += r[id] * zv;
                if (!first) v[1] += zv * kp[id];
            }
        }
    double tot[2];
    if (laneGridReduce<2, RB>(v, 0u, partials, ticket, tot)) {
        const int qq = threadIdx.x;
        if (qq < RB && rhsRunning(bs, qq)) {
            bs->beta[qq] = first ? 0.0 : fmax(0.0, -bs->alpha[qq] * tot[1] / bs->rz[qq]);
            bs->rz[qq] = tot[0];
        }
    }
}

// p = z + beta p at free DOFs of running right-hand sides
template <int RB>
__global__ void kb_cg_p(const int* __restrict__ act, int nAct, const uint8_t* __restrict__ nmask, const float* __restrict__ z32,
                        const double* __restrict__ z64, double* __restrict__ p, const BlockState* bs, Ctl ctl) {
    if (skipped(ctl)) return;
    constexpr int NPW = 32 / RB;
    const int lane = threadIdx.x & 31, q = lane % RB, sub = lane / RB;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((long long)gridDim.x * blockDim.x) >> 5;
    if (!rhsRunning(bs, q)) return;
    const double inv = 1.0 / bs->vscale[q], beta = bs->beta[q];
    const bool first = bs->first;
    for (long long t = warp * NPW + sub; t < nAct; t += nw * NPW) {
        const long long n = act[t];
        const uint8_t mask = nmask[n];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            if (fixedDof(mask, c)) continue;
            const long long id = (3 * n + c) * RB + q;
            const double zv = z64 ? z64[id] : double(z32[id]) * inv;
            p[id] = first ? zv : zv + beta * p[id];
        }
    }
}

__global__ void kb_clear_first(BlockState* bs) { bs->first = 0; }

// true residual per right-hand side after the loop: ||f - K x||_free / bnorm (voxel_fea.cpp:921-925)
template <int RB>
__global__ void kb_final(const int* __restrict__ act, int nAct, const uint8_t* __restrict__ nmask, const double* __restrict__ f,
                         const double* __restrict__ kx, BlockState* bs, double* partials, unsigned* ticket) {
    constexpr int NPW = 32 / RB;
    const int lane = threadIdx.x & 31, q = lane % RB, sub = lane / RB;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((long long)gridDim.x * blockDim.x) >> 5;
    double v[1] = {0};
    for (long long t = warp * NPW + sub; t < nAct; t += nw * NPW) {
        const long long n = act[t];
        const uint8_t mask = nmask[n];
#pragma unroll
        for (int c = 0; c < 3; c++)
            if (!fixedDof(mask, c)) {
                const long long id = (3 * n + c) * RB + q;
                const double rv = f[id] - kx[id];
                v[0] += rv * rv;
            }
    }
    double tot[1];
    if (laneGridReduce<1, RB>(v, 0u, partials, ticket, tot)) {
        const int qq = threadIdx.x;
        if (qq < RB && qq < bs->nrhs) bs->rel[qq] = bs->bnorm[qq] > 0 ? sqrt(tot[0]) / bs->bnorm[qq] : 0.0;
    }
}

// max |r_free| per right-hand side into rmax / scale (the block preconditioner's entry). nvec comes as an argument: the call returns
// before the GPU has run it, so a state copied from a host buffer could be the next call's.
template <int RB>
__global__ void kb_rmax(const int* __restrict__ act, int nAct, const uint8_t* __restrict__ nmask, const double* __restrict__ r, int nvec,
                        BlockState* bs, double* partials, unsigned* ticket) {
    constexpr int NPW = 32 / RB;
    const int lane = threadIdx.x & 31, q = lane % RB, sub = lane / RB;
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((long long)gridDim.x * blockDim.x) >> 5;
    double v[1] = {0};
    for (long long t = warp * NPW + sub; t < nAct; t += nw * NPW) {
        const long long n = act[t];
        const uint8_t mask = nmask[n];
#pragma unroll
        for (int c = 0; c < 3; c++)
            if (!fixedDof(mask, c)) v[0] = fmax(v[0], fabs(r[(3 * n + c) * RB + q]));
    }
    double tot[1];
    if (laneGridReduce<1, RB>(v, 1u, partials, ticket, tot)) {
        const int qq = threadIdx.x;
        if (qq < RB) {
            bs->rmax[qq] = tot[0];
            bs->scale[qq] = tot[0] > 0 ? 1.0 / tot[0] : 1.0;
            bs->done[qq] = (qq < nvec && tot[0] > 0) ? 0 : 1;  // a zero vector gives z = 0
        }
        if (qq == 0) bs->nrhs = nvec;
    }
}

// ---- the C ABI's dense vectors (nrhs consecutive vectors of 3 NX NY NZ values, node i + NX (j + NY k))
// <-> the block layout over pitched nodes; 2048 values at a time (PACK_DOFS consecutive dense DOFs x RB right-hand sides)
// through shared memory, so both sides are read and written contiguously, eight independent values a thread, and a
// DOF's place is computed once for its right-hand sides. Right-hand sides q >= nrhs read as 0 and are not written back.
// (32-bit index arithmetic where the vector allows it: a 64-bit division is a long software sequence)
__device__ __forceinline__ long long pitchedDof(long long e, int NX, int PX) {
    if (e <= 0xffffffffLL) {
        const unsigned u = unsigned(e), nd = u / 3u, row = nd / unsigned(NX);
        return 3 * ((long long)(nd - row * unsigned(NX)) + (long long)PX * row) + (u - 3u * nd);
    }
    const long long nd = e / 3, row = nd / NX;
    return 3 * ((nd - row * NX) + (long long)PX * row) + (e - 3 * nd);
}
template <int RB> __host__ __device__ constexpr int packDofs() { return 2048 / RB; }
template <int RB>
__global__ void __launch_bounds__(256) kb_pack(double* __restrict__ dense, int nrhs, long long nDense, double* __restrict__ blk, int NX,
                                               int PX, int toBlock) {
    constexpr int PK = packDofs<RB>();
    __shared__ double tile[RB][PK + 1];
    __shared__ long long pos[PK];
    for (long long e0 = (long long)blockIdx.x * PK; e0 < nDense; e0 += (long long)gridDim.x * PK) {
        if (threadIdx.x < PK) pos[threadIdx.x] = e0 + threadIdx.x < nDense ? pitchedDof(e0 + threadIdx.x, NX, PX) : -1;
        if (toBlock) {
#pragma unroll
            for (int w = threadIdx.x; w < 2048; w += 256) {
                const int q = w / PK, de = w % PK;
                tile[q][de] = (q < nrhs && e0 + de < nDense) ? dense[(long long)q * nDense + e0 + de] : 0.0;
            }
            __syncthreads();
#pragma unroll
            for (int w = threadIdx.x; w < 2048; w += 256) {
                const int de = w / RB, q = w % RB;
                if (pos[de] >= 0) blk[pos[de] * RB + q] = tile[q][de];
            }
        } else {
            __syncthreads();
#pragma unroll
            for (int w = threadIdx.x; w < 2048; w += 256) {
                const int de = w / RB, q = w % RB;
                tile[q][de] = pos[de] >= 0 ? blk[pos[de] * RB + q] : 0.0;
            }
            __syncthreads();
#pragma unroll
            for (int w = threadIdx.x; w < 2048; w += 256) {
                const int q = w / PK, de = w % PK;
                if (q < nrhs && e0 + de < nDense) dense[(long long)q * nDense + e0 + de] = tile[q][de];
            }
        }
        __syncthreads();
    }
}

// the block preconditioner's result to the caller's dense vectors: z = z32 / vscale at active nodes (voxel_fea.cpp:859-860),
// 0 elsewhere and for zero vectors
template <int RB>
__global__ void __launch_bounds__(256) kb_unpack_z(double* __restrict__ dense, int nvec, long long nDense, const float* __restrict__ z32,
                                                   const uint8_t* __restrict__ nmask, int NX, int PX, const BlockState* bs) {
    constexpr int PK = packDofs<RB>();
    __shared__ float tile[RB][PK + 1];
    __shared__ long long pos[PK];
    __shared__ double scale[RB];  // vscale, or 0 for a zero vector
    if (threadIdx.x < RB) scale[threadIdx.x] = rhsRunning(bs, threadIdx.x) ? bs->vscale[threadIdx.x] : 0.0;
    for (long long e0 = (long long)blockIdx.x * PK; e0 < nDense; e0 += (long long)gridDim.x * PK) {
        if (threadIdx.x < PK) {
            long long p = e0 + threadIdx.x < nDense ? pitchedDof(e0 + threadIdx.x, NX, PX) : -1;
            if (p >= 0 && !(nmask[p / 3] & NM_ACTIVE)) p = -1;
            pos[threadIdx.x] = p;
        }
        __syncthreads();
#pragma unroll
        for (int w = threadIdx.x; w < 2048; w += 256) {
            const int de = w / RB, q = w % RB;
            tile[q][de] = pos[de] >= 0 ? z32[pos[de] * RB + q] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int w = threadIdx.x; w < 2048; w += 256) {
            const int q = w / PK, de = w % PK;
            if (q < nvec && e0 + de < nDense) dense[(long long)q * nDense + e0 + de] = scale[q] != 0.0 ? double(tile[q][de]) / scale[q] : 0.0;
        }
        __syncthreads();
    }
}

// held DOFs of every right-hand side set to 0 over all pitched nodes (a warm start's held values)
template <int RB>
__global__ void kb_mask_fixed(long long nNodes, const uint8_t* __restrict__ nmask, double* __restrict__ x) {
    const long long total = nNodes * 3 * RB;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
        const long long dof = e / RB, n = dof / 3;
        if (fixedDof(nmask[n], int(dof - 3 * n))) x[e] = 0.0;
    }
}

// right-hand side q of a block vector set to 0
template <int RB>
__global__ void kb_zero_rhs(long long nNodes, double* __restrict__ x, int q) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nNodes * 3; e += (long long)gridDim.x * blockDim.x) x[e * RB + q] = 0.0;
}

}  // namespace dev
}  // namespace psfea
