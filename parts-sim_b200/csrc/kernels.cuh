// Device code of the voxel solve (sm_100a). Included by solver.cu only.
//
// Data layout in HBM, per level: xyz-interleaved DOF vectors (DOF 3n + d) over pitched node rows,
// node n = i + PX (j + NY k) with the row pitch PX = NX rounded up to a multiple of 4, so that every
// row of 3 PX values starts on a 16-byte boundary (the rule of tensor-memory-access copies); the
// padding nodes i >= NX are inactive with all DOFs held, and stay 0 in every vector. One 32-bit word
// per voxel (0 empty, float bits of s for s * Kb, OWN_BIT | index of an own 24x24 matrix) over rows
// of px = nx rounded up to a multiple of 4 words (padding words 0), one mask byte per node (fixed
// DOFs, active, uniform). The reference's dense layout (pitch NX) exists only at the C ABI.
// The level's Kb (576) and its assembled 27-point stencil (243) travel as kernel parameters, so
// every coefficient is a constant-bank operand of the FMA that uses it.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cstdint>

namespace psfea {
namespace dev {

constexpr uint32_t OWN_BIT = 0x80000000u;
constexpr uint8_t NM_ACTIVE = 8, NM_UNIFORM = 16, NM_PLAIN = 32;

struct LevelView {
    int nx, ny, nz, NX, NY, NZ;  // voxel and node counts per axis
    int PX, px;                  // row pitches: nodes (PX >= NX) and voxel words (px >= nx), multiples of 4
    long long nNodes;            // PX NY NZ: the length of every per-node array
    const uint32_t* word;
    const uint8_t* nmask;
    const float* own;       // own matrices, 32-bit
    const __half* own16;    // the same as halves times hs (mixed precision), or null
    float hs;
    const double* dadd;     // diagonal shift per DOF, or null
    const float* dadd32;
    const float* invD;      // 1 / diag per DOF (0 where fixed), 32-bit
    __host__ __device__ long long wi(int i, int j, int k) const { return i + (long long)px * (j + (long long)ny * k); }
};

template <class T>
struct Coefs {
    alignas(16) T Kb[576];  // row-major 24x24 (16-byte aligned: read as pairs by the paired FMAs)
    T S[243];               // [m][3 d + c], m = (ox+1) + 3 (oy+1) + 9 (oz+1)
};
// corner index of the unit offset (x, y, z)
__host__ __device__ constexpr int cornerOf(int x, int y, int z) { return (y ? (x ? 2 : 3) : (x ? 1 : 0)) + 4 * z; }

// the three rows of corner a of a 24x24 matrix times the 24 corner values xe, added to t[3]:
//   Kb (the level's uniform matrix, kernel parameter): 32-bit values pair consecutive columns in
//   paired FMAs (__ffma2_rn; the pair's two partial sums are added at the end)
//   own16 (FP16 Galerkin matrices): 16-byte loads of eight halves each, widened to the value type
template <class T>
__device__ __forceinline__ void kbRows(const T* Kb, int a, const T xe[24], T t[3]) {
    if constexpr (sizeof(T) == 4) {
        const float2* K2 = reinterpret_cast<const float2*>(Kb) + 36 * a;
        float2 p0 = make_float2(0.f, 0.f), p1 = p0, p2 = p0;
#pragma unroll
        for (int q = 0; q < 12; q++) {
            const float2 xq = make_float2(xe[2 * q], xe[2 * q + 1]);
            p0 = __ffma2_rn(K2[q], xq, p0);
            p1 = __ffma2_rn(K2[12 + q], xq, p1);
            p2 = __ffma2_rn(K2[24 + q], xq, p2);
        }
        t[0] = p0.x + p0.y;
        t[1] = p1.x + p1.y;
        t[2] = p2.x + p2.y;
    } else {
        T t0 = 0, t1 = 0, t2 = 0;
#pragma unroll
        for (int q = 0; q < 24; q++) {
            t0 += Kb[(3 * a + 0) * 24 + q] * xe[q];
            t1 += Kb[(3 * a + 1) * 24 + q] * xe[q];
            t2 += Kb[(3 * a + 2) * 24 + q] * xe[q];
        }
        t[0] = t0;
        t[1] = t1;
        t[2] = t2;
    }
}
// SMEM: M is in shared memory (plain loads; the read-only global path otherwise)
template <class T, bool SMEM = false>
__device__ __forceinline__ void own16Rows(const __half* M, const T xe[24], T t[3]) {
    const uint4* K16 = reinterpret_cast<const uint4*>(M);  // 72 halves: rows d at [24 d, 24 d + 24)
#pragma unroll
    for (int d = 0; d < 3; d++) {
        T acc = 0;
#pragma unroll
        for (int g = 0; g < 3; g++) {
            const uint4 u = SMEM ? K16[3 * d + g] : __ldg(K16 + 3 * d + g);
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float2 kv = __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
                acc += T(kv.x) * xe[8 * g + 2 * e] + T(kv.y) * xe[8 * g + 2 * e + 1];
            }
        }
        t[d] = acc;
    }
}

// (K x) at node (i, j, k). Uniform nodes: s times the assembled stencil, structural zeros skipped
// (entry (d, c) of neighbour o is zero by the cube's reflection symmetry unless d == c or both
// o_d and o_c are nonzero: 153 of 243). Others: the rows of the node's corner in each of its up
// to 8 voxels (native/src/fea/voxel_fea.cpp:422-486 computes the same sums).
//
// DIFF: every value enters as its difference from the node's own value, x_m - x_n. Rows of K
// annihilate rigid translations, so the product is unchanged in exact arithmetic, but its 32-bit
// rounding error then scales with the field's local variation instead of its magnitude: what keeps
// the FP32 CG accurate on smooth search directions. (The reference's WGSL kernel forms its
// products the same way, native/shaders/fea.wgsl:91-92.) The diagonal shift is not a
// translation-free term and always uses x_n itself.
//
// x is read at node index n with row pitch XP (L.PX for the level's own vectors); the diagonal
// shift at the level's node index nm. S: the stride between consecutive DOFs of x (1 for one
// vector; the block width for the RHS-minor layout of a multi-RHS block, x then pointing at the
// lane's right-hand side). SMEM: L.own / L.own16 point at a copy in shared memory.
template <class T, bool OWN16, bool DIFF = false, int S = 1, bool SMEM = false>
__device__ __forceinline__ void applyAt(const LevelView& L, const Coefs<T>& C, const T* x, int i, int j, int k,
                                        long long n, uint8_t mask, T acc[3], long long XP, long long nm) {
    acc[0] = acc[1] = acc[2] = T(0);
    if (!(mask & NM_ACTIVE)) return;
    const long long NX = XP, NXY = XP * L.NY;
    T own0 = 0, own1 = 0, own2 = 0;
    if (DIFF) {
        own0 = x[3 * S * n];
        own1 = x[3 * S * n + S];
        own2 = x[3 * S * n + 2 * S];
    }
    if (mask & NM_UNIFORM) {
        const float s = __uint_as_float(__ldg(L.word + L.wi(i - 1, j - 1, k - 1)));
        T a0 = 0, a1 = 0, a2 = 0;
#pragma unroll
        for (int m = 0; m < 27; m++) {
            const int ox = m % 3 - 1, oy = (m / 3) % 3 - 1, oz = m / 9 - 1;
            if (DIFF && m == 13) continue;  // the node itself: a zero difference
            const T* xp = x + 3 * S * (n + ox + oy * NX + oz * NXY);
            const T x0 = xp[0] - own0, x1 = xp[S] - own1, x2 = xp[2 * S] - own2;
            a0 += C.S[m * 9 + 0] * x0;
            a1 += C.S[m * 9 + 4] * x1;
            a2 += C.S[m * 9 + 8] * x2;
            if (ox && oy) { a0 += C.S[m * 9 + 1] * x1; a1 += C.S[m * 9 + 3] * x0; }
            if (ox && oz) { a0 += C.S[m * 9 + 2] * x2; a2 += C.S[m * 9 + 6] * x0; }
            if (oy && oz) { a1 += C.S[m * 9 + 5] * x2; a2 += C.S[m * 9 + 7] * x1; }
        }
        acc[0] = T(s) * a0;
        acc[1] = T(s) * a1;
        acc[2] = T(s) * a2;
    } else {
#pragma unroll
        for (int v = 0; v < 8; v++) {
            const int di = v & 1, dj = (v >> 1) & 1, dk = v >> 2;
            const int ei = i - 1 + di, ej = j - 1 + dj, ek = k - 1 + dk;
            if (ei < 0 || ej < 0 || ek < 0 || ei >= L.nx || ej >= L.ny || ek >= L.nz) continue;
            const uint32_t w = __ldg(L.word + L.wi(ei, ej, ek));
            if (w == 0) continue;
            const int a = cornerOf(1 - di, 1 - dj, 1 - dk);
            // the voxel's 8 corner values
            T xe[24];
#pragma unroll
            for (int b = 0; b < 8; b++) {
                const int bx = (b == 1 || b == 2 || b == 5 || b == 6), by = (b == 2 || b == 3 || b == 6 || b == 7), bz = b >> 2;
                const T* xp = x + 3 * S * (n + (di + bx - 1) + (dj + by - 1) * NX + (dk + bz - 1) * NXY);
                xe[3 * b] = xp[0] - own0;
                xe[3 * b + 1] = xp[S] - own1;
                xe[3 * b + 2] = xp[2 * S] - own2;
            }
            if (!(w & OWN_BIT)) {
                T t[3];
                kbRows<T>(C.Kb, a, xe, t);
                const T s = T(__uint_as_float(w));
                acc[0] += s * t[0];
                acc[1] += s * t[1];
                acc[2] += s * t[2];
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
        }
    }
    if (L.dadd) {
#pragma unroll
        for (int d = 0; d < 3; d++) acc[d] += (sizeof(T) == 8 ? T(L.dadd[3 * nm + d]) : T(L.dadd32[3 * nm + d])) * x[(3 * n + d) * S];
    }
}

// An entry of a solve's vector as T: FP32 / FP64 storage as is, FP16 storage converted. Plain loads, and no const __restrict__ on the
// vectors the kernels of an iteration read: the read-only path (__ldg, and what the compiler makes of const
// __restrict__) asks for data that nothing writes while the kernel is resident, and a programmatically launched kernel is
// resident while the one before it still writes them. Masks, words, lists, matrices, stencils and 1/diag keep that path.
template <class T>
__device__ __forceinline__ T ldv(const float* p) { return T(*p); }
template <class T>
__device__ __forceinline__ T ldv(const double* p) { return T(*p); }
template <class T>
__device__ __forceinline__ T ldv(const __half* p) { return T(__half2float(*p)); }
__device__ __forceinline__ void stv(float* p, float v) { *p = v; }
__device__ __forceinline__ void stv(__half* p, float v) { *p = __float2half_rn(v); }

// Layout: coefficient c = 9 m + 3 p + q (m the neighbour (ox + 1) + 3 (oy + 1) + 9 (oz + 1), p the
// row and q the column component) of listed node t sits in chunk c / CW of CW consecutive values
// (16 bytes: CW = 4 floats or 8 halves), chunks stored chunk-major over the nodes, so that a warp
// reads one chunk of 32 consecutive nodes as 512 contiguous bytes. The tail of the last chunk is 0.
template <int CW>
__host__ __device__ constexpr int stnChunks() { return (243 + CW - 1) / CW; }
template <int CW>
__host__ __device__ __forceinline__ long long stnAt(int c, long long t, long long count) { return ((c / CW) * count + t) * CW + c % CW; }

// one 16-byte chunk of coefficients as floats
__device__ __forceinline__ void ldChunk(const float* p, float (&v)[4]) {
    const float4 u = __ldcs(reinterpret_cast<const float4*>(p));
    v[0] = u.x;
    v[1] = u.y;
    v[2] = u.z;
    v[3] = u.w;
}
__device__ __forceinline__ void ldChunk(const __half* p, float (&v)[8]) {
    const uint4 u = __ldcs(reinterpret_cast<const uint4*>(p));
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
        v[2 * e] = f.x;
        v[2 * e + 1] = f.y;
    }
}

__device__ __forceinline__ void ldChunk(const double* p, double (&v)[2]) {
    const double2 u = __ldcs(reinterpret_cast<const double2*>(p));
    v[0] = u.x;
    v[1] = u.y;
}

__device__ __forceinline__ void nodeCoords(const LevelView& L, long long n, int& i, int& j, int& k) {
    if (n <= 0xffffffffLL) {  // two 32-bit divisions: a 64-bit one is a long software sequence
        const unsigned u = unsigned(n), px = unsigned(L.PX), ny = unsigned(L.NY);
        const unsigned row = u / px, kk = row / ny;
        i = int(u - row * px);
        j = int(row - kk * ny);
        k = int(kk);
        return;
    }
    const long long row = n / L.PX;
    i = int(n - row * L.PX);
    j = int(row % L.NY);
    k = int(row / L.NY);
}

// ---- deterministic grid reductions: per-block tree sums, the last block folds the partials in
// block order (so results are bitwise reproducible for a given launch shape) ----

template <int K>
__device__ __forceinline__ void warpReduce(double (&v)[K], unsigned maxMask) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < K; q++) {
            const double w = __shfl_down_sync(0xffffffffu, v[q], o);
            v[q] = ((maxMask >> q) & 1) ? fmax(v[q], w) : v[q] + w;
        }
}

// Reduces v over the block into out (thread 0's copy valid). sh: 32 * K doubles of shared memory.
template <int K>
__device__ __forceinline__ void blockReduce(double (&v)[K], unsigned maxMask, double* sh) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    warpReduce<K>(v, maxMask);
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < K; q++) sh[wid * K + q] = v[q];
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int q = 0; q < K; q++) v[q] = lane < nw ? sh[lane * K + q] : 0.0;
        warpReduce<K>(v, maxMask);
    }
}

// Whole-grid reduction: every block writes its partial; returns true in the last block to finish,
// where out[] (in every thread) holds the totals. ticket must start at 0 and is left at 0.
template <int K>
__device__ bool gridReduce(double (&v)[K], unsigned maxMask, double* partials, unsigned* ticket, double (&out)[K]) {
    __shared__ double sh[32 * K];
    __shared__ bool last;
    blockReduce<K>(v, maxMask, sh);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < K; q++) partials[(size_t)blockIdx.x * K + q] = v[q];
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double acc[K];
#pragma unroll
    for (int q = 0; q < K; q++) acc[q] = 0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x)
#pragma unroll
        for (int q = 0; q < K; q++) {
            const double p = __ldcg(partials + (size_t)b * K + q);
            acc[q] = ((maxMask >> q) & 1) ? fmax(acc[q], p) : acc[q] + p;
        }
    __syncthreads();
    blockReduce<K>(acc, maxMask, sh);
    __shared__ double res[K];
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < K; q++) res[q] = acc[q];
        *ticket = 0;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < K; q++) out[q] = res[q];
    return true;
}

}  // namespace dev
}  // namespace psfea

namespace psfea {
namespace dev {

// ---------------------------------------------------------------- shared by the operator kernels

// epilogues of the operator passes over a large level's nodes
enum { TOP_APPLY = 0, TOP_CHEB = 1, TOP_RESID = 2, TOP_DOT = 3 };

struct MarchIO {
    float c1, c2;      // CHEB: d = c1 d + c2 D^-1 (r - K x)
    int raw;           // APPLY: keep held DOFs
    int partial;       // DOT: leave the step to the list kernel (st->pqPart holds the marched share)
    unsigned outBit;   // the mask bit of the nodes to compute
    int nTiles;        // DENSE: the tiles of the list, and where x . y goes
    double* dotOut;
};

__host__ __device__ constexpr uint32_t packTile(int tx, int ty, int tz) { return uint32_t(tx) | (uint32_t(ty) << 11) | (uint32_t(tz) << 22); }

__host__ __device__ constexpr size_t align128(size_t b) { return (b + 127) & ~size_t(127); }

// Bound on the polls of a shared-memory barrier. A wait that never completes (it cannot in a correct
// launch) is given up: the CTA records ST_ERR_STAGING in st->err and ends the solve.
constexpr unsigned TILE_WAIT_POLLS = 1u << 22;
constexpr int ST_ERR_STAGING = 1;

// ---- shared-memory barrier primitives (PTX, sm_90 and later)
__device__ __forceinline__ unsigned smemAddr(const void* p) { return unsigned(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbarInit(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smemAddr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ bool mbarTryWait(uint64_t* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smemAddr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded wait for the completion of the barrier phase with the given parity: false after `limit`
// polls (each poll may suspend the thread for a hardware-defined time)
__device__ __forceinline__ bool mbarWaitParity(uint64_t* bar, unsigned parity, unsigned limit) {
    for (unsigned it = 0; it < limit; it++)
        if (mbarTryWait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ bool mbarWait(uint64_t* bar, unsigned limit) { return mbarWaitParity(bar, 0, limit); }

}  // namespace dev
}  // namespace psfea
