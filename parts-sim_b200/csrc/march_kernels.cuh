// The operator of a large level by reflection modes, marched along z. Included by solver.cu only.
//
// y = K x over a level's voxels with one scale s per voxel (a voxel with an own matrix counts as empty
// here; the list kernels take the nodes that touch one). The element of a cube of isotropic material
// commutes with the reflections x -> 1 - x, y -> 1 - y, z -> 1 - z and with permutations of the axes,
// the Galerkin coarse element of a uniform grid too. In the basis of sums and differences along the axes
// (mode a = (ax, ay, az): u_c[a] = sum over the corners of (+-1)^a u_c) the 24 x 24 matrix therefore
// falls apart into eight blocks of at most 3 x 3 with eight distinct numbers (ModeCoefs), where the
// row-by-row product takes 576 multiply-adds per voxel and the assembled 27-point stencil 153 per
// node. The sums and differences are shared between neighbouring voxels: per voxel 24 operations form the
// four in-plane modes of a plane of its corners, 27 combine two planes, 41 apply the blocks, 30 go back
// to the planes and 24 to the nodes: 146 in all, whatever the scales of the neighbours, so that
// graded grids, thin walls and solid parts cost the same.
//
// Every mode but the sums starts from differences of neighbouring values (the sum over a face enters
// as 4 x one corner + differences), so the rounding error scales with the field's local variation and a
// rigid translation gives exact zeros: what keeps the FP32 CG accurate on smooth search directions.
//
// One CTA computes a tile of 30 x 14 nodes (30 x 18 where a level has several waves of them; 64-bit: 30 x 10) over a range of z planes. Lane l of a warp holds the
// nodes i = 30 tx - 1 + l and the voxels right of them (lanes 0 and 31 are halo), warp w the node row
// j = (ROWS - 2) ty - 1 + w and the voxels above it (the first and last warp are halo). Planes of x are staged into a ring
// in shared memory by asynchronous copies of one value each (zeros at inactive nodes, which are not read), two planes
// ahead; a plane's in-plane modes stay in registers until the next plane has come. Finished sums go to shared
// memory once (node order in, DOF order out), from where the epilogue runs in DOF order: r, d, 1/diag and the results
// move in fully coalesced accesses, at output nodes only, so that the empty space of a lattice costs no memory
// traffic beyond whole 32-byte sectors. Sums run in a fixed order: bitwise reproducible.
//
// What bounds it: latency and issue at one CTA (16, 20 or 12 warps) an SM, not DRAM (SIMP 192x96x96: 111 MB in 43 us; warps
// issue in 68 % of the cycles, the rest goes to the turn's barrier and to the latency of the staged planes).
// The modes of two planes, the sums and the epilogue operands take 96-109 (64-bit: 143-156) registers; any spill costs
// more than the warps it buys (64 registers and 32 warps: 117 us; 64-bit at 16 rows and 128 registers:
// 92-110 us against 68 us). Two rows a thread in paired 32-bit instructions, which on this GPU run at half the rate of
// single ones, measured 83 us, 8 rows at two CTAs an SM 64 us, 10 rows 56 us, two planes a turn without register
// copies 64 us. Smoothing step, SIMP 192x96x96 / gyroid 256x256x128 / the same FP64 products: 97 / 254 / 184 / 522 us
// for 32 x 8 x 4 tiles with the 27-point stencil and per-voxel gathers before, 43 / 170 / 63 / 252 us here (43 / 190 with 14 output
// rows on both grids; 48 / 207 / 68 / 285 us with turns that branch on their position and masks loaded where they are used).
#pragma once

#include "kernels.cuh"

namespace psfea {
namespace dev {

constexpr int MARCH_NX = 30;  // output nodes of a tile along x
template <class T> __host__ __device__ constexpr int marchRows() { return sizeof(T) == 4 ? 16 : 12; }  // node rows of a tile, a warp each
constexpr int MARCH_ROWS_TALL = 20;                                                                    // the same of a tall tile (32-bit only)
constexpr double MARCH_TALL_STEP = 1.15;                                                               // a tall tile's time for a plane, of a low one's
template <class T> __host__ __device__ constexpr int marchThreads() { return 32 * marchRows<T>(); }
constexpr int MARCH_PREFETCH = 2, MARCH_STAGES = MARCH_PREFETCH + 2;  // planes of x in flight; ring slots (a power of two)
constexpr int MARCH_ROW = 96;                                         // values of a staged row: 32 nodes
constexpr int MARCH_BITS = 8;                                         // ring of output-node bits (a power of two > STAGES)
// shared memory: the ring of x planes, the finished sums of two planes (a warp's own row and its share of the next
// one), the output bits
template <class T> __host__ __device__ constexpr size_t marchSmemBytes(int rows = marchRows<T>()) {
    return (sizeof(T) * MARCH_ROW * (MARCH_STAGES + 4) + 4 * MARCH_BITS) * rows;
}

// the level's element in the reflection basis (see above), made from Kb on the host (marchCoefs)
template <class T>
struct ModeCoefs {
    T b0, a0;  // normal strains: b0 on every pair, a0 extra on the diagonal
    T a1, b1;  // the two bending modes of a block
    T c2, e2;  // shear strain, hourglass
    T b3, a3;  // twists: as the normal strains
};

// a tile: its (tx, ty) and the output planes [k0, k1)
constexpr uint16_t MARCH_EMPTY = 0x8000;  // in tx: no active node (lists over the whole grid)
struct MarchTile {
    uint16_t tx, ty, k0, k1;
};

// A plain load that stays where it stands in the turn: left to the compiler, the residual's loads went in between the epilogue's
// stores (SIMP 192x96x96 smoothing step 49.2 us, 43.0 with this). Not the read-only path: see ldv.
__device__ __forceinline__ float ldHere(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];\n" : "=f"(v) : "l"(p));
    return v;
}

// asynchronous copy of one value, or zeros (the source is then not read)
template <class T>
__device__ __forceinline__ void cpAsyncOr0(T* dst, const T* src, bool take) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(smemAddr(dst)), "l"(src), "n"(int(sizeof(T))),
                 "r"(take ? int(sizeof(T)) : 0)
                 : "memory");
}
__device__ __forceinline__ void cpAsyncCommit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpAsyncWait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// in-plane modes of the face over four nodes, lo0 lo1 (x, x + 1 of the lower row), hi0 hi1: the differences along x,
// along y, along both, and the sum; 32-bit: as the corner lo0 itself and D, 4 lo0 + D = the sum
template <class T>
struct FaceModes {
    static constexpr bool REL = sizeof(T) == 4;
    T u[3], D[REL ? 3 : 1], f10[3], f01[3], f11[3];
    __device__ __forceinline__ void make(int c, T lo0, T lo1, T hi0, T hi1) {
        const T dl = lo1 - lo0, dh = hi1 - hi0;
        f10[c] = dl + dh;
        f11[c] = dh - dl;
        if constexpr (REL) {
            const T e0 = hi0 - lo0, e1 = hi1 - lo1;
            f01[c] = e0 + e1;
            D[c] = fma(T(2), e0, f10[c]);
            u[c] = lo0;
        } else {
            const T sl = lo1 + lo0, sh = hi1 + hi0;
            f01[c] = sh - sl;
            u[c] = sh + sl;
        }
    }
    // difference of the face sums of two planes
    static __device__ __forceinline__ T sumDiff(const FaceModes& Q, const FaceModes& P, int c) {
        if constexpr (REL) return fma(T(4), Q.u[c] - P.u[c], Q.D[c] - P.D[c]);
        else return Q.u[c] - P.u[c];
    }
};

// F: the in-plane modes (00, 10, 01, 11 per component) of the plane below gathered so far. Adds to it the layer of
// voxels of scale s between the planes with modes P (below) and Q (above): G, and leaves the layer's share of
// the plane above in F.
template <class T>
__device__ __forceinline__ void marchLayer(const ModeCoefs<T>& K, T s, const FaceModes<T>& P, const FaceModes<T>& Q,
                                           T (&F)[3][4], T (&G)[3][4]) {
    T s10[3], s01[3], s11[3], d00[3], d10[3], d01[3], d11[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        s10[c] = P.f10[c] + Q.f10[c];
        s01[c] = P.f01[c] + Q.f01[c];
        s11[c] = P.f11[c] + Q.f11[c];
        d00[c] = FaceModes<T>::sumDiff(Q, P, c);
        d10[c] = Q.f10[c] - P.f10[c];
        d01[c] = Q.f01[c] - P.f01[c];
        d11[c] = Q.f11[c] - P.f11[c];
    }
    // z parts of the plane modes: o the even one (on both planes alike), w the odd one (minus below, plus above)
    auto put = [&](int c, int m, T o, T w) {
        G[c][m] = F[c][m] + o - w;
        F[c][m] = o + w;
    };
    auto put0 = [&](int c, T w) {
        G[c][0] = F[c][0] - w;
        F[c][0] = w;
    };
    const T a1 = s * K.a1, b1 = s * K.b1, e2 = s * K.e2;
    const T a0 = s * K.a0, tn = s * K.b0 * (s10[0] + s01[1] + d00[2]);
    const T a3 = s * K.a3, tt = s * K.b3 * (d01[0] + d10[1] + s11[2]);
    const T c2 = s * K.c2;
    const T gxy = c2 * (s01[0] + s10[1]), gxz = c2 * (d00[0] + s10[2]), gyz = c2 * (d00[1] + s01[2]);
    put0(0, gxz);
    put0(1, gyz);
    put0(2, fma(a0, d00[2], tn));
    put(0, 1, fma(a0, s10[0], tn), fma(a1, d10[0], b1 * d01[1]));
    put(1, 2, fma(a0, s01[1], tn), fma(a1, d01[1], b1 * d10[0]));
    put(0, 2, gxy, fma(a3, d01[0], tt));
    put(1, 1, gxy, fma(a3, d10[1], tt));
    put(2, 3, fma(a3, s11[2], tt), e2 * d11[2]);
    put(0, 3, fma(a1, s11[0], b1 * d01[2]), e2 * d11[0]);
    put(2, 2, gyz, fma(a1, d01[2], b1 * s11[0]));
    put(1, 3, fma(a1, s11[1], b1 * d10[2]), e2 * d11[1]);
    put(2, 1, gxz, fma(a1, d10[2], b1 * s11[1]));
}

// One pass y = K x with an epilogue (TOP_*; io and st as in the list kernels):
//   TOP_APPLY  y = K x (held DOFs 0 unless raw)
//   TOP_CHEB   d = c1 d + c2 D^-1 (r - K x); y = x + d      (Chebyshev / Jacobi step, 32-bit)
//   TOP_RESID  y = r - K x
//   TOP_DOT    y = K x and the CG step alpha = rz / (x . y); x . y <= 0 is a breakdown
//              (voxel_fea.cpp:902-905); held DOFs of y, where x is 0, are left with K x
// at the nodes whose mask has the bit `outBit`; the other nodes' y and d are not touched. Held DOFs have
// x = r = d = 1/diag = 0, so the smoother leaves zeros there.
// DENSE (TOP_DOT, 64-bit): the caller's vectors instead, in the reference's layout (rows of NX nodes): y is written at
// every node of the grid (0 at held DOFs and inactive nodes; a tile of the list with MARCH_EMPTY set has only those),
// x . y goes to io.dotOut, and the CTAs take the tiles in turn.
template <class T, int MODE, bool DENSE = false, int ROWS = marchRows<T>()>
__global__ void __launch_bounds__(32 * ROWS, 1)
    k_march(LevelView L, ModeCoefs<T> K, const MarchTile* __restrict__ tiles, const T* x, T* __restrict__ y,
            const float* r, float* __restrict__ d, MarchIO io, SolveState* st, double* partials, unsigned* ticket, Ctl ctl) {
    if (skipped(ctl)) return;
    constexpr int PLANE = ROWS * MARCH_ROW;
    constexpr bool CHEB = MODE == TOP_CHEB, RESID = MODE == TOP_RESID, DOT = MODE == TOP_DOT, APPLY = MODE == TOP_APPLY;
    constexpr bool MASKED = RESID || APPLY || DENSE;  // held DOFs of the result set to 0 by the masks
    extern __shared__ __align__(16) unsigned char marchSmem[];
    T* ring = reinterpret_cast<T*>(marchSmem);                       // [STAGES][ROWS][96]
    T* sums = ring + MARCH_STAGES * PLANE;                           // [2][own row, share of the next row][ROWS][96]
    unsigned* bits = reinterpret_cast<unsigned*>(sums + 4 * PLANE);  // [BITS][ROWS]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double dot = 0.0;
    // (one tile a CTA, or, DENSE, every gridDim.x-th)
    for (unsigned tileAt = blockIdx.x; tileAt == blockIdx.x || (DENSE && tileAt < unsigned(io.nTiles)); tileAt += gridDim.x) {
        if (DENSE) __syncthreads();  // the tile before is done with the shared memory
        const MarchTile tile = tiles[tileAt];
        const int k0 = tile.k0, k1 = tile.k1;
        const int i = MARCH_NX * int(tile.tx & ~MARCH_EMPTY) - 1 + lane;      // the lane's node and voxel along x
        const int j = (ROWS - 2) * int(tile.ty) - 1 + warp;  // the warp's node row
        const int XROW = DENSE ? L.NX : L.PX;  // the vectors' row pitch
        const long long PXY = (long long)L.PX * L.NY, XXY = (long long)XROW * L.NY, WXY = (long long)L.px * L.ny;  // mask, vector and word planes
        const bool nodeIn = i >= 0 && i < L.NX && j >= 0 && j < L.NY, nextIn = i >= 0 && i < L.NX && j + 1 >= 0 && j + 1 < L.NY;
        // the last lane's and the last row's voxels lack a corner: they count as empty (and shape halo nodes only)
        const bool voxIn = i >= 0 && i < L.nx && lane < 31 && j >= 0 && j < L.ny && warp < ROWS - 1;
        const bool outRow = warp > 0 && warp < ROWS - 1;
        // offsets within a plane: the lane's node, its voxel, and the row's value `lane` in DOF order; the row's values
        // lane + 32 q belong to the nodes at bits mq[q]
        const int nodeAt = i + L.PX * j, wordAt = i + L.px * j, valueAt = 3 * (i - lane + XROW * j) + lane;
        unsigned mq[3];
#pragma unroll
        for (int q = 0; q < 3; q++) mq[q] = 1u << ((lane + 32 * q) / 3);
        auto maskAt = [&](bool in, int at, int k) -> unsigned {  // of a node of plane k, 0 outside the grid
            const uint8_t* m = L.nmask + k * PXY;
            return (in && unsigned(k) < unsigned(L.NZ)) ? unsigned(__ldg(m + at)) : 0u;
        };
        auto stage = [&](int k, unsigned mk) {
            T* dst = ring + ((k + 1) & (MARCH_STAGES - 1)) * PLANE + warp * MARCH_ROW + lane;
            const unsigned act = __ballot_sync(0xffffffffu, mk & NM_ACTIVE), out = __ballot_sync(0xffffffffu, DENSE ? nodeIn : (mk & io.outBit) != 0);
            if (lane == 0) bits[((k + 1) & (MARCH_BITS - 1)) * ROWS + warp] = (outRow && k >= k0 && k < k1) ? out & 0x7ffffffeu : 0u;
            const T* src = x + 3 * k * XXY + valueAt;  // (read at the active nodes only)
#pragma unroll
            for (int q = 0; q < 3; q++) cpAsyncOr0(dst + 32 * q, src + 32 * q, act & mq[q]);
            cpAsyncCommit();
        };

        T F[3][4] = {};
        float er[3] = {}, ed[3] = {}, ei[3] = {};  // epilogue operands of the plane being completed, loaded a step ahead
        unsigned eb = 0, mkNext;
        unsigned holdAhead = 0, holdNextAhead = 0;  // the masks of the warp's own row and the next, a step ahead
        uint32_t wNext = 0;  // the voxel word above the plane, a step ahead; used as loaded only then

        // the finished sums of plane k (in shared memory) through the epilogue
        auto finish = [&](int k) {
            const T* sm = sums + ((k + 1) & 1) * 2 * PLANE + warp * MARCH_ROW + lane;
            const T* own = ring + ((k + 1) & (MARCH_STAGES - 1)) * PLANE + warp * MARCH_ROW + lane;
            T kx[3], xv[3];
#pragma unroll
            for (int q = 0; q < 3; q++) {
                kx[q] = sm[32 * q];
                xv[q] = own[32 * q];
            }
            if (warp > 0)
#pragma unroll
                for (int q = 0; q < 3; q++) kx[q] += sm[PLANE - MARCH_ROW + 32 * q];  // the warp below's share
            if (L.dadd) {
#pragma unroll
                for (int q = 0; q < 3; q++)
                    if (eb & mq[q]) {
                        const long long id = 3 * (k * PXY + nodeAt - lane) + lane + 32 * q, n = id / 3;  // (pitched)
                        // (a held DOF keeps its 0: the solver's x is 0 there)
                        if (!((APPLY || DENSE) && !io.raw && fixedDof(__ldg(L.nmask + n), int(id - 3 * n))))
                            kx[q] += (sizeof(T) == 8 ? T(L.dadd[id]) : T(L.dadd32[id])) * xv[q];
                    }
            }
            T* yr = y + 3 * k * XXY + valueAt;
            float* dr = d + 3 * k * XXY + valueAt;
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const bool p = eb & mq[q];
                if constexpr (CHEB) {
                    const float dn = io.c1 * ed[q] + io.c2 * ei[q] * (er[q] - float(kx[q]));
                    if (p) dr[32 * q] = dn;
                    if (p) yr[32 * q] = xv[q] + T(dn);
                } else if constexpr (RESID) {
                    if (p) yr[32 * q] = T(er[q]) - kx[q];
                } else {
                    if (p) yr[32 * q] = kx[q];
                    if (DOT && p) dot += double(xv[q]) * double(kx[q]);
                }
            }
        };

        if (DENSE && (tile.tx & MARCH_EMPTY)) {  // no active node: zeros
            if (outRow && j < L.NY)
                for (int k = k0; k < k1; k++)
#pragma unroll
                    for (int q = 0; q < 3; q++)
                        if (__ballot_sync(0xffffffffu, nodeIn) & 0x7ffffffeu & mq[q]) y[3 * k * XXY + valueAt + 32 * q] = T(0);
            continue;
        }

        // planes k0 - 1 .. k1, PREFETCH of them in flight
#pragma unroll
        for (int p = 0; p < MARCH_PREFETCH; p++) stage(k0 - 1 + p, maskAt(nodeIn, nodeAt, k0 - 1 + p));
        mkNext = maskAt(nodeIn, nodeAt, k0 - 1 + MARCH_PREFETCH);
        if (lane == 0) bits[((k0 - 1) & (MARCH_BITS - 1)) * ROWS + warp] = 0u;  // plane k0 - 2
        FaceModes<T> P{}, Q;  // the modes of planes k - 1 and k
        // The turns at both ends run the whole body too: planes outside [k0, k1) have no output bits, the layer below
        // plane k0 - 1 has scale 0 and planes past k1 are staged as zeros. Without branches the compiler can spread the loads and
        // the epilogue over the arithmetic.
#pragma unroll 2  // (the modes change places without copies)
        for (int k = k0 - 1; k <= k1; k++) {
            cpAsyncWait<MARCH_PREFETCH - 1>();
            __syncthreads();
            finish(k - 2);
            __syncwarp();
            stage(k + MARCH_PREFETCH, mkNext);  // into the slot of plane k - 2, whose last reader was this warp, just now
            mkNext = maskAt(nodeIn && k + MARCH_PREFETCH < k1, nodeAt, k + MARCH_PREFETCH + 1);
            eb = bits[(k & (MARCH_BITS - 1)) * ROWS + warp];
            const long long at = 3 * (k - 1) * XXY + valueAt;
            if (CHEB || RESID)
#pragma unroll
                for (int q = 0; q < 3; q++)
                    if (eb & mq[q]) er[q] = ldHere(r + at + 32 * q);
            if (CHEB) {
#pragma unroll
                for (int q = 0; q < 3; q++)
                    if (eb & mq[q]) ed[q] = d[at + 32 * q];
#pragma unroll
                for (int q = 0; q < 3; q++)
                    if (eb & mq[q]) ei[q] = __ldg(L.invD + at + 32 * q);
            }
            const unsigned hold = holdAhead, holdNext = holdNextAhead;  // plane k - 1
            if (MASKED && !io.raw) {
                holdAhead = maskAt(nodeIn, nodeAt, k);
                holdNextAhead = maskAt(nextIn, nodeAt + L.PX, k);
            }
            const T s = T(fmaxf(__uint_as_float(wNext), 0.f));  // of the layer below (an own matrix's word is a negative float or NaN: 0)
            wNext = (voxIn && unsigned(k) < unsigned(L.nz)) ? __ldg(L.word + k * WXY + wordAt) : 0u;
            const T* pl = ring + ((k + 1) & (MARCH_STAGES - 1)) * PLANE + warp * MARCH_ROW + 3 * lane;
            const int right = lane < 31 ? 3 : 0, up = warp < ROWS - 1 ? MARCH_ROW : 0;
#pragma unroll
            for (int c = 0; c < 3; c++) Q.make(c, pl[c], pl[c + right], pl[up + c], pl[up + c + right]);
            T G[3][4];
            if (sizeof(T) == 4 || s != T(0)) {
                marchLayer<T>(K, s, P, Q, F, G);
            } else {  // an empty voxel (64-bit: whatever x holds at its corners, infinities too, stays out)
#pragma unroll
                for (int c = 0; c < 3; c++)
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        G[c][m] = F[c][m];
                        F[c][m] = T(0);
                    }
            }
            // plane k - 1 back to its nodes: x neighbours by shuffles, the next row's share to its warp
            T* sm = sums + (k & 1) * 2 * PLANE + warp * MARCH_ROW + 3 * lane;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const T s0 = G[c][0] - G[c][2], s1 = G[c][0] + G[c][2], t0 = G[c][1] - G[c][3], t1 = G[c][1] + G[c][3];
                T own = s0 - t0 + __shfl_up_sync(0xffffffffu, s0 + t0, 1);
                T next = s1 - t1 + __shfl_up_sync(0xffffffffu, s1 + t1, 1);
                if (MASKED && !io.raw && ((hold >> c) & 1u)) own = T(0);
                if (MASKED && !io.raw && ((holdNext >> c) & 1u)) next = T(0);
                sm[c] = own;
                sm[PLANE + c] = next;
            }
            P = Q;
        }
        cpAsyncWait<0>();
        __syncthreads();
        finish(k1 - 1);
    }
    if (DOT) {
        double vv[1] = {dot};
        double tot[1];
        if (gridReduce<1>(vv, 0u, partials, ticket, tot) && threadIdx.x == 0) {
            const double pq = tot[0];
            if (DENSE) {
                *io.dotOut = pq;
                return;
            }
            if (io.partial) {  // the list kernel adds its share and finishes the step
                st->pqPart = pq;
                return;
            }
            st->pq = pq;
            if (!(pq > 0)) {
                st->status = ST_BREAKDOWN;
                if (st->mixed) st->fold = 1;  // fold what there is, then stop
                else st->done = 1;
            } else {
                st->alpha = st->rz / pq;
            }
        }
    }
}

}  // namespace dev
}  // namespace psfea
