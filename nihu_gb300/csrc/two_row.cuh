// The column loop shared by the FP32 regular kernels whose threads own two
// test rows: a warp owns 64 consecutive rows (lane and lane + 32, so that its
// stores are two full 256-byte runs of a column whatever the leading
// dimension), a block TWO_ROW_WARPS warps and up to TWO_ROW_COLS columns.
// The two rows are the halves of packed FP32 pairs (f32x2.cuh), the column's
// values are staged twice over, so that one instruction serves two pairs.
//
// Far rows of a column are evaluated in the loop.  The others are appended to
// the warp's lists in shared memory (a 16-bit code, row and column), each
// list one kind of work, and worked through every TWO_ROW_CHUNK columns, one
// pair per lane: a warp runs one scheme with full lanes, where a direct
// dispatch would make every lane wait for the largest point count of its 32
// neighbours.  Lists hold every pair of a chunk, so they cannot overflow; warps
// do not wait for one another.
//
// K, the operator, provides
//   struct Extra                    what it keeps of the thread's two rows; Extra extra(int i0, int i1)
//   bool far(Extra, c, q, r2)       q = (d/D)^2 of a pair, r2 = d^2: certainly the one-point rule
//   int list(float q)               of a pair that is not: 0, 1, 2, or -1 (left to the singular kernel)
//   void far_eval(Extra, c, dx, dy, dz, r2, Val &)  both rows' far values in column c of the block
//   void put<H>(Val, c, i)          stores half H (0, 1) at row i
//   void pair<LIST>(i, c)           evaluates and stores a pair of list 0 or 1
//   void general(i, c)              evaluates and stores a pair of list 2, called by GENERAL_LANES lanes
#pragma once

#include <cuda_runtime.h>

#include "f32x2.cuh"
#include "kernels.h"

namespace nihu {

constexpr int TWO_ROW_WARPS = 4;
constexpr int TWO_ROW_THREADS = 32 * TWO_ROW_WARPS;
constexpr int TWO_ROW_ROWS = 64 * TWO_ROW_WARPS;
constexpr int TWO_ROW_COLS = 16;
constexpr int TWO_ROW_CHUNK = 8;
constexpr int TWO_ROW_LIST = 64 * TWO_ROW_CHUNK;

// one column's values, each as a pair of equal halves
struct TwoRowCol {
    f2 hx, hy, hz, iw;  // centre (hi), 1/D^2
    f2 lx, ly, lz, w4;  // centre (lo), w J / (4 pi) of the one-point rule
    f2 nx, ny, nz, nw4; // unit normal, -w4
    __device__ __forceinline__ static float first(f2 x)
    {
        float a, b;
        f2_unpack(x, a, b);
        return a;
    }
    // the same as one scalar each
    __device__ __forceinline__ float4 hi() const { return make_float4(first(hx), first(hy), first(hz), first(iw)); }
    __device__ __forceinline__ float3 lo() const { return make_float3(first(lx), first(ly), first(lz)); }
    __device__ __forceinline__ float4 p0() const { return make_float4(first(w4), first(nx), first(ny), first(nz)); }
    // c_j - x_i from the hi/lo centres
    __device__ __forceinline__ float3 diff(const DevMesh &test, int i) const
    {
        const float4 ih = test.chi[i], il = test.clo[i], h = hi();
        const float3 l = lo();
        return make_float3((h.x - ih.x) + (l.x - il.x), (h.y - ih.y) + (l.y - il.y), (h.z - ih.z) + (l.z - il.z));
    }
};

// lists 0 (from the front) and 2 (from the back) share an array: together at
// most every pair of a chunk
struct TwoRowShared {
    TwoRowCol col[TWO_ROW_COLS];
    unsigned short ac[TWO_ROW_WARPS][TWO_ROW_LIST], b[TWO_ROW_WARPS][TWO_ROW_LIST];
    // stages column j of the trial mesh (call by one thread per column, then __syncthreads)
    __device__ __forceinline__ void stage(int c, const DevMesh &trial, int j)
    {
        constexpr float INV4PI = 0.0795774715459476679f;
        const float4 h = trial.chi[j], l = trial.clo[j], p = trial.p0[j];
        TwoRowCol &t = col[c];
        t.hx = f2_dup(h.x);
        t.hy = f2_dup(h.y);
        t.hz = f2_dup(h.z);
        t.iw = f2_dup(h.w);
        t.lx = f2_dup(l.x);
        t.ly = f2_dup(l.y);
        t.lz = f2_dup(l.z);
        t.w4 = f2_dup(p.x * INV4PI);
        t.nx = f2_dup(p.y);
        t.ny = f2_dup(p.z);
        t.nz = f2_dup(p.w);
        t.nw4 = f2_dup(-p.x * INV4PI);
    }
};

// what a block takes of an SM's shared memory, 1 KB of it the runtime's own
constexpr size_t TWO_ROW_SMEM = sizeof(TwoRowShared) + 1024;
// the shared-memory carveout, in per cent of 228 KB, that the kernels with two rows
// a thread and the singular ones beside them ask for alike: the 100 KB
// configuration, which holds the eight blocks an SM that launch bounds allow
constexpr int TWO_ROW_CARVEOUT = 44;
static_assert(8 * TWO_ROW_SMEM <= 100 * 1024, "eight blocks in the 100 KB configuration");

// columns per block: all TWO_ROW_COLS, or on a small mesh as few as keep
// about four blocks per SM (320 elements: one column, 320 blocks; the regular
// kernel 110 -> 13 us)
inline int two_row_cols(int n_rows, int n_cols, int sms)
{
    const int64_t rb = (n_rows + TWO_ROW_ROWS - 1) / TWO_ROW_ROWS;
    const int64_t c = rb * n_cols / (4 * (int64_t)sms);
    return (int)(c < 1 ? 1 : (c > TWO_ROW_COLS ? TWO_ROW_COLS : c));
}

// the launches that cover columns [j0, j1), launch(first column, end, grid, columns
// per block) each: one, or beyond a million columns (a few field points of a
// very large mesh) as many as grid.y, 65 535 column blocks, asks for
template <class F>
inline cudaError_t two_row_launches(int n_rows, int j0, int j1, F &&launch)
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int cols = two_row_cols(n_rows, j1 - j0, sms);
    const unsigned rows = (unsigned)((n_rows + TWO_ROW_ROWS - 1) / TWO_ROW_ROWS);
    for (int64_t j = j0; j < j1; j += 65535 * (int64_t)cols) {
        const int end = (int)(j1 - j < 65535 * (int64_t)cols ? j1 : j + 65535 * (int64_t)cols);
        launch((int)j, end, dim3(rows, (unsigned)((end - j + cols - 1) / cols)), cols);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <bool FULL, class K>
__device__ __forceinline__ void two_row_columns(const K &op, TwoRowShared &sh, const DevMesh &test, int ib, int ncols)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = test.n;
    const int i0 = ib + 64 * warp + lane, i1 = i0 + 32;
    const bool ok0 = FULL || i0 < n, ok1 = FULL || i1 < n;
    const int r0 = ok0 ? i0 : n - 1, r1 = ok1 ? i1 : n - 1;
    f2 nhx, nhy, nhz, nlx, nly, nlz;  // the rows' centres, negated
    {
        const float4 h0 = test.chi[r0], h1 = test.chi[r1], l0 = test.clo[r0], l1 = test.clo[r1];
        nhx = f2_pack(-h0.x, -h1.x);
        nhy = f2_pack(-h0.y, -h1.y);
        nhz = f2_pack(-h0.z, -h1.z);
        nlx = f2_pack(-l0.x, -l1.x);
        nly = f2_pack(-l0.y, -l1.y);
        nlz = f2_pack(-l0.z, -l1.z);
    }
    const typename K::Extra ex = op.extra(r0, r1);
    unsigned short *la = sh.ac[warp], *lb = sh.b[warp];
    const unsigned lt = (1u << lane) - 1u;
    for (int c0 = 0; c0 < ncols; c0 += TWO_ROW_CHUNK) {
        const int c1 = min(ncols, c0 + TWO_ROW_CHUNK);
        int nA = 0, nB = 0, nC = 0;  // warp-uniform
        for (int c = c0; c < c1; ++c) {
            const TwoRowCol &t = sh.col[c];
            // hi/lo centre differences: FP32 relative accuracy of r
            const f2 dx = (t.hx + nhx) + (t.lx + nlx), dy = (t.hy + nhy) + (t.ly + nly), dz = (t.hz + nhz) + (t.lz + nlz);
            // rounded in the order of the frequency batch's kernel: at large k r one
            // more ulp of r is a visible phase
            const f2 r2 = f2_fma(dz, dz, f2_fma(dx, dx, dy * dy));
            float qa, qb;
            f2_unpack(r2 * t.iw, qa, qb);
            float ra, rb;
            f2_unpack(r2, ra, rb);
            const bool fa = op.far(ex, c, qa, ra), fb = op.far(ex, c, qb, rb);
            const bool all = __all_sync(0xffffffffu, fa && fb);
            if (all || __any_sync(0xffffffffu, fa || fb)) {
                typename K::Val v;
                op.far_eval(ex, c, dx, dy, dz, r2, v);
                if (fa && ok0) op.template put<0>(v, c, i0);
                if (fb && ok1) op.template put<1>(v, c, i1);
            }
            if (all) continue;
            const int ka = fa || !ok0 ? -1 : op.list(qa), kb = fb || !ok1 ? -1 : op.list(qb);
            const unsigned short ca = (unsigned short)(lane | (c << 6)), cb = (unsigned short)((lane + 32) | (c << 6));
            const unsigned a0 = __ballot_sync(0xffffffffu, ka == 0), a1 = __ballot_sync(0xffffffffu, kb == 0);
            const unsigned b0 = __ballot_sync(0xffffffffu, ka == 1), b1 = __ballot_sync(0xffffffffu, kb == 1);
            const unsigned d0 = __ballot_sync(0xffffffffu, ka == 2), d1 = __ballot_sync(0xffffffffu, kb == 2);
            if (ka == 0) la[nA + __popc(a0 & lt)] = ca;
            if (ka == 1) lb[nB + __popc(b0 & lt)] = ca;
            if (ka == 2) la[TWO_ROW_LIST - 1 - (nC + __popc(d0 & lt))] = ca;
            nA += __popc(a0);
            nB += __popc(b0);
            nC += __popc(d0);
            if (kb == 0) la[nA + __popc(a1 & lt)] = cb;
            if (kb == 1) lb[nB + __popc(b1 & lt)] = cb;
            if (kb == 2) la[TWO_ROW_LIST - 1 - (nC + __popc(d1 & lt))] = cb;
            nA += __popc(a1);
            nB += __popc(b1);
            nC += __popc(d1);
        }
        if (nA + nB + nC) {
            const int wb = ib + 64 * warp;
            __syncwarp();  // the entries are visible to the whole warp
            for (int t = lane; t < nA; t += 32) op.template pair<0>(wb + (la[t] & 63), la[t] >> 6);
            for (int t = lane; t < nB; t += 32) op.template pair<1>(wb + (lb[t] & 63), lb[t] >> 6);
            // G lanes per entry of list 2
            constexpr int G = K::GENERAL_LANES;
            for (int t0 = 0; t0 < nC; t0 += 32 / G) {
                const int t = t0 + lane / G;
                if (t < nC) op.general(wb + (la[TWO_ROW_LIST - 1 - t] & 63), la[TWO_ROW_LIST - 1 - t] >> 6);
            }
            __syncwarp();  // read before the next chunk appends
        }
    }
}

}  // namespace nihu
