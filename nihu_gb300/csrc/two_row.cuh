// The column loop shared by the FP32 regular kernels whose threads own two
// test rows: a warp owns 64 consecutive rows (lane and lane + 32, so that its
// stores are two full 256-byte runs of a column whatever the leading
// dimension), a block TWO_ROW_WARPS warps and up to TWO_ROW_COLS columns.
//
// A column whose 64 pairs are all far takes one vote and one evaluation per
// row.  Otherwise its far rows are evaluated there, and the others appended
// to the warp's lists in shared memory (a 16-bit code, row and column), each
// list one kind of work, and worked through every TWO_ROW_CHUNK columns, one
// pair per lane: a warp runs one scheme with full lanes, where a direct
// dispatch would make every lane wait for the largest point count of its 32
// neighbours.  Lists hold every pair of a chunk, so they cannot overflow; warps
// do not wait for one another.
//
// K, the operator, provides
//   struct Row                      a test row's data, Row load(int i)
//   bool far(float q)               q = (d/D)^2 of a pair: certainly the one-point rule
//   int list(float q)               of a pair that is not: 0, 1, 2, or -1 (left to the singular kernel)
//   void far_pair(Row, c, dx, dy, dz, i)  evaluates and stores a far pair of column c (in the block)
//   void pair<LIST>(i, c)           evaluates and stores a listed pair
#pragma once

#include <cuda_runtime.h>

namespace nihu {

constexpr int TWO_ROW_WARPS = 8;
constexpr int TWO_ROW_THREADS = 32 * TWO_ROW_WARPS;
constexpr int TWO_ROW_ROWS = 64 * TWO_ROW_WARPS;
constexpr int TWO_ROW_COLS = 32;
constexpr int TWO_ROW_CHUNK = 8;
constexpr int TWO_ROW_LIST = 64 * TWO_ROW_CHUNK;

// lists 0 (from the front) and 2 (from the back) share an array: together at
// most every pair of a chunk
struct TwoRowLists {
    unsigned short ac[TWO_ROW_WARPS][TWO_ROW_LIST], b[TWO_ROW_WARPS][TWO_ROW_LIST];
};

// columns per block: all TWO_ROW_COLS, or on a small mesh as few as keep
// about four blocks per SM (one column: 320 elements, 320 blocks)
inline int two_row_cols(int n_rows, int n_cols, int sms)
{
    const int64_t rb = (n_rows + TWO_ROW_ROWS - 1) / TWO_ROW_ROWS;
    const int64_t c = rb * n_cols / (4 * (int64_t)sms);
    return (int)(c < 1 ? 1 : (c > TWO_ROW_COLS ? TWO_ROW_COLS : c));
}

template <bool FULL, class K>
__device__ __forceinline__ void two_row_columns(const K &op, TwoRowLists &lists, const float4 *s_hi, const float4 *s_lo,
                                                int ib, int n, int ncols)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i0 = ib + 64 * warp + lane, i1 = i0 + 32;
    const bool ok0 = FULL || i0 < n, ok1 = FULL || i1 < n;
    const typename K::Row r0 = op.load(ok0 ? i0 : n - 1), r1 = op.load(ok1 ? i1 : n - 1);
    unsigned short *la = lists.ac[warp], *lb = lists.b[warp];
    const unsigned lt = (1u << lane) - 1u;
    for (int c0 = 0; c0 < ncols; c0 += TWO_ROW_CHUNK) {
        const int c1 = min(ncols, c0 + TWO_ROW_CHUNK);
        int nA = 0, nB = 0, nC = 0;  // warp-uniform
        for (int c = c0; c < c1; ++c) {
            const float4 h = s_hi[c], l = s_lo[c];
            // hi/lo centre differences: FP32 relative accuracy of r
            const float ax = (h.x - r0.hi.x) + (l.x - r0.lo.x), ay = (h.y - r0.hi.y) + (l.y - r0.lo.y),
                        az = (h.z - r0.hi.z) + (l.z - r0.lo.z);
            const float bx = (h.x - r1.hi.x) + (l.x - r1.lo.x), by = (h.y - r1.hi.y) + (l.y - r1.lo.y),
                        bz = (h.z - r1.hi.z) + (l.z - r1.lo.z);
            const float qa = (ax * ax + ay * ay + az * az) * h.w, qb = (bx * bx + by * by + bz * bz) * h.w;
            const bool fa = op.far(qa), fb = op.far(qb);
            if (__all_sync(0xffffffffu, fa && fb)) {
                if (FULL || ok0) op.far_pair(r0, c, ax, ay, az, i0);
                if (FULL || ok1) op.far_pair(r1, c, bx, by, bz, i1);
                continue;
            }
            if (fa && ok0) op.far_pair(r0, c, ax, ay, az, i0);
            if (fb && ok1) op.far_pair(r1, c, bx, by, bz, i1);
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
            for (int t = lane; t < nC; t += 32)
                op.template pair<2>(wb + (la[TWO_ROW_LIST - 1 - t] & 63), la[TWO_ROW_LIST - 1 - t] >> 6);
            __syncwarp();  // read before the next chunk appends
        }
    }
}

}  // namespace nihu
