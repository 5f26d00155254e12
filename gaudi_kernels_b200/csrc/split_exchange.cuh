// Exchange of fp32 partial tiles inside a thread-block cluster whose CTAs took equal slices of one tile's K range.
//
// A 128 x 256 tile is cut into 32 units of 8 columns; CTA o of a cluster of cs owns units [32 o / cs, 32 (o + 1) / cs)
// (any cs up to 8, 4 to 16 units each).  Every CTA writes each unit of its partial tile into its owner's shared memory as
// 16-byte vectors, laid out [source rank][4-column group q][row ^ (q & 7)]: a warp that sends one group of 32 rows and a
// warp that receives consecutive groups of one row both touch every bank group once.  The owner adds the slices in rank
// order, which is K order: a fixed order, results do not depend on timing.  It walks its columns with consecutive lanes
// on consecutive columns, so the stores to global memory are contiguous (one row per lane took 2.1 us of a 14.7 us
// launch at M=300, K=N=4096, and 9.7 us with fp32 results).  The receive area (at most 144 KB) reuses the pipeline
// buffers: the caller puts one cluster barrier before the first send and one before finish().
#pragma once

#include "common.cuh"
#include "ptx.cuh"

namespace bfp8 {
namespace split {

constexpr int kRows = 128;
constexpr int kUnits = 32;                       // 8-column units of a 256-column tile
constexpr int kMaxCluster = 8;

__device__ __forceinline__ int first_unit(int owner, int cs) { return owner * kUnits / cs; }
// Most units one CTA owns, hence the layout's pitch: the same for every owner.
__device__ __forceinline__ int units_pitch(int cs) { return (kUnits + cs - 1) / cs; }

// Send unit `c8` (columns 8 c8 .. 8 c8 + 7) of row `row`.
__device__ __forceinline__ void send(uint32_t recv_base, int cs, int crank, int c8, int row, const float (&v)[8]) {
  const int owner = ((c8 + 1) * cs - 1) >> 5;
  const int q = (c8 - first_unit(owner, cs)) * 2;
  const uint32_t at = recv_base + static_cast<uint32_t>(crank * units_pitch(cs) * 2 + q) * (kRows * 16u);
  const uint32_t lo = (row ^ (q & 7)) * 16u, hi = kRows * 16u + (row ^ ((q + 1) & 7)) * 16u;
  if (owner == crank) {                          // own columns: plain stores, the path through the cluster is slower
    ptx::st_shared_f32x4(at + lo, v[0], v[1], v[2], v[3]);
    ptx::st_shared_f32x4(at + hi, v[4], v[5], v[6], v[7]);
  } else {
    const uint32_t to = ptx::cluster_map(at, static_cast<uint32_t>(owner));
    ptx::st_cluster_f32x4(to + lo, v[0], v[1], v[2], v[3]);
    ptx::st_cluster_f32x4(to + hi, v[4], v[5], v[6], v[7]);
  }
}

// Sums this CTA's columns of the tile over the cluster and stores them: `threads` threads call it together.  row0 / col0
// are the tile's first output row and column; apply(row, col, x) turns the sum of one element into its result.
template <bool kBf16, typename Apply>
__device__ __forceinline__ void finish(const uint8_t* recv, int cs, int crank, int tid, int threads, void* out,
                                       int64_t ldo, int row0, int col0, int m, int n, Apply apply) {
  const int u0 = first_unit(crank, cs), groups = (first_unit(crank + 1, cs) - u0) * 2, pitch = units_pitch(cs) * 2;
  const int rows = min(kRows, m - row0);
  const float4* src = reinterpret_cast<const float4*>(recv);
  int row = tid / groups, q = tid - row * groups;
  const int step_row = threads / groups, step_q = threads - step_row * groups;
  constexpr int kAhead = 4;                      // vectors summed side by side: their load and add chains overlap
  while (row < rows) {
    float v[kAhead][4];
    int at_row[kAhead], at_q[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      at_row[i] = row;
      at_q[i] = q;
      v[i][0] = v[i][1] = v[i][2] = v[i][3] = 0.0f;
      row += step_row;
      q += step_q;
      if (q >= groups) { q -= groups; ++row; }
    }
    for (int r = 0; r < cs; ++r) {
#pragma unroll
      for (int i = 0; i < kAhead; ++i) {
        // rows beyond the tile's last one are in the receive area too as long as they are below kRows
        const int rr = min(at_row[i], kRows - 1);
        const float4 p = src[(r * pitch + at_q[i]) * kRows + (rr ^ (at_q[i] & 7))];
        v[i][0] += p.x; v[i][1] += p.y; v[i][2] += p.z; v[i][3] += p.w;
      }
    }
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const int col = col0 + u0 * 8 + at_q[i] * 4;
      const int valid = at_row[i] < rows ? min(4, n - col) : 0;
      const int64_t at_out = static_cast<int64_t>(row0 + at_row[i]) * ldo + col;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < valid) v[i][j] = apply(row0 + at_row[i], col + j, v[i][j]);
      if (kBf16) {
        uint16_t* o = reinterpret_cast<uint16_t*>(out) + at_out;     // rows of bf16 results are 16-byte aligned
        if (valid == 4) {
          *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf16x2(v[i][0], v[i][1]), pack_bf16x2(v[i][2], v[i][3]));
        } else {
#pragma unroll
          for (int j = 0; j < 3; ++j)
            if (j < valid) o[j] = static_cast<uint16_t>(float_to_bf16_bits(v[i][j]));
        }
      } else {
        float* o = reinterpret_cast<float*>(out) + at_out;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j < valid) o[j] = v[i][j];
      }
    }
  }
}

}  // namespace split
}  // namespace bfp8
