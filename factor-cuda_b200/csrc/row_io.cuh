// row_io.cuh -- one section (a date's row of N columns) held in registers: the
// vector layout the shared-memory rank kernels share, its loads and stores,
// the compaction offsets and the shared-memory layout of the radix forms.
#pragma once

#include "block_sort.cuh"
#include "fcb_kernels.h"

namespace fcb {

__host__ __device__ inline size_t al16(size_t x) { return (x + 15) & ~size_t(15); }

// Row loads in the vector layout: thread tid owns columns 4*(j*NT + tid) + k.
template <int NT, int V, bool STREAM>
FCB_DEV void load_row_f32(const float* __restrict__ row, int N, float (&x)[4 * V]) {
  const bool al = (reinterpret_cast<uintptr_t>(row) & 15u) == 0;
  const float qnan = __uint_as_float(kQuietNanBits);
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int i0 = 4 * (j * NT + static_cast<int>(threadIdx.x));
    if (al && i0 + 3 < N) {
      const float4* p = reinterpret_cast<const float4*>(row + i0);
      const float4 q = STREAM ? __ldcs(p) : __ldg(p);
      x[4 * j] = q.x;
      x[4 * j + 1] = q.y;
      x[4 * j + 2] = q.z;
      x[4 * j + 3] = q.w;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) x[4 * j + k] = (i0 + k < N) ? row[i0 + k] : qnan;
    }
  }
}

template <int NT, int V>
FCB_DEV void load_words(const uint32_t* __restrict__ row, int N, uint32_t (&w)[4 * V]) {
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int i0 = 4 * (j * NT + static_cast<int>(threadIdx.x));
    if (i0 + 3 < N) {
      const uint4 q = __ldg(reinterpret_cast<const uint4*>(row + i0));
      w[4 * j] = q.x;
      w[4 * j + 1] = q.y;
      w[4 * j + 2] = q.z;
      w[4 * j + 3] = q.w;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) w[4 * j + k] = (i0 + k < N) ? row[i0 + k] : 0u;
    }
  }
}

// 0/1 bytes in the vector layout (all ones when there is no mask).
template <int NT, int V>
FCB_DEV void load_mask4(const uint8_t* __restrict__ row, int N, uint32_t (&m)[4 * V]) {
  const bool al = (reinterpret_cast<uintptr_t>(row) & 3u) == 0;
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int i0 = 4 * (j * NT + static_cast<int>(threadIdx.x));
    if (row == nullptr) {
#pragma unroll
      for (int k = 0; k < 4; ++k) m[4 * j + k] = (i0 + k < N) ? 1u : 0u;
    } else if (al && i0 + 3 < N) {
      const uint32_t q = __ldcs(reinterpret_cast<const unsigned int*>(row + i0));
#pragma unroll
      for (int k = 0; k < 4; ++k) m[4 * j + k] = ((q >> (8 * k)) & 0xFFu) ? 1u : 0u;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) m[4 * j + k] = (i0 + k < N && row[i0 + k] != 0) ? 1u : 0u;
    }
  }
}

// Columns i0 .. i0+3 of a row (al: the row is 16-byte aligned).
FCB_DEV void store_quad(float* __restrict__ row, bool al, int N, int i0, float4 v) {
  if (al && i0 + 3 < N) {
    __stcs(reinterpret_cast<float4*>(row + i0), v);
  } else {
    if (i0 < N) row[i0] = v.x;
    if (i0 + 1 < N) row[i0 + 1] = v.y;
    if (i0 + 2 < N) row[i0 + 2] = v.z;
    if (i0 + 3 < N) row[i0 + 3] = v.w;
  }
}

template <int NT, int V>
FCB_DEV void store_row_f32v(float* __restrict__ row, int N, const float (&v)[4 * V]) {
  const bool al = (reinterpret_cast<uintptr_t>(row) & 15u) == 0;
#pragma unroll
  for (int j = 0; j < V; ++j)
    store_quad(row, al, N, 4 * (j * NT + static_cast<int>(threadIdx.x)),
               make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
}

// key_f32 of a value known to be finite: x + 0 folds -0 into +0.
FCB_DEV uint32_t key_finite_f32(float x) {
  const uint32_t b = __float_as_uint(x + 0.0f);
  return b ^ (static_cast<uint32_t>(static_cast<int>(b) >> 31) | 0x80000000u);
}

// Order-preserving compaction offsets in the vector layout: the column order
// is the (j, tid, k) order, so cell (j, k) of this thread goes to
//   sum_{j' < j} total_j' + (flagged cells of vector j in threads < tid)
//   + (flagged cells k' < k of this thread's vector j).
// Per-vector counts (0..4 per thread, <= 4*NT per block) are packed into
// 12-bit fields (13-bit from 1024 threads on), five (four) per 64-bit word, so
// one block scan serves that many vectors.
// Returns the block total; base[j] receives the first two terms.
template <int NT, int V>
FCB_DEV int compact_bases(uint32_t flags, int (&base)[V], unsigned long long* scratch) {
  static_assert(4 * NT < 8192, "13-bit count fields");
  static_assert(4 * V <= 32, "one flag bit per cell");
  constexpr int FB = 4 * NT < 4096 ? 12 : 13, PER = 60 / FB, K = (V + PER - 1) / PER;
  int run = 0;
#pragma unroll
  for (int q = 0; q < K; ++q) {
    unsigned long long packed = 0;
#pragma unroll
    for (int jj = 0; jj < PER; ++jj) {
      const int j = q * PER + jj;
      if (j < V) packed |= static_cast<unsigned long long>(__popc((flags >> (4 * j)) & 0xFu)) << (FB * jj);
    }
    unsigned long long tot;
    const unsigned long long ex = block_exclusive_sum(packed, scratch, tot);
#pragma unroll
    for (int jj = 0; jj < PER; ++jj) {
      const int j = q * PER + jj;
      if (j < V) {
        base[j] = run + static_cast<int>((ex >> (FB * jj)) & ((1ull << FB) - 1));
        run += static_cast<int>((tot >> (FB * jj)) & ((1ull << FB) - 1));
      }
    }
  }
  return run;
}

// Words of a bitmap over sorted positions 0 .. n (see mark_set), or of one bit
// per position with room to spare.
__host__ __device__ inline int mark_words(int n) { return n / 16 + 2; }

// Shared-memory layout of the radix-sorted forms (bytes; every region 16-aligned)
// with keys of K bytes.
template <int NT, int K = 4>
struct SortedLayout {
  size_t red, dw, dw2, scratch, k0, k1, i0, i1, total;
  __host__ __device__ explicit SortedLayout(int n) {
    size_t o = 0;
    red = o; o += 1024;
    dw = o; o = al16(o + size_t(mark_words(n)) * 4);   // two bitmaps over positions
    dw2 = o; o = al16(o + size_t(mark_words(n)) * 4);  // for the kernels' own use
    scratch = o; o = al16(o + SortScratch<NT>::bytes);
    k0 = o; o = al16(o + size_t(n) * K + 16);
    k1 = o; o = al16(o + size_t(n) * K + 16);
    i0 = o; o = al16(o + size_t(n) * 2 + 16);
    i1 = o; o = al16(o + size_t(n) * 2 + 16);
    total = o;
  }
};

}  // namespace fcb
