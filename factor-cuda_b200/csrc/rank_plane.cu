// rank_plane.cu -- cs_rank and parameter_scan of one plane, one CTA per date,
// for sm_100a.
//
//  k_csr    cs_rank: each valid cell's rank from the section's value-spread
//           buckets (section_rank.cuh).
//  k_pscan  parameter_scan: the same buckets of the finite cells give all four
//           groups (ascending / descending x masked / unmasked).
//
// Sections whose buckets come out crowded take the radix-sorted form of the
// same kernel (csr_radix, pscan_radix).
//
// Measured on a B200 against the radix forms alone (256 threads, three CTAs
// per SM): cs_rank of 1218 x 5000 169 -> 51.6 us, parameter_scan of
// 1001 x 4733 (four groups) 190 -> 76.6 us, one date of 5000 31 -> 17 us.
// What bounds them is instruction issue (about 140 instructions per cell at
// 60 % of the issue slots; 8 HBM bytes per cell take a sixth of the time).  A
// plane of nothing but ties pays for finding that out, and sorts with two CTAs of
// 448 threads per SM: cs_rank of integers 0..6 takes 64 us against 56, of values
// rounded to 1e-1 and 1e-2 93 and 117 against 84 and 101, with 30 % zeros 153
// against 141; with 3 % zeros, or rounded to 1e-3, 64 and 56 us against 174 and
// 121.  (The keys go to the sort from registers; read and tested again they cost
// 5 us more.)
#include "section_rank.cuh"

namespace fcb {
namespace {

// compact_bases, and the bits in which the flagged cells' keys differ.  scratch:
// 128 words.
template <int NT, int V>
FCB_DEV uint32_t compact_bits(const uint32_t (&key)[4 * V], uint32_t flags, int (&base)[V], int& m,
                              unsigned long long* scratch) {
  constexpr int NW = NT / 32;
  uint32_t* red = reinterpret_cast<uint32_t*>(scratch + 33);  // past block_exclusive_sum's words
  uint32_t all = 0xFFFFFFFFu, any = 0u;
#pragma unroll
  for (int c = 0; c < 4 * V; ++c)
    if ((flags >> c) & 1u) {
      all &= key[c];
      any |= key[c];
    }
  all = __reduce_and_sync(kFull, all);
  any = __reduce_or_sync(kFull, any);
  if (lane_id() == 0) {
    red[threadIdx.x >> 5] = all;
    red[32 + (threadIdx.x >> 5)] = any;
  }
  m = compact_bases<NT, V>(flags, base, scratch);  // its barriers publish the words
  return __reduce_and_sync(kFull, lane_id() < NW ? red[lane_id()] : 0xFFFFFFFFu) ^
         __reduce_or_sync(kFull, lane_id() < NW ? red[32 + lane_id()] : 0u);
}

// cs_rank by radix: the valid cells (key <= range, as spread_place left them) are
// compacted in column order, radix-sorted by key, and each cell's rank is its
// sorted position + 1.  A section of one value is in order as it is.
template <int NT, int V>
__device__ __noinline__ void csr_radix(const uint32_t* keys, uint32_t range, int N, float* __restrict__ out,
                                       uint8_t* sm) {
  constexpr int C = 4 * V;
  uint32_t key[C];
#pragma unroll
  for (int c = 0; c < C; ++c) key[c] = keys[c];
  const SortedLayout<NT> L(N);
  unsigned long long* scan64 = reinterpret_cast<unsigned long long*>(sm + L.red);
  uint32_t* k0 = reinterpret_cast<uint32_t*>(sm + L.k0);
  uint32_t* k1 = reinterpret_cast<uint32_t*>(sm + L.k1);
  uint16_t* i0 = reinterpret_cast<uint16_t*>(sm + L.i0);
  uint16_t* i1 = reinterpret_cast<uint16_t*>(sm + L.i1);
  const int tid = static_cast<int>(threadIdx.x);
  const float qnan = __uint_as_float(kQuietNanBits);
  uint32_t valid = 0u;
#pragma unroll
  for (int c = 0; c < C; ++c) valid |= (key[c] <= range ? 1u : 0u) << c;
  int base[V], m;
  const uint32_t diff = compact_bits<NT, V>(key, valid, base, m, scan64);
  float v[C];
  if (diff == 0u || m < 2) {
#pragma unroll
    for (int j = 0; j < V; ++j) {
      int p = base[j];
#pragma unroll
      for (int k = 0; k < 4; ++k) v[4 * j + k] = (valid >> (4 * j + k)) & 1u ? static_cast<float>(++p) : qnan;
    }
    store_row_f32v<NT, V>(out, N, v);
    return;
  }
#pragma unroll
  for (int j = 0; j < V; ++j) {
    int p = base[j];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * j + k;
      if ((valid >> c) & 1u) {
        k0[p] = key[c];
        i0[p] = static_cast<uint16_t>(4 * (j * NT + tid) + k);
        ++p;
      }
    }
  }
  __syncthreads();
  uint32_t* ks;
  uint16_t* is;
  block_radix_sort_bits<NT, C, uint32_t>(k0, i0, k1, i1, m, diff, sm + L.scratch, &ks, &is);
  uint32_t* RK = (ks == k0) ? k1 : k0;
  for (int p = tid; p < m; p += NT) RK[is[p]] = static_cast<uint32_t>(p + 1);
  __syncthreads();
#pragma unroll
  for (int c = 0; c < C; ++c)
    v[c] = ((valid >> c) & 1u) ? static_cast<float>(RK[4 * ((c >> 2) * NT + tid) + (c & 3)]) : qnan;
  store_row_f32v<NT, V>(out, N, v);
}

// parameter_scan by radix, of the cells that spread_place left (out_of_mask: bit c,
// cell c is finite but not in the mask): one ascending sort of the finite cells serves all four
// groups (asc / desc x masked / unmasked).  With S the start and E the end of
// a cell's tie group in sorted order, C the count of masked-valid cells before
// a sorted position and m / mt the finite / masked-valid totals:
//   asc unmasked  p + 1                  asc masked   C[p] + 1
//   desc unmasked m - E + (p - S) + 1    desc masked  mt - C[E] + (C[p] - C[S]) + 1
// (descending ranks keep ties by ascending column).  Shared memory stays at
// the sort's 12 bytes per cell: tie-group starts go to a bitmap (the sorted
// keys are then free for C and E), and the ascending and descending pairs of
// ranks pass through one per-column buffer in turn.
template <int NT, int V>
__device__ __noinline__ void pscan_radix(const uint32_t* keys, uint32_t range, uint32_t out_of_mask, int N,
                                         const ScanOut& outs, uint8_t* sm) {
  constexpr int C = 4 * V;
  const SortedLayout<NT> L(N);
  unsigned long long* scan64 = reinterpret_cast<unsigned long long*>(sm + L.red);
  uint32_t* scan32 = reinterpret_cast<uint32_t*>(sm + L.red);
  uint32_t* bits = reinterpret_cast<uint32_t*>(sm + L.dw);  // tie-group start per sorted position
  uint32_t* k0 = reinterpret_cast<uint32_t*>(sm + L.k0);
  uint32_t* k1 = reinterpret_cast<uint32_t*>(sm + L.k1);
  uint16_t* i0 = reinterpret_cast<uint16_t*>(sm + L.i0);
  uint16_t* i1 = reinterpret_cast<uint16_t*>(sm + L.i1);
  const int tid = static_cast<int>(threadIdx.x);
  const size_t row = static_cast<size_t>(blockIdx.x) * N;
  for (int k = tid; k < (N + 31) / 32 + 1; k += NT) bits[k] = 0u;
  uint32_t key[C], fin = 0u;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    key[c] = keys[c];
    fin |= (key[c] <= range ? 1u : 0u) << c;
  }
  int base[V], m;
  const uint32_t diff = compact_bits<NT, V>(key, fin, base, m, scan64);  // its barriers publish the bitmap clear
#pragma unroll
  for (int j = 0; j < V; ++j) {
    int p = base[j];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * j + k;
      if ((fin >> c) & 1u) {
        k0[p] = key[c];
        i0[p] = static_cast<uint16_t>((4 * (j * NT + tid) + k) | (((~out_of_mask >> c) & 1u) << 15));
        ++p;
      }
    }
  }
  __syncthreads();
  uint32_t* ks;
  uint16_t* is;
  block_radix_sort_bits<NT, C, uint32_t>(k0, i0, k1, i1, m, diff, sm + L.scratch, &ks, &is);
  uint16_t* S = (is == i0) ? i1 : i0;                                // group start per sorted position
  uint32_t* O = (ks == k0) ? k1 : k0;                                // two ranks per column
  uint16_t* Cn = reinterpret_cast<uint16_t*>(ks);                    // m + 1 entries, over the sorted keys
  uint16_t* GE = reinterpret_cast<uint16_t*>(ks) + (N + 1);          // group end by group start
  // pass 1: per chunk, masked-valid count, last group start, start bits
  const int per = (m + NT - 1) / NT;
  const int b0 = tid * per, b1 = min(m, b0 + per);
  uint32_t cm = 0;
  int last = -1;
  for (int p = b0; p < b1; ++p) {
    cm += is[p] >> 15;
    if (p == 0 || ks[p] != ks[p - 1]) {
      last = p;
      atomicOr(&bits[p >> 5], 1u << (p & 31));
    }
  }
  uint32_t mt;
  uint32_t c = block_exclusive_sum(cm, scan32, mt);  // barriers: ks reads done, bits complete
  // exclusive max-scan of the chunks' last group starts (identity -1)
  int inc = last;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(kFull, inc, o);
    if (lane_id() >= static_cast<unsigned>(o)) inc = max(inc, u);
  }
  const int wi = tid >> 5;
  int* sc = reinterpret_cast<int*>(scan64);
  if (lane_id() == 31) sc[wi] = inc;
  __syncthreads();
  int carry = -1;
  for (int i = 0; i < wi; ++i) carry = max(carry, sc[i]);
  const int up = __shfl_up_sync(kFull, inc, 1);
  if (lane_id() > 0) carry = max(carry, up);
  // pass 2: S, the masked-valid prefix C and the group ends E
  auto is_start = [&](int p) { return ((bits[p >> 5] >> (p & 31)) & 1u) != 0u; };
  for (int p = b0; p < b1; ++p) {
    if (is_start(p)) carry = p;
    S[p] = static_cast<uint16_t>(carry);
    Cn[p] = static_cast<uint16_t>(c);
    c += is[p] >> 15;
    if (p == m - 1 || is_start(p + 1)) GE[carry] = static_cast<uint16_t>(p + 1);
  }
  if (tid == 0) Cn[m] = static_cast<uint16_t>(mt);
  __syncthreads();
  const float qnan = __uint_as_float(kQuietNanBits);
  // pass 3, twice: the ascending pair (groups 0 | 1), then the descending pair
  // (groups 2 | 3), each stored by column and written out
  for (int half = 0; half < 2; ++half) {
    if (outs.out[2 * half] == nullptr && outs.out[2 * half + 1] == nullptr) continue;  // uniform
    for (int p = tid; p < m; p += NT) {
      const uint32_t id = is[p];
      const uint32_t cp = Cn[p];
      uint32_t lo = 0u, hi;
      if (half == 0) {
        hi = static_cast<uint32_t>(p + 1);
        if (id & 0x8000u) lo = cp + 1u;
      } else {
        const int s0 = S[p], e0 = GE[s0];
        hi = static_cast<uint32_t>(m - e0 + (p - s0) + 1);
        if (id & 0x8000u) lo = mt - Cn[e0] + (cp - Cn[s0]) + 1u;
      }
      O[id & 0x3FFFu] = lo | (hi << 16);
    }
    __syncthreads();
#pragma unroll
    for (int g2 = 0; g2 < 2; ++g2) {
      float* dst = outs.out[2 * half + g2];
      if (dst == nullptr) continue;  // uniform
      const int sh = g2 ? 16 : 0;
      float v[C];
#pragma unroll
      for (int cc = 0; cc < C; ++cc) {
        const uint32_t r =
            ((fin >> cc) & 1u) ? ((O[4 * ((cc >> 2) * NT + tid) + (cc & 3)] >> sh) & 0xFFFFu) : 0u;
        v[cc] = r ? static_cast<float>(r) : qnan;
      }
      store_row_f32v<NT, V>(dst + row, N, v);
    }
    __syncthreads();  // O is rewritten by the second half
  }
}

// cs_rank: valid = finite & mask; a cell's rank is the number of smaller valid
// keys (of -x for descending) plus its ties at smaller columns plus one
// (replaces cs_rank_gpu, src/cross_sectional_rank.cu:228-372, which runs CUB's
// global segmented sort).
template <int NT, int V>
__global__ void __launch_bounds__(NT, kSmThreads / NT) k_csr(const float* __restrict__ X, const uint8_t* __restrict__ mask,
                                                       int N, int desc, float* __restrict__ out) {
  constexpr int C = 4 * V;
  extern __shared__ __align__(16) uint8_t sm[];
  const SpreadLayout<NT, V> L(N);
  const size_t row = static_cast<size_t>(blockIdx.x) * N;
  uint32_t key[C], W[C];
  {
    float x[C];
    uint32_t mk[C];
    load_row_f32<NT, V, true>(X + row, N, x);
    load_mask4<NT, V>(mask != nullptr ? mask + row : nullptr, N, mk);
#pragma unroll
    for (int c = 0; c < C; ++c)
      key[c] = finite_f32(x[c]) && mk[c] ? key_finite_f32(desc ? -x[c] : x[c]) : kInvalidKey32;
  }
  SpreadTotals T;
  if (!spread_place<NT, V>(key, L, sm, W, T)) {
    uint32_t kk[C];  // (the keys stay in registers but for this call)
#pragma unroll
    for (int c = 0; c < C; ++c) kk[c] = key[c];
    csr_radix<NT, V>(kk, T.range, N, out + row, sm);
    return;
  }
  spread_positions<NT, V, false>(L, sm, T.m, T.heavy, key, W);
  float v[C];
#pragma unroll
  for (int c = 0; c < C; ++c)
    v[c] = key[c] <= T.range && T.m != 0 ? static_cast<float>(W[c] + 1u) : __uint_as_float(kQuietNanBits);
  store_row_f32v<NT, V>(out + row, N, v);
}

// parameter_scan: the finite cells' buckets serve all four groups.  With less,
// q and t of spread_positions, U[p] the finite cells outside the mask among the
// first p sorted positions (a bitmap over positions) and m / mu the finite
// cells / those outside the mask:
//   asc unmasked  less + t + 1           asc masked   the same - U[less + t]
//   desc unmasked m - (less + q) + t + 1 desc masked  the same - (mu - U[less + q]) - (U[less + t] - U[less])
// (descending ranks keep ties by ascending column, the contract of
// fc/_cpu_core.py:57-78 / :295-301; replaces the reference's four rank
// pipelines, src/cross_sectional_rank.cu:401-664).
template <int NT, int V>
__global__ void __launch_bounds__(NT, kSmThreads / NT) k_pscan(const float* __restrict__ X, const uint8_t* __restrict__ mask,
                                                         int N, ScanOut outs) {
  constexpr int C = 4 * V;
  extern __shared__ __align__(16) uint8_t sm[];
  const SpreadLayout<NT, V> L(N);
  const int tid = static_cast<int>(threadIdx.x);
  const size_t row = static_cast<size_t>(blockIdx.x) * N;
  uint32_t* bits = reinterpret_cast<uint32_t*>(sm + L.bits);
  const int nbw = mark_words(N);
  for (int k = tid; k < nbw; k += NT) bits[k] = 0u;  // spread_place's barriers publish the clear
  uint32_t key[C], W[C], out_of_mask = 0u;
  {
    float x[C];
    uint32_t mk[C];
    load_row_f32<NT, V, true>(X + row, N, x);
    load_mask4<NT, V>(mask != nullptr ? mask + row : nullptr, N, mk);
#pragma unroll
    for (int c = 0; c < C; ++c) {
      out_of_mask |= ((finite_f32(x[c]) && !mk[c]) ? 1u : 0u) << c;
      key[c] = finite_f32(x[c]) ? key_finite_f32(x[c]) : kInvalidKey32;
    }
  }
  SpreadTotals T;
  if (!spread_place<NT, V>(key, L, sm, W, T)) {
    uint32_t kk[C];  // (the keys stay in registers but for this call)
#pragma unroll
    for (int c = 0; c < C; ++c) kk[c] = key[c];
    pscan_radix<NT, V>(kk, T.range, out_of_mask, N, outs, sm);
    return;
  }
  static_assert(kSpreadMaxBucket < 512, "ties fit 9-bit fields");
  // W[c] becomes less | t << 14 | q << 23, q = 0 for the cells not ranked
  spread_positions<NT, V, true>(L, sm, T.m, T.heavy, key, W);
#pragma unroll
  for (int c = 0; c < C; ++c)
    if ((out_of_mask >> c) & 1u) mark_set(bits, (W[c] & 0x3FFFu) + ((W[c] >> 14) & 0x1FFu));
  if (__syncthreads_or(out_of_mask != 0u)) {
    if (tid < 32) mark_prefix(bits, nbw);
    __syncthreads();
  }
  const uint32_t m = static_cast<uint32_t>(T.m);
  const uint32_t mu = marks_before(bits, m);
  // key[c] becomes the ascending pair of ranks (unmasked | masked << 16, 0 =
  // not ranked) and W[c] the descending pair
#pragma unroll
  for (int c = 0; c < C; ++c) {
    uint32_t asc = 0u, des = 0u;
    const uint32_t less = W[c] & 0x3FFFu, t = (W[c] >> 14) & 0x1FFu, q = W[c] >> 23;
    if (q != 0u) {
      asc = less + t + 1u;
      des = m - (less + q) + t + 1u;
      uint32_t am = asc, dm = des;
      if (mu != 0u) {  // uniform
        const uint32_t u = marks_before(bits, less + t);
        am -= u;
        dm -= mu - marks_before(bits, less + q);
        if (t != 0u) dm -= u - marks_before(bits, less);
        if ((out_of_mask >> c) & 1u) am = dm = 0u;
      }
      asc |= am << 16;
      des |= dm << 16;
    }
    key[c] = asc;
    W[c] = des;
  }
  // one group of outputs at a time: the masked ones are the upper halves
  auto store = [&](float* dst, const uint32_t (&r2)[C], int shift) {
    if (dst == nullptr) return;  // uniform
    const float qnan = __uint_as_float(kQuietNanBits);
    float v[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const uint32_t r = (r2[c] >> shift) & 0xFFFFu;
      v[c] = r != 0u ? static_cast<float>(r) : qnan;
    }
    store_row_f32v<NT, V>(dst + row, N, v);
  };
  store(outs.out[0], key, 16);
  store(outs.out[1], key, 0);
  store(outs.out[2], W, 16);
  store(outs.out[3], W, 0);
}

// the radix form of a crowded section needs its own layout in the same memory
template <int NT, int V>
size_t plane_smem(int N) {
  const size_t a = SpreadLayout<NT, V>(N).total, b = SortedLayout<NT>(N).total;
  return a > b ? a : b;
}
template <int NT, int V>
cudaError_t csr_launch(const float* X, const uint8_t* mask, int T, int N, int desc, float* out, cudaStream_t st) {
  const size_t smem = plane_smem<NT, V>(N);
  if (smem > kMaxSmemPerBlock) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(k_csr<NT, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  k_csr<NT, V><<<T, NT, smem, st>>>(X, mask, N, desc, out);
  return cudaGetLastError();
}
template <int NT, int V>
cudaError_t pscan_launch(const float* X, const uint8_t* mask, int T, int N, ScanOut outs, cudaStream_t st) {
  const size_t smem = plane_smem<NT, V>(N);
  if (smem > kMaxSmemPerBlock) return cudaErrorInvalidValue;
  cudaError_t e =
      cudaFuncSetAttribute(k_pscan<NT, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  k_pscan<NT, V><<<T, NT, smem, st>>>(X, mask, N, outs);
  return cudaGetLastError();
}
}  // namespace


// The per-date rank kernels stage nothing through mbarriers, so `status` has
// nothing to report; it is kept for the callers' uniform interface.
cudaError_t launch_cs_rank(const float* X, const uint8_t* mask, int T, int N, int desc, float* out, int* status,
                           cudaStream_t st) {
  (void)status;
  if (N < 1 || N > kSmemRankCap) return cudaErrorInvalidValue;
  auto go = [&](auto shape) {
    return csr_launch<decltype(shape)::kThreads, decltype(shape)::kVectors>(X, mask, T, N, desc, out, st);
  };
  return T <= kFewSections ? section_shape_few(N, go) : section_shape(N, go);
}

cudaError_t launch_param_scan(const float* X, const uint8_t* mask, int T, int N, ScanOut outs, int* status,
                              cudaStream_t st) {
  (void)status;
  if (N < 1 || N > kSmemRankCap) return cudaErrorInvalidValue;
  auto go = [&](auto shape) {
    return pscan_launch<decltype(shape)::kThreads, decltype(shape)::kVectors>(X, mask, T, N, outs, st);
  };
  return T <= kFewSections ? section_shape_few(N, go) : section_shape(N, go);
}


}  // namespace fcb
