// SC projector over several rotated views of one matrix: F = A X^T (bins x views), Q = Y / F,
// U = A^T Q (views x voxels), weight += scale * sum_r P_r^-1 u_r
// (the rotation loop of osem_bin_mode, recon_osem_plane.py:49-53). Views are taken in blocks of at
// most 20, each block padded to NB in {2, 4, 8, 12, 16, 20} with zero views:
//   sc_views_gather   xt[j][r] = image value of voxel j in view r (voxel-major, rows of XS floats)
//   sc_views_forward  CTA = column slice x row groups; the slice of xt sits in shared memory, a warp
//                     holds TM x NB sums in registers and its lanes own adjacent columns, so an
//                     element of A meets all NB views as it arrives and nothing of A is staged:
//                     TM * NB FMAs on TM loads of A and NB / 4 16-byte reads of x. One transposing
//                     butterfly per row group; partial sums per slice
//   sc_views_ratio    q[b][r] = y[b, r] / f, slices in order (or f itself)
//   sc_views_back     CTA = 128 (or 256) columns x a chunk of rows; a lane holds 4 NB (8 NB) sums, a row's NB ratios
//                     are one broadcast; the eight warps take every eighth row and add up in warp order
// then sc_reduce_scatter_kernel (views and chunks in order).
// Bound: HBM below about 8 views, the FP32 pipe (2 NB flops an element and pass at 80 TFLOP/s) and
// the reads of x and q from shared memory above. Weight of 512 x 36,000 float32 rows, 20 views: 82 us
// (forward 28, back 33) against 334 us for passes of 8 views whose image reads went through L1 once a
// row; 4,096 rows, 20 views 1,681 -> 357 us; 128 x 4,800, 10 views 95 -> 35 us.
// All sums have one fixed order (no atomics).
#pragma once

namespace jscc {

constexpr int kSvWarps = 8;
constexpr int kSvThreads = kSvWarps * 32;
constexpr int kSvMaxViews = 20;             // views of a block
constexpr size_t kSvSmem = 220u * 1024u;    // forward: shared memory of the CTAs of an SM

// Elements of A travel in units of four bytes (one float32 or two BF16 columns) by cp.async into a
// ring of shared-memory stages that only the lane itself reads, so that several stages are in
// flight at any alignment of four bytes without registers or barriers. RING = false (BF16 rows off
// four-byte boundaries): plain two-byte loads, one stage ahead.
template <typename T, int NB, bool RING>
struct SvTraits {
  static constexpr int kRows = NB == 2 ? 16 : 8;  // rows of a warp's tile: kRows * NB is a multiple of 32
  // floats between voxels of the staged slice: an odd number of 16-byte units, so that eight lanes'
  // 16-byte reads fall into different banks (NB = 2: 8-byte reads, no padding needed)
  static constexpr int kPitch = NB == 2 ? 2 : ((NB / 4) % 2 ? NB : NB + 4);
  static constexpr int kUnit = RING ? 4 / (int)sizeof(T) : 1;    // columns of a lane's unit
  static constexpr int kFwdCtas = NB <= 8 ? 2 : 1;  // CTAs an SM
  static constexpr int kFwdStages = NB <= 8 ? 4 : 8;
  static constexpr int kFwdRing = RING ? kSvWarps * kFwdStages * kRows * 128 : 0;  // bytes of a CTA
};

// Columns of a back pass's tile. Aligned BF16 rows of few views: 256, so that a warp reads 512 bytes of a
// row, as it does of float32: 256 bytes at a time ran at 2.6 to 3.8 TB/s, 512 at 5.1 to 5.4 (back projection
// of two views, 41,666 x 4,800: 153 -> 75 us, 5,555 x 36,000: 126 -> 79 us). The sums of more views leave no
// registers for that.
constexpr int sv_back_cols(int nb, size_t el, bool aligned) { return aligned && el == 2 && nb <= 4 ? 256 : 128; }

// The back pass's copies. COPY 0: plain loads, a row ahead; 1: four-byte cp.async units; 2: a lane's
// columns in one cp.async of 16 bytes (8 for BF16 of more views), for rows on such boundaries.
template <typename T, int NB, int COPY>
struct SvBack {
  static constexpr int kCols = sv_back_cols(NB, sizeof(T), COPY == 2) / 32;  // columns of a lane
  static constexpr int kUnit = COPY == 2 ? kCols : COPY == 1 ? 4 / (int)sizeof(T) : 1;  // columns of a copy
  static constexpr int kUnits = kCols / kUnit;
  static constexpr int kStages = 32 * kCols * sizeof(T) == 256 ? 16 : 8;
  // a row's ratios (in whole 16 bytes), then its units
  static constexpr int kRatioBytes = (NB * 4 + 15) / 16 * 16;
  static constexpr int kStage = 32 * kCols * (int)sizeof(T) + kRatioBytes;
  static constexpr int kRing = COPY ? kSvWarps * kStages * kStage : 0;
  static constexpr int kSum = kSvWarps * NB * 32 * kCols * 4;
  static constexpr int kSmem = kRing > kSum ? kRing : kSum;
};

// the columns of a unit as floats
template <typename T, int UNIT>
__device__ __forceinline__ void sv_unpack(uint32_t u, float (&v)[UNIT]) {
  if constexpr (UNIT == 2) {
    v[0] = bf16_lo(u);
    v[1] = bf16_hi(u);
  } else if constexpr (sizeof(T) == 4) {
    v[0] = __uint_as_float(u);
  } else {
    v[0] = bf16_lo(u);
  }
}

__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
template <int BYTES>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

inline int sv_pad(int views) {
  return views <= 2 ? 2 : views <= 4 ? 4 : views <= 8 ? 8 : views <= 12 ? 12 : views <= 16 ? 16 : 20;
}
inline int sv_pitch(int nb) { return nb == 2 ? 2 : ((nb / 4) % 2 ? nb : nb + 4); }
inline int sv_rows(int nb) { return nb == 2 ? 16 : 8; }
inline int sv_fwd_ctas(int nb) { return nb <= 8 ? 2 : 1; }
constexpr int sv_back_ctas(int nb) { return nb <= 4 ? 3 : nb <= 12 ? 2 : 1; }
inline size_t sv_fwd_ring(int nb) { return (size_t)kSvWarps * (nb <= 8 ? 4 : 8) * sv_rows(nb) * 128; }

// xt[j * pitch + r] = img[rotmat[j, r0 + r] - 1] (the image itself without a table), 0 for r >= nr
__global__ void sc_views_gather_kernel(const float* __restrict__ img, const int64_t* __restrict__ rotmat,
                                       int64_t ld_rot, int r0, int nr, int pitch, int64_t V, float* __restrict__ xt) {
  const int64_t total = V * pitch;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = t / pitch;
    const int r = (int)(t - j * pitch);
    float v = 0.f;
    if (r < nr) {
      int64_t src = j;
      if (rotmat != nullptr) src = rotmat[j * ld_rot + r0 + r] - 1;
      if (src < 0 || src >= V) atomicAdd(&g_bad_index_count, 1u);
      else v = img[src];
    }
    xt[t] = v;
  }
}

// Sums of a[0..M) over the warp's lanes; lane l is left with the M / 32 sums of the indexes
// sv_index(l, i). Halving: at each step a lane keeps one half of its values and adds the other
// lane's copies of it.
template <int M, int STEP = 0, int N>
__device__ __forceinline__ void sv_transpose_sum(float (&a)[N], int lane) {
  static_assert(N % 32 == 0, "whole lanes");
  if constexpr (STEP < 5) {
    constexpr int w = 16 >> STEP, half = M / 2;
    const bool up = (lane & w) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float send = up ? a[i] : a[i + half];
      const float mine = up ? a[i + half] : a[i];
      a[i] = mine + __shfl_xor_sync(0xffffffffu, send, w);
    }
    sv_transpose_sum<half, STEP + 1>(a, lane);
  }
}
template <int M>
__device__ __forceinline__ int sv_index(int lane, int i) {
  int at = i;
#pragma unroll
  for (int step = 0; step < 5; ++step)
    if (lane & (16 >> step)) at += M >> (step + 1);
  return at;
}

// part[(s * n_bins + b) * NB + r] = sum over the columns of slice s of A[row(b), j] xt[j][r].
// Slice s holds the 64-column blocks [blocks * s / n_slices, blocks * (s + 1) / n_slices), taken in
// pieces of piece_cols columns (one piece: staged once for all row groups of the CTA). With units of
// two columns the staged voxels of a 64-column block stand even columns first, so that the lanes'
// reads are those of adjacent voxels either way.
template <typename T, int NB, bool RING>
__global__ void __launch_bounds__(kSvThreads, SvTraits<T, NB, RING>::kFwdCtas)
sc_views_forward_kernel(const T* __restrict__ A, int64_t lda, const int64_t* __restrict__ row_idx, int64_t n_bins,
                        int64_t V, const float* __restrict__ xt, int n_slices, int piece_cols,
                        float* __restrict__ part) {
  using Tr = SvTraits<T, NB, RING>;
  constexpr int TM = Tr::kRows, XS = Tr::kPitch, M = TM * NB, NP = NB / 2, E = Tr::kUnit, W = 32 * E;
  constexpr int D = Tr::kFwdStages;
  extern __shared__ __align__(128) unsigned char sv_smem[];
  float* xs = reinterpret_cast<float*>(sv_smem + Tr::kFwdRing);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t* ring = reinterpret_cast<const uint32_t*>(sv_smem) + warp * (D * TM * 32) + lane;
  const uint32_t ring_at = smem_u32(ring);
  const int s = blockIdx.x;
  const int64_t blocks = (V + 63) / 64;
  const int64_t j0 = blocks * s / n_slices * 64;
  int64_t j1 = blocks * (s + 1) / n_slices * 64;
  if (j1 > V) j1 = V;
  const int64_t len_all = j1 > j0 ? j1 - j0 : 0;
  const int pieces = len_all > piece_cols ? (int)((len_all + piece_cols - 1) / piece_cols) : 1;
  auto slot = [](int c) { return E == 2 ? (c & ~63) | ((c & 1) << 5) | ((c & 63) >> 1) : c; };
  auto stage = [&](int p) {
    const int64_t a = j0 + (int64_t)p * piece_cols;
    const int len = (int)(j1 - a < piece_cols ? j1 - a : piece_cols);
    if constexpr (NB == 2) {
      const float2* src = reinterpret_cast<const float2*>(xt) + a;
#pragma unroll 8
      for (int c = tid; c < len; c += kSvThreads) reinterpret_cast<float2*>(xs)[slot(c)] = __ldg(src + c);
    } else {
      constexpr int Q = XS / 4;
      const float4* src = reinterpret_cast<const float4*>(xt) + a * Q;
#pragma unroll 8
      for (int i = tid; i < len * Q; i += kSvThreads) {
        const int c = i / Q;
        reinterpret_cast<float4*>(xs)[slot(c) * Q + (i - c * Q)] = __ldg(src + i);
      }
    }
    return len;
  };
  int len = (int)len_all;
  if (pieces == 1) {
    if (len > 0) stage(0);
    __syncthreads();
  }
  const int64_t groups = (n_bins + kSvWarps * TM - 1) / (kSvWarps * TM);
  for (int64_t g = blockIdx.y; g < groups; g += gridDim.y) {
    const int64_t b0 = (g * kSvWarps + warp) * TM;
    const T* rowp[TM];
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int64_t b = b0 + i < n_bins ? b0 + i : n_bins - 1;  // rows past the end repeat the last one
      rowp[i] = A + (row_idx ? row_idx[b] : b) * lda + j0;
    }
    float2 acc[TM][NP];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int k = 0; k < NP; ++k) acc[i][k] = make_float2(0.f, 0.f);
    for (int p = 0; p < pieces; ++p) {
      if (pieces > 1) {
        __syncthreads();
        len = stage(p);
        __syncthreads();
      }
      const int full = len / W;
      auto accumulate = [&](const float* xp, const float (&a)[TM]) {
        float2 x[NP];
        if constexpr (NB == 2) {
          x[0] = *reinterpret_cast<const float2*>(xp);
        } else {
#pragma unroll
          for (int k = 0; k < NP; k += 2) {
            const float4 v = *reinterpret_cast<const float4*>(xp + 2 * k);
            x[k] = make_float2(v.x, v.y);
            x[k + 1] = make_float2(v.z, v.w);
          }
        }
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const float2 aa = make_float2(a[i], a[i]);
#pragma unroll
          for (int k = 0; k < NP; ++k) acc[i][k] = __ffma2_rn(aa, x[k], acc[i][k]);
        }
      };
      const float* xp = xs + lane * XS;
      if constexpr (RING) {
        auto issue = [&](int it) {
          const uint32_t at = ring_at + (uint32_t)(it % D) * (TM * 128);
#pragma unroll
          for (int i = 0; i < TM; ++i) cp_async4(at + i * 128, rowp[i] + it * W + lane * E);
        };
#pragma unroll
        for (int it = 0; it < D - 1; ++it) {
          if (it < full) issue(it);
          cp_async_commit();
        }
        for (int it = 0; it < full; ++it) {
          cp_async_wait<D - 2>();
          uint32_t u[TM];
#pragma unroll
          for (int i = 0; i < TM; ++i) u[i] = ring[(it % D) * (TM * 32) + i * 32];
          if (it + D - 1 < full) issue(it + D - 1);
          cp_async_commit();
          float a[E][TM];
#pragma unroll
          for (int i = 0; i < TM; ++i) {
            float v[E];
            sv_unpack<T, E>(u[i], v);
#pragma unroll
            for (int e = 0; e < E; ++e) a[e][i] = v[e];
          }
#pragma unroll
          for (int e = 0; e < E; ++e) accumulate(xp + e * 32 * XS, a[e]);
          xp += W * XS;
        }
      } else {
        // the next 32 columns are loaded while these are used
        float a[TM];
#pragma unroll
        for (int i = 0; i < TM; ++i) a[i] = full > 0 ? load_elem(rowp[i], lane) : 0.f;
        for (int it = 0; it < full; ++it) {
          float an[TM];
          const int next = (it + 1 < full ? it + 1 : it) * W + lane;
#pragma unroll
          for (int i = 0; i < TM; ++i) an[i] = load_elem(rowp[i], next);
          accumulate(xp, a);
          xp += W * XS;
#pragma unroll
          for (int i = 0; i < TM; ++i) a[i] = an[i];
        }
      }
      // the columns past the last whole unit row of the matrix, one a lane and turn (a lane past the end
      // adds nothing: 0 times another lane's image value would be NaN where that is infinite)
      for (int c = full * W + lane; c < len; c += 32) {
        float a[TM];
#pragma unroll
        for (int i = 0; i < TM; ++i) a[i] = load_elem(rowp[i], c);
        accumulate(xs + slot(c) * XS, a);
      }
#pragma unroll
      for (int i = 0; i < TM; ++i) rowp[i] += len;
    }
    float v[M];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int k = 0; k < NP; ++k) {
        v[i * NB + 2 * k] = acc[i][k].x;
        v[i * NB + 2 * k + 1] = acc[i][k].y;
      }
    sv_transpose_sum<M>(v, lane);
#pragma unroll
    for (int i = 0; i < M / 32; ++i) {
      const int at = sv_index<M>(lane, i);
      const int64_t b = b0 + at / NB;
      if (b < n_bins) part[((int64_t)s * n_bins + b) * NB + at % NB] = v[i];
    }
  }
}

// f[b][r] = the slices' partial sums; ratio[b * nb + r] = proj[row(b), r0 + r] / max(f, floor) (0 for
// the padding views; or another row_ratio), and, with `raw`, raw[b * ld_raw + r0 + r] = f. 32 sums a block: each of eight
// warps adds one eighth of the slices, the eight sums are added in warp order.
__global__ void __launch_bounds__(kSvThreads)
sc_views_ratio_kernel(const float* __restrict__ part, int n_slices, int64_t n_bins, int nb, int nr, int r0,
                      const int64_t* __restrict__ row_idx, const float* __restrict__ proj, int64_t ld_proj,
                      int mode, float floor_v, float* __restrict__ ratio, float* __restrict__ raw,
                      int64_t ld_raw) {
  __shared__ float red[kSvWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t total = n_bins * nb;
  const int64_t t = (int64_t)blockIdx.x * 32 + lane;
  const int s0 = n_slices * warp / kSvWarps, s1 = n_slices * (warp + 1) / kSvWarps;
  const int64_t b = t / nb;
  const int r = (int)(t - b * nb);
  const bool in = t < total && r < nr;
  float f = 0.f, y = 0.f;
  if (in) {
    if (warp == 0 && ratio != nullptr) y = proj[(row_idx ? row_idx[b] : b) * ld_proj + r0 + r];
#pragma unroll 4
    for (int s = s0; s < s1; ++s) f += part[(int64_t)s * total + t];
  }
  red[warp][lane] = f;
  __syncthreads();
  if (warp != 0 || t >= total) return;
#pragma unroll
  for (int w = 1; w < kSvWarps; ++w) f += red[w][lane];
  if (raw != nullptr && in) raw[b * ld_raw + r0 + r] = f;
  if (ratio != nullptr) ratio[t] = in ? row_ratio(y, f, mode, floor_v) : 0.f;
}

// part[(chunk * NB + r) * ldp + j] = sum over the chunk's rows b of A[row(b), j] ratio[b * NB + r]
template <typename T, int NB, int COPY>
__global__ void __launch_bounds__(kSvThreads, sv_back_ctas(NB))
sc_views_back_kernel(const T* __restrict__ A, int64_t lda, const int64_t* __restrict__ row_idx, int64_t n_bins,
                     int64_t V, const float* __restrict__ ratio, int64_t rows_per_chunk, float* __restrict__ part,
                     int64_t ldp) {
  using Tr = SvBack<T, NB, COPY>;
  constexpr int COLS = 32 * Tr::kCols;
  constexpr int TC = Tr::kCols, NP = NB / 2, E = Tr::kUnit, TU = Tr::kUnits, D = Tr::kStages;
  extern __shared__ __align__(128) unsigned char sv_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t c0 = (int64_t)blockIdx.x * COLS;
  const int64_t b_begin = (int64_t)blockIdx.y * rows_per_chunk;
  const int64_t b_end = b_begin + rows_per_chunk < n_bins ? b_begin + rows_per_chunk : n_bins;
  // the lane's column t * E + e stands at (32 t + lane) E + e of the tile
  auto column = [&](int i) { return (32 * (i / E) + lane) * E + i % E; };
  float2 acc[TC][NP];
#pragma unroll
  for (int t = 0; t < TC; ++t)
#pragma unroll
    for (int k = 0; k < NP; ++k) acc[t][k] = make_float2(0.f, 0.f);
  const int n_rows = b_end > b_begin + warp ? (int)((b_end - b_begin - warp + kSvWarps - 1) / kSvWarps) : 0;
  auto row_of = [&](int k) {
    const int64_t b = b_begin + warp + (int64_t)k * kSvWarps;
    return A + (row_idx ? row_idx[b] : b) * lda;
  };
  auto take_q = [&](const float* r, float2 (&q)[NP]) {
    if constexpr (NB == 2) {
      q[0] = *reinterpret_cast<const float2*>(r);
    } else {
#pragma unroll
      for (int i = 0; i < NP; i += 2) {
        const float4 v = *reinterpret_cast<const float4*>(r + 2 * i);
        q[i] = make_float2(v.x, v.y);
        q[i + 1] = make_float2(v.z, v.w);
      }
    }
  };
  auto add = [&](const float (&a)[TC], const float2 (&q)[NP]) {
#pragma unroll
    for (int t = 0; t < TC; ++t) {
      const float2 aa = make_float2(a[t], a[t]);
#pragma unroll
      for (int k = 0; k < NP; ++k) acc[t][k] = __ffma2_rn(aa, q[k], acc[t][k]);
    }
  };
  // a tile whose last columns fill no whole unit takes the plain loads
  const bool whole = E == 1 || V - c0 >= COLS || (V - c0) % E == 0;
  if (COPY != 0 && whole) {
    int64_t col[TU];  // units past the matrix repeat its last one (their sums are not written)
#pragma unroll
    for (int t = 0; t < TU; ++t) {
      col[t] = c0 + (int64_t)(32 * t + lane) * E;
      if (col[t] + E > V) col[t] = V - E;
    }
    // the ratios travel in the ring too: a CTA reads each row's once, from L2, and loaded on demand
    // they cost every row that latency
    const unsigned char* ring = sv_smem + warp * (D * Tr::kStage);
    const uint32_t ring_at = smem_u32(ring);
    const float* rq = ratio + (b_begin + warp) * NB + lane;
    auto issue = [&](int k) {
      const uint32_t at = ring_at + (uint32_t)(k % D) * Tr::kStage;
      const T* rp = row_of(k);
      if (lane < NB) cp_async<4>(at + lane * 4, rq + (int64_t)k * (kSvWarps * NB));
#pragma unroll
      for (int t = 0; t < TU; ++t)
        cp_async<E * (int)sizeof(T)>(at + Tr::kRatioBytes + (32 * t + lane) * (E * (int)sizeof(T)), rp + col[t]);
    };
#pragma unroll
    for (int k = 0; k < D - 1; ++k) {
      if (k < n_rows) issue(k);
      cp_async_commit();
    }
    for (int k = 0; k < n_rows; ++k) {
      cp_async_wait<D - 2>();
      __syncwarp();  // the other lanes' copies of the ratios; their reads of the stage refilled below
      const unsigned char* st = ring + (k % D) * Tr::kStage;
      if (k + D - 1 < n_rows) issue(k + D - 1);
      cp_async_commit();
      float2 q[NP];
      take_q(reinterpret_cast<const float*>(st), q);
      float a[TC];
      st += Tr::kRatioBytes;
      if constexpr (COPY == 2 && sizeof(T) == 4) {
        const float4 v = *reinterpret_cast<const float4*>(st + lane * 16);
        a[0] = v.x; a[1] = v.y; a[2] = v.z; a[3] = v.w;
      } else if constexpr (COPY == 2 && TC == 8) {
        const uint4 v = *reinterpret_cast<const uint4*>(st + lane * 16);
        a[0] = bf16_lo(v.x); a[1] = bf16_hi(v.x); a[2] = bf16_lo(v.y); a[3] = bf16_hi(v.y);
        a[4] = bf16_lo(v.z); a[5] = bf16_hi(v.z); a[6] = bf16_lo(v.w); a[7] = bf16_hi(v.w);
      } else if constexpr (COPY == 2) {
        const uint2 v = *reinterpret_cast<const uint2*>(st + lane * 8);
        a[0] = bf16_lo(v.x); a[1] = bf16_hi(v.x); a[2] = bf16_lo(v.y); a[3] = bf16_hi(v.y);
      } else {
#pragma unroll
        for (int t = 0; t < TU; ++t) {
          float v[E];
          sv_unpack<T, E>(*reinterpret_cast<const uint32_t*>(st + (32 * t + lane) * 4), v);
#pragma unroll
          for (int e = 0; e < E; ++e) a[t * E + e] = v[e];
        }
      }
      add(a, q);
    }
    cp_async_wait<0>();
  } else {
    constexpr int U = TC == 8 ? 1 : 4;  // rows loaded together
    int64_t cs[TC];
#pragma unroll
    for (int t = 0; t < TC; ++t) cs[t] = c0 + column(t) < V ? c0 + column(t) : V - 1;
    const float* rq = ratio + (b_begin + warp) * NB;
    int k = 0;
    for (; k + U <= n_rows; k += U) {
      float a[U][TC];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const T* rp = row_of(k + u);
#pragma unroll
        for (int t = 0; t < TC; ++t) a[u][t] = load_elem(rp, cs[t]);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float2 q[NP];
        take_q(rq + (int64_t)(k + u) * (kSvWarps * NB), q);
        add(a[u], q);
      }
    }
    for (; k < n_rows; ++k) {
      float a[TC];
      const T* rp = row_of(k);
#pragma unroll
      for (int t = 0; t < TC; ++t) a[t] = load_elem(rp, cs[t]);
      float2 q[NP];
      take_q(rq + (int64_t)k * (kSvWarps * NB), q);
      add(a, q);
    }
  }
  __syncthreads();  // the rings are free
  float(*red)[NB][COLS] = reinterpret_cast<float(*)[NB][COLS]>(sv_smem);
#pragma unroll
  for (int t = 0; t < TC; ++t)
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      red[warp][2 * k][column(t)] = acc[t][k].x;
      red[warp][2 * k + 1][column(t)] = acc[t][k].y;
    }
  __syncthreads();
  for (int i = tid; i < NB * COLS; i += kSvThreads) {
    const int r = i / COLS, c = i % COLS;
    if (c0 + c >= V) continue;
    float sum = red[0][r][c];
#pragma unroll
    for (int w = 1; w < kSvWarps; ++w) sum += red[w][r][c];
    part[((int64_t)blockIdx.y * NB + r) * ldp + c0 + c] = sum;
  }
}

// How a call of several views is split: views in equal blocks, slices and row splits of the forward
// pass and row chunks of the back pass for about one wave of CTAs, within `cap` bytes.
struct SvPlan {
  int blocks, per, nb, pitch;  // views: blocks of `per` (padded to nb)
  int slices, piece_cols, row_splits;
  int64_t chunks, rows_per_chunk, ldp;
  int64_t ranges;  // warps of the one-view forward kernel, where two views may take it (0: they do not)
  int maxp;        // and its row pieces a warp
  size_t bytes;
};

// Two views of float32 rows on 16-byte boundaries take the one-view forward kernel with both images in
// shared memory where they fit and the matrix is past 96 MB: it reads whole stretches of rows, 5.6 TB/s
// (projection of 20,833 x 4,800: 71 against 89 us, 6,944 x 14,400 71 and 88), the kernel of several views 128
// bytes of 16 rows at a time. From L2 that is the faster (1,666 x 4,800: 12.0 against 13.4 us), as it
// is for BF16, of three views on, and past 25,600 voxels (2,777 x 36,000: 87 against 95 us).
constexpr int64_t kSvSplitBytes = 96000000;
constexpr size_t kSvSplitSmem = 200 * 1024;
constexpr double kSvPlanBytes = 24e6;  // smaller matrices: the host's time for the search is not won back

static size_t sv_forward_floats(const SvPlan& p, int64_t n_bins) {
  const size_t views = (size_t)p.slices * n_bins * p.nb, split = (size_t)p.ranges * p.maxp * 2;
  return views > split ? views : split;
}

static size_t sv_bytes(const SvPlan& p, int64_t n_bins, int64_t V) {
  size_t b = align_up((size_t)V * p.pitch * sizeof(float), 256);
  b += align_up((size_t)n_bins * p.nb * sizeof(float), 256);                      // ratios
  b += align_up(sv_forward_floats(p, n_bins) * sizeof(float), 256);               // forward partials
  b += align_up((size_t)p.chunks * p.nb * (size_t)p.ldp * sizeof(float), 256);    // back partials
  return b + 256;
}

template <typename T>
static bool sv_aligned(const T* A, int64_t lda) {
  return (lda * (int64_t)sizeof(T)) % 16 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0;
}

// el: bytes of a value of A; 0: the most that a plan for any type and alignment takes.
static SvPlan plan_views(int64_t n_bins, int64_t V, int n_rot, size_t cap, size_t el, bool aligned) {
  const int64_t sms = num_sms();
  SvPlan p{};
  p.ldp = (int64_t)align_up((size_t)V, 8);
  if (n_rot == 2 && el != sizeof(__nv_bfloat16) && (size_t)p.ldp * 2 * sizeof(float) <= kSvSplitSmem &&
      n_bins * V * (int64_t)sizeof(float) >= kSvSplitBytes) {
    p.ranges = sms * 32;
    p.maxp = (int)((n_bins + p.ranges - 1) / p.ranges) + 2;
  }
  for (int blocks = (n_rot + kSvMaxViews - 1) / kSvMaxViews;; ++blocks) {
    p.blocks = blocks;
    p.per = (n_rot + blocks - 1) / blocks;
    p.nb = sv_pad(p.per);
    p.pitch = sv_pitch(p.nb);
    const int64_t units = (V + 63) / 64;
    const int64_t group = (int64_t)kSvWarps * sv_rows(p.nb);
    const int64_t groups = (n_bins + group - 1) / group;
    // forward: at least the slices that fit shared memory whole, more while row groups leave SMs idle
    const int64_t wave = sms * sv_fwd_ctas(p.nb);
    const int64_t cols_fit =
        (int64_t)((kSvSmem / sv_fwd_ctas(p.nb) - sv_fwd_ring(p.nb)) / (p.pitch * sizeof(float))) / 64 * 64;
    int64_t slices = (V + cols_fit - 1) / cols_fit;
    const int64_t want = wave / (groups < wave ? groups : wave);
    if (slices < want) slices = want;
    if (slices > units) slices = units;
    // back: about two CTAs an SM, at least eight rows a warp
    const int64_t tile = sv_back_cols(p.nb, el ? el : sizeof(__nv_bfloat16), aligned), tiles = (V + tile - 1) / tile;
    const int64_t most = (n_bins + 63) / 64;
    int64_t chunks = (2 * sms + tiles - 1) / tiles;
    if (chunks > most) chunks = most;
    // Then a few more of either where they fill the rounds of CTAs better: the passes' bytes over the share of
    // the CTA slots that work, a round's start and end (about 1 us + 0.1 us a view at 6.5 TB/s) and the partial
    // sums written and read. Two views: projection of 20,833 float32 rows of 4,800 voxels 146 -> 89 us (one
    // slice: 163 CTAs on 304 slots; nine: five rounds, 97% of them at work), weight of 2,777 x 36,000 164 -> 158.
    const double work = (double)n_bins * (double)V * (double)el, turn = 0.65e6 * (double)(10 + p.nb);
    auto cheapest = [](int64_t first, int64_t last, auto cost) {
      int64_t best = first;
      double least = cost(first);
      for (int64_t k = first + 1; k <= last; ++k) {
        const double c = cost(k);
        if (c < least) {
          least = c;
          best = k;
        }
      }
      return best;
    };
    const int64_t slices_to = slices + 8 < units ? slices + 8 : units, chunks_to = chunks + 8 < most ? chunks + 8 : most;
    if (el == 0) {
      slices = slices_to;
      chunks = chunks_to;
    }
    if (work >= kSvPlanBytes) slices = cheapest(slices, slices_to, [&](int64_t k) {
      const int64_t splits = wave / k < 1 ? 1 : (wave / k < groups ? wave / k : groups);
      const double rounds = (double)((groups + splits - 1) / splits) * (double)((k * splits + wave - 1) / wave);
      return work * rounds * (double)wave / (double)(groups * k) + turn * rounds +
             8.0 * (double)(k * n_bins * p.nb);
    });
    const int64_t slots = sms * sv_back_ctas(p.nb);
    if (work >= kSvPlanBytes) chunks = cheapest(chunks, chunks_to, [&](int64_t k) {
      // (two CTAs of three already draw the full rate: a last round of fewer takes as long as theirs)
      const int64_t full = tiles * k / slots, rest = tiles * k % slots, least = 2 * slots / 3;
      const double share = (double)(full * slots + (rest == 0 ? 0 : rest < least ? least : rest));
      return work * share / (double)(tiles * k) + turn * (double)(full + (rest > 0)) +
             8.0 * (double)(k * p.nb) * (double)V;
    });
    for (;;) {
      p.slices = (int)slices;
      p.rows_per_chunk = (n_bins + chunks - 1) / chunks;
      p.chunks = (n_bins + p.rows_per_chunk - 1) / p.rows_per_chunk;
      p.bytes = sv_bytes(p, n_bins, V);
      if (p.bytes > cap && p.ranges > 0) {
        p.ranges = 0;
        continue;
      }
      if (p.bytes <= cap || (slices == 1 && chunks == 1)) break;
      if (slices > 1) slices = (slices + 1) / 2;
      else chunks = (chunks + 1) / 2;
    }
    const int64_t cols = (units + p.slices - 1) / p.slices * 64;
    p.piece_cols = (int)(cols < cols_fit ? cols : cols_fit);
    int64_t splits = wave / p.slices;
    if (splits > groups) splits = groups;
    p.row_splits = (int)(splits < 1 ? 1 : (splits > 65535 ? 65535 : splits));
    if (p.bytes <= cap || p.per == 1) return p;
  }
}

template <typename T, int NB, bool RING>
static int sv_launch_block(const T* A, int64_t lda, const int64_t* row_idx, int64_t n_bins, int64_t V,
                           const SvPlan& p, const float* xt, float* ratio, float* fpart, float* part, int r0, int nr,
                           const float* proj, int64_t ld_proj, int mode, float floor_v, int stage, float* fout,
                           int64_t ld_fout, cudaStream_t st) {
  using Tr = SvTraits<T, NB, RING>;
  const bool split = NB == 2 && sizeof(T) == 4 && p.ranges > 0 && sv_aligned(A, lda);
  if (stage != 2 && split) {
    if constexpr (NB == 2 && sizeof(T) == 4) {
      const int64_t nvr = (V + 3) / 4, L = (n_bins * nvr + p.ranges - 1) / p.ranges;
      auto kernel = sc_forward_split_kernel<T, true, true, 1024, 2>;
      JSCC_CUDA_CHECK(allow_smem(kernel));
      JSCC_TIMED("sc_forward_split", st,
                 (kernel<<<(unsigned)(p.ranges / 32), 1024, (size_t)p.ldp * 2 * sizeof(float), st>>>(
                     A, lda, row_idx, n_bins, V, xt, nvr, L, p.maxp, fpart)));
      JSCC_LAUNCH_CHECK();
      const unsigned blocks = (unsigned)((2 * n_bins + 255) / 256);
      if (stage == 1)
        JSCC_TIMED("sc_finish_raw", st,
                   (sc_finish_raw_kernel<2><<<blocks, 256, 0, st>>>(fpart, n_bins, nvr, L, p.maxp, fout, ld_fout)));
      else
        JSCC_TIMED("sc_finish_ratio", st,
                   (sc_finish_ratio_kernel<2><<<blocks, 256, 0, st>>>(fpart, n_bins, nvr, L, p.maxp, row_idx, proj,
                                                                      ld_proj, mode, floor_v, ratio, fout, ld_fout)));
      JSCC_LAUNCH_CHECK();
    }
    if (stage == 1) return JSCC_OK;
  } else if (stage != 2) {
    const size_t smem = Tr::kFwdRing + align_up((size_t)p.piece_cols * p.pitch * sizeof(float), 16);
    JSCC_CUDA_CHECK(allow_smem(sc_views_forward_kernel<T, NB, RING>));
    JSCC_TIMED("sc_views_forward", st,
               (sc_views_forward_kernel<T, NB, RING><<<dim3((unsigned)p.slices, (unsigned)p.row_splits), kSvThreads,
                                                       smem, st>>>(A, lda, row_idx, n_bins, V, xt, p.slices,
                                                                   p.piece_cols, fpart)));
    JSCC_LAUNCH_CHECK();
    JSCC_TIMED("sc_views_ratio", st,
               (sc_views_ratio_kernel<<<(unsigned)((n_bins * NB + 31) / 32), kSvThreads, 0, st>>>(
                   fpart, p.slices, n_bins, NB, nr, r0, row_idx, proj, ld_proj, mode, floor_v, stage == 1 ? nullptr : ratio,
                   fout, ld_fout)));
    JSCC_LAUNCH_CHECK();
    if (stage == 1) return JSCC_OK;
  }
  auto back = [&](auto kernel, int smem, int cols) {
    cudaError_t e = allow_smem(kernel);
    if (e != cudaSuccess) return e;
    JSCC_TIMED("sc_views_back", st,
               (kernel<<<dim3((unsigned)((V + cols - 1) / cols), (unsigned)p.chunks), kSvThreads, smem, st>>>(
                   A, lda, row_idx, n_bins, V, ratio, p.rows_per_chunk, part, p.ldp)));
    return cudaSuccess;
  };
  using Wide = SvBack<T, NB, 2>;
  const int unit = Wide::kUnit * (int)sizeof(T);
  const bool whole = (lda * (int64_t)sizeof(T)) % unit == 0 && reinterpret_cast<uintptr_t>(A) % unit == 0;
  // rows on odd boundaries: four-byte copies pay from 12 views on, where the plain loads' registers
  // leave one CTA an SM (2,048 x 35,343 float32, 8 views: plain 68 us, copies 125 us; 512 rows, 20
  // views: copies 51 us)
  constexpr int kOdd = (RING && NB >= 12) ? 1 : 0;
  JSCC_CUDA_CHECK(whole ? back(sc_views_back_kernel<T, NB, 2>, Wide::kSmem, 32 * Wide::kCols)
                        : back(sc_views_back_kernel<T, NB, kOdd>, SvBack<T, NB, kOdd>::kSmem,
                               32 * SvBack<T, NB, kOdd>::kCols));
  JSCC_LAUNCH_CHECK();
  return JSCC_OK;
}

// The weight (stage 0), the projection into fout (1) or the back-projection of gin (2) of n_rot >= 2
// views, within `ws_bytes` of workspace.
template <typename T>
static int sc_views(const T* A, int64_t lda, const int64_t* row_idx, int64_t n_bins, int64_t V, const float* proj,
                    int64_t ld_proj, int n_rot, const float* img, const int64_t* rotmat, const int64_t* rotinv,
                    int64_t ld_rot, int mode, float floor_v, int has_scale, float scale, float* weight,
                    void* ws, size_t ws_bytes, cudaStream_t st, int stage, float* fout, int64_t ld_fout,
                    const float* gin, int64_t ld_gin) {
  const SvPlan p = plan_views(n_bins, V, n_rot, ws_bytes, sizeof(T), sv_aligned(A, lda));
  JSCC_REQUIRE(p.bytes <= ws_bytes, "SC projector: %d views need %zu bytes of workspace (%zu given)", n_rot, p.bytes,
               ws_bytes);
  Carver cv(ws, ws_bytes);
  float* xt = cv.take<float>((size_t)V * p.pitch);
  float* ratio = cv.take<float>((size_t)n_bins * p.nb);
  float* fpart = cv.take<float>(sv_forward_floats(p, n_bins));
  float* part = cv.take<float>((size_t)p.chunks * p.nb * (size_t)p.ldp);
  JSCC_REQUIRE(cv.ok(), "SC projector: workspace carve overflow");
  const int64_t cap = (int64_t)num_sms() * 16;
  // rows on four-byte boundaries (always for float32)
  [[maybe_unused]] const bool ring = (lda * (int64_t)sizeof(T)) % 4 == 0 && reinterpret_cast<uintptr_t>(A) % 4 == 0;
  for (int r0 = 0; r0 < n_rot; r0 += p.per) {
    const int nr = n_rot - r0 < p.per ? n_rot - r0 : p.per;
    if (stage != 2) {
      int64_t blocks = (V * p.pitch + 255) / 256;
      if (blocks > cap) blocks = cap;
      JSCC_TIMED("sc_gather_rot", st,
                 (sc_views_gather_kernel<<<(unsigned)blocks, 256, 0, st>>>(img, rotmat, ld_rot, r0, nr, p.pitch, V,
                                                                           xt)));
      JSCC_LAUNCH_CHECK();
    } else {
      int64_t blocks = (n_bins * p.nb + 255) / 256;
      if (blocks > cap) blocks = cap;
      JSCC_TIMED("sc_load_ratio", st,
                 (sc_load_ratio_kernel<<<(unsigned)blocks, 256, 0, st>>>(gin, ld_gin, n_bins, r0, nr, p.nb, ratio)));
      JSCC_LAUNCH_CHECK();
    }
#define JSCC_SV_LAUNCH(NB, RING)                                                                                 \
  sv_launch_block<T, NB, RING>(A, lda, row_idx, n_bins, V, p, xt, ratio, fpart, part, r0, nr, proj, ld_proj,     \
                               mode, floor_v, stage, fout, ld_fout, st)
#define JSCC_SV(NB)                                                                                              \
  case NB:                                                                                                       \
    if constexpr (sizeof(T) == 2) rc = ring ? JSCC_SV_LAUNCH(NB, true) : JSCC_SV_LAUNCH(NB, false);              \
    else rc = JSCC_SV_LAUNCH(NB, true);                                                                          \
    break
    int rc = JSCC_OK;
    switch (p.nb) {
      JSCC_SV(2);
      JSCC_SV(4);
      JSCC_SV(8);
      JSCC_SV(12);
      JSCC_SV(16);
      JSCC_SV(20);
    }
#undef JSCC_SV
#undef JSCC_SV_LAUNCH
    if (rc != JSCC_OK) return rc;
    if (stage == 1) continue;
    rc = launch_reduce_scatter(part, p.ldp, (int)p.chunks, nr, p.nb, rotinv, ld_rot, r0, V, has_scale, scale, weight,
                               st);
    if (rc != JSCC_OK) return rc;
  }
  return JSCC_OK;
}

}  // namespace jscc
