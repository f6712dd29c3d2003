// Single-photon (self-collimation, SC) projector: w += scale * sum_r P_r^-1 A^T (y_r / A P_r x).
//
// Reference semantics: recon_osem_plane.py:28-30 (get_weight_single) inside the
// rotation loop of osem_bin_mode (recon_osem_plane.py:49-53); the clamped form of
// recon_osem_local_cntstat.py:6-8.
//
// GB300 design
//  * Several views: all of a block of up to 20 share each pass over the subset matrix A
//    (sc_views.cuh: a skinny FP32 GEMM in registers instead of R GEMVs).
//  * One view: the single-read kernel (sc_fused.cuh) where a row half fits its registers;
//    otherwise, and for the projector's halves on their own, the two passes below:
//    forward: persistent grid, 128-bit streaming loads of A that bypass L1, balanced
//    contiguous ranges per warp; back: CTA per (1024-column tile x row chunk), each thread
//    owns 4 (fp32) or 8 (bf16) adjacent columns and walks its rows in order.
//  * Reduce pass: the chunk partials in a fixed order, the inverse rotation gather,
//    accumulated into `weight`.
//  No float atomics anywhere: every sum has one fixed order, so results are
//  bit-reproducible run to run.
#include "jscc_common.cuh"

#include <mutex>

#include "sc_fused.cuh"

namespace jscc {

constexpr int kRotBlock = 8;          // most rotations the minimum workspace provides for
constexpr int kColTile = 1024;        // columns per back-pass CTA
constexpr int kTargetCtas = 1216;     // back-pass grid target (8 CTAs x 152 SMs)

__device__ unsigned int g_bad_index_count = 0;  // out-of-range rotation indices seen

// ------------------------------------------------------------------ gather
__global__ void sc_gather_rot_kernel(const float* __restrict__ img, const int64_t* __restrict__ rotmat,
                                     int64_t ld_rot, int r0, int nr, int64_t V, int64_t ldx,
                                     float* __restrict__ xr) {
  const int64_t total = (int64_t)nr * V;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(t / V);
    const int64_t j = t - (int64_t)r * V;
    int64_t src = j;
    if (rotmat != nullptr) {
      src = rotmat[j * ld_rot + r0 + r] - 1;
      if (src < 0 || src >= V) {
        atomicAdd(&g_bad_index_count, 1u);
        xr[(int64_t)r * ldx + j] = 0.f;
        continue;
      }
    }
    xr[(int64_t)r * ldx + j] = img[src];
  }
}

// ------------------------------------------------------------------ forward
template <typename T>
struct VecTraits;
template <>
struct VecTraits<float> {
  static constexpr int kVec = 4;  // elements per 16-byte load
};
template <>
struct VecTraits<__nv_bfloat16> {
  static constexpr int kVec = 8;
};

template <typename T>
__device__ __forceinline__ void load_vec(const T* p, float (&v)[VecTraits<T>::kVec]);

template <>
__device__ __forceinline__ void load_vec<float>(const float* p, float (&v)[4]) {
  float4 a = ld_stream_f4(p);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
template <>
__device__ __forceinline__ void load_vec<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[8]) {
  uint4 u = ld_stream_u4(p);
  v[0] = bf16_lo(u.x); v[1] = bf16_hi(u.x);
  v[2] = bf16_lo(u.y); v[3] = bf16_hi(u.y);
  v[4] = bf16_lo(u.z); v[5] = bf16_hi(u.z);
  v[6] = bf16_lo(u.w); v[7] = bf16_hi(u.w);
}

template <typename T>
__device__ __forceinline__ void unpack_vec(const uint4& u, float (&v)[VecTraits<T>::kVec]) {
  if constexpr (sizeof(T) == 4) {
    v[0] = __uint_as_float(u.x); v[1] = __uint_as_float(u.y);
    v[2] = __uint_as_float(u.z); v[3] = __uint_as_float(u.w);
  } else {
    v[0] = bf16_lo(u.x); v[1] = bf16_hi(u.x);
    v[2] = bf16_lo(u.y); v[3] = bf16_hi(u.y);
    v[4] = bf16_lo(u.z); v[5] = bf16_hi(u.z);
    v[6] = bf16_lo(u.w); v[7] = bf16_hi(u.w);
  }
}

// acc + sum_k a[k] * x[k] over one 16-byte vector of A held as raw bits.
template <typename T>
__device__ __forceinline__ float fma_raw(const uint4& u, const float* x, float acc);
template <>
__device__ __forceinline__ float fma_raw<float>(const uint4& u, const float* x, float acc) {
  const float4 xv = *reinterpret_cast<const float4*>(x);
  acc = fmaf(__uint_as_float(u.x), xv.x, acc);
  acc = fmaf(__uint_as_float(u.y), xv.y, acc);
  acc = fmaf(__uint_as_float(u.z), xv.z, acc);
  acc = fmaf(__uint_as_float(u.w), xv.w, acc);
  return acc;
}
template <>
__device__ __forceinline__ float fma_raw<__nv_bfloat16>(const uint4& u, const float* x, float acc) {
  const float4 x0 = *reinterpret_cast<const float4*>(x);
  const float4 x1 = *reinterpret_cast<const float4*>(x + 4);
  acc = fmaf(bf16_lo(u.x), x0.x, acc);
  acc = fmaf(bf16_hi(u.x), x0.y, acc);
  acc = fmaf(bf16_lo(u.y), x0.z, acc);
  acc = fmaf(bf16_hi(u.y), x0.w, acc);
  acc = fmaf(bf16_lo(u.z), x1.x, acc);
  acc = fmaf(bf16_hi(u.z), x1.y, acc);
  acc = fmaf(bf16_lo(u.w), x1.z, acc);
  acc = fmaf(bf16_hi(u.w), x1.w, acc);
  return acc;
}

// ------------------------------------------------------------------ forward, balanced split
// The subset matrix is viewed as n_bins x nvr vector units (nvr = ceil(V / NV)). Every
// warp of the persistent grid owns one contiguous range of L units (the last warp
// fewer), so all warps stream the same number of bytes. A range crosses at most a
// few row boundaries; for each row piece the warp writes one partial dot product
// to part[g][k]. sc_finish_ratio_kernel sums a row's partials in warp order. The image is staged
// in shared memory when it fits. VIEWS = 2: two images, x[j][2], with two partials a piece (staged one after
// the other, xs[r][ldx]).
template <typename T, bool VEC, bool SMEM_X, int THREADS, int VIEWS = 1>
__global__ void __launch_bounds__(THREADS)
sc_forward_split_kernel(const T* __restrict__ A, int64_t lda, const int64_t* __restrict__ row_idx,
                        int64_t n_bins, int64_t V, const float* __restrict__ x, int64_t nvr, int64_t L, int maxp,
                        float* __restrict__ part) {
  constexpr int NV = VEC ? VecTraits<T>::kVec : 1;
  constexpr int WARPS = THREADS / 32;
  extern __shared__ float4 xs4[];
  float* xs = reinterpret_cast<float*>(xs4);
  const int lane = threadIdx.x & 31;
  const int64_t g = (int64_t)blockIdx.x * WARPS + (threadIdx.x >> 5);
  static_assert(VIEWS == 1 || SMEM_X, "two images are staged");
  const int ldx = VIEWS == 1 ? 0 : (int)((V + 7) / 8 * 8);
  if (SMEM_X) {
    for (int64_t i = threadIdx.x; i < V; i += THREADS)
#pragma unroll
      for (int r = 0; r < VIEWS; ++r) xs[r * ldx + i] = __ldg(x + i * VIEWS + r);
    __syncthreads();
  }
  const float* xsrc = SMEM_X ? xs : x;
  const int64_t U = n_bins * nvr;
  int64_t u = g * L;
  const int64_t u_end = (u + L < U) ? u + L : U;
  int64_t row = u < U ? u / nvr : 0;
  int k = 0;
  while (u < u_end) {
    const int64_t row_end = (row + 1) * nvr;
    const int64_t piece_end = row_end < u_end ? row_end : u_end;
    const T* rowp = A + (row_idx ? row_idx[row] : row) * lda;
    const int64_t ubase = row * nvr;
    float acc[VIEWS];
#pragma unroll
    for (int r = 0; r < VIEWS; ++r) acc[r] = 0.f;
    int64_t uu = u + lane;
    if constexpr (VEC) {
      // 4 independent 16-byte loads in flight per lane; raw registers, converted on use.
      // Only whole vectors here (32-bit column arithmetic); the row's partial last
      // vector, if any, is left to the loop below.
      const int64_t full_end_u = ubase + V / NV;
      const int64_t fe = piece_end < full_end_u ? piece_end : full_end_u;
      if (uu + 96 < fe) {
        const T* rp = rowp;
        const float* xp0 = xsrc;
        int col = (int)(uu - ubase) * NV;
        const int n_iter = (int)((fe - uu - 96 + 127) / 128);
        for (int it = 0; it < n_iter; ++it, col += 128 * NV) {
          uint4 raw[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) raw[q] = ld_stream_u4(rp + col + 32 * NV * q);
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int r = 0; r < VIEWS; ++r) acc[r] = fma_raw<T>(raw[q], xp0 + r * ldx + col + 32 * NV * q, acc[r]);
        }
        uu += (int64_t)n_iter * 128;
      }
    }
    for (; uu < piece_end; uu += 32) {
      const int64_t col = (uu - ubase) * NV;
      bool done = false;
      if constexpr (VEC) {
        if (col + NV <= V) {
          float a[NV];
          load_vec<T>(rowp + col, a);
#pragma unroll
          for (int r = 0; r < VIEWS; ++r)
#pragma unroll
            for (int kk = 0; kk < NV; ++kk) acc[r] = fmaf(a[kk], xsrc[r * ldx + col + kk], acc[r]);
          done = true;
        }
      }
      if (!done) {
        const int64_t cend = (col + NV < V) ? col + NV : V;
        for (int64_t c = col; c < cend; ++c) {
          const float a = load_elem(rowp, c);
#pragma unroll
          for (int r = 0; r < VIEWS; ++r) acc[r] = fmaf(a, xsrc[r * ldx + c], acc[r]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < VIEWS; ++r) {
      const float sum = warp_sum(acc[r]);
      if (lane == 0) part[(g * maxp + k) * VIEWS + r] = sum;
    }
    ++k;
    ++row;
    u = piece_end;
  }
}

// f of row b (in view r): the row's partials in warp order
template <int VIEWS>
__device__ __forceinline__ float row_sum(const float* __restrict__ part, int64_t b, int r, int64_t nvr, int64_t L,
                                         int maxp) {
  const int64_t g0 = (b * nvr) / L;
  const int64_t g1 = ((b + 1) * nvr - 1) / L;
  float f = 0.f;
  for (int64_t g = g0; g <= g1; ++g) {
    const int64_t first_row = (g * L) / nvr;
    f += part[((g * maxp) + (b - first_row)) * VIEWS + r];
  }
  return f;
}

// ratio[b] = row_ratio(proj[b], f), and f_out[b] = f where it is given (of two views: [b][2], columns 0 and 1
// of proj and f_out)
template <int VIEWS>
__global__ void sc_finish_ratio_kernel(const float* __restrict__ part, int64_t n_bins, int64_t nvr,
                                       int64_t L, int maxp, const int64_t* __restrict__ row_idx,
                                       const float* __restrict__ proj, int64_t ld_proj, int mode, float floor_v,
                                       float* __restrict__ ratio, float* __restrict__ f_out, int64_t ld_f) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_bins * VIEWS;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = t / VIEWS;
    const int r = (int)(t % VIEWS);
    const float f = row_sum<VIEWS>(part, b, r, nvr, L, maxp);
    const int64_t pb = row_idx ? row_idx[b] : b;
    if (f_out != nullptr) f_out[b * ld_f + r] = f;
    ratio[t] = row_ratio(proj[pb * ld_proj + r], f, mode, floor_v);
  }
}

// out[b][r] = f(b, r) (the forward projection itself, no ratio)
template <int VIEWS>
__global__ void sc_finish_raw_kernel(const float* __restrict__ part, int64_t n_bins, int64_t nvr, int64_t L,
                                     int maxp, float* __restrict__ out, int64_t ld_out) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_bins * VIEWS;
       t += (int64_t)gridDim.x * blockDim.x)
    out[t / VIEWS * ld_out + t % VIEWS] = row_sum<VIEWS>(part, t / VIEWS, (int)(t % VIEWS), nvr, L, maxp);
}

// ratio[b * nb + r] = g[b][r0 + r] (a caller-given vector to back-project), 0 for r >= nr
__global__ void sc_load_ratio_kernel(const float* __restrict__ g, int64_t ld_g, int64_t n_bins, int r0, int nr,
                                     int nb, float* __restrict__ ratio) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_bins * nb;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = t / nb;
    const int r = (int)(t % nb);
    ratio[t] = r < nr ? g[b * ld_g + r0 + r] : 0.f;
  }
}

// ------------------------------------------------------------------ back (partials)
// part[chunk][col] = sum_{b in chunk} A[b, col] * ratio[b]. Bound by HBM once enough rows are in flight: a
// thread loads kBackRows of them before it uses the first, within the registers that keep five (float32) or eight
// CTAs an SM. 5,555 BF16 rows of 36,000 voxels: four rows at a time 85 us, eight 71 (5.6 TB/s); 2,777 float32
// rows: four 68, eight without the bound, so four CTAs an SM and three rounds, 80, six 61 us (6.5 TB/s).
template <typename T>
constexpr int kBackRows = sizeof(T) == 2 ? 8 : 6;

template <typename T, bool VEC>
__global__ void __launch_bounds__(kColTile / VecTraits<T>::kVec, sizeof(T) == 2 ? 8 : 5)
sc_back_partial_kernel(const T* __restrict__ A, int64_t lda, const int64_t* __restrict__ row_idx,
                       int64_t n_bins, int64_t V, const float* __restrict__ ratio, int64_t rows_per_chunk,
                       float* __restrict__ part, int64_t ldp) {
  constexpr int NV = VecTraits<T>::kVec;
  const int64_t col = (int64_t)blockIdx.x * kColTile + (int64_t)threadIdx.x * NV;
  const int64_t b_begin = (int64_t)blockIdx.y * rows_per_chunk;
  int64_t b_end = b_begin + rows_per_chunk;
  if (b_end > n_bins) b_end = n_bins;
  if (col >= V) return;
  const bool full = VEC && (col + NV <= V);
  const int ncol = (int)((V - col) < NV ? (V - col) : NV);

  float acc[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) acc[k] = 0.f;

  if (full) {
    int64_t b = b_begin;
    auto rows = [&](auto count) {  // that many rows, loaded together
      constexpr int N = decltype(count)::value;
      uint4 raw[N];
#pragma unroll
      for (int u = 0; u < N; ++u) raw[u] = ld_stream_u4(A + (row_idx ? row_idx[b + u] : b + u) * lda + col);
#pragma unroll
      for (int u = 0; u < N; ++u) {
        const float q = __ldg(ratio + b + u);
        float a[NV];
        unpack_vec<T>(raw[u], a);
#pragma unroll
        for (int k = 0; k < NV; ++k) acc[k] = fmaf(a[k], q, acc[k]);
      }
      b += N;
    };
    while (b + kBackRows<T> <= b_end) rows(std::integral_constant<int, kBackRows<T>>{});
    if (b + 4 <= b_end) rows(std::integral_constant<int, 4>{});
    while (b < b_end) rows(std::integral_constant<int, 1>{});
  } else {
    for (int64_t b = b_begin; b < b_end; ++b) {
      const T* rowb = A + (row_idx ? row_idx[b] : b) * lda;
      const float q = __ldg(ratio + b);
#pragma unroll
      for (int k = 0; k < NV; ++k)
        if (k < ncol) acc[k] = fmaf(load_elem(rowb, col + k), q, acc[k]);
    }
  }

  float* dst = part + (int64_t)blockIdx.y * ldp + col;
#pragma unroll
  for (int k = 0; k < NV; ++k)
    if (k < ncol) dst[k] = acc[k];
}

// ------------------------------------------------------------------ compensated column sums
// Kahan summation (Kahan 1965): s accumulates, c carries the rounding error of each add with
// the opposite sign; every add is an explicit round-to-nearest op so nothing is contracted.
__device__ __forceinline__ void kahan_add(float& s, float& c, float v) {
  const float y = __fsub_rn(v, c);
  const float t = __fadd_rn(s, y);
  c = __fsub_rn(__fsub_rn(t, s), y);
  s = t;
}

// sum[chunk][col] / comp[chunk][col]: compensated column sums of the chunk's rows of A. Bound by
// the rows' bytes once enough of them are in flight: a thread loads kSumRows rows before it adds them
// (20,480 x 36,000 floats: one row at a time 535 us, 5.5 TB/s; eight, in one wave of CTAs, 430 us,
// 6.9 TB/s).
constexpr int kSumRows = 8;

template <typename T, bool VEC>
__global__ void __launch_bounds__(kColTile / VecTraits<T>::kVec)
sc_colsum_kahan_kernel(const T* __restrict__ A, int64_t lda, const int64_t* __restrict__ row_idx, int64_t n_bins,
                       int64_t V, int64_t rows_per_chunk, float* __restrict__ sum, float* __restrict__ comp,
                       int64_t ldp) {
  constexpr int NV = VecTraits<T>::kVec;
  const int64_t col = (int64_t)blockIdx.x * kColTile + (int64_t)threadIdx.x * NV;
  const int64_t b_begin = (int64_t)blockIdx.y * rows_per_chunk;
  int64_t b_end = b_begin + rows_per_chunk;
  if (b_end > n_bins) b_end = n_bins;
  if (col >= V) return;
  const int ncol = (int)((V - col) < NV ? (V - col) : NV);
  float sa[NV], ca[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) sa[k] = ca[k] = 0.f;
  if (VEC && ncol == NV) {
    int64_t b = b_begin;
    for (; b + kSumRows <= b_end; b += kSumRows) {
      uint4 v[kSumRows];
#pragma unroll
      for (int u = 0; u < kSumRows; ++u)
        v[u] = ld_stream_u4(A + (row_idx ? row_idx[b + u] : b + u) * lda + col);
#pragma unroll
      for (int u = 0; u < kSumRows; ++u) {
        float a[NV];
        unpack_vec<T>(v[u], a);
#pragma unroll
        for (int k = 0; k < NV; ++k) kahan_add(sa[k], ca[k], a[k]);
      }
    }
    for (; b < b_end; ++b) {
      float a[NV];
      load_vec<T>(A + (row_idx ? row_idx[b] : b) * lda + col, a);
#pragma unroll
      for (int k = 0; k < NV; ++k) kahan_add(sa[k], ca[k], a[k]);
    }
  } else {
    for (int64_t b = b_begin; b < b_end; ++b) {
      const T* rowb = A + (row_idx ? row_idx[b] : b) * lda;
#pragma unroll
      for (int k = 0; k < NV; ++k)
        if (k < ncol) kahan_add(sa[k], ca[k], load_elem(rowb, col + k));
    }
  }
  float* ds = sum + (int64_t)blockIdx.y * ldp + col;
  float* dc = comp + (int64_t)blockIdx.y * ldp + col;
#pragma unroll
  for (int k = 0; k < NV; ++k)
    if (k < ncol) {
      ds[k] = sa[k];
      dc[k] = ca[k];
    }
}

// ------------------------------------------------------------------ reduce + inverse rotation
// weight[j] += scale * sum_r sum_c part[c][r][src(j, r)] over the nr rotations of the block and their
// chunks. SPLIT threads of a block share a voxel: each adds one contiguous part of the (rotation, chunk)
// terms and the parts' sums are added in order (one fixed order), so the partial images are read with SPLIT
// times the loads in flight of one thread per voxel (bound by latency, not bytes: 76 images of 21,252
// voxels 14.1 -> 8.0 us between events, of which about 5 are the events'). Eight threads where the voxels are
// few; from kRedFewVoxels on four, as eight then fill the chip's threads by themselves (back projection of
// 1,777 BF16 rows, split 8 / 4 / 2: 36,000 voxels 29.9 / 27.8 / 27.8 us, weight of 5,555 87.0 / 86.2 / 87.6;
// 14,400 voxels 154.5 / 155.3 / 156.8).
constexpr int kRedThreads = 256;
constexpr int64_t kRedFewVoxels = 24000;

template <int SPLIT>
__global__ void __launch_bounds__(kRedThreads)
sc_reduce_scatter_kernel(const float* __restrict__ part, int64_t ldp, int chunks, int nr, int rb_stride,
                         const int64_t* __restrict__ rotinv, int64_t ld_rot, int r0, int64_t V, int has_scale,
                         float scale, float* __restrict__ weight) {
  constexpr int VOX = kRedThreads / SPLIT;  // voxels of a block
  __shared__ float red[SPLIT][VOX];
  const int vox = threadIdx.x % VOX, share = threadIdx.x / VOX;
  const int64_t j = (int64_t)blockIdx.x * VOX + vox;
  const int terms = nr * chunks;
  const int t0 = (int)((int64_t)terms * share / SPLIT), t1 = (int)((int64_t)terms * (share + 1) / SPLIT);
  float s = 0.f;
  if (j < V) {
    for (int t = t0; t < t1;) {
      const int r = t / chunks, c_begin = t - r * chunks;
      const int c_end = (t1 - t) < (chunks - c_begin) ? c_begin + (t1 - t) : chunks;
      int64_t src = j;
      if (rotinv != nullptr) src = rotinv[j * ld_rot + r0 + r] - 1;
      if (src < 0 || src >= V) {
        if (c_begin == 0) atomicAdd(&g_bad_index_count, 1u);  // counted by the share that starts the rotation
      } else {
#pragma unroll 8
        for (int c = c_begin; c < c_end; ++c) s += part[((int64_t)c * rb_stride + r) * ldp + src];
      }
      t += c_end - c_begin;
    }
  }
  if constexpr (SPLIT > 1) {
    red[share][vox] = s;
    __syncthreads();
  }
  if (share != 0 || j >= V) return;
#pragma unroll
  for (int w = 1; w < SPLIT; ++w) s += red[w][vox];
  weight[j] = has_scale ? __fadd_rn(weight[j], __fmul_rn(scale, s)) : __fadd_rn(weight[j], s);
}

int launch_reduce_scatter(const float* part, int64_t ldp, int chunks, int nr, int rb_stride, const int64_t* rotinv,
                          int64_t ld_rot, int r0, int64_t V, int has_scale, float scale, float* weight,
                          cudaStream_t st) {
  auto launch = [&](auto kernel, int split) {
    const int vox = kRedThreads / split;
    JSCC_TIMED("sc_reduce_scatter", st,
               (kernel<<<(unsigned)((V + vox - 1) / vox), kRedThreads, 0, st>>>(
                   part, ldp, chunks, nr, rb_stride, rotinv, ld_rot, r0, V, has_scale, scale, weight)));
  };
  if (V < kRedFewVoxels) launch(sc_reduce_scatter_kernel<8>, 8);
  else launch(sc_reduce_scatter_kernel<4>, 4);
  JSCC_LAUNCH_CHECK();
  return JSCC_OK;
}

// SC sensitivity: s[j] += (sum_r colsum[rotinv[j, r] - 1]) / n_rot, colsum[c] = the chunk
// partials of column c and their carried errors summed in chunk order with compensation
// (rotations summed first, then divided, as main_local_cntstat.py:140-146 does).
__device__ __forceinline__ float fold_chunks(const float* sum, const float* comp, int64_t ldp, int chunks, int64_t c) {
  float s = 0.f, e = 0.f;
#pragma unroll 8
  for (int k = 0; k < chunks; ++k) {
    kahan_add(s, e, sum[(int64_t)k * ldp + c]);
    kahan_add(s, e, -comp[(int64_t)k * ldp + c]);
  }
  return __fsub_rn(s, e);
}

// The column sums in place of the first chunk's: several rotations fold each column once instead of
// once a rotation (20 rotations of 36,000 voxels, 16 chunks: 33 us in one kernel, 18 us in two).
__global__ void sc_fold_kernel(float* __restrict__ sum, const float* __restrict__ comp, int64_t ldp, int chunks,
                               int64_t V) {
  const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (c < V) sum[c] = fold_chunks(sum, comp, ldp, chunks, c);
}

// FOLDED: `sum` holds the column sums, else the chunks' sums (one rotation)
template <bool FOLDED>
__global__ void sc_sensitivity_kernel(const float* __restrict__ sum, const float* __restrict__ comp, int64_t ldp,
                                      int chunks, const int64_t* __restrict__ rotinv, int64_t ld_rot, int n_rot,
                                      int64_t V, float* __restrict__ weight) {
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (j >= V) return;
  float acc = 0.f, acc_c = 0.f;
#pragma unroll 4
  for (int r = 0; r < n_rot; ++r) {
    int64_t src = rotinv != nullptr ? rotinv[j * ld_rot + r] - 1 : j;
    const bool ok = src >= 0 && src < V;
    if (!ok) {
      atomicAdd(&g_bad_index_count, 1u);
      continue;
    }
    kahan_add(acc, acc_c, FOLDED ? sum[src] : fold_chunks(sum, comp, ldp, chunks, src));
  }
  weight[j] = __fadd_rn(weight[j], __fdiv_rn(__fsub_rn(acc, acc_c), (float)n_rot));
}

}  // namespace jscc

#include "sc_views.cuh"

namespace jscc {

// ------------------------------------------------------------------ host planning
struct ScPlan {
  int rb;                  // rotations the minimum workspace provides for (1, 2, 4, 8)
  int64_t ldx;             // padded voxel stride of X / partials
  int64_t col_tiles;       // back pass: 1024-column tiles
  int64_t chunks;          // back pass: row chunks
  int64_t rows_per_chunk;
  int64_t fwd_warps;       // forward pass: warps of the persistent grid (32 per SM)
  int fwd_maxp;            // forward pass: row pieces per warp (upper bound)
  size_t ws_bytes;         // the minimum workspace (the one-view two-pass kernels fill it)
  int64_t fs_clusters;     // fused single-read path (one rotation): clusters of two CTAs
  size_t fs_bytes;         // its partial images, after the two-pass carve
};

static int pow2_block(int n_rot) {
  int rb = 1;
  while (rb < n_rot && rb < kRotBlock) rb <<= 1;
  return rb;
}

static ScPlan plan_sc(int64_t n_bins, int64_t V, int32_t n_rot) {
  ScPlan p{};
  p.rb = pow2_block(n_rot < 1 ? 1 : n_rot);
  p.ldx = (int64_t)align_up((size_t)(V > 0 ? V : 1), 8);
  p.col_tiles = (V + kColTile - 1) / kColTile;
  if (p.col_tiles < 1) p.col_tiles = 1;
  int64_t chunks = (kTargetCtas + p.col_tiles - 1) / p.col_tiles;
  int64_t max_chunks = (n_bins + 15) / 16;  // at least 16 rows per chunk
  if (max_chunks < 1) max_chunks = 1;
  if (chunks > max_chunks) chunks = max_chunks;
  if (chunks < 1) chunks = 1;
  p.rows_per_chunk = (n_bins + chunks - 1) / chunks;
  if (p.rows_per_chunk < 1) p.rows_per_chunk = 1;
  p.chunks = (n_bins + p.rows_per_chunk - 1) / p.rows_per_chunk;
  if (p.chunks < 1) p.chunks = 1;
  p.fwd_warps = (int64_t)num_sms() * 32;
  p.fwd_maxp = (int)((n_bins + p.fwd_warps - 1) / p.fwd_warps) + 2;
  size_t bytes = 0;
  bytes += align_up((size_t)p.fwd_warps * p.fwd_maxp * p.rb * sizeof(float), 256);  // fwd partials
  bytes += align_up((size_t)p.rb * p.ldx * sizeof(float), 256);                   // X
  bytes += align_up((size_t)(n_bins > 0 ? n_bins : 1) * p.rb * sizeof(float), 256);  // ratio
  bytes += align_up((size_t)p.chunks * p.rb * p.ldx * sizeof(float), 256);          // partials
  p.ws_bytes = bytes + 256;
  p.fs_clusters = n_rot == 1 ? (int64_t)num_sms() / 2 : 0;
  if (p.fs_clusters > n_bins) p.fs_clusters = n_bins;
  p.fs_bytes = p.fs_clusters > 0 ? align_up((size_t)p.fs_clusters * p.ldx * sizeof(float), 256) + 256 : 0;
  return p;
}

int set_sc_poll_limit(uint32_t polls, bool reset) {
  const uint32_t v = reset ? kFsMaxPolls : polls;
  JSCC_CUDA_CHECK(cudaMemcpyToSymbol(g_sc_poll_limit, &v, sizeof(v)));
  return JSCC_OK;
}

int take_sc_timeout_count(unsigned int* out) {
  unsigned int h = 0, zero = 0;
  JSCC_CUDA_CHECK(cudaMemcpyFromSymbol(&h, g_sc_timeout_count, sizeof(h)));
  JSCC_CUDA_CHECK(cudaMemcpyToSymbol(g_sc_timeout_count, &zero, sizeof(zero)));
  *out = h;
  return JSCC_OK;
}

// The fused single-read path's partial images: after the two-pass carve `cv` when the
// workspace holds them, else nullptr (the two-pass kernels run).
static float* fused_partials(const ScPlan& p, Carver cv) {
  if (p.fs_bytes == 0) return nullptr;
  float* f = cv.take<float>((size_t)p.fs_clusters * p.ldx);
  return cv.ok() ? f : nullptr;
}

// One view. stage 0: forward, ratio, back (the weight); 1: forward only into fout; 2: back-project gin
template <typename T>
static int sc_one_view(const T* A, int64_t lda, const int64_t* row_idx, int64_t n_bins, int64_t V, const float* proj,
                       int64_t ld_proj, const float* img, const int64_t* rotmat, const int64_t* rotinv,
                       int64_t ld_rot, int mode, float floor_v, int has_scale, float scale, float* weight,
                       const ScPlan& p, float* xr, float* ratio, float* part, float* fpart, float* fs_part,
                       cudaStream_t st, int stage, float* fout, int64_t ld_fout, const float* gin, int64_t ld_gin) {
  constexpr int NV = VecTraits<T>::kVec;
  const bool vec_ok = ((lda * (int64_t)sizeof(T)) % 16 == 0) &&
                      (reinterpret_cast<uintptr_t>(A) % 16 == 0);
  const int sms = num_sms();
  const float* x = img;
  if (stage != 2 && (rotmat != nullptr || reinterpret_cast<uintptr_t>(img) % 16 != 0)) {
    int64_t blocks = (V + 255) / 256;
    if (blocks > (int64_t)sms * 16) blocks = (int64_t)sms * 16;
    JSCC_TIMED("sc_gather_rot", st,
               sc_gather_rot_kernel<<<(unsigned)blocks, 256, 0, st>>>(img, rotmat, ld_rot, 0, 1, V, p.ldx, xr));
    JSCC_LAUNCH_CHECK();
    x = xr;
  }
  // fused single-read path: the weight, row halves that fit the consumer registers, at least two
  // stages of a row half. Rows of whole 16-byte units on 16-byte boundaries take the plain form,
  // others the LOOSE one (its extra stage bytes hold the values before and after a row half's
  // whole blocks).
  if (stage == 0 && fs_part != nullptr && p.fs_clusters > 0) {
    const int64_t el = 16 / (int64_t)sizeof(T);
    const bool loose = !(vec_ok && V % el == 0);
    const int64_t split = loose ? (V + 1) / 2 : (V / 2 + el - 1) / el * el;
    const uint32_t stride = (uint32_t)align_up((size_t)split * sizeof(T) + (loose ? 128 : 0), 128);
    int stages = (int)((227u * 1024u - kFsHeader) / stride);
    if (stages > kFsMaxStages) stages = kFsMaxStages;
    int batch = stages / 2 < kFsMaxBatch ? stages / 2 : kFsMaxBatch;
    if (split <= kFsHalfMax && V - split <= kFsHalfMax && V - split > 0 && stages >= 2 && batch >= 1) {
      const size_t smem = kFsHeader + (size_t)stages * stride;
      auto launch = [&](auto kernel) {
        cudaError_t e = allow_smem(kernel);
        if (e != cudaSuccess) return e;
        JSCC_TIMED("sc_fused", st,
                   (kernel<<<(unsigned)(2 * p.fs_clusters), kFsThreads, smem, st>>>(
                       A, lda, row_idx, n_bins, V, split, x, proj, ld_proj, mode, floor_v, fout, ld_fout, fs_part, p.ldx,
                       stages, batch, stride)));
        return cudaSuccess;
      };
      if (mode == kRatioLog || mode == kRatioLogMinus || fout != nullptr)
        JSCC_CUDA_CHECK(loose ? launch(sc_fused_kernel<T, true, true>) : launch(sc_fused_kernel<T, false, true>));
      else
        JSCC_CUDA_CHECK(loose ? launch(sc_fused_kernel<T, true, false>) : launch(sc_fused_kernel<T, false, false>));
      JSCC_LAUNCH_CHECK();
      return launch_reduce_scatter(fs_part, p.ldx, (int)p.fs_clusters, 1, 1, rotinv, ld_rot, 0, V, has_scale, scale,
                                   weight, st);
    }
  }
  int64_t row_blocks = (n_bins + 255) / 256;
  if (row_blocks > (int64_t)sms * 8) row_blocks = (int64_t)sms * 8;
  if (stage == 2) {
    JSCC_TIMED("sc_load_ratio", st,
               (sc_load_ratio_kernel<<<(unsigned)row_blocks, 256, 0, st>>>(gin, ld_gin, n_bins, 0, 1, 1, ratio)));
    JSCC_LAUNCH_CHECK();
  } else {
    // forward: balanced contiguous split over warps, then fixed-order row finish
    const int64_t nvr = vec_ok ? (V + NV - 1) / NV : V;
    const int64_t U = n_bins * nvr;
    const int64_t G = p.fwd_warps;
    const int64_t L = (U + G - 1) / G;
    const size_t xbytes = (size_t)p.ldx * sizeof(float);
    const bool smem_x = vec_ok && xbytes <= 200 * 1024;
    const unsigned grid = (unsigned)(G / 32);
    auto launch = [&](auto kernel, size_t sh) {
      cudaError_t e = allow_smem(kernel);
      if (e != cudaSuccess) return e;
      JSCC_TIMED("sc_forward_split", st,
                 (kernel<<<grid, 1024, sh, st>>>(A, lda, row_idx, n_bins, V, x, nvr, L, p.fwd_maxp, fpart)));
      return cudaSuccess;
    };
    JSCC_CUDA_CHECK(smem_x   ? launch(sc_forward_split_kernel<T, true, true, 1024>, xbytes)
                    : vec_ok ? launch(sc_forward_split_kernel<T, true, false, 1024>, 0)
                             : launch(sc_forward_split_kernel<T, false, false, 1024>, 0));
    JSCC_LAUNCH_CHECK();
    if (stage == 1) {
      JSCC_TIMED("sc_finish_raw", st,
                 (sc_finish_raw_kernel<1><<<(unsigned)row_blocks, 256, 0, st>>>(fpart, n_bins, nvr, L, p.fwd_maxp, fout,
                                                                                ld_fout)));
      JSCC_LAUNCH_CHECK();
      return JSCC_OK;
    }
    JSCC_TIMED("sc_finish_ratio", st,
               (sc_finish_ratio_kernel<1><<<(unsigned)row_blocks, 256, 0, st>>>(
                   fpart, n_bins, nvr, L, p.fwd_maxp, row_idx, proj, ld_proj, mode, floor_v, ratio, fout, ld_fout)));
    JSCC_LAUNCH_CHECK();
  }
  const dim3 grid((unsigned)p.col_tiles, (unsigned)p.chunks);
  const int threads = kColTile / NV;
  JSCC_TIMED("sc_back_partial", st, {
    if (vec_ok)
      sc_back_partial_kernel<T, true><<<grid, threads, 0, st>>>(A, lda, row_idx, n_bins, V, ratio, p.rows_per_chunk,
                                                                part, p.ldx);
    else
      sc_back_partial_kernel<T, false><<<grid, threads, 0, st>>>(A, lda, row_idx, n_bins, V, ratio, p.rows_per_chunk,
                                                                 part, p.ldx);
  });
  JSCC_LAUNCH_CHECK();
  return launch_reduce_scatter(part, p.ldx, (int)p.chunks, 1, 1, rotinv, ld_rot, 0, V, has_scale, scale, weight, st);
}

// One view takes the kernels of several views (padded to two) where they are the faster ones.
// The weight: the fused kernel costs a row 8.7 + 0.2 V / 1000 ns, 13 + 0.3 V / 1000 with rows off
// 16-byte boundaries, mostly its exchange, however short the row is; the two passes cost 1.7 V / 1000
// (float32; 2.25 for aligned rows taken by their ids, out of order) or 1.3 V / 1000 ns (BF16) and three
// launches more: about 6 us there, and as much again in updates short enough (up to about 45 us) for the host
// to set their pace: two joint subsets of 3,280 BF16 rows of 5,440 voxels 237 us so, 217 us with the fused
// kernel, though that is 9 us slower by itself. Rows off 16-byte boundaries: 693 float32 rows of 1,441 voxels 17.5 against 11.8 us. 12,000 float32 rows of 1,440 voxels: 114 against 34 us; of 5,280 voxels 120
// against 108, by their ids 126 against 135; of 8,000 voxels 127 against 162; BF16 128 against 66 us of 5,280
// voxels, 131 against 93 of 8,000. The halves on their own: rows off 16-byte boundaries, which the one-view
// forward pass reads a value at a time.
template <typename T>
static bool one_view_by_views(const T* A, int64_t lda, bool ids, int64_t n_bins, int64_t V, int stage) {
  const bool vec_ok = (lda * (int64_t)sizeof(T)) % 16 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0;
  if (stage != 0) return !vec_ok;
  const double k = (double)V / 1000.0;
  const bool loose = !vec_ok || V % (16 / (int64_t)sizeof(T)) != 0;
  const double fused = loose ? 13.0 + 0.3 * k : 8.7 + 0.2 * k;
  const double views = (sizeof(T) == 2 ? 1.3 : ids && !loose ? 2.25 : 1.7) * k;
  const double gain = (double)n_bins * (fused - views);
  return gain > (loose || (double)n_bins * fused > 45000.0 ? 6000.0 : 12000.0);
}

// The weight or one of its halves (stage as in sc_one_view) for any number of views, in a
// caller workspace of at least plan_sc(...).ws_bytes.
template <typename T>
static int sc_run(const T* A, int64_t lda, const int64_t* row_idx, int64_t n_bins, int64_t V, const float* proj,
                  int64_t ld_proj, int n_rot, const float* img, const int64_t* rotmat, const int64_t* rotinv,
                  int64_t ld_rot, int mode, float floor_v, float scale, float* weight, const ScPlan& p, void* ws,
                  size_t ws_bytes, cudaStream_t st, int stage, float* fout, int64_t ld_fout, const float* gin,
                  int64_t ld_gin) {
  const int has_scale = scale != 1.0f;
  // (one view in less than its padding to two takes goes the way that the smallest workspace is made for)
  if (n_rot > 1 || (one_view_by_views<T>(A, lda, row_idx != nullptr, n_bins, V, stage) &&
                    plan_views(n_bins, V, 1, ws_bytes, sizeof(T), sv_aligned(A, lda)).bytes <= ws_bytes))
    return sc_views<T>(A, lda, row_idx, n_bins, V, proj, ld_proj, n_rot, img, rotmat, rotinv, ld_rot, mode,
                       floor_v, has_scale, scale, weight, ws, ws_bytes, st, stage, fout, ld_fout, gin, ld_gin);
  Carver cv(ws, ws_bytes);
  float* xr = cv.take<float>((size_t)p.ldx);
  float* ratio = cv.take<float>((size_t)n_bins);
  float* part = cv.take<float>((size_t)p.chunks * p.ldx);
  float* fpart = cv.take<float>((size_t)p.fwd_warps * p.fwd_maxp);
  JSCC_REQUIRE(cv.ok(), "SC projector: workspace carve overflow");
  float* fs_part = stage == 0 ? fused_partials(p, cv) : nullptr;
  return sc_one_view<T>(A, lda, row_idx, n_bins, V, proj, ld_proj, img, rotmat, rotinv, ld_rot, mode, floor_v,
                        has_scale, scale, weight, p, xr, ratio, part, fpart, fs_part, st, stage, fout, ld_fout, gin,
                        ld_gin);
}

size_t rows_weight_bytes(int64_t n_rows, int64_t V) { return jscc_sc_weight_workspace_bytes(n_rows, V, 1); }

int launch_rows_weight(const float* A, int64_t lda, int64_t n_rows, int64_t V, const float* one, const float* x,
                       const int64_t* rotinv, int64_t ld_rot, int mode, float floor_v, float scale, float* weight,
                       float* f_out, void* ws, size_t ws_bytes, cudaStream_t st) {
  return sc_run<float>(A, lda, nullptr, n_rows, V, one, 0, 1, x, nullptr, rotinv, ld_rot, mode, floor_v, scale, weight,
                       plan_sc(n_rows, V, 1), ws, ws_bytes, st, 0, f_out, 1, nullptr, 0);
}

template <typename T>
static int sc_sensitivity_typed(const T* A, int64_t lda, const int64_t* row_idx, int64_t n_bins, int64_t V,
                                int n_rot, const int64_t* rotinv, int64_t ld_rot, float* weight, int64_t col_tiles,
                                int64_t chunks, int64_t rows_per_chunk, int64_t ldp, float* sum, float* comp,
                                cudaStream_t st) {
  constexpr int NV = VecTraits<T>::kVec;
  const bool vec_ok = ((lda * (int64_t)sizeof(T)) % 16 == 0) && (reinterpret_cast<uintptr_t>(A) % 16 == 0);
  dim3 grid((unsigned)col_tiles, (unsigned)chunks);
  const int threads = kColTile / NV;
  JSCC_TIMED("sc_colsum_kahan", st, {
    if (vec_ok)
      sc_colsum_kahan_kernel<T, true><<<grid, threads, 0, st>>>(A, lda, row_idx, n_bins, V, rows_per_chunk, sum,
                                                                comp, ldp);
    else
      sc_colsum_kahan_kernel<T, false><<<grid, threads, 0, st>>>(A, lda, row_idx, n_bins, V, rows_per_chunk, sum,
                                                                 comp, ldp);
  });
  JSCC_LAUNCH_CHECK();
  const unsigned blocks = (unsigned)((V + 127) / 128);
  if (n_rot > 1) {
    JSCC_TIMED("sc_fold", st, (sc_fold_kernel<<<blocks, 128, 0, st>>>(sum, comp, ldp, (int)chunks, V)));
    JSCC_LAUNCH_CHECK();
  }
  JSCC_TIMED("sc_sensitivity", st, {
    if (n_rot > 1)
      sc_sensitivity_kernel<true><<<blocks, 128, 0, st>>>(sum, comp, ldp, (int)chunks, rotinv, ld_rot, n_rot, V,
                                                          weight);
    else
      sc_sensitivity_kernel<false><<<blocks, 128, 0, st>>>(sum, comp, ldp, (int)chunks, rotinv, ld_rot, n_rot, V,
                                                           weight);
  });
  JSCC_LAUNCH_CHECK();
  return JSCC_OK;
}

// ------------------------------------------------------------------ FP64 evaluation
// Reference-grade projector halves for gradient checks (sums in double; not a hot path).
// f[b, r] = sum_j A[rb, j] x[rot[j, r] - 1]: one warp per (b, r).
template <typename T>
__global__ void sc_project_f64_kernel(const T* __restrict__ A, int64_t lda, const int64_t* __restrict__ row_idx,
                                      int64_t n_bins, int64_t V, int n_rot, const double* __restrict__ x,
                                      const int64_t* __restrict__ rotmat, int64_t ld_rot, double* __restrict__ out,
                                      int64_t ld_out) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; w < n_bins * n_rot; w += warps) {
    const int64_t b = w / n_rot;
    const int r = (int)(w % n_rot);
    const T* row = A + (row_idx ? row_idx[b] : b) * lda;
    double acc = 0.0;
    for (int64_t j = lane; j < V; j += 32) {
      int64_t src = j;
      if (rotmat) {
        src = rotmat[j * ld_rot + r] - 1;
        if (src < 0 || src >= V) {
          atomicAdd(&g_bad_index_count, 1u);
          continue;
        }
      }
      acc += (double)load_elem(row, j) * x[src];
    }
    acc = warp_sum_d(acc);
    if (lane == 0) out[b * ld_out + r] = acc;
  }
}

// u[r][c] = sum_b A[rb, c] g[b, r]
template <typename T>
__global__ void sc_colsum_f64_kernel(const T* __restrict__ A, int64_t lda, const int64_t* __restrict__ row_idx,
                                     int64_t n_bins, int64_t V, int n_rot, const double* __restrict__ g, int64_t ld_g,
                                     double* __restrict__ u) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < V * n_rot;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(t / V);
    const int64_t c = t % V;
    double acc = 0.0;
    for (int64_t b = 0; b < n_bins; ++b) acc += (double)load_elem(A + (row_idx ? row_idx[b] : b) * lda, c) * g[b * ld_g + r];
    u[(int64_t)r * V + c] = acc;
  }
}

// weight[j] += scale * sum_r u[r][rotinv[j, r] - 1]
__global__ void sc_gather_f64_kernel(const double* __restrict__ u, int64_t V, int n_rot,
                                     const int64_t* __restrict__ rotinv, int64_t ld_rot, double scale,
                                     double* __restrict__ weight) {
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < V; j += (int64_t)gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int r = 0; r < n_rot; ++r) {
      int64_t src = j;
      if (rotinv) {
        src = rotinv[j * ld_rot + r] - 1;
        if (src < 0 || src >= V) {
          atomicAdd(&g_bad_index_count, 1u);
          continue;
        }
      }
      acc += u[(int64_t)r * V + src];
    }
    weight[j] += scale * acc;
  }
}

}  // namespace jscc

using namespace jscc;

extern "C" {

int jscc_sc_sensitivity(const void* A, int32_t a_dtype, int64_t lda, const int64_t* row_idx, int64_t n_bins,
                        int64_t n_vox, int32_t n_rot, const int64_t* rotmat_inv, int64_t ld_rot, float* weight,
                        void* workspace, size_t workspace_bytes, void* stream) {
  JSCC_REQUIRE(n_bins >= 0 && n_vox >= 0, "jscc_sc_sensitivity: negative size");
  JSCC_REQUIRE(n_rot >= 1, "jscc_sc_sensitivity: n_rot must be >= 1 (got %d)", n_rot);
  JSCC_REQUIRE(a_dtype == JSCC_DTYPE_F32 || a_dtype == JSCC_DTYPE_BF16, "jscc_sc_sensitivity: unsupported a_dtype %d",
               a_dtype);
  if (n_bins == 0 || n_vox == 0) return JSCC_OK;
  JSCC_REQUIRE(A && weight, "jscc_sc_sensitivity: null pointer argument");
  JSCC_REQUIRE(lda >= n_vox, "jscc_sc_sensitivity: lda (%lld) < n_vox (%lld)", (long long)lda, (long long)n_vox);
  JSCC_REQUIRE(rotmat_inv != nullptr || n_rot == 1, "jscc_sc_sensitivity: n_rot > 1 needs rotmat_inv");
  JSCC_REQUIRE(rotmat_inv == nullptr || ld_rot >= n_rot, "jscc_sc_sensitivity: ld_rot (%lld) < n_rot (%d)",
               (long long)ld_rot, n_rot);
  const ScPlan p = plan_sc(n_bins, n_vox, 1);
  JSCC_REQUIRE(workspace != nullptr && workspace_bytes >= p.ws_bytes,
               "jscc_sc_sensitivity: workspace too small (%zu < %zu bytes)", workspace_bytes, p.ws_bytes);
  // compensated sums: half as many row chunks as the back pass, so the sums and their carried
  // errors (2 x chunks x ldx floats) fit in the same workspace (>= (chunks + 1) x ldx floats)
  int64_t chunks = (p.chunks + 1) / 2;
  // and no more than the CTAs that run at once (64 registers: 1,024 threads an SM): no second wave
  const int64_t wave = num_sms() * (int64_t)(a_dtype == JSCC_DTYPE_F32 ? 4 : 8) / p.col_tiles;
  if (chunks > wave) chunks = wave;
  if (chunks < 1) chunks = 1;
  const int64_t rows_per_chunk = (n_bins + chunks - 1) / chunks;
  chunks = (n_bins + rows_per_chunk - 1) / rows_per_chunk;
  Carver cv(workspace, workspace_bytes);
  float* sum = cv.take<float>((size_t)chunks * p.ldx);
  float* comp = cv.take<float>((size_t)chunks * p.ldx);
  JSCC_REQUIRE(cv.ok(), "jscc_sc_sensitivity: workspace carve overflow");
  cudaStream_t st = as_stream(stream);
  if (a_dtype == JSCC_DTYPE_F32)
    return sc_sensitivity_typed<float>(static_cast<const float*>(A), lda, row_idx, n_bins, n_vox, n_rot, rotmat_inv,
                                       ld_rot, weight, p.col_tiles, chunks, rows_per_chunk, p.ldx, sum, comp, st);
  return sc_sensitivity_typed<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(A), lda, row_idx, n_bins, n_vox,
                                             n_rot, rotmat_inv, ld_rot, weight, p.col_tiles, chunks, rows_per_chunk,
                                             p.ldx, sum, comp, st);
}

size_t jscc_sc_weight_workspace_bytes(int64_t n_bins, int64_t n_vox, int32_t n_rot) {
  const ScPlan p = plan_sc(n_bins, n_vox, n_rot);
  const size_t one = p.ws_bytes + p.fs_bytes;
  if (n_rot < 1 || n_bins < 1 || n_vox < 1) return one;
  const size_t views = plan_views(n_bins, n_vox, n_rot, SIZE_MAX, 0, true).bytes;
  return views > one ? views : one;
}

int jscc_sc_weight(const void* A, int32_t a_dtype, int64_t lda, const int64_t* row_idx,
                   int64_t n_bins, int64_t n_vox,
                   const float* proj, int64_t ld_proj, int32_t n_rot, const float* img,
                   const int64_t* rotmat, const int64_t* rotmat_inv, int64_t ld_rot,
                   int32_t use_floor, float floor_v, float scale, float* weight, void* workspace,
                   size_t workspace_bytes, void* stream) {
  JSCC_REQUIRE(n_bins >= 0 && n_vox >= 0, "jscc_sc_weight: negative size");
  JSCC_REQUIRE(n_rot >= 1, "jscc_sc_weight: n_rot must be >= 1 (got %d)", n_rot);
  JSCC_REQUIRE(a_dtype == JSCC_DTYPE_F32 || a_dtype == JSCC_DTYPE_BF16,
               "jscc_sc_weight: unsupported a_dtype %d", a_dtype);
  if (n_bins == 0 || n_vox == 0) return JSCC_OK;  // nothing to add
  JSCC_REQUIRE(A && proj && img && weight, "jscc_sc_weight: null pointer argument");
  JSCC_REQUIRE(lda >= n_vox, "jscc_sc_weight: lda (%lld) < n_vox (%lld)", (long long)lda,
               (long long)n_vox);
  JSCC_REQUIRE(ld_proj >= n_rot, "jscc_sc_weight: ld_proj (%lld) < n_rot (%d)",
               (long long)ld_proj, n_rot);
  JSCC_REQUIRE((rotmat == nullptr && rotmat_inv == nullptr) || ld_rot >= n_rot,
               "jscc_sc_weight: ld_rot (%lld) < n_rot (%d)", (long long)ld_rot, n_rot);
  const ScPlan p = plan_sc(n_bins, n_vox, n_rot);
  JSCC_REQUIRE(workspace != nullptr && workspace_bytes >= p.ws_bytes,
               "jscc_sc_weight: workspace too small (%zu < %zu bytes)", workspace_bytes,
               p.ws_bytes);
  if (a_dtype == JSCC_DTYPE_F32)
    return sc_run<float>(static_cast<const float*>(A), lda, row_idx, n_bins, n_vox, proj, ld_proj, n_rot, img, rotmat,
                         rotmat_inv, ld_rot, use_floor ? kRatioFloor : kRatio, floor_v, scale, weight, p, workspace, workspace_bytes,
                         as_stream(stream), 0, nullptr, 0, nullptr, 0);
  return sc_run<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(A), lda, row_idx, n_bins, n_vox, proj, ld_proj, n_rot,
                               img, rotmat, rotmat_inv, ld_rot, use_floor ? kRatioFloor : kRatio, floor_v, scale, weight, p, workspace,
                               workspace_bytes, as_stream(stream), 0, nullptr, 0, nullptr, 0);
}

int jscc_sc_loglik(const void* A, int32_t a_dtype, int64_t lda, int64_t n_bins, int64_t n_vox, const float* proj,
                   int64_t ld_proj, int32_t n_rot, const float* img, const int64_t* rotmat, const int64_t* rotmat_inv,
                   int64_t ld_rot, float eps, float* f, int64_t ld_f, float* grad, void* workspace,
                   size_t workspace_bytes, void* stream) {
  const char* what = "jscc_sc_loglik";
  JSCC_REQUIRE(n_bins >= 0 && n_vox >= 0, "%s: negative size", what);
  JSCC_REQUIRE(n_rot >= 1, "%s: n_rot must be >= 1 (got %d)", what, n_rot);
  JSCC_REQUIRE(a_dtype == JSCC_DTYPE_F32 || a_dtype == JSCC_DTYPE_BF16, "%s: unsupported a_dtype %d", what, a_dtype);
  if (n_bins == 0 || n_vox == 0) return JSCC_OK;
  JSCC_REQUIRE(A && proj && img && f && grad, "%s: null pointer argument", what);
  JSCC_REQUIRE(lda >= n_vox, "%s: lda (%lld) < n_vox (%lld)", what, (long long)lda, (long long)n_vox);
  JSCC_REQUIRE(ld_proj >= n_rot && ld_f >= n_rot, "%s: ld_proj or ld_f < n_rot (%d)", what, n_rot);
  JSCC_REQUIRE((rotmat == nullptr) == (rotmat_inv == nullptr), "%s: give both rotation tables", what);
  JSCC_REQUIRE(rotmat ? ld_rot >= n_rot : n_rot == 1, "%s: ld_rot (%lld) < n_rot (%d)", what, (long long)ld_rot, n_rot);
  const ScPlan p = plan_sc(n_bins, n_vox, n_rot);
  JSCC_REQUIRE(workspace != nullptr && workspace_bytes >= p.ws_bytes, "%s: workspace too small (%zu < %zu bytes)", what,
               workspace_bytes, p.ws_bytes);
  if (a_dtype == JSCC_DTYPE_F32)
    return sc_run<float>(static_cast<const float*>(A), lda, nullptr, n_bins, n_vox, proj, ld_proj, n_rot, img, rotmat,
                         rotmat_inv, ld_rot, kRatioLogMinus, eps, 1.0f, grad, p, workspace, workspace_bytes,
                         as_stream(stream), 0, f, ld_f, nullptr, 0);
  return sc_run<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(A), lda, nullptr, n_bins, n_vox, proj, ld_proj, n_rot,
                               img, rotmat, rotmat_inv, ld_rot, kRatioLogMinus, eps, 1.0f, grad, p, workspace,
                               workspace_bytes, as_stream(stream), 0, f, ld_f, nullptr, 0);
}

// The two halves of jscc_sc_weight on their own (the differentiable projector's forward and
// backward): out[b * ld_out + r] = A[rb] . rot_r(img), and weight += scale * sum_r
// rotinv_r(A^T g[:, r]). Same workspace as jscc_sc_weight for the same sizes.
static int sc_stage_entry(const char* what, int stage, const void* A, int32_t a_dtype, int64_t lda,
                          const int64_t* row_idx, int64_t n_bins, int64_t n_vox, int32_t n_rot, const float* img,
                          const int64_t* rotmat, const int64_t* rotmat_inv, int64_t ld_rot, float* out,
                          int64_t ld_out, const float* g, int64_t ld_g, float scale, float* weight, void* workspace,
                          size_t workspace_bytes, void* stream) {
  JSCC_REQUIRE(n_bins >= 0 && n_vox >= 0, "%s: negative size", what);
  JSCC_REQUIRE(n_rot >= 1, "%s: n_rot must be >= 1 (got %d)", what, n_rot);
  JSCC_REQUIRE(a_dtype == JSCC_DTYPE_F32 || a_dtype == JSCC_DTYPE_BF16, "%s: unsupported a_dtype %d", what, a_dtype);
  if (n_bins == 0 || n_vox == 0) return JSCC_OK;
  JSCC_REQUIRE(A, "%s: null matrix", what);
  JSCC_REQUIRE(lda >= n_vox, "%s: lda (%lld) < n_vox (%lld)", what, (long long)lda, (long long)n_vox);
  if (stage == 1) {
    JSCC_REQUIRE(img && out && ld_out >= n_rot, "%s: null image/output or ld_out < n_rot", what);
    JSCC_REQUIRE(rotmat != nullptr || n_rot == 1, "%s: n_rot > 1 needs rotmat", what);
  } else {
    JSCC_REQUIRE(g && weight && ld_g >= n_rot, "%s: null input/weight or ld_g < n_rot", what);
    JSCC_REQUIRE(rotmat_inv != nullptr || n_rot == 1, "%s: n_rot > 1 needs rotmat_inv", what);
  }
  JSCC_REQUIRE(ld_rot >= n_rot || (rotmat == nullptr && rotmat_inv == nullptr), "%s: ld_rot < n_rot", what);
  const ScPlan p = plan_sc(n_bins, n_vox, n_rot);
  JSCC_REQUIRE(workspace != nullptr && workspace_bytes >= p.ws_bytes, "%s: workspace too small (%zu < %zu bytes)",
               what, workspace_bytes, p.ws_bytes);
  if (a_dtype == JSCC_DTYPE_F32)
    return sc_run<float>(static_cast<const float*>(A), lda, row_idx, n_bins, n_vox, nullptr, 0, n_rot, img, rotmat,
                         rotmat_inv, ld_rot, 0, 0.f, scale, weight, p, workspace, workspace_bytes, as_stream(stream),
                         stage, out, ld_out, g, ld_g);
  return sc_run<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(A), lda, row_idx, n_bins, n_vox, nullptr, 0, n_rot,
                               img, rotmat, rotmat_inv, ld_rot, 0, 0.f, scale, weight, p, workspace, workspace_bytes,
                               as_stream(stream), stage, out, ld_out, g, ld_g);
}

int jscc_sc_project(const void* A, int32_t a_dtype, int64_t lda, const int64_t* row_idx, int64_t n_bins,
                    int64_t n_vox, int32_t n_rot, const float* img, const int64_t* rotmat, int64_t ld_rot, float* out,
                    int64_t ld_out, void* workspace, size_t workspace_bytes, void* stream) {
  return sc_stage_entry("jscc_sc_project", 1, A, a_dtype, lda, row_idx, n_bins, n_vox, n_rot, img, rotmat, nullptr,
                        ld_rot, out, ld_out, nullptr, 0, 1.f, nullptr, workspace, workspace_bytes, stream);
}

int jscc_sc_backproject(const void* A, int32_t a_dtype, int64_t lda, const int64_t* row_idx, int64_t n_bins,
                        int64_t n_vox, int32_t n_rot, const float* g, int64_t ld_g, const int64_t* rotmat_inv,
                        int64_t ld_rot, float scale, float* weight, void* workspace, size_t workspace_bytes,
                        void* stream) {
  return sc_stage_entry("jscc_sc_backproject", 2, A, a_dtype, lda, row_idx, n_bins, n_vox, n_rot, nullptr, nullptr,
                        rotmat_inv, ld_rot, nullptr, 0, g, ld_g, scale, weight, workspace, workspace_bytes, stream);
}

size_t jscc_sc_f64_workspace_bytes(int64_t n_vox, int32_t n_rot) {
  return align_up((size_t)(n_vox > 0 ? n_vox : 1) * (size_t)(n_rot > 0 ? n_rot : 1) * sizeof(double), 256) + 256;
}

int jscc_sc_project_f64(const void* A, int32_t a_dtype, int64_t lda, const int64_t* row_idx, int64_t n_bins,
                        int64_t n_vox, int32_t n_rot, const double* img, const int64_t* rotmat, int64_t ld_rot,
                        double* out, int64_t ld_out, void* stream) {
  JSCC_REQUIRE(n_bins >= 0 && n_vox >= 0 && n_rot >= 1, "jscc_sc_project_f64: bad sizes");
  JSCC_REQUIRE(a_dtype == JSCC_DTYPE_F32 || a_dtype == JSCC_DTYPE_BF16, "jscc_sc_project_f64: bad a_dtype");
  JSCC_REQUIRE(rotmat != nullptr || n_rot == 1, "jscc_sc_project_f64: n_rot > 1 needs rotmat");
  if (n_bins == 0 || n_vox == 0) return JSCC_OK;
  JSCC_REQUIRE(A && img && out && lda >= n_vox && ld_out >= n_rot, "jscc_sc_project_f64: bad argument");
  cudaStream_t st = as_stream(stream);
  int64_t blocks = (n_bins * n_rot + 7) / 8;  // 8 warps per block
  if (blocks > (int64_t)num_sms() * 16) blocks = (int64_t)num_sms() * 16;
  if (a_dtype == JSCC_DTYPE_F32)
    JSCC_TIMED("sc_project_f64", st,
               (sc_project_f64_kernel<float><<<(unsigned)blocks, 256, 0, st>>>(
                   static_cast<const float*>(A), lda, row_idx, n_bins, n_vox, n_rot, img, rotmat, ld_rot, out, ld_out)));
  else
    JSCC_TIMED("sc_project_f64", st,
               (sc_project_f64_kernel<__nv_bfloat16><<<(unsigned)blocks, 256, 0, st>>>(
                   static_cast<const __nv_bfloat16*>(A), lda, row_idx, n_bins, n_vox, n_rot, img, rotmat, ld_rot, out,
                   ld_out)));
  JSCC_LAUNCH_CHECK();
  return JSCC_OK;
}

int jscc_sc_backproject_f64(const void* A, int32_t a_dtype, int64_t lda, const int64_t* row_idx, int64_t n_bins,
                            int64_t n_vox, int32_t n_rot, const double* g, int64_t ld_g, const int64_t* rotmat_inv,
                            int64_t ld_rot, double scale, double* weight, void* workspace, size_t workspace_bytes,
                            void* stream) {
  JSCC_REQUIRE(n_bins >= 0 && n_vox >= 0 && n_rot >= 1, "jscc_sc_backproject_f64: bad sizes");
  JSCC_REQUIRE(a_dtype == JSCC_DTYPE_F32 || a_dtype == JSCC_DTYPE_BF16, "jscc_sc_backproject_f64: bad a_dtype");
  JSCC_REQUIRE(rotmat_inv != nullptr || n_rot == 1, "jscc_sc_backproject_f64: n_rot > 1 needs rotmat_inv");
  if (n_bins == 0 || n_vox == 0) return JSCC_OK;
  JSCC_REQUIRE(A && g && weight && lda >= n_vox && ld_g >= n_rot, "jscc_sc_backproject_f64: bad argument");
  JSCC_REQUIRE(workspace && workspace_bytes >= jscc_sc_f64_workspace_bytes(n_vox, n_rot),
               "jscc_sc_backproject_f64: workspace too small");
  Carver cv(workspace, workspace_bytes);
  double* u = cv.take<double>((size_t)n_vox * n_rot);
  JSCC_REQUIRE(cv.ok(), "jscc_sc_backproject_f64: workspace carve overflow");
  cudaStream_t st = as_stream(stream);
  int64_t blocks = (n_vox * n_rot + 255) / 256;
  if (blocks > (int64_t)num_sms() * 16) blocks = (int64_t)num_sms() * 16;
  if (a_dtype == JSCC_DTYPE_F32)
    JSCC_TIMED("sc_colsum_f64", st,
               (sc_colsum_f64_kernel<float><<<(unsigned)blocks, 256, 0, st>>>(
                   static_cast<const float*>(A), lda, row_idx, n_bins, n_vox, n_rot, g, ld_g, u)));
  else
    JSCC_TIMED("sc_colsum_f64", st,
               (sc_colsum_f64_kernel<__nv_bfloat16><<<(unsigned)blocks, 256, 0, st>>>(
                   static_cast<const __nv_bfloat16*>(A), lda, row_idx, n_bins, n_vox, n_rot, g, ld_g, u)));
  JSCC_LAUNCH_CHECK();
  blocks = (n_vox + 255) / 256;
  if (blocks > (int64_t)num_sms() * 16) blocks = (int64_t)num_sms() * 16;
  JSCC_TIMED("sc_gather_f64", st,
             (sc_gather_f64_kernel<<<(unsigned)blocks, 256, 0, st>>>(u, n_vox, n_rot, rotmat_inv, ld_rot, scale,
                                                                     weight)));
  JSCC_LAUNCH_CHECK();
  return JSCC_OK;
}

int jscc_take_bad_index_count(unsigned int* out) {
  unsigned int h = 0, zero = 0;
  JSCC_CUDA_CHECK(cudaMemcpyFromSymbol(&h, g_bad_index_count, sizeof(h)));
  JSCC_CUDA_CHECK(cudaMemcpyToSymbol(g_bad_index_count, &zero, sizeof(zero)));
  h += jscc::take_prior_bad_index_count();
  if (out) *out = h;
  return JSCC_OK;
}

}  // extern "C"

// ============================================================================
// No-allocation variant of jscc_sc_weight.
//
// Some callers cannot hand this library a workspace: a host framework that owns all
// device memory through its own pool and forbids allocations from plugins, a language
// runtime driving the library through a bare FFI without any device allocator, or a
// latency-critical loop that must not pay cudaMalloc's implicit synchronisation. For
// them the scratch of the SC weight lives in one fixed file-scope device array,
// allocated when the library's device code is loaded on a GPU and held until the
// process exits.
//
// The array's name is only a host-side stand-in in host code: its device address is
// obtained once per device with cudaGetSymbolAddress (the first call on each device
// does this, with that device current) and that address is what the kernels get.
// Every call shares the one array: calls that may overlap on the GPU (different
// streams, or concurrent host threads) race on it and must be serialised by the
// caller. No byte of the scratch needs to start at zero: each call writes every
// scratch element before it reads it.
// ============================================================================

namespace jscc {

static __device__ __align__(256) unsigned char g_sc_noalloc_scratch[JSCC_SC_NOALLOC_SCRATCH_BYTES];

static std::mutex g_noalloc_mu;
static void* g_noalloc_ptr[64] = {nullptr};

static int noalloc_scratch_address(void** out) {
  int dev = -1;
  JSCC_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    set_error("jscc_sc_weight_noalloc: device ordinal %d outside the supported range", dev);
    return JSCC_ERR_INVALID;
  }
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (g_noalloc_ptr[dev] == nullptr) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_sc_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) {
      set_error("jscc_sc_weight_noalloc: cudaGetSymbolAddress of the scratch array failed on device %d: %s",
                dev, cudaGetErrorString(e));
      return JSCC_ERR_CUDA;
    }
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return JSCC_OK;
}

}  // namespace jscc

extern "C" int jscc_sc_weight_noalloc(const void* A, int32_t a_dtype, int64_t lda, const int64_t* row_idx,
                                      int64_t n_bins, int64_t n_vox, const float* proj, int64_t ld_proj,
                                      int32_t n_rot, const float* img, const int64_t* rotmat,
                                      const int64_t* rotmat_inv, int64_t ld_rot, int32_t use_floor,
                                      float floor_v, float scale, float* weight, void* stream) {
  JSCC_REQUIRE(n_bins >= 0 && n_vox >= 0, "jscc_sc_weight_noalloc: negative size");
  JSCC_REQUIRE(n_rot >= 1, "jscc_sc_weight_noalloc: n_rot must be >= 1 (got %d)", n_rot);
  JSCC_REQUIRE(a_dtype == JSCC_DTYPE_F32 || a_dtype == JSCC_DTYPE_BF16,
               "jscc_sc_weight_noalloc: unsupported a_dtype %d", a_dtype);
  if (n_bins == 0 || n_vox == 0) return JSCC_OK;
  JSCC_REQUIRE(A && proj && img && weight, "jscc_sc_weight_noalloc: null pointer argument");
  JSCC_REQUIRE(lda >= n_vox, "jscc_sc_weight_noalloc: lda (%lld) < n_vox (%lld)", (long long)lda,
               (long long)n_vox);
  JSCC_REQUIRE(ld_proj >= n_rot, "jscc_sc_weight_noalloc: ld_proj (%lld) < n_rot (%d)",
               (long long)ld_proj, n_rot);
  JSCC_REQUIRE((rotmat == nullptr && rotmat_inv == nullptr) || ld_rot >= n_rot,
               "jscc_sc_weight_noalloc: ld_rot (%lld) < n_rot (%d)", (long long)ld_rot, n_rot);
  const ScPlan p = plan_sc(n_bins, n_vox, n_rot);
  JSCC_REQUIRE(p.ws_bytes <= (size_t)JSCC_SC_NOALLOC_SCRATCH_BYTES,
               "jscc_sc_weight_noalloc: this problem (%lld bins x %lld voxels, %d rotations) needs %zu "
               "bytes of scratch but the fixed scratch array holds %zu bytes; call jscc_sc_weight with a "
               "caller-provided workspace instead",
               (long long)n_bins, (long long)n_vox, n_rot, p.ws_bytes,
               (size_t)JSCC_SC_NOALLOC_SCRATCH_BYTES);
  void* scratch = nullptr;
  const int rc = noalloc_scratch_address(&scratch);
  if (rc != JSCC_OK) return rc;
  const size_t bytes = (size_t)JSCC_SC_NOALLOC_SCRATCH_BYTES;
  if (a_dtype == JSCC_DTYPE_F32)
    return sc_run<float>(static_cast<const float*>(A), lda, row_idx, n_bins, n_vox, proj, ld_proj, n_rot, img, rotmat,
                         rotmat_inv, ld_rot, use_floor ? kRatioFloor : kRatio, floor_v, scale, weight, p, scratch, bytes, as_stream(stream), 0,
                         nullptr, 0, nullptr, 0);
  return sc_run<__nv_bfloat16>(static_cast<const __nv_bfloat16*>(A), lda, row_idx, n_bins, n_vox, proj, ld_proj, n_rot,
                               img, rotmat, rotmat_inv, ld_rot, use_floor ? kRatioFloor : kRatio, floor_v, scale, weight, p, scratch, bytes,
                               as_stream(stream), 0, nullptr, 0, nullptr, 0);
}
