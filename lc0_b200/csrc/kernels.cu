// Memory-bound and small kernels of the evaluation path.
#include "kernels.cuh"

namespace b200 {

thread_local bool t_dependent_launch = false;

// ------------------------------------------------------------------------------------------------
// Plane expansion (reference: BlasComputation::EncodePlanes, backends/blas/network_blas.cc:973-981;
// GPU twin expandPlanes_kernel_NCHW, backends/cuda/common_kernels.cu:484-521).
// ------------------------------------------------------------------------------------------------
template <typename T>
__global__ void expand_planes_kernel(const uint64_t* __restrict__ masks, const float* __restrict__ values,
                                     long long total_planes, T* __restrict__ out) {
  // One thread writes 8 consecutive squares (one 16-byte store for 16-bit types).
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long plane = idx >> 3;
  if (plane >= total_planes) return;
  const int part = int(idx & 7);
  const uint64_t m = masks[plane] >> (part * 8);
  const float v = values[plane];
  __align__(16) T vals[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) vals[i] = from_f<T>(((m >> i) & 1) ? v : 0.f);
  T* dst = out + plane * 64 + part * 8;
  if (sizeof(T) == 2) {
    *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(vals);
  } else {
    reinterpret_cast<uint4*>(dst)[0] = reinterpret_cast<const uint4*>(vals)[0];
    reinterpret_cast<uint4*>(dst)[1] = reinterpret_cast<const uint4*>(vals)[1];
  }
}

template <typename T>
cudaError_t launch_expand_planes(const uint64_t* masks, const float* values, int n, T* out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const long long planes = (long long)n * 112;
  const long long threads = planes * 8;
  expand_planes_kernel<T><<<ceil_div(threads, 256), 256, 0, s>>>(masks, values, planes, out);
  return cudaGetLastError();
}

// Token-major expansion with positional-encoding concat (reference: network_blas.cc:631-652; GPU twin
// preprocess_for_attention_body_kernel, backends/cuda/common_kernels.cu:1203-1244).
template <typename T> struct __align__(16) Vec8 { T v[8]; };

// Clears what later launches add to or leave out: a position's row statistics (two doubles per token) and its q, d, m.
__device__ __forceinline__ void clear_position(int n, double2* stats, float* qdm) {
  if (stats && threadIdx.x < 64) stats[(long long)n * 64 + threadIdx.x] = make_double2(0.0, 0.0);
  if (qdm && threadIdx.x < 3) qdm[(long long)n * 3 + threadIdx.x] = 0.f;
}

template <typename T>
__global__ void expand_tokens_kernel(const uint64_t* __restrict__ masks, const float* __restrict__ values,
                                     const float* __restrict__ pe_static, const T* __restrict__ pe_dense,
                                     int pe_ch, int cin, T* __restrict__ out, double2* stats, float* qdm) {
  __shared__ uint64_t sm[112];
  __shared__ float sv[112];
  const int n = blockIdx.x;
  grid_dependency_wait();
  grid_launch_dependents();
  clear_position(n, stats, qdm);
  for (int i = threadIdx.x; i < 112; i += blockDim.x) {
    sm[i] = masks[(long long)n * 112 + i];
    sv[i] = values[(long long)n * 112 + i];
  }
  __syncthreads();
  T* o = out + (long long)n * 64 * cin;
  const int total = 64 * cin;
  for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
    const int sq = idx / cin, c = idx - sq * cin;
    float v = 0.f;
    if (c < 112) {
      v = ((sm[c] >> sq) & 1) ? sv[c] : 0.f;
    } else if (c < 112 + pe_ch) {
      const int j = c - 112;
      v = pe_dense ? to_f(pe_dense[((long long)n * 64 + sq) * pe_ch + j]) : pe_static[sq * pe_ch + j];
    }
    o[idx] = from_f<T>(v);
  }
}

// Same for row widths and encoding widths that are multiples of 8: a thread writes 8 channels (16 bytes for
// 16-bit storage) at a time, dense positional encodings are copied as 16-byte pieces.
template <typename T>
__global__ void __launch_bounds__(256)
expand_tokens_vec_kernel(const uint64_t* __restrict__ masks, const float* __restrict__ values,
                         const float* __restrict__ pe_static, const T* __restrict__ pe_dense, int pe_ch, int cin,
                         T* __restrict__ out, double2* stats, float* qdm) {
  __shared__ uint64_t sm[112];
  __shared__ float sv[112];
  const int n = blockIdx.x;
  grid_dependency_wait();
  grid_launch_dependents();
  if (blockIdx.y == 0) clear_position(n, stats, qdm);
  for (int i = threadIdx.x; i < 112; i += blockDim.x) {
    sm[i] = masks[(long long)n * 112 + i];
    sv[i] = values[(long long)n * 112 + i];
  }
  __syncthreads();
  T* o = out + (long long)n * 64 * cin;
  const int vec_per_row = cin >> 3, rows = 64 / gridDim.y, sq0 = blockIdx.y * rows;
  for (int idx = threadIdx.x; idx < rows * vec_per_row; idx += blockDim.x) {
    const int r0 = idx / vec_per_row, sq = sq0 + r0, c = (idx - r0 * vec_per_row) << 3;
    Vec8<T> r;
    if (c < 112) {
#pragma unroll
      for (int i = 0; i < 8; ++i) r.v[i] = from_f<T>(((sm[c + i] >> sq) & 1) ? sv[c + i] : 0.f);
    } else if (c < 112 + pe_ch) {
      const int j = c - 112;
      if (pe_dense) {
        r = *reinterpret_cast<const Vec8<T>*>(pe_dense + ((long long)n * 64 + sq) * pe_ch + j);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) r.v[i] = from_f<T>(pe_static[sq * pe_ch + j + i]);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) r.v[i] = from_f<T>(0.f);
    }
    *reinterpret_cast<Vec8<T>*>(o + (long long)sq * cin + c) = r;
  }
}

template <typename T>
cudaError_t launch_expand_tokens(const uint64_t* masks, const float* values, int n, const float* pe_static,
                                 const T* pe_dense, int pe_ch, int cin, T* out, double* stats, float* qdm, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  double2* st2 = reinterpret_cast<double2*>(stats);
  const bool aligned = (reinterpret_cast<uintptr_t>(out) & 15) == 0 && (reinterpret_cast<uintptr_t>(pe_dense) & 15) == 0;
  if ((cin & 7) == 0 && (pe_ch & 7) == 0 && aligned)
    // Few positions: eight (four) CTAs to a position, 8 (16) squares each; one CTA took 16 us for one position's 80 KB.
    return launch_dependent(expand_tokens_vec_kernel<T>, dim3(n, n <= 148 ? 8 : n <= 592 ? 4 : 1), dim3(256), 0, s, masks, values,
                            pe_static, pe_dense, pe_ch, cin, out, st2, qdm);
  return launch_dependent(expand_tokens_kernel<T>, dim3(n), dim3(256), 0, s, masks, values, pe_static, pe_dense, pe_ch, cin, out,
                          st2, qdm);
}

// First 12 planes, square-major (reference: network_blas.cc:613-621).
template <typename T>
__global__ void expand_pre12_kernel(const uint64_t* __restrict__ masks, const float* __restrict__ values, int n,
                                    T* __restrict__ out) {
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= (long long)n * 768) return;
  const int s = int(idx / 768), r = int(idx - (long long)s * 768);
  const int sq = r / 12, j = r - sq * 12;
  const uint64_t m = masks[(long long)s * 112 + j];
  out[idx] = from_f<T>(((m >> sq) & 1) ? values[(long long)s * 112 + j] : 0.f);
}

template <typename T>
cudaError_t launch_expand_pre12(const uint64_t* masks, const float* values, int n, T* out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  expand_pre12_kernel<T><<<ceil_div((long long)n * 768, 256), 256, 0, s>>>(masks, values, n, out);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------
// LayerNorm with skip connection (reference: LayerNorm2DWithSkipConnection, backends/blas/encoder.h:29-78;
// GPU twin layer_norm_kernel, backends/cuda/common_kernels.cu:932-1081).  One CTA per row, the row is held
// in registers (8 contiguous elements per thread per step), two-pass mean / variance, warp-shuffle sums.
// ------------------------------------------------------------------------------------------------
template <int kThreads>
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (l < kThreads / 32) ? red[l] : 0.f;
  t = warp_sum(t);
  __syncthreads();
  return t;
}


template <typename T, int kThreads, int kSteps>
__global__ void __launch_bounds__(kThreads)
layer_norm_kernel(T* __restrict__ out, const T* __restrict__ x, const T* __restrict__ skip,
                  const float* __restrict__ gamma, const float* __restrict__ beta,
                  const float* __restrict__ gate_mult, const float* __restrict__ gate_add, int C,
                  float alpha, float eps) {
  __shared__ float red[32];
  grid_dependency_wait();
  grid_launch_dependents();
  const long long row = blockIdx.x;
  const T* xr = x + row * C;
  const T* sr = skip ? skip + row * C : nullptr;
  float v[kSteps][8];
  float sum = 0.f;
#pragma unroll
  for (int s = 0; s < kSteps; ++s) {
    const int c = (s * kThreads + threadIdx.x) * 8;
    if (c < C) {
      Vec8<T> a = *reinterpret_cast<const Vec8<T>*>(xr + c);
      Vec8<T> b;
      if (sr) b = *reinterpret_cast<const Vec8<T>*>(sr + c);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float t = to_f(a.v[i]) * alpha;
        if (sr) t += to_f(b.v[i]);
        v[s][i] = t;
        sum += t;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[s][i] = 0.f;
    }
  }
  const float mean = block_sum<kThreads>(sum, red) / C;
  float var = 0.f;
#pragma unroll
  for (int s = 0; s < kSteps; ++s) {
    const int c = (s * kThreads + threadIdx.x) * 8;
    if (c < C) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float d = v[s][i] - mean;
        var += d * d;
      }
    }
  }
  var = block_sum<kThreads>(var, red) / C;
  const float den = 1.0f / sqrtf(var + eps);
  const int sq = int(row & 63);
#pragma unroll
  for (int s = 0; s < kSteps; ++s) {
    const int c = (s * kThreads + threadIdx.x) * 8;
    if (c < C) {
      const float4 g0 = *reinterpret_cast<const float4*>(gamma + c), g1 = *reinterpret_cast<const float4*>(gamma + c + 4);
      const float4 b0 = *reinterpret_cast<const float4*>(beta + c), b1 = *reinterpret_cast<const float4*>(beta + c + 4);
      const float gg[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
      const float bb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
      Vec8<T> o;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float t = bb[i] + gg[i] * (v[s][i] - mean) * den;
        if (gate_mult) t = t * gate_mult[(long long)sq * C + c + i] + gate_add[(long long)sq * C + c + i];
        o.v[i] = from_f<T>(t);
      }
      *reinterpret_cast<Vec8<T>*>(out + row * C + c) = o;
    }
  }
}

// Warp-per-row variant for C <= 2048: a lane holds kChunks 16-byte pieces of the row (piece index
// lane + 32 * i), the reductions are pure shuffles and a 128-thread CTA normalises four rows.
template <typename T, int kChunks>
__global__ void __launch_bounds__(128)
layer_norm_warp_kernel(T* __restrict__ out, const T* __restrict__ x, const T* __restrict__ skip,
                       const float* __restrict__ gamma, const float* __restrict__ beta,
                       const float* __restrict__ gate_mult, const float* __restrict__ gate_add, int rows, int C,
                       float alpha, float eps) {
  grid_dependency_wait();
  grid_launch_dependents();
  const long long row = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int lane = threadIdx.x & 31;
  const T* xr = x + row * C;
  const T* sr = skip ? skip + row * C : nullptr;
  Vec8<T> a[kChunks], b[kChunks];
#pragma unroll
  for (int i = 0; i < kChunks; ++i) {
    const int c = (lane + 32 * i) * 8;
    if (c < C) {
      a[i] = *reinterpret_cast<const Vec8<T>*>(xr + c);
      if (sr) b[i] = *reinterpret_cast<const Vec8<T>*>(sr + c);
    }
  }
  float v[kChunks][8];
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < kChunks; ++i) {
    const int c = (lane + 32 * i) * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float t = 0.f;
      if (c < C) {
        t = to_f(a[i].v[j]) * alpha;
        if (sr) t += to_f(b[i].v[j]);
      }
      v[i][j] = t;
      sum += t;
    }
  }
  const float mean = warp_sum(sum) / C;
  float var = 0.f;
#pragma unroll
  for (int i = 0; i < kChunks; ++i) {
    const int c = (lane + 32 * i) * 8;
    if (c < C) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float d = v[i][j] - mean;
        var += d * d;
      }
    }
  }
  var = warp_sum(var) / C;
  const float den = 1.0f / sqrtf(var + eps);
  const int sq = int(row & 63);
#pragma unroll
  for (int i = 0; i < kChunks; ++i) {
    const int c = (lane + 32 * i) * 8;
    if (c < C) {
      const float4 g0 = *reinterpret_cast<const float4*>(gamma + c), g1 = *reinterpret_cast<const float4*>(gamma + c + 4);
      const float4 b0 = *reinterpret_cast<const float4*>(beta + c), b1 = *reinterpret_cast<const float4*>(beta + c + 4);
      const float gg[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
      const float bb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
      float gm[8] = {1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f}, ga[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (gate_mult) {
        const float4 m0 = *reinterpret_cast<const float4*>(gate_mult + (long long)sq * C + c);
        const float4 m1 = *reinterpret_cast<const float4*>(gate_mult + (long long)sq * C + c + 4);
        const float4 a0 = *reinterpret_cast<const float4*>(gate_add + (long long)sq * C + c);
        const float4 a1 = *reinterpret_cast<const float4*>(gate_add + (long long)sq * C + c + 4);
        gm[0] = m0.x; gm[1] = m0.y; gm[2] = m0.z; gm[3] = m0.w; gm[4] = m1.x; gm[5] = m1.y; gm[6] = m1.z; gm[7] = m1.w;
        ga[0] = a0.x; ga[1] = a0.y; ga[2] = a0.z; ga[3] = a0.w; ga[4] = a1.x; ga[5] = a1.y; ga[6] = a1.z; ga[7] = a1.w;
      }
      Vec8<T> o;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float t = bb[j] + gg[j] * (v[i][j] - mean) * den;
        t = t * gm[j] + ga[j];
        o.v[j] = from_f<T>(t);
      }
      *reinterpret_cast<Vec8<T>*>(out + row * C + c) = o;
    }
  }
}

template <typename T>
cudaError_t launch_layer_norm(T* out, const T* x, const T* skip, const float* gamma, const float* beta,
                              const float* gate_mult, const float* gate_add, int rows, int C, float alpha,
                              float eps, cudaStream_t s) {
  if (rows <= 0) return cudaSuccess;
  if (C % 8 != 0 || C > 8192) return cudaErrorInvalidValue;
#define LNW_LAUNCH(CH)                                                                                      \
  le = launch_dependent(layer_norm_warp_kernel<T, CH>, dim3(ceil_div(rows, 4)), dim3(128), 0, s, out, x, skip, \
                        gamma, beta, gate_mult, gate_add, rows, C, alpha, eps)
#define LN_LAUNCH(TH, ST)                                                                                     \
  le = launch_dependent(layer_norm_kernel<T, TH, ST>, dim3(rows), dim3(TH), 0, s, out, x, skip, gamma, beta, \
                        gate_mult, gate_add, C, alpha, eps)
  cudaError_t le = cudaSuccess;
  if (C <= 256) LNW_LAUNCH(1);
  else if (C <= 512) LNW_LAUNCH(2);
  else if (C <= 1024) LNW_LAUNCH(4);
  else if (C <= 2048) LNW_LAUNCH(8);
  else if (C <= 4096) LN_LAUNCH(256, 2);  // few, wide rows (smolgen): 256 threads, several 16-byte pieces each
  else LN_LAUNCH(256, 4);
#undef LN_LAUNCH
#undef LNW_LAUNCH
  return le;
}

// Input gating x * mult + add (reference: network_blas.cc:669-682; gates re-laid out [64][C] at load).
// Memory-bound.  The vector form gates eight channels of one square in kGateBoards positions per thread, so that the gates
// (fp32, [64][C]) are read once for all of them; the scalar form takes widths that are no multiple of eight.
constexpr int kGateBoards = 4;
template <typename T>
__global__ void gate_kernel(T* __restrict__ x, const float* __restrict__ mult, const float* __restrict__ add,
                            long long total, int C) {
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const long long row = idx / C;
  const int c = int(idx - row * C);
  const long long g = (row & 63) * C + c;
  x[idx] = from_f<T>(to_f(x[idx]) * mult[g] + add[g]);
}
template <typename T>
__global__ void __launch_bounds__(256)
gate_vec_kernel(T* __restrict__ x, const float* __restrict__ mult, const float* __restrict__ add, int boards, int C) {
  const int piece = blockIdx.x * 256 + threadIdx.x;  // piece of eight channels of a board
  if (piece >= 8 * C) return;
  const long long board = 64LL * C;
  float m[8], a[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    m[i] = __ldg(mult + piece * 8 + i);
    a[i] = __ldg(add + piece * 8 + i);
  }
  grid_dependency_wait();
  grid_launch_dependents();
  T* p = x + (long long)piece * 8;
  const int b0 = blockIdx.y * kGateBoards, b1 = b0 + kGateBoards < boards ? b0 + kGateBoards : boards;
  Vec8<T> v[kGateBoards];
#pragma unroll
  for (int i = 0; i < kGateBoards; ++i)
    if (b0 + i < b1) v[i] = *reinterpret_cast<const Vec8<T>*>(p + (b0 + i) * board);
#pragma unroll
  for (int i = 0; i < kGateBoards; ++i) {
    if (b0 + i >= b1) break;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[i].v[j] = from_f<T>(to_f(v[i].v[j]) * m[j] + a[j]);
    *reinterpret_cast<Vec8<T>*>(p + (b0 + i) * board) = v[i];
  }
}

template <typename T>
cudaError_t launch_gate(T* x, const float* gate_mult, const float* gate_add, int rows, int C, cudaStream_t s) {
  const long long total = (long long)rows * C;
  if (total <= 0) return cudaSuccess;
  if ((C & 7) == 0 && (rows & 63) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0)
    return launch_dependent(gate_vec_kernel<T>, dim3(ceil_div(8LL * C, 256), ceil_div(rows / 64, kGateBoards)), dim3(256), 0, s,
                            x, gate_mult, gate_add, rows / 64, C);
  gate_kernel<T><<<ceil_div(total, 256), 256, 0, s>>>(x, gate_mult, gate_add, total, C);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------
// 64-token attention, one CTA per (sample, head), fp32 arithmetic in shared memory
// (reference: network_blas.cc:352-439; GPU twins are two batched cuBLAS calls + softmax_opt_64_kernel).
// ------------------------------------------------------------------------------------------------
// Bound by the FMA pipe and shared-memory reads.  A thread owns four query rows (16 threads to a row) and four keys
// 16 apart, later four rows and two channels 16 apart, and reads every operand as 16-byte pieces along the contraction; rows of
// depth + 4 (68 for the probabilities and the transposed V) floats put eight neighbouring rows on different banks.
// The fp32 mode uses expf for parity with the CPU oracle.
template <typename T>
__global__ void __launch_bounds__(256)
attention_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, long long ld,
                 const T* __restrict__ bias, T* __restrict__ out, long long ldo, int heads, int depth,
                 float scale) {
  constexpr bool kFast = sizeof(T) == 2;
  constexpr int kLdP = 68;
  extern __shared__ __align__(16) float smem[];
  const int d4 = (depth + 3) >> 2, dp = d4 * 4 + 4;
  float* sq = smem;              // [64][dp]
  float* sk = sq + 64 * dp;      // [64][dp]
  float* sp = smem;              // [64][kLdP], over Q and K once they have been read
  float* sv = smem + (2 * dp > kLdP ? 2 * dp : kLdP) * 64;  // [depth][kLdP], transposed
  grid_dependency_wait();
  grid_launch_dependents();
  const int tid = threadIdx.x;
  const int n = blockIdx.x / heads, h = blockIdx.x - n * heads;
  const long long base = (long long)n * 64 * ld + (long long)h * depth;
  // Four numbers in one load where every row's pieces are whole and aligned (uniform over the launch).  With the bias asked for
  // ahead of the product it belongs to, 512 heads of depth 32 in fp32 take 16.9 us instead of 19.4.
  constexpr size_t kPiece = 4 * sizeof(T);
  const bool pieces = !(depth & 3) && !(ld & 3) && !((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) |
                                                      reinterpret_cast<uintptr_t>(v)) & (kPiece - 1));
  struct __align__(4 * sizeof(T)) Four { T v[4]; };
  const int tx = tid & 15, row0 = (tid >> 4) * 4;
  T bv[4][4];  // the scores' bias, in flight under the loads and the first product
  if (bias) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) bv[i][j] = bias[(((long long)n * heads + h) * 64 + row0 + i) * 64 + tx + 16 * j];
  }
  if (pieces) {
#pragma unroll 2
    for (int i = tid; i < 64 * d4; i += 256) {
      const int r = i / d4, c = (i - r * d4) * 4;
      const Four a = *reinterpret_cast<const Four*>(q + base + r * ld + c), b = *reinterpret_cast<const Four*>(k + base + r * ld + c);
      *reinterpret_cast<float4*>(sq + r * dp + c) = make_float4(to_f(a.v[0]), to_f(a.v[1]), to_f(a.v[2]), to_f(a.v[3]));
      *reinterpret_cast<float4*>(sk + r * dp + c) = make_float4(to_f(b.v[0]), to_f(b.v[1]), to_f(b.v[2]), to_f(b.v[3]));
    }
#pragma unroll 2
    for (int i = tid; i < 64 * d4; i += 256) {
      const int r = i & 63, c = (i >> 6) * 4;
      const Four a = *reinterpret_cast<const Four*>(v + base + r * ld + c);
#pragma unroll
      for (int e = 0; e < 4; ++e) sv[(c + e) * kLdP + r] = to_f(a.v[e]);
    }
  } else {
    for (int i = tid; i < 64 * d4; i += 256) {
      const int r = i / d4, c = (i - r * d4) * 4;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const bool in = c + e < depth;
        sq[r * dp + c + e] = in ? to_f(q[base + r * ld + c + e]) : 0.f;
        sk[r * dp + c + e] = in ? to_f(k[base + r * ld + c + e]) : 0.f;
      }
    }
    for (int i = tid; i < 64 * d4; i += 256) {
      const int r = i & 63, c = (i >> 6) * 4;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (c + e < depth) sv[(c + e) * kLdP + r] = to_f(v[base + r * ld + c + e]);
    }
  }
  __syncthreads();
  float sc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) sc[i][j] = 0.f;
#pragma unroll 2
  for (int c = 0; c < d4 * 4; c += 4) {
    float4 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(sq + (row0 + i) * dp + c);
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(sk + (tx + 16 * j) * dp + c);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        sc[i][j] = fmaf(a[i].w, b[j].w, fmaf(a[i].z, b[j].z, fmaf(a[i].y, b[j].y, fmaf(a[i].x, b[j].x, sc[i][j]))));
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float mx = -3.0e38f, sum = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      sc[i][j] *= scale;
      if (bias) sc[i][j] += to_f(bv[i][j]);
      mx = fmaxf(mx, sc[i][j]);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      sc[i][j] = kFast ? __expf(sc[i][j] - mx) : expf(sc[i][j] - mx);
      sum += sc[i][j];
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
#pragma unroll
    for (int j = 0; j < 4; ++j) sc[i][j] = sc[i][j] / sum;
  }
  __syncthreads();  // Q and K have been read
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) sp[(row0 + i) * kLdP + tx + 16 * j] = sc[i][j];
  __syncthreads();
  for (int c0 = tx; c0 < depth; c0 += 32) {
    const int c1 = c0 + 16 < depth ? c0 + 16 : c0;
    float o[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i][0] = o[i][1] = 0.f;
#pragma unroll 4
    for (int j = 0; j < 64; j += 4) {
      const float4 v0 = *reinterpret_cast<const float4*>(sv + c0 * kLdP + j);
      const float4 v1 = *reinterpret_cast<const float4*>(sv + c1 * kLdP + j);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(sp + (row0 + i) * kLdP + j);
        o[i][0] = fmaf(a.w, v0.w, fmaf(a.z, v0.z, fmaf(a.y, v0.y, fmaf(a.x, v0.x, o[i][0]))));
        o[i][1] = fmaf(a.w, v1.w, fmaf(a.z, v1.z, fmaf(a.y, v1.y, fmaf(a.x, v1.x, o[i][1]))));
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      T* dst = out + ((long long)n * 64 + row0 + i) * ldo + (long long)h * depth;
      dst[c0] = from_f<T>(o[i][0]);
      if (c0 + 16 < depth) dst[c0 + 16] = from_f<T>(o[i][1]);
    }
  }
}

template <typename T>
cudaError_t launch_attention(const T* q, const T* k, const T* v, long long ld, const T* bias, T* out,
                             long long ldo, int n, int heads, int depth, float scale, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  constexpr int kMaxDepth = 128;
  if (depth > kMaxDepth) return cudaErrorInvalidValue;
  auto bytes = [](int d) {
    const int dp = ceil_div(d, 4) * 4 + 4;
    return (size_t)(64 * (2 * dp > 68 ? 2 * dp : 68) + d * 68) * sizeof(float);
  };
  const size_t smem = bytes(depth);
  if (smem > 48 * 1024) {
    cudaError_t e = raise_smem_limit<&attention_kernel<T>>((int)bytes(kMaxDepth));
    if (e != cudaSuccess) return e;
  }
  return launch_dependent(attention_kernel<T>, dim3(n * heads), dim3(256), smem, s, q, k, v, ld, bias, out, ldo, heads, depth,
                          scale);
}

// ------------------------------------------------------------------------------------------------
// Attention policy tail: promotion offsets + gather of the 1858 move logits
// (reference: network_blas.cc:873-914; GPU twins promotion_logits_kernel and policyMap_kernel,
// backends/cuda/common_kernels.cu:1116-1201 and :703-734).  One CTA per sample.
// src_slot[j] is the slot (0..4287) of the 64*64 + 8*24 raw vector that feeds policy index j.
// ------------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
policy_attn_gather_kernel(const float* __restrict__ logits, const T* __restrict__ kp,
                          const float* __restrict__ w4, int dm, const short* __restrict__ src_slot,
                          float* __restrict__ policy) {
  __shared__ float off[4][8];
  const int n = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  grid_dependency_wait();
  grid_launch_dependents();
  // 32 dot products (4 promotion rows x 8 files), 4 per warp with one row of w4 between them; eight steps of loads in flight
  {
    const int i = warp >> 1, j0 = (warp & 1) * 4;
    const T* key = kp + ((long long)n * 64 + 56 + j0) * dm;
    float a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int c = lane; c < dm; c += 32) {
      const float w = w4[i * dm + c];
#pragma unroll
      for (int j = 0; j < 4; ++j) a[j] = fmaf(to_f(key[(long long)j * dm + c]), w, a[j]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      a[j] = warp_sum(a[j]);
      if (lane == 0) off[i][j0 + j] = a[j];
    }
  }
  __syncthreads();
  const float* lg = logits + (long long)n * 4096;
  for (int j = threadIdx.x; j < 1858; j += 256) {
    const int slot = src_slot[j];
    float v;
    if (slot < 4096) {
      v = lg[slot];
    } else {
      const int r = slot - 4096;  // 24*k + 3*file + i
      const int kf = r / 24, rem = r - kf * 24, jf = rem / 3, i = rem - jf * 3;
      v = lg[(48 + kf) * 64 + 56 + jf] + off[i][jf] + off[3][jf];
    }
    policy[(long long)n * 1858 + j] = v;
  }
}

template <typename T>
cudaError_t launch_policy_attn_gather(const float* logits, const T* kp, const float* w4, int dm,
                                      const short* src_slot, int n, float* policy, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  return launch_dependent(policy_attn_gather_kernel<T>, dim3(n), dim3(256), 0, s, logits, kp, w4, dm, src_slot, policy);
}

template <typename T>
__global__ void policy_gather_kernel(const T* __restrict__ raw, long long ld, const short* __restrict__ src,
                                     float* __restrict__ policy) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int n = blockIdx.x;
  for (int j = threadIdx.x; j < 1858; j += blockDim.x)
    policy[(long long)n * 1858 + j] = to_f(raw[(long long)n * ld + src[j]]);
}

template <typename T>
cudaError_t launch_policy_gather(const T* raw, long long ld, const short* src_slot, int n, float* policy,
                                 cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  return launch_dependent(policy_gather_kernel<T>, dim3(n), dim3(256), 0, s, raw, ld, src_slot, policy);
}

// ------------------------------------------------------------------------------------------------
// Last layer of the value / moves-left heads (reference: network_blas.cc:747-772 and :797-802;
// the reference CUDA backend leaves the WDL softmax to the host, network_cuda.cc:991-1014).
// ------------------------------------------------------------------------------------------------
template <typename T>
__global__ void head_final_kernel(const T* __restrict__ h, int k, const float* __restrict__ w,
                                  const float* __restrict__ b, int mode, int n, float* __restrict__ qdm) {
  grid_dependency_wait();
  grid_launch_dependents();
  const int sample = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (sample >= n) return;
  const T* hr = h + (long long)sample * k;
  const int outs = mode == 0 ? 3 : 1;
  float o[3] = {0.f, 0.f, 0.f};
  for (int i = 0; i < outs; ++i) {
    float a = 0.f;
    for (int c = lane; c < k; c += 32) a = fmaf(to_f(hr[c]), w[i * k + c], a);
    o[i] = warp_sum(a) + b[i];
  }
  if (lane != 0) return;
  float* dst = qdm + (long long)sample * 3;
  if (mode == 0) {
    const float mx = fmaxf(o[0], fmaxf(o[1], o[2]));
    const float e0 = expf(o[0] - mx), e1 = expf(o[1] - mx), e2 = expf(o[2] - mx);
    const float s = e0 + e1 + e2;
    dst[0] = e0 / s - e2 / s;
    dst[1] = e1 / s;
  } else if (mode == 1) {
    dst[0] = tanhf(o[0]);
    dst[1] = 0.f;
  } else {
    dst[2] = o[0] > 0.f ? o[0] : 0.f;
  }
}

template <typename T>
cudaError_t launch_head_final(const T* h, int k, const float* w, const float* b, int mode, int n, float* qdm,
                              cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  return launch_dependent(head_final_kernel<T>, dim3(ceil_div(n, 4)), dim3(128), 0, s, h, k, w, b, mode, n, qdm);
}

// ------------------------------------------------------------------------------------------------
// Residual tower on NHWC activations [n*64][C].
// Squeeze-excitation block, one CTA per sample (reference: ApplySEUnit, backends/blas/se_unit.cc:31-91;
// GPU twin SE_Layer_NHWC, backends/cuda/fp16_kernels.cu:55-136).
template <typename T, bool kFast>
__global__ void __launch_bounds__(256)
se_kernel(const T* __restrict__ x, const float* __restrict__ conv_bias, const T* __restrict__ skip,
          const float* __restrict__ w1, const float* __restrict__ b1, const float* __restrict__ w2,
          const float* __restrict__ b2, T* __restrict__ y, int C, int se_k, int act) {
  extern __shared__ float sm[];
  float* pool = sm;           // [C]
  float* hid = pool + C;      // [se_k]
  float* z = hid + se_k;      // [2C]
  const int n = blockIdx.x;
  const T* xs = x + (long long)n * 64 * C;
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    float a = 0.f;
    for (int sq = 0; sq < 64; ++sq) a += to_f(xs[sq * C + c]);
    pool[c] = a / 64.0f + conv_bias[c];
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int o = warp; o < se_k; o += nw) {
    float a = 0.f;
    for (int c = lane; c < C; c += 32) a = fmaf(pool[c], w1[o * C + c], a);
    a = warp_sum(a);
    if (lane == 0) hid[o] = activate<false>(a + b1[o], act);
  }
  __syncthreads();
  for (int o = threadIdx.x; o < 2 * C; o += blockDim.x) {
    float a = b2[o];
    for (int c = 0; c < se_k; ++c) a = fmaf(hid[c], w2[o * se_k + c], a);
    z[o] = a;
  }
  __syncthreads();
  const T* ss = skip + (long long)n * 64 * C;
  T* ys = y + (long long)n * 64 * C;
  for (int i = threadIdx.x; i < 64 * C; i += blockDim.x) {
    const int c = i % C;
    const float g = 1.0f / (1.0f + expf(-z[c]));
    const float v = g * to_f(xs[i]) + to_f(ss[i]) + z[C + c] + g * conv_bias[c];
    ys[i] = from_f<T>(activate<kFast>(v, act));
  }
}

// Vectorised variant (C % 8 == 0): 16-byte loads, the sample's 64 x C tile is kept in shared memory between the
// pooling pass and the scaling pass, partial sums over square groups are reduced through shared memory.
template <typename T, bool kFast>
__global__ void __launch_bounds__(256)
se_vec_kernel(const T* __restrict__ x, const float* __restrict__ conv_bias, const T* __restrict__ skip,
              const float* __restrict__ w1, const float* __restrict__ b1, const float* __restrict__ w2,
              const float* __restrict__ b2, T* __restrict__ y, int C, int se_k, int act) {
  extern __shared__ __align__(16) uint8_t se_sm[];
  T* xs = reinterpret_cast<T*>(se_sm);                          // [64][C]
  float* partial = reinterpret_cast<float*>(xs + 64 * C);       // [nsqg][C]  (nsqg * C == 2048)
  float* pool = partial + 2048;                                 // [C]
  float* hid = pool + C;                                        // [se_k]
  float* z = hid + se_k;                                        // [2C]
  const int n = blockIdx.x, tid = threadIdx.x;
  const int cgs = C / 8;            // channel groups of 8
  const int nsqg = 256 / cgs;       // square groups working in parallel
  const int cg = tid % cgs, sqg = tid / cgs;
  const T* xg = x + (long long)n * 64 * C;
  if (sqg < nsqg) {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int sq = sqg; sq < 64; sq += nsqg) {
      const Vec8<T> v = *reinterpret_cast<const Vec8<T>*>(xg + sq * C + cg * 8);
      *reinterpret_cast<Vec8<T>*>(xs + sq * C + cg * 8) = v;
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += to_f(v.v[j]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) partial[sqg * C + cg * 8 + j] = acc[j];
  }
  __syncthreads();
  for (int c = tid; c < C; c += 256) {
    float a = 0.f;
    for (int g = 0; g < nsqg; ++g) a += partial[g * C + c];
    pool[c] = a / 64.0f + conv_bias[c];
  }
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31;
  for (int o = warp; o < se_k; o += 8) {
    float a = 0.f;
    for (int c = lane; c < C; c += 32) a = fmaf(pool[c], w1[o * C + c], a);
    a = warp_sum(a);
    if (lane == 0) hid[o] = activate<false>(a + b1[o], act);
  }
  __syncthreads();
  for (int o = tid; o < 2 * C; o += 256) {
    float a = b2[o];
    for (int c = 0; c < se_k; ++c) a = fmaf(hid[c], w2[o * se_k + c], a);
    // first C outputs become the sigmoid gate, the rest the shift (with the gate times the conv bias folded in)
    z[o] = a;
  }
  __syncthreads();
  for (int c = tid; c < C; c += 256) {
    const float g = 1.0f / (1.0f + expf(-z[c]));
    z[C + c] += g * conv_bias[c];
    z[c] = g;
  }
  __syncthreads();
  const T* sg = skip + (long long)n * 64 * C;
  T* yg = y + (long long)n * 64 * C;
  if (sqg < nsqg) {
    float g[8], sh[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      g[j] = z[cg * 8 + j];
      sh[j] = z[C + cg * 8 + j];
    }
    for (int sq = sqg; sq < 64; sq += nsqg) {
      const Vec8<T> v = *reinterpret_cast<const Vec8<T>*>(xs + sq * C + cg * 8);
      const Vec8<T> r = *reinterpret_cast<const Vec8<T>*>(sg + sq * C + cg * 8);
      Vec8<T> o;
#pragma unroll
      for (int j = 0; j < 8; ++j) o.v[j] = from_f<T>(activate<kFast>(g[j] * to_f(v.v[j]) + to_f(r.v[j]) + sh[j], act));
      *reinterpret_cast<Vec8<T>*>(yg + sq * C + cg * 8) = o;
    }
  }
}

// The same with everything that the chain reads in shared memory: w2 comes as [se_k / 4][2C][4] (a row per thread makes every
// load of a warp touch 32 lines), the matrices are asked for ahead of the wait for the convolution, the tile and (`stage_skip`:
// where it fits) the skip input in one piece behind it.  A block's work is a chain of short sums, bound by its round trips to L2:
// with 128 channels, 32 hidden units, fp32 and 64 boards it adds 6.3 us behind the convolution, se_vec_kernel 12.5 us; the
// 10 x 128 network takes, us, se_vec_kernel / this one: 1 board 499 / 422, 64 602 / 537, 512 2691 / 2595.
__device__ __forceinline__ void copy_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
template <typename T, bool kFast>
__global__ void __launch_bounds__(256)
se_staged_kernel(const T* __restrict__ x, const float* __restrict__ conv_bias, const T* __restrict__ skip,
                 const float* __restrict__ w1, const float* __restrict__ b1, const float* __restrict__ w2q,
                 const float* __restrict__ b2, T* __restrict__ y, int C, int se_k, int act, int stage_skip) {
  extern __shared__ __align__(16) uint8_t se_sm[];
  float* w1s = reinterpret_cast<float*>(se_sm);                 // [se_k][C]
  float* w2s = w1s + se_k * C;                                  // [se_k / 4][2C][4]
  T* xs = reinterpret_cast<T*>(w2s + 2 * se_k * C);             // [64][C]
  T* ss = xs + 64 * C;                                          // [64][C] if stage_skip
  float* partial = reinterpret_cast<float*>(stage_skip ? ss + 64 * C : ss);  // [nsqg][C]  (nsqg * C == 2048)
  float* z = partial + 2048;                                    // [2C]
  float* pool = z + 2 * C;                                      // [C]
  float* hid = pool + C;                                        // [se_k]
  float* cb = hid + se_k;                                       // conv_bias [C], b1 [se_k], b2 [2C]
  float* b1s = cb + C;
  float* b2s = b1s + se_k;
  const int n = blockIdx.x, tid = threadIdx.x;
  const int cgs = C / 8, nsqg = 256 / cgs, cg = tid % cgs, sqg = tid / cgs;
  for (int i = tid; i < se_k * C / 4; i += 256) copy_async16(w1s + 4 * i, w1 + 4 * i);
  for (int i = tid; i < se_k * C / 2; i += 256) copy_async16(w2s + 4 * i, w2q + 4 * i);
  for (int i = tid; i < C; i += 256) cb[i] = conv_bias[i];
  for (int i = tid; i < se_k; i += 256) b1s[i] = b1[i];
  for (int i = tid; i < 2 * C; i += 256) b2s[i] = b2[i];
  grid_dependency_wait();
  grid_launch_dependents();
  const T* xg = x + (long long)n * 64 * C;
  const T* sg = skip + (long long)n * 64 * C;
  constexpr int kPiece = 16 / sizeof(T);
  for (int i = tid; i < 64 * C / kPiece; i += 256) copy_async16(xs + kPiece * i, xg + kPiece * i);
  asm volatile("cp.async.commit_group;" ::: "memory");
  if (stage_skip)
    for (int i = tid; i < 64 * C / kPiece; i += 256) copy_async16(ss + kPiece * i, sg + kPiece * i);
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncthreads();
  {
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int sq = sqg; sq < 64; sq += nsqg) {
      const Vec8<T> v = *reinterpret_cast<const Vec8<T>*>(xs + sq * C + cg * 8);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += to_f(v.v[j]);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) partial[sqg * C + cg * 8 + j] = acc[j];
  }
  __syncthreads();
  for (int c = tid; c < C; c += 256) {
    float a = 0.f;
    for (int g = 0; g < nsqg; ++g) a += partial[g * C + c];
    pool[c] = a / 64.0f + cb[c];
  }
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31;
  for (int o = warp; o < se_k; o += 8) {
    float a = 0.f;
    for (int c = lane; c < C; c += 32) a = fmaf(pool[c], w1s[o * C + c], a);
    a = warp_sum(a);
    if (lane == 0) hid[o] = activate<false>(a + b1s[o], act);
  }
  __syncthreads();
  for (int o = tid; o < 2 * C; o += 256) {
    float a = b2s[o];
    for (int c = 0; c < se_k / 4; ++c) {
      const float4 w = *reinterpret_cast<const float4*>(w2s + ((long long)c * 2 * C + o) * 4);
      a = fmaf(hid[4 * c], w.x, a);
      a = fmaf(hid[4 * c + 1], w.y, a);
      a = fmaf(hid[4 * c + 2], w.z, a);
      a = fmaf(hid[4 * c + 3], w.w, a);
    }
    z[o] = a;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  for (int c = tid; c < C; c += 256) {  // the gate, and the shift with the gate times the convolution's bias folded in
    const float g = 1.0f / (1.0f + expf(-z[c]));
    z[C + c] += g * cb[c];
    z[c] = g;
  }
  __syncthreads();
  T* yg = y + (long long)n * 64 * C;
  const T* sr = stage_skip ? ss : sg;
  float g[8], sh[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    g[j] = z[cg * 8 + j];
    sh[j] = z[C + cg * 8 + j];
  }
#pragma unroll 4
  for (int sq = sqg; sq < 64; sq += nsqg) {
    const Vec8<T> v = *reinterpret_cast<const Vec8<T>*>(xs + sq * C + cg * 8);
    const Vec8<T> r = *reinterpret_cast<const Vec8<T>*>(sr + sq * C + cg * 8);
    Vec8<T> o;
#pragma unroll
    for (int j = 0; j < 8; ++j) o.v[j] = from_f<T>(activate<kFast>(g[j] * to_f(v.v[j]) + to_f(r.v[j]) + sh[j], act));
    *reinterpret_cast<Vec8<T>*>(yg + sq * C + cg * 8) = o;
  }
}

template <typename T>
cudaError_t launch_se(const T* x, const float* conv_bias, const T* skip, const float* w1, const float* b1,
                      const float* w2, const float* w2q, const float* b2, T* y, int C, int se_k, int n, int act, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  constexpr size_t kMaxSmem = 200 * 1024;
  const int cgs = C / 8;
  // w2q and se_k % 4: every piece of the copies is 16 aligned bytes (C % 8 == 0 here)
  if (w2q && se_k % 4 == 0 && C % 8 == 0 && cgs >= 1 && cgs <= 256 && 256 % cgs == 0) {
    const size_t tile = (size_t)64 * C * sizeof(T), rest = (size_t)(3 * se_k * C + 2048 + 6 * C + 2 * se_k) * sizeof(float);
    const int stage_skip = rest + 2 * tile <= kMaxSmem;
    const size_t smem = rest + (stage_skip ? 2 : 1) * tile;
    // Of 512 channels an SM holds one block of this kernel and two of se_vec_kernel: where the skip input is not staged either, more
    // than a round of them (148 SMs) is behind.  16 bits, 12 hidden units, four blocks of 512 filters, us, se_vec_kernel / this one: 64
    // boards 346 / 332, 148 490 / 481, 200 726 / 759, 512 1490 / 1555, 1000 2740 / 2881.  256 channels stay ahead (fp32, 32
    // units, 1 to 2 % of the network at every size).
    if (smem <= kMaxSmem && (stage_skip || C <= 256 || n <= 148)) {
      const auto kernel = se_staged_kernel<T, (sizeof(T) == 2)>;
      if (smem > 48 * 1024) {
        cudaError_t e = raise_smem_limit<&se_staged_kernel<T, (sizeof(T) == 2)>>((int)kMaxSmem);
        if (e != cudaSuccess) return e;
      }
      return launch_dependent(kernel, dim3(n), dim3(256), smem, s, x, conv_bias, skip, w1, b1, w2q, b2, y, C, se_k, act,
                              stage_skip);
    }
  }
  if (C % 8 == 0 && cgs <= 256 && 256 % cgs == 0) {
    const size_t smem = (size_t)64 * C * sizeof(T) + (size_t)(2048 + 3 * C + se_k) * sizeof(float);
    if (smem <= kMaxSmem) {
      if (smem > 48 * 1024) {
        cudaError_t e = raise_smem_limit<&se_vec_kernel<T, (sizeof(T) == 2)>>((int)kMaxSmem);
        if (e != cudaSuccess) return e;
      }
      se_vec_kernel<T, (sizeof(T) == 2)><<<n, 256, smem, s>>>(x, conv_bias, skip, w1, b1, w2, b2, y, C, se_k, act);
      return cudaGetLastError();
    }
  }
  const size_t smem = (size_t)(3 * C + se_k) * sizeof(float);
  se_kernel<T, (sizeof(T) == 2)><<<n, 256, smem, s>>>(x, conv_bias, skip, w1, b1, w2, b2, y, C, se_k, act);
  return cudaGetLastError();
}

template <typename T, bool kFast>
__global__ void bias_skip_act_kernel(const T* __restrict__ x, const float* __restrict__ bias,
                                     const T* __restrict__ skip, T* __restrict__ y, int C, long long total,
                                     int act) {
  const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (idx >= total) return;
  float v = to_f(x[idx]) + bias[idx % C];
  if (skip) v += to_f(skip[idx]);
  y[idx] = from_f<T>(activate<kFast>(v, act));
}

template <typename T>
cudaError_t launch_bias_skip_act(const T* x, const float* bias, const T* skip, T* y, int C, int rows, int act,
                                 cudaStream_t s) {
  const long long total = (long long)rows * C;
  if (total <= 0) return cudaSuccess;
  bias_skip_act_kernel<T, (sizeof(T) == 2)><<<ceil_div(total, 256), 256, 0, s>>>(x, bias, skip, y, C, total, act);
  return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------
// Legal-move softmax (reference: NetworkAsBackendComputation::SoftmaxPolicy, neural/wrapper.cc:135-156).
// One warp per position.  The exponential is the reference's FastExp restated with explicitly unfused
// multiplies and adds, and the total is accumulated sequentially in move order, so that the result is
// bit-identical to the host formula applied to the same logits.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ float fast_exp_ref(float x) {
  const float a = __fmul_rn(1.442695040f, x);
  int e;
  if (a < 0.f) {
    if (a < -126.f) return 0.f;
    e = (int)__fadd_rn(a, -1.0f);
  } else {
    e = (int)a;
  }
  float out = __fadd_rn(a, -(float)e);
  out = __fadd_rn(1.0f, __fmul_rn(out, __fadd_rn(0.6602339f, __fmul_rn(0.33976606f, out))));
  return __int_as_float(__float_as_int(out) + (int)((unsigned)e << 23));
}

__global__ void __launch_bounds__(128)
legal_softmax_kernel(const float* __restrict__ policy, const unsigned short* __restrict__ move_ids,
                     const int* __restrict__ n_moves, int n, float inv_t, float* __restrict__ probs) {
  __shared__ float vals[4][kLegalStride];
  grid_dependency_wait();
  grid_launch_dependents();
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sample = blockIdx.x * 4 + w;
  if (sample >= n) return;
  int cnt = n_moves[sample];
  cnt = cnt < 0 ? 0 : (cnt > kLegalStride ? kLegalStride : cnt);
  const unsigned short* ids = move_ids + (long long)sample * kLegalStride;
  const float* pol = policy + (long long)sample * 1858;
  float mx = -INFINITY;
  for (int i = lane; i < cnt; i += 32) {
    const int id = ids[i] < 1858 ? ids[i] : 1857;
    const float v = pol[id];
    vals[w][i] = v;
    mx = fmaxf(mx, v);
  }
  mx = warp_max(mx);
  __syncwarp();
  for (int i = lane; i < cnt; i += 32) vals[w][i] = fast_exp_ref(__fmul_rn(__fadd_rn(vals[w][i], -mx), inv_t));
  __syncwarp();
  float total = 0.f;
  if (lane == 0)
    for (int i = 0; i < cnt; ++i) total = __fadd_rn(total, vals[w][i]);
  total = __shfl_sync(0xffffffffu, total, 0);
  const float scale = total > 0.f ? __fdiv_rn(1.0f, total) : 1.0f;
  float* out = probs + (long long)sample * kLegalStride;
  for (int i = lane; i < cnt; i += 32) out[i] = __fmul_rn(vals[w][i], scale);
}

cudaError_t launch_legal_softmax(const float* policy, const unsigned short* move_ids, const int* n_moves, int n,
                                 float inv_temperature, float* probs, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  return launch_dependent(legal_softmax_kernel, dim3(ceil_div(n, 4)), dim3(128), 0, s, policy, move_ids, n_moves, n,
                          inv_temperature, probs);
}

#define INSTANTIATE(T)                                                                                        \
  template cudaError_t launch_expand_planes<T>(const uint64_t*, const float*, int, T*, cudaStream_t);         \
  template cudaError_t launch_expand_tokens<T>(const uint64_t*, const float*, int, const float*, const T*,    \
                                               int, int, T*, double*, float*, cudaStream_t);                  \
  template cudaError_t launch_expand_pre12<T>(const uint64_t*, const float*, int, T*, cudaStream_t);          \
  template cudaError_t launch_layer_norm<T>(T*, const T*, const T*, const float*, const float*, const float*, \
                                            const float*, int, int, float, float, cudaStream_t);              \
  template cudaError_t launch_gate<T>(T*, const float*, const float*, int, int, cudaStream_t);                \
  template cudaError_t launch_attention<T>(const T*, const T*, const T*, long long, const T*, T*, long long,  \
                                           int, int, int, float, cudaStream_t);                               \
  template cudaError_t launch_policy_attn_gather<T>(const float*, const T*, const float*, int, const short*,  \
                                                    int, float*, cudaStream_t);                               \
  template cudaError_t launch_policy_gather<T>(const T*, long long, const short*, int, float*, cudaStream_t); \
  template cudaError_t launch_head_final<T>(const T*, int, const float*, const float*, int, int, float*,      \
                                            cudaStream_t);                                                    \
  template cudaError_t launch_se<T>(const T*, const float*, const T*, const float*, const float*, const float*, \
                                    const float*, const float*, T*, int, int, int, int, cudaStream_t);        \
  template cudaError_t launch_bias_skip_act<T>(const T*, const float*, const T*, T*, int, int, int,           \
                                               cudaStream_t);

INSTANTIATE(float)
INSTANTIATE(__half)
INSTANTIATE(__nv_bfloat16)

}  // namespace b200
