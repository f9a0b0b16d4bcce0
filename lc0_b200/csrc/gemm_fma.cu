// FMA matrix kernel: the fp32 verification mode's products with fewer than 32 rows per position, its layers of shapes that
// gemm_f32.cu does not take (and all of it with the tensor cores switched off), and 16-bit products of shapes that the TMA path
// does not take (leading dimensions that are no multiple of 8, stacked products, products in fp32 storage).
// (reference: FullyConnectedLayer::Forward1D, backends/blas/fully_connected_layer.cc:50-106;
// WinogradConvolution3::Forward, backends/blas/winograd_convolution3.cc:47-57, same sums through F(2x2,3x3) transforms)
//
// Bound by the FMA pipe (74 TFLOP/s at 1.965 GHz), for few rows by the latency of the K loop.  Operands are staged
// K-contiguous as they lie in memory (16-byte cp.async, four floats of one row) in three stages; rows are padded by four floats
// so that eight rows of a quarter warp fall on different banks.  A thread owns TM x TN outputs whose rows are 8 and whose
// columns 4 apart and reads TM + TN 16-byte pieces per four k for 4 TM TN FMAs.  Two groups of warps take alternate pieces of k, so
// that a tile that has an SM to itself still has two warps per scheduler; their sums are added at the end.
// A sum does not depend on the number of rows: the K range is summed in pieces whose number follows from N and K alone
// (k_pieces), a piece group by group, and the pieces' sums are added one after the other.  A tile that leaves SMs idle has a CTA
// of a cluster for every piece or pair of pieces, whose sums meet through distributed shared memory; otherwise one CTA takes
// the pieces in turn and keeps the total in shared memory, which costs up to 4 % against one running sum (4096x3072x1024 in two
// pieces 676 -> 678 us, 1024x1024x1024 in four 69.4 -> 69.8, 1024x1536x1024 in four 102.5 -> 106.6).
// Rows that do not start on 16-byte boundaries move in 4-byte cp.async (16-bit storage: plain loads), in a kernel of their own: with
// both forms of staging in one, the aligned products were 3 - 5 % slower; 4096x1024x1022 336 -> 290 us.
#include <atomic>
#include <type_traits>

#include "kernels.cuh"

namespace b200 {
namespace {

constexpr int kStages = 3;

struct FmaParams {
  const void* A; long long lda, strideA;
  const void* W; long long ldw, strideW;
  const float* bias;
  void* C; long long ldc, strideC;
  const void* skip; long long ldskip;
  int M, N, K, act, out_f32, w_const;
  int pieces, ks;  // pieces of the K range that are summed one by one; CTAs per tile: pieces, pieces / 2 or 1
  float scale, alpha;
  int vec;       // rows start on 16-byte (16-bit storage: 8-byte) boundaries: operands move as pieces of four elements
  int conv_cin;  // convolution: A is [M][cin] on 8x8 boards, W is [9][N][cin]
  int conv_kt;   // ... and k runs over nine taps of conv_kt = cin rounded up to pieces of four
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ float4 ld_cluster_v4(uint32_t local, uint32_t rank) {
  uint32_t a;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Four elements from `src` into shared memory as floats; those from `left` on are zeros (left may be anything).
template <bool kVec, typename T>
__device__ __forceinline__ void stage4(float* dst, const T* src, int left) {
  if constexpr (sizeof(T) == 4) {
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (kVec) {
      cp_async16(to, src, min(max(left, 0), 4) * 4);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) cp_async4(to + 4 * i, i < left ? src + i : src, i < left ? 4 : 0);
    }
    return;
  }
  if (kVec && left >= 4) {
    const uint2 u = *reinterpret_cast<const uint2*>(src);
    const T* e = reinterpret_cast<const T*>(&u);
    *reinterpret_cast<float4*>(dst) = make_float4(to_f(e[0]), to_f(e[1]), to_f(e[2]), to_f(e[3]));
    return;
  }
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = i < left ? to_f(src[i]) : 0.f;
  *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
}

template <typename T, bool kFast, int BM, int BN, int TM, int TN, int kBK, int kGroups, int kMinCtas, bool kConv, bool kTotals, bool kVec>
__global__ void __launch_bounds__(kGroups * (BM / TM) * (BN / TN), kMinCtas)
gemm_fma_kernel(const FmaParams p) {
  constexpr int kGroupThreads = (BM / TM) * (BN / TN), kThreads = kGroups * kGroupThreads;
  constexpr int kWarpM = 8 * TM, kWarpN = 4 * TN;  // outputs of a warp
  constexpr int kLd = kBK + 4, kLdOut = BN + 4, kPieces = kBK / 4;
  constexpr int kRowStep = kThreads / kPieces;     // rows staged at a time
  static_assert(BM % kWarpM == 0 && BN % kWarpN == 0, "whole warps");
  extern __shared__ __align__(16) float sm[];      // [stages][BM + BN][kLd]; afterwards [1 or 2][BM][kLdOut] sums
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)blockIdx.x % p.ks;
  const int n0 = (int)blockIdx.x / p.ks * BN, m0 = blockIdx.y * BM;
  const T* A = reinterpret_cast<const T*>(p.A) + (long long)blockIdx.z * p.strideA;
  const T* W = reinterpret_cast<const T*>(p.W) + (long long)blockIdx.z * p.strideW;
  const int k_blocks = (p.K + kBK - 1) / kBK;
  auto piece_start = [&](int j) { return (int)((long long)k_blocks * j / p.pieces); };
  const int first = kTotals ? rank * (p.pieces / p.ks) : rank, own_pieces = kTotals ? p.pieces / p.ks : 1;  // of this CTA
  const int kb0 = piece_start(first), kbn = piece_start(first + own_pieces) - kb0;

  // This thread stages the four k from lk on of rows lr, lr + kRowStep, ... of both tiles.
  constexpr int kRowsA = (BM + kRowStep - 1) / kRowStep, kRowsW = (BN + kRowStep - 1) / kRowStep;
  const int lr = tid / kPieces, lk = tid % kPieces * 4;
  long long off_a[kRowsA], off_w[kRowsW];
  uint32_t ok_a[kRowsA], ok_w = 0;  // convolution: bit t of ok_a = tap t of that row lies on the board
#pragma unroll
  for (int r = 0; r < kRowsA; ++r) {
    const int m = m0 + lr + r * kRowStep;
    const bool in = m < p.M && lr + r * kRowStep < BM;
    off_a[r] = in ? (long long)m * p.lda : 0;
    ok_a[r] = in ? 1 : 0;
    if constexpr (kConv) {
      ok_a[r] = 0;
      for (int t = 0; t < 9; ++t) {
        const int y = ((m >> 3) & 7) + t / 3 - 1, x = (m & 7) + t % 3 - 1;
        if (in && (unsigned)y < 8u && (unsigned)x < 8u) ok_a[r] |= 1u << t;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kRowsW; ++r) {
    const int n = n0 + lr + r * kRowStep;
    const bool in = n < p.N && lr + r * kRowStep < BN;
    off_w[r] = in ? (long long)n * p.ldw : 0;
    if (in) ok_w |= 1u << r;
  }
  auto stage_w = [&](int i) {
    if (i >= kbn) return;
    float* dst = sm + (i % kStages) * (BM + BN) * kLd + (BM + lr) * kLd + lk;
    int k = (kb0 + i) * kBK + lk, left = p.K - k;
    const T* w = W;
    if constexpr (kConv) {
      const int tap = k / p.conv_kt;
      k -= tap * p.conv_kt;
      left = tap < 9 ? p.conv_cin - k : 0;
      if (tap < 9) w += (long long)tap * p.N * p.conv_cin;
    }
    if (left > 0) w += k;
#pragma unroll
    for (int r = 0; r < kRowsW; ++r)
      if (BN % kRowStep == 0 || lr + r * kRowStep < BN)
        stage4<kVec>(dst + r * kRowStep * kLd, w + off_w[r], (ok_w >> r) & 1 ? left : 0);
  };
  auto stage_a = [&](int i) {
    if (i >= kbn) return;
    float* dst = sm + (i % kStages) * (BM + BN) * kLd + lr * kLd + lk;
    const int k = (kb0 + i) * kBK + lk;
    int left = p.K - k, tap = 0;
    long long at = k;
    if constexpr (kConv) {
      tap = k / p.conv_kt;
      const int c = k - tap * p.conv_kt;
      left = tap < 9 ? p.conv_cin - c : 0;
      at = ((tap / 3 - 1) * 8 + tap % 3 - 1) * p.conv_cin + c;
    }
#pragma unroll
    for (int r = 0; r < kRowsA; ++r)
      if (BM % kRowStep == 0 || lr + r * kRowStep < BM) {
        const bool in = (ok_a[r] >> tap) & 1 && left > 0;
        stage4<kVec>(dst + r * kRowStep * kLd, in ? A + off_a[r] + at : A, in ? left : 0);
      }
  };

  // weights do not depend on the kernel before this one (w_const): they are requested while it is still running
  if (p.w_const) {
    for (int i = 0; i < kStages - 1; ++i) stage_w(i);
  }
  grid_dependency_wait();
  grid_launch_dependents();
  for (int i = 0; i < kStages - 1; ++i) {
    if (!p.w_const) stage_w(i);
    stage_a(i);
    cp_async_commit();  // the first group also holds the weights requested above
  }

  constexpr int kWarpsN = BN / kWarpN;
  const int group = tid / kGroupThreads, gw = warp - group * (kGroupThreads / 32);
  const int wm = gw / kWarpsN * kWarpM + (lane & 7), wn = gw % kWarpsN * kWarpN + (lane >> 3);
  float acc[TM][TN];
  auto clear = [&] {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  };
  clear();
  static_assert(kGroups == 2 && TN == 4, "held_at: one float4 per row of a thread");
  // kTotals: [TM][threads], of the rows that a thread's group owns the total so far, of the others the last piece
  auto held_at = [&](int t) { return reinterpret_cast<float4*>(sm + kStages * (BM + BN) * kLd) + t; };
  int i = 0;
  for (int piece = 1;; ++piece) {
    const int end = kTotals ? piece_start(first + piece) - kb0 : kbn;
#pragma unroll 1
    for (; i < end; ++i) {
      cp_async_wait<kStages - 2>();
      __syncthreads();  // stage i has landed; every thread is done with the stage that is filled next
      stage_w(i + kStages - 1);
      stage_a(i + kStages - 1);
      cp_async_commit();
      const float* as = sm + (i % kStages) * (BM + BN) * kLd + wm * kLd;
      const float* ws = sm + (i % kStages) * (BM + BN) * kLd + BM * kLd + wn * kLd;
#pragma unroll
      for (int kk = 0; kk < kBK; kk += 4 * kGroups) {
        const int k = kk + group * 4;
        float4 a[TM];
#pragma unroll
        for (int r = 0; r < TM; ++r) a[r] = *reinterpret_cast<const float4*>(as + r * 8 * kLd + k);
#pragma unroll
        for (int c0 = 0; c0 < TN; c0 += 4) {
          float4 w[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) w[c] = *reinterpret_cast<const float4*>(ws + (c0 + c) * 4 * kLd + k);
#pragma unroll
          for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int r = 0; r < TM; ++r)
#pragma unroll
              for (int c = 0; c < 4; ++c)
                acc[r][c0 + c] = fmaf(reinterpret_cast<const float*>(&a[r])[e], reinterpret_cast<const float*>(&w[c])[e], acc[r][c0 + c]);
        }
      }
    }
    if (end == kbn) break;
    // The piece is complete: a row's sums of both groups are added to the total in the group that owns the row.  The
    // thread's index is read again here: kept through the main loop it cost 1.5 %.
    uint32_t t0;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t0));
    const int grp = t0 / kGroupThreads, partner = grp == 0 ? kGroupThreads : -kGroupThreads;
    float4* held = held_at(t0);
#pragma unroll
    for (int r = 0; r < TM; ++r)
      if (r % 2 != grp) held[r * kThreads] = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < TM; ++r) {
      if (r % 2 != grp) continue;
      const float4 o = held[r * kThreads + partner];
      float4 t = make_float4(acc[r][0] + o.x, acc[r][1] + o.y, acc[r][2] + o.z, acc[r][3] + o.w);
      if (piece > 1) {
        const float4 b = held[r * kThreads];
        t = make_float4(b.x + t.x, b.y + t.y, b.z + t.z, b.w + t.w);
      }
      held[r * kThreads] = t;
    }
    clear();
  }

  const T* skip = reinterpret_cast<const T*>(p.skip);
  auto finish = [&](int m, int n, float v) {
    if (m >= p.M || n >= p.N) return;
    v *= p.scale;
    if (p.bias) v += __ldg(p.bias + n);
    v = activate<kFast>(v, p.act);
    if (skip) v = p.alpha * v + to_f(skip[(long long)m * p.ldskip + n]);
    const long long o = (long long)blockIdx.z * p.strideC + (long long)m * p.ldc + n;
    if (p.out_f32) reinterpret_cast<float*>(p.C)[o] = v;
    else reinterpret_cast<T*>(p.C)[o] = from_f<T>(v);
  };

  // The sums go through shared memory, so that whole rows are written, and with a cut K range to the other CTAs.
  cp_async_wait<0>();
  __syncthreads();
#pragma unroll
  for (int g = kGroups - 1; g >= 0; --g) {
    if (group == g) {
#pragma unroll
      for (int r = 0; r < TM; ++r) {
        float4 total = make_float4(0.f, 0.f, 0.f, 0.f);
        if (kTotals && g == 0) total = held_at(tid)[r * kThreads + (r % 2 == 0 ? 0 : kGroupThreads)];
#pragma unroll
        for (int c = 0; c < TN; ++c) {
          float* o = sm + (wm + r * 8) * kLdOut + wn + c * 4;
          float v = g == kGroups - 1 ? acc[r][c] : acc[r][c] + *o;
          if (kTotals && g == 0) {
            const float t = reinterpret_cast<const float*>(&total)[c];
            if (p.ks == 1) v = t + v;
            else o[BM * kLdOut] = t;  // two pieces of a cut range stay apart: the total is the first one
          }
          *o = v;
        }
      }
    }
    if (g > 0) __syncthreads();
  }
  if (p.ks == 1) {
    __syncthreads();
    for (int e = tid; e < BM * BN; e += kThreads) finish(m0 + e / BN, n0 + e % BN, sm[e / BN * kLdOut + e % BN]);
    return;
  }
  cluster_sync();
  const int slice = BM * BN / p.ks;  // a power of two and at least 64
  for (int e = rank * slice + tid * 4; e < (rank + 1) * slice; e += kThreads * 4) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(sm + e / BN * kLdOut + e % BN);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j = 0; j < p.ks; ++j) {
      if (kTotals) {
        const float4 u = ld_cluster_v4(at + BM * kLdOut * 4, j);
        v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
      }
      const float4 u = ld_cluster_v4(at, j);
      v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
    }
    const int m = m0 + e / BN, n = n0 + e % BN;
    finish(m, n, v.x);
    finish(m, n + 1, v.y);
    finish(m, n + 2, v.z);
    finish(m, n + 3, v.w);
  }
  cluster_sync();  // the others may still be reading this CTA's sums
}

template <typename T, int BM, int BN, int TM, int TN, int kBK, int kGroups, int kMinCtas, bool kConv, bool kTotals, bool kVec>
cudaError_t launch_kernel(const FmaParams& p, int batch, cudaStream_t s) {
  constexpr int ring = kStages * (BM + BN) * (kBK + 4) * 4, out = BM * (BN + 4) * 4;
  static_assert(ring >= 2 * out, "the sums take the place of the ring");
  constexpr int smem = ring + (kTotals ? kGroups * BM * BN * 4 : 0);
  auto kernel = gemm_fma_kernel<T, (sizeof(T) == 2), BM, BN, TM, TN, kBK, kGroups, kMinCtas, kConv, kTotals, kVec>;
  static std::atomic<unsigned long long> attr_mask{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (!(attr_mask.load() >> (dev & 63) & 1ull)) {
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
    attr_mask.fetch_or(1ull << (dev & 63));
  }
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(ceil_div(p.N, BN) * p.ks, ceil_div(p.M, BM), batch);
  lc.blockDim = dim3(kGroups * (BM / TM) * (BN / TN));
  lc.dynamicSmemBytes = smem;
  lc.stream = s;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (p.ks > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = p.ks;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  }
  if (t_dependent_launch) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  lc.attrs = attr;
  lc.numAttrs = na;
  return cudaLaunchKernelEx(&lc, kernel, p);
}

template <typename T, int BM, int BN, int TM, int TN, int kBK, int kGroups, int kMinCtas, bool kConv>
cudaError_t launch_tile(const FmaParams& p, int batch, cudaStream_t s) {
  auto launch = [&](auto totals, auto vec) {
    return launch_kernel<T, BM, BN, TM, TN, kBK, kGroups, kMinCtas, kConv, decltype(totals)::value, decltype(vec)::value>(p, batch, s);
  };
  using Yes = std::true_type;
  using No = std::false_type;
  if (p.ks == p.pieces) return p.vec ? launch(No(), Yes()) : launch(No(), No());
  return p.vec ? launch(Yes(), Yes()) : launch(Yes(), No());
}

// Pieces of the K range: from N and K alone, so that every number of rows has the same sums.  As many as give the column tiles of
// one row block work for 64 CTAs (128 when there are 64 k-blocks of 32 and more), of four k-blocks at least.
int k_pieces(int N, int K) {
  const int k_blocks = ceil_div(K, 32), n_tiles = ceil_div(N, 64), want = k_blocks >= 64 ? 128 : 64;
  int pieces = 1;
  while (pieces < 8 && pieces * n_tiles < want && k_blocks >= pieces * 8) pieces *= 2;
  return pieces;
}

// CTAs per tile: one for each piece or for each pair of pieces, while that finds SMs with little to do.  Measured in us at 1 / 2 / 4 /
// 8 CTAs per tile (fp32): 64x64 tiles 256x1024x1024 38 / 23 / 21 / 26, 256x3072x1024 67 / 57 / 60 / 73, 1024x1024x1024 67 / 73 /
// 76 / 94, 64x1024x1024 37 / 22 / 13 / 13, 64x3072x1024 37 / 23 / 21 / 24; 32x64 tiles 16x256x2048 45 / 25 / 15 / 10,
// 16x8192x256 8 / 9 / 13.  Uncut, 149 - 200 tiles take two rounds of SMs: 200 tiles of a 3x3 convolution of 128 channels at four CTAs
// each, ten of them 1.89 instead of 2.17 ms.
int cuts(const FmaParams& p, int bm, int batch) {
  const long long tiles = (long long)ceil_div(p.N, 64) * ceil_div(p.M, bm) * batch;
  auto fits = [&](int ks) { return tiles * ks <= (bm < 64 || ks == 8 ? 148 : 400); };
  if (fits(p.pieces)) return p.pieces;
  return p.pieces >= 4 && (fits(p.pieces / 2) || (bm == 64 && tiles > 148 && tiles <= 200)) ? p.pieces / 2 : 1;
}

template <typename T, bool kConv>
cudaError_t launch_fma(FmaParams p, int batch, cudaStream_t s) {
  p.pieces = k_pieces(p.N, p.K);
  const int bm = kConv || p.M > 32 ? 64 : p.M > 8 ? 32 : 8;  // a convolution has whole boards of 64 rows
  p.ks = cuts(p, bm, batch);
  if constexpr (!kConv) {
    if (bm == 8) return launch_tile<T, 8, 64, 1, 4, 32, 2, 2, false>(p, batch, s);
    if (bm == 32) return launch_tile<T, 32, 64, 4, 4, 32, 2, 2, false>(p, batch, s);
  }
  return launch_tile<T, 64, 64, 8, 4, 32, 2, 2, kConv>(p, batch, s);
}

template <typename T> bool aligned4(const void* ptr, long long ld, long long stride) {
  return (reinterpret_cast<uintptr_t>(ptr) % (4 * sizeof(T))) == 0 && ld % 4 == 0 && stride % 4 == 0;
}

}  // namespace

template <typename T>
cudaError_t launch_gemm_fma(const GemmParams& g, cudaStream_t s) {
  if (g.M <= 0 || g.N <= 0 || g.batch <= 0) return cudaSuccess;
  FmaParams p = {};
  p.A = g.A; p.lda = g.lda; p.strideA = g.strideA;
  p.W = g.W; p.ldw = g.ldw; p.strideW = g.strideW;
  p.bias = g.bias;
  p.C = g.C; p.ldc = g.ldc; p.strideC = g.strideC;
  p.skip = g.skip; p.ldskip = g.ldskip;
  p.M = g.M; p.N = g.N; p.K = g.K; p.act = g.act; p.out_f32 = g.out_f32;
  p.scale = g.scale; p.alpha = g.alpha;
  p.vec = aligned4<T>(g.A, g.lda, g.strideA) && aligned4<T>(g.W, g.ldw, g.strideW);
  p.w_const = g.w_const;
  return launch_fma<T, false>(p, g.batch, s);
}

template <typename T>
cudaError_t launch_conv3x3(const T* x, int cin, const T* w, const float* bias, T* y, int cout, int n, int act,
                           cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  FmaParams p = {};
  p.A = x; p.lda = cin; p.W = w; p.ldw = cin; p.bias = bias; p.C = y; p.ldc = cout;
  p.M = n * 64; p.N = cout; p.act = act; p.conv_cin = cin; p.conv_kt = ceil_div(cin, 4) * 4; p.K = 9 * p.conv_kt;
  p.scale = 1.f; p.alpha = 1.f; p.w_const = 1;
  p.vec = aligned4<T>(x, cin, 0) && aligned4<T>(w, cin, 0);
  return launch_fma<T, true>(p, 1, s);
}

#define INSTANTIATE(T)                                                          \
  template cudaError_t launch_gemm_fma<T>(const GemmParams&, cudaStream_t);     \
  template cudaError_t launch_conv3x3<T>(const T*, int, const T*, const float*, T*, int, int, int, cudaStream_t);
INSTANTIATE(float)
INSTANTIATE(__half)
INSTANTIATE(__nv_bfloat16)

}  // namespace b200
