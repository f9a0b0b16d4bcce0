// Products and 3x3 convolutions of the fp32 verification mode on tensor cores.
//
// Every fp32 operand is cut into three bf16 pieces, x = x1 + x2 + x3, each the rounding of what the ones before it leave: 24
// significant bits, so the pieces hold x exactly (short of underflow).  A product of two pieces is exact in fp32, and of the nine the
// six of order 2^-16 and above are summed:
//   a1 w1                      order 1
//   a1 w2 + a2 w1              order 2^-9
//   a1 w3 + a2 w2 + a3 w1      order 2^-18;  what is left out is below 2^-26 of |a||w|
// The tensor core adds to its accumulator with truncation, which over a long K range would cost more digits than an FMA chain
// has to lose.  So the sums of order 1 stay in tensor memory for 64 k only and are then added, rounded, in registers; the
// small orders may stay there for the whole range, where truncation at 2^-9 of their size does not count.  A row's sum is taken in the
// same order at every number of rows, tile width and grid.
//
// Measured against sums in 64 bits, relative 2-norm of the error, this kernel / FMA kernel: see DESIGN; the network's outputs too.
//
// Bound by the tensor pipe (six MMAs for one: 277 TFLOP/s at the measured bf16 rate; the FMA pipe has 74) with the operand
// traffic close behind: an A tile of 128 x 64 arrives as 32 KB of fp32 and is cut by the CTA itself, the weights' pieces are
// made once at load and arrive by TMA (24 KB per k-block at 64 columns, 48 KB at 128).
//   warps 0-7    fp32 rows of A -> registers (one k-block ahead) -> three bf16 pieces -> swizzled operand tiles
//   warp 8       TMA of the weights' pieces
//   warp 9       tcgen05.mma (cta_group::1).  Pieces of W lie one behind the other, so a1 [w2 w3] and a2 [w1 w2] are one MMA each
//                of twice the width: four MMAs per 16 k instead of six, the narrow ones being bound by the reads of A
//   warps 10-17  after every k-block: order-1 sums of one of two accumulators -> added in registers; at the end the small
//                orders, then through shared memory to whole rows: scale, bias, activation, skip
// Infinities: inf times a piece that is zero would be NaN, and a value may round to an infinite piece; an output that comes
// out non-finite is therefore computed again from the fp32 operands, by FMAs.
// Every wait is bounded like those of gemm_tc.cu.
#include <atomic>

#include "kernels.cuh"
#include "tcgen05.cuh"

namespace b200 {
namespace {

constexpr int kF32Threads = 576;

struct F32Params {
  const float* A; long long lda;
  const float* W; long long ldw;
  const float* bias;
  float* C; long long ldc;
  const float* skip; long long ldskip;
  int M, N, K, act;
  float scale, alpha;
  int conv_cin;   // convolution: A is [M][cin] on 8x8 boards, W [9][N][cin]
  int cblocks;    // ... k-blocks per tap
  int k_blocks;
  int vec_c;      // C may be written, skip and bias read in 16-byte pieces
  int* status;
};

template <int BN> struct F32Tile {
  static constexpr int kA = 3 * 128 * 128, kW = 3 * BN * 128;  // bytes of a k-block's pieces
  static constexpr int kStage = kA + kW;
  static constexpr int kStages = BN == 128 ? 2 : 3;
  static constexpr int kOut = 128 * (BN + 4) * 4;  // the tile's sums, in place of the ring
  static constexpr int kBytes = kStages * kStage + 1024 /*alignment*/ + 256 /*barriers*/;
  static_assert(kStages * kStage >= kOut, "the sums take the place of the ring");
};

// The three bf16 pieces of two values (the first in the lower half).
__device__ __forceinline__ void split3(float x, float y, uint32_t& u1, uint32_t& u2, uint32_t& u3) {
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(u1) : "f"(y), "f"(x));
  x = __fsub_rn(x, __uint_as_float(u1 << 16));
  y = __fsub_rn(y, __uint_as_float(u1 & 0xffff0000u));
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(u2) : "f"(y), "f"(x));
  x = __fsub_rn(x, __uint_as_float(u2 << 16));
  y = __fsub_rn(y, __uint_as_float(u2 & 0xffff0000u));
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(u3) : "f"(y), "f"(x));
}

// W [count] -> planes [3][count]
__global__ void __launch_bounds__(256) split_weights_kernel(const float* __restrict__ w, long long count, __nv_bfloat16* __restrict__ out) {
  const long long i = blockIdx.x * 256LL + threadIdx.x;
  if (i >= count) return;
  uint32_t u1, u2, u3;
  split3(w[i], 0.f, u1, u2, u3);
  out[i] = __ushort_as_bfloat16((unsigned short)u1);
  out[count + i] = __ushort_as_bfloat16((unsigned short)u2);
  out[2 * count + i] = __ushort_as_bfloat16((unsigned short)u3);
}

__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Row m, column n of the product from the fp32 operands, by a whole warp.
template <bool kConv>
__device__ __forceinline__ float warp_dot(const F32Params& p, int m, int n) {
  const int lane = threadIdx.x & 31;
  float v = 0.f;
  if constexpr (kConv) {
    for (int t = 0; t < 9; ++t) {
      const int y = ((m >> 3) & 7) + t / 3 - 1, x = (m & 7) + t % 3 - 1;
      if ((unsigned)y >= 8u || (unsigned)x >= 8u) continue;
      const float* a = p.A + (long long)(m + (t / 3 - 1) * 8 + t % 3 - 1) * p.conv_cin;
      const float* w = p.W + ((long long)t * p.N + n) * p.conv_cin;
      for (int k = lane; k < p.conv_cin; k += 32) v = fmaf(a[k], w[k], v);
    }
  } else {
    for (int k = lane; k < p.K; k += 32) v = fmaf(p.A[m * p.lda + k], p.W[n * p.ldw + k], v);
  }
  return warp_sum(v);
}

template <int BN, bool kConv>
__global__ void __launch_bounds__(kF32Threads, 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap tmap_w, const F32Params p) {
  using L = F32Tile<BN>;
  constexpr int S = L::kStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S * L::kStage);  // [S] eight converter warps and the weights
  uint64_t* empty_bar = full_bar + S;                                      // [S] the k-block's MMAs are done
  uint64_t* hfull_bar = empty_bar + S;                                     // [2] order-1 sums complete
  uint64_t* hempty_bar = hfull_bar + 2;                                    // [2] ... and read by eight warps
  uint64_t* xfull_bar = hempty_bar + 2;                                    // every MMA done
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(xfull_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int n0 = (int)blockIdx.x * BN, m0 = (int)blockIdx.y * 128;
  const int kbn = p.k_blocks;

  if (tid == 256) {
    tma_prefetch_map(&tmap_w);
    for (int i = 0; i < S; ++i) {
      mbar_init(smem_u32(&full_bar[i]), 9);
      mbar_init(smem_u32(&empty_bar[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&hfull_bar[i]), 1);
      mbar_init(smem_u32(&hempty_bar[i]), 8);
    }
    mbar_init(smem_u32(xfull_bar), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)(4 * BN))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  // after the allocation: the next kernel's CTAs must not take the tensor memory that this one still waits for
  grid_launch_dependents();
  const uint32_t tmem = *tmem_slot;  // order-1 sums of even k-blocks, of odd ones, order 2^-9, order 2^-18: BN columns each

  if (warp < 8) {
    // ---------------- A: fp32 rows -> pieces ----------------
    const int lr = tid >> 3, lp = tid & 7;  // rows lr, lr + 32, ...; eight k from 8 lp on
    long long off[4];
    uint32_t ok[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int m = m0 + lr + 32 * r;
      const bool in = m < p.M;
      off[r] = in ? (long long)m * p.lda + lp * 8 : 0;
      ok[r] = in ? 1 : 0;
      if constexpr (kConv) {
        ok[r] = 0;
        for (int t = 0; t < 9; ++t) {
          const int y = ((m >> 3) & 7) + t / 3 - 1, x = (m & 7) + t % 3 - 1;
          if (in && (unsigned)y < 8u && (unsigned)x < 8u) ok[r] |= 1u << t;
        }
      }
    }
    float4 next[4][2];
    auto load = [&](int i) {
      int tap = 0, c = i * 64;
      long long at = c;
      bool in_k;
      if constexpr (kConv) {
        tap = i / p.cblocks;
        c = (i - tap * p.cblocks) * 64;
        at = ((tap / 3 - 1) * 8 + tap % 3 - 1) * p.lda + c;
        in_k = c + lp * 8 < p.conv_cin;
      } else {
        in_k = c + lp * 8 < p.K;
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float4* src = reinterpret_cast<const float4*>(p.A + off[r] + at);
        const bool in = in_k && ((ok[r] >> tap) & 1);
        next[r][0] = in ? src[0] : make_float4(0.f, 0.f, 0.f, 0.f);
        next[r][1] = in ? src[1] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    grid_dependency_wait();
    load(0);
    int s = 0;
    uint32_t ph = 0;
    for (int i = 0; i < kbn; ++i) {
      float4 cur[4][2];
#pragma unroll
      for (int r = 0; r < 4; ++r) { cur[r][0] = next[r][0]; cur[r][1] = next[r][1]; }
      if (i + 1 < kbn) load(i + 1);
      if (i >= S && !mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1, abort_flag, 1)) break;
      const uint32_t st = smem_u32(smem + s * L::kStage) + lr * 128 + ((lp ^ (lr & 7)) << 4);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        uint32_t u[3][4];
        split3(cur[r][0].x, cur[r][0].y, u[0][0], u[1][0], u[2][0]);
        split3(cur[r][0].z, cur[r][0].w, u[0][1], u[1][1], u[2][1]);
        split3(cur[r][1].x, cur[r][1].y, u[0][2], u[1][2], u[2][2]);
        split3(cur[r][1].z, cur[r][1].w, u[0][3], u[1][3], u[2][3]);
#pragma unroll
        for (int j = 0; j < 3; ++j) st_shared_v4(st + j * 16384 + r * 4096, u[j][0], u[j][1], u[j][2], u[j][3]);
      }
      fence_async_smem();  // the tensor core reads the pieces through the asynchronous proxy
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&full_bar[s]));
      if (++s == S) { s = 0; ph ^= 1; }
    }
  } else if (warp == 8) {
    // ---------------- weights: loaded once, requested while the kernel before this one is still running ----------------
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      for (int i = 0; i < kbn; ++i) {
        if (i >= S && !mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1, abort_flag, 2)) break;
        const uint32_t fb = smem_u32(&full_bar[s]), dst = smem_u32(smem + s * L::kStage) + L::kA;
        mbar_expect_tx(fb, L::kW);
        int row = n0, x = i * 64, plane = p.N;
        if constexpr (kConv) {
          const int tap = i / p.cblocks;
          x = (i - tap * p.cblocks) * 64;
          row += tap * p.N;
          plane = 9 * p.N;
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) tma_load_2d(dst + j * BN * 128, &tmap_w, x, row + j * plane, fb);
        if (++s == S) { s = 0; ph ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 9) {
    // ---------------- MMA issuer ----------------
    if (elect_one()) {
      constexpr uint32_t one = make_idesc<__nv_bfloat16, BN>(), two = make_idesc<__nv_bfloat16, 2 * BN>();
      bool good = true;
      int s = 0;
      uint32_t ph = 0;
      for (int i = 0; i < kbn; ++i) {
        const int b = i & 1;
        if (i >= 2 && !mbar_wait(smem_u32(&hempty_bar[b]), ((i >> 1) & 1) ^ 1, abort_flag, 3)) { good = false; break; }
        if (!mbar_wait(smem_u32(&full_bar[s]), ph, abort_flag, 4)) { good = false; break; }
        tcgen05_fence_after();
        const uint32_t sa = smem_u32(smem + s * L::kStage);
        const uint64_t a1 = make_smem_desc(sa), a2 = make_smem_desc(sa + 16384), a3 = make_smem_desc(sa + 32768);
        const uint64_t w1 = make_smem_desc(sa + L::kA), w2 = make_smem_desc(sa + L::kA + BN * 128);
#pragma unroll
        for (int k = 0; k < 4; ++k) tcgen05_mma_f16(tmem + b * BN, a1 + 2 * k, w1 + 2 * k, one, k > 0 ? 1u : 0u);
        tcgen05_commit(smem_u32(&hfull_bar[b]));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          tcgen05_mma_f16(tmem + 2 * BN, a1 + 2 * k, w2 + 2 * k, two, (i > 0 || k > 0) ? 1u : 0u);
          tcgen05_mma_f16(tmem + 2 * BN, a2 + 2 * k, w1 + 2 * k, two, 1u);
          tcgen05_mma_f16(tmem + 3 * BN, a3 + 2 * k, w1 + 2 * k, one, 1u);
        }
        tcgen05_commit(smem_u32(&empty_bar[s]));
        if (++s == S) { s = 0; ph ^= 1; }
      }
      if (good) tcgen05_commit(smem_u32(xfull_bar));
    }
    __syncwarp();
  } else {
    // ---------------- sums ----------------
    constexpr int kCols = BN / 2;  // columns of this warp: its half of the tile, 32 rows
    const int quarter = warp & 3, half = (warp - 10) >> 2;
    const uint32_t ta = tmem + ((uint32_t)(quarter * 32) << 16) + half * kCols;
    float acc[kCols];
#pragma unroll
    for (int j = 0; j < kCols; ++j) acc[j] = 0.f;
    auto add = [&](uint32_t at, float* to) {
#pragma unroll
      for (int c = 0; c < kCols; c += 16) {
        uint32_t r[16];
        tmem_ld16(at + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) to[c + j] = __fadd_rn(to[c + j], __uint_as_float(r[j]));
      }
    };
    bool good = true;
    for (int i = 0; i < kbn; ++i) {
      const int b = i & 1;
      if (!mbar_wait(smem_u32(&hfull_bar[b]), (i >> 1) & 1, abort_flag, 5)) { good = false; break; }
      tcgen05_fence_after();
      add(ta + b * BN, acc);
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&hempty_bar[b]));
    }
    if (good) good = mbar_wait(smem_u32(xfull_bar), 0, abort_flag, 6);
    tcgen05_fence_after();
    // the small orders, smallest first; the ring is free, the sums go through it
    float* out = reinterpret_cast<float*>(smem);
    {
      float* row = out + (quarter * 32 + lane) * (BN + 4) + half * kCols;
#pragma unroll
      for (int c = 0; c < kCols; c += 16) {
        uint32_t x1[16], x2[16];
        tmem_ld16(ta + 2 * BN + c, x1);
        tmem_ld16(ta + 3 * BN + c, x2);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
          float4 v;
          v.x = __fadd_rn(acc[c + j], __fadd_rn(__uint_as_float(x1[j]), __uint_as_float(x2[j])));
          v.y = __fadd_rn(acc[c + j + 1], __fadd_rn(__uint_as_float(x1[j + 1]), __uint_as_float(x2[j + 1])));
          v.z = __fadd_rn(acc[c + j + 2], __fadd_rn(__uint_as_float(x1[j + 2]), __uint_as_float(x2[j + 2])));
          v.w = __fadd_rn(acc[c + j + 3], __fadd_rn(__uint_as_float(x1[j + 3]), __uint_as_float(x2[j + 3])));
          *reinterpret_cast<float4*>(row + c + j) = v;
        }
      }
    }
    tcgen05_fence_before();
    asm volatile("bar.sync 1, 256;" ::: "memory");
    grid_dependency_wait();  // the residual input
    const int t = tid - 320;
#pragma unroll 1
    for (int e = t * 4; e < 128 * BN; e += 1024) {
      const int r = e / BN, c = e % BN, m = m0 + r, n = n0 + c;
      const float4 q = *reinterpret_cast<const float4*>(out + r * (BN + 4) + c);
      float v[4] = {q.x, q.y, q.z, q.w};
      const bool in = m < p.M && n < p.N;
      bool again = false;
#pragma unroll
      for (int j = 0; j < 4; ++j) again |= in && n + j < p.N && !(fabsf(v[j]) <= 3.402823466e38f);
      for (uint32_t todo = __ballot_sync(0xffffffffu, again); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        const int mm = __shfl_sync(0xffffffffu, m, src), nn = __shfl_sync(0xffffffffu, n, src);
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
          const float d = nn + j < p.N ? warp_dot<kConv>(p, mm, nn + j) : 0.f;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (lane == src && k == j) v[k] = d;
        }
      }
      if (!in) continue;
      const bool whole = p.vec_c && n + 4 <= p.N;
      float b4[4] = {0.f, 0.f, 0.f, 0.f}, s4[4] = {0.f, 0.f, 0.f, 0.f};
      const float* skip = p.skip ? p.skip + (long long)m * p.ldskip + n : nullptr;
      if (whole) {
        if (p.bias) *reinterpret_cast<float4*>(b4) = __ldg(reinterpret_cast<const float4*>(p.bias + n));
        if (skip) *reinterpret_cast<float4*>(s4) = *reinterpret_cast<const float4*>(skip);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (p.bias && n + j < p.N) b4[j] = __ldg(p.bias + n + j);
          if (skip && n + j < p.N) s4[j] = skip[j];
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[j] *= p.scale;
        if (p.bias) v[j] += b4[j];
        v[j] = activate<false>(v[j], p.act);
        if (skip) v[j] = p.alpha * v[j] + s4[j];
      }
      float* o = p.C + (long long)m * p.ldc + n;
      if (whole) {
        *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n + j < p.N) o[j] = v[j];
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 9) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)(4 * BN)) : "memory");
  }
  if (*abort_flag) {
    // Give copies that may still be in flight time to land before the CTA's shared memory is released.
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    if (tid == 0 && p.status) atomicCAS(p.status, 0, 600 + *abort_flag);
  }
}

template <int BN, bool kConv>
cudaError_t launch_f32_bn(const F32Params& p, const void* planes, cudaStream_t s) {
  using L = F32Tile<BN>;
  auto kernel = gemm_f32_kernel<BN, kConv>;
  static std::atomic<unsigned long long> attr_mask{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (!(attr_mask.load() >> (dev & 63) & 1ull)) {
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes)) != cudaSuccess) return e;
    attr_mask.fetch_or(1ull << (dev & 63));
  }
  CUtensorMap mw;
  const int rows = 3 * (kConv ? 9 : 1) * p.N, cols = kConv ? p.conv_cin : p.K;
  if ((e = gemm_tensor_map(planes, cols, rows, cols, BN, TypeTag<__nv_bfloat16>::prec, &mw)) != cudaSuccess) return e;
  return launch_dependent(kernel, dim3(ceil_div(p.N, BN), ceil_div(p.M, 128)), dim3(kF32Threads), L::kBytes, s, mw, p);
}

// Tile width: the least time of a round of tiles (one per SM) times the rounds.  Cycles of a k-block are those of its MMAs
// (128 x N x 16: 40 / 48 / 64 / 126 at N = 32 / 64 / 128 / 256); a tile's start and end take what is added.
template <bool kConv>
cudaError_t launch_f32(const F32Params& p, const void* planes, int sm_count, cudaStream_t s) {
  const long long m_tiles = ceil_div(p.M, 128);
  auto cost = [&](int bn, int block, int ends) {
    return (long long)ceil_div(m_tiles * ceil_div(p.N, bn), sm_count) * ((long long)p.k_blocks * block + ends);
  };
  const long long c32 = cost(32, 710, 5000), c64 = cost(64, 900, 6000), c128 = cost(128, 1520, 8000);
  if (c32 < c64 && c32 < c128) return launch_f32_bn<32, kConv>(p, planes, s);
  if (c64 <= c128) return launch_f32_bn<64, kConv>(p, planes, s);
  return launch_f32_bn<128, kConv>(p, planes, s);
}

bool al16(const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; }

}  // namespace

cudaError_t launch_split_weights(const float* w, long long count, void* planes, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  split_weights_kernel<<<ceil_div(count, 256), 256, 0, s>>>(w, count, static_cast<__nv_bfloat16*>(planes));
  return cudaGetLastError();
}

bool gemm_f32_supported(const GemmParams& g) {
  const int k = g.conv_cin > 0 ? g.conv_cin : g.K;
  return g.W3 && g.batch == 1 && g.batch_rows == 0 && k >= 8 && (k % 8) == 0 && (g.lda % 4) == 0 && (g.conv_cin > 0 || g.ldw == g.K) &&
         al16(g.A) && al16(g.W3) && !g.a_stats && !g.res && !g.out_stats && g.n_split == 0 && g.se_k == 0 && !g.ln_gamma;
}

cudaError_t launch_gemm_f32(const GemmParams& g, int* status, int sm_count, cudaStream_t s) {
  if (g.M <= 0 || g.N <= 0) return cudaSuccess;
  if (!gemm_f32_supported(g)) return cudaErrorInvalidValue;
  F32Params p = {};
  p.A = static_cast<const float*>(g.A); p.lda = g.conv_cin > 0 ? g.conv_cin : g.lda;
  p.W = static_cast<const float*>(g.W); p.ldw = g.ldw;
  p.bias = g.bias;
  p.C = static_cast<float*>(g.C); p.ldc = g.ldc;
  p.skip = static_cast<const float*>(g.skip); p.ldskip = g.ldskip;
  p.M = g.M; p.N = g.N; p.K = g.K; p.act = g.act; p.scale = g.scale; p.alpha = g.alpha;
  p.conv_cin = g.conv_cin;
  p.cblocks = ceil_div(g.conv_cin, 64);
  p.k_blocks = g.conv_cin > 0 ? 9 * p.cblocks : ceil_div(g.K, 64);
  p.vec_c = al16(g.C) && g.ldc % 4 == 0 && (!g.skip || (al16(g.skip) && g.ldskip % 4 == 0)) && (!g.bias || al16(g.bias));
  p.status = status;
  return g.conv_cin > 0 ? launch_f32<true>(p, g.W3, sm_count, s) : launch_f32<false>(p, g.W3, sm_count, s);
}

}  // namespace b200
