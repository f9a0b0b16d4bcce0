// Tensor-core GEMM for products of few rows: C[M][N] = epilogue(A[M][K] . W[N][K]^T), the shapes a search's small batches
// send (64 rows and up for the token-wise layers, 1 row and up for the layers that see one row per position).
//
// Such a product is bound by latency and by how many SMs pull weights, not by the tensor pipe: with one 128x256 tile per
// CTA the 1024x1024 projection of one position ran on 4 SMs.  Here a tile is 128 (or 64) rows x BN columns and its K range
// is cut over the CTAs of a cluster (split-K), so that about one CTA per SM has a few k-blocks each, all of them in
// flight at once.  Tiles of loaded weights (GemmParams::w_const) do not depend on the kernel before this one: they are requested
// before griddepcontrol.wait, i.e. while that kernel is still running (two CTAs fit on an SM).
//   warp 8      TMA producer (W ahead of the grid dependency, then A)
//   warp 9      tcgen05.mma issuer (cta_group::1, 128xBNx16), accumulator in tensor memory
//   warps 0-7   accumulator -> fp32 partial tiles in shared memory; with split-K each CTA of the cluster owns a slice of
//               the tile's rows and every CTA pushes its partial sums of that slice there (st.shared::cluster); then
//               a fixed-order sum over the partials and the epilogue (scale, folded LayerNorm, bias, activation,
//               residual, row statistics) on eight columns per thread, written as 16-byte pieces of whole rows.
// A tile of at most 64 rows loads 64-row boxes of A; the upper half of the 128-row MMA then reads whatever follows in
// shared memory and its results are never looked at.
// Chains of dependent launches, before (one 128xBN tile per CTA of gemm_tc.cu's kernel, FMA kernel below 64 rows) and now:
// 64x1024x1024 15 -> 5.9 us, 1x256x2048 135 -> 5.3 us, 1x8192x256 21 -> 4.5 us, 32x4096x256 24 -> 4.2 us; with everything in this file one
// position of the BT4-class network 4.37 -> 0.81 ms, 24 positions 4.47 -> 1.71 ms.  (Net does not cut the K range of products with 64
// rows per position: one position's 1024-wide ones take 7.8 us for 5.9.)
// With a LayerNorm in front (GemmParams::ln_gamma; 256-wide rows, smolgen's two inner LayerNorms) warps 0-7 load the 64 rows of
// A themselves, normalise them in registers and write them to the operand tiles in the swizzle TMA would have used; gamma and
// beta arrive by bulk copy ahead of the grid dependency.  A LayerNorm vector may span several rows of A (smolgen's
// second one: 32 heads x 256), as long as a tile holds whole vectors.  Every column tile repeats the LayerNorm: worth it
// while a launch costs more than that (Net::gemm_with_ln has the line); beyond, ln_rows_kernel does it with the same results.
// Every wait is bounded by wall-clock time like those of gemm_tc.cu; the cluster barriers are reached by all threads
// whatever happened before them.
#include <atomic>

#include "kernels.cuh"
#include "tcgen05.cuh"

namespace b200 {
namespace {

constexpr int kSplitThreads = 320;

struct SplitCfg {
  int stages;  // shared-memory stages
  int a_rows;  // 64 or 128: rows of an A box = rows of the tile that exist
  int ks;      // CTAs per tile (cluster size)
  // LayerNorm in front of the product (kLN): x [M][256], vectors of `group` consecutive rows
  const void* x;
  const float* gamma;
  const float* beta;
  int group;
  float eps;
};
constexpr int kLnK = 256;  // row width of A with a LayerNorm: four k-blocks, all of them resident
constexpr int kLnMaxGroup = 32;

__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void load8(const float* src, int col, int n, float (&v)[8]) {
  if (col + 8 <= n && (reinterpret_cast<uintptr_t>(src + col) & 15) == 0) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(src + col)), b = __ldg(reinterpret_cast<const float4*>(src + col + 4));
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = col + i < n ? __ldg(src + col + i) : 0.f;
  }
}

template <int BN> struct SplitTile {
  static constexpr int kTail = 8 * 1024;  // what the 128-row MMA over a 64-row box may read behind the last stage
  static constexpr int kMisc = 1024 /*alignment*/ + 256 /*barriers*/ + 128 * 16 /*row vectors*/;
  __host__ __device__ static constexpr int stage_bytes(int a_rows) { return (a_rows + BN) * 128; }
  __host__ __device__ static constexpr int bytes(int a_rows, int stages) {
    const int ring = stages * stage_bytes(a_rows), part = a_rows * BN * 4;  // the partial tiles reuse the ring
    return (ring > part ? ring : part) + kTail + kMisc;
  }
  __host__ __device__ static constexpr int ln_bytes(int group) { return group * kLnK * 8; }  // gamma and beta
};

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}
// Sum over the rows of a LayerNorm vector of each row's `v` (four lanes per row, eight rows per warp, 64 rows per CTA): over
// lanes by shuffles, over warps (vectors of more than eight rows) through red[8].  All 256 threads call it.
__device__ __forceinline__ float ln_sum(float v, int group, float* red) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  for (int o = 1; o < group && o < 8; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, 4 * o);
  if (group > 8) {
    const int warp = threadIdx.x >> 5, span = group >> 3;
    if ((threadIdx.x & 31) == 0) red[warp] = v;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    v = 0.f;
    for (int w = warp & ~(span - 1), e = w + span; w < e; ++w) v += red[w];
  }
  return v;
}

// LayerNorm of 64 rows by 256 threads: this thread's 16-byte pieces q, q + 4, ..., q + 28 of row tid / 4 (q = tid % 4), and the
// mean and reciprocal deviation of the row's vector.  The product and ln_rows_kernel must agree to the last bit, hence the explicit
// fused multiply-adds.
template <typename T>
__device__ __forceinline__ void ln_rows_load(const void* x, int m, int M, int group, float eps, float* red, uint4 (&u)[8], float& mean,
                                             float& rstd) {
  const int q = threadIdx.x & 3;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    u[i] = m < M ? *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(x) + (long long)m * kLnK + (q + 4 * i) * 8)
                 : make_uint4(0, 0, 0, 0);
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) sum += to_f(reinterpret_cast<const T*>(&u[i])[j]);
  const float inv = 1.0f / (float)(group * kLnK);  // a power of two
  mean = ln_sum(sum, group, red) * inv;
  float var = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float d = to_f(reinterpret_cast<const T*>(&u[i])[j]) - mean;
      var = fmaf(d, d, var);
    }
  rstd = 1.0f / sqrtf(fmaf(ln_sum(var, group, red + 8), inv, eps));
}
// Eight values normalised; gamma and beta point at theirs.
template <typename T>
__device__ __forceinline__ uint4 ln_piece(const uint4& u, const float* gamma, const float* beta, float mean, float rstd) {
  const T* e = reinterpret_cast<const T*>(&u);
  float v[8], g[8], b[8];
  *reinterpret_cast<float4*>(g) = *reinterpret_cast<const float4*>(gamma);
  *reinterpret_cast<float4*>(g + 4) = *reinterpret_cast<const float4*>(gamma + 4);
  *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(beta);
  *reinterpret_cast<float4*>(b + 4) = *reinterpret_cast<const float4*>(beta + 4);
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = fmaf(g[j] * (to_f(e[j]) - mean), rstd, b[j]);
  return make_uint4(pack_pair<T>(v[0], v[1]), pack_pair<T>(v[2], v[3]), pack_pair<T>(v[4], v[5]), pack_pair<T>(v[6], v[7]));
}

// The same LayerNorm as a launch of its own, where the product has too many column tiles to repeat it in.  Latency-bound: 64 rows of
// 512 bytes per CTA, all loads of a thread in flight at once.
template <typename T>
__global__ void __launch_bounds__(256)
ln_rows_kernel(const T* x, T* out, const float* __restrict__ gamma, const float* __restrict__ beta, int group, float eps, int M) {
  __shared__ float red[16];
  grid_dependency_wait();
  grid_launch_dependents();
  const int row = threadIdx.x >> 2, q = threadIdx.x & 3, m = (int)blockIdx.x * 64 + row;
  uint4 u[8];
  float mean, rstd;
  ln_rows_load<T>(x, m, M, group, eps, red, u, mean, rstd);
  if (m >= M) return;
  const int at = (row & (group - 1)) * kLnK;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int c = (q + 4 * i) * 8;
    *reinterpret_cast<uint4*>(out + (long long)m * kLnK + c) = ln_piece<T>(u[i], gamma + at + c, beta + at + c, mean, rstd);
  }
}

template <typename T, int BN, bool kLN>
__global__ void __launch_bounds__(kSplitThreads)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w, const TcParams p,
                  const SplitCfg cfg) {
  constexpr int kMaxStages = 12;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int stage_bytes = SplitTile<BN>::stage_bytes(cfg.a_rows);
  const int ring = cfg.stages * stage_bytes, part_bytes = cfg.a_rows * BN * 4;
  uint8_t* misc = smem + (ring > part_bytes ? ring : part_bytes) + SplitTile<BN>::kTail;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(misc);       // [kMaxStages]
  uint64_t* empty_bar = full_bar + kMaxStages;                   // [kMaxStages]
  uint64_t* tfull_bar = empty_bar + kMaxStages;                  // accumulator complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint64_t* gb_bar = reinterpret_cast<uint64_t*>(misc + 216);    // kLN: gamma and beta have landed
  uint64_t* a_bar = gb_bar + 1;                                  // kLN: the normalised rows are in place
  float4* rowv = reinterpret_cast<float4*>(misc + 256);          // [rows of this CTA's slice] mean_a, rstd_a, mean_r, rstd_r
  float* ln_gb = reinterpret_cast<float*>(misc + 256 + 128 * 16);  // kLN: gamma [group * 256], beta [group * 256]

  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int ks = cfg.ks, rank = ks > 1 ? (int)cluster_ctarank() : 0;
  const int n0 = ((int)blockIdx.x / ks) * BN, m0 = (int)blockIdx.y * cfg.a_rows;
  const int k_blocks = (p.K + BK - 1) / BK;
  const int kb0 = k_blocks * rank / ks, kbn = k_blocks * (rank + 1) / ks - kb0;
  const int S = cfg.stages;

  if (tid == 256) {
    tma_prefetch_map(&tmap_w);
    tma_prefetch_map(&tmap_a);
    for (int i = 0; i < S; ++i) {
      mbar_init(smem_u32(&full_bar[i]), 1);
      mbar_init(smem_u32(&empty_bar[i]), 1);
    }
    mbar_init(smem_u32(tfull_bar), 1);
    if (kLN) {
      mbar_init(smem_u32(gb_bar), 1);
      mbar_init(smem_u32(a_bar), 256);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  // after the allocation: the next kernel's CTAs must not take the tensor memory that this one still waits for
  grid_launch_dependents();
  const uint32_t tmem = *tmem_slot;

  // ---- the eight columns this thread finishes, of rows r0, r0 + kRowStep, ... of the CTA's slice ----
  constexpr int kGroups = BN / 8, kRowStep = 256 / kGroups;
  const int rp = cfg.a_rows / ks;  // rows of the slice
  const int cg = tid % kGroups, r0 = tid / kGroups, col = n0 + cg * 8;
  float vb[8], vc[8], vg[8], ve[8];

  if (warp == 8) {
    // ---------------- TMA producer ----------------
    if (elect_one()) {
      const int early = kbn < S ? kbn : S;
      if (!p.w_const) grid_dependency_wait();
      for (int i = 0; i < early; ++i) {
        const uint32_t fb = smem_u32(&full_bar[i]);
        mbar_expect_tx(fb, kLN ? BN * 128 : stage_bytes);
        tma_load_2d(smem_u32(smem + i * stage_bytes) + cfg.a_rows * 128, &tmap_w, (kb0 + i) * BK, n0, fb);
      }
      if constexpr (kLN) {
        const uint32_t bytes = cfg.group * kLnK * 4, gb = smem_u32(gb_bar);
        mbar_expect_tx(gb, 2 * bytes);
        bulk_load(smem_u32(ln_gb), cfg.gamma, bytes, gb);
        bulk_load(smem_u32(ln_gb) + bytes, cfg.beta, bytes, gb);
      }
      grid_dependency_wait();
      int s = 0;
      uint32_t ph = 0;
      for (int i = 0; !kLN && i < kbn; ++i) {
        const uint32_t fb = smem_u32(&full_bar[s]), sa = smem_u32(smem + s * stage_bytes);
        if (i >= early) {
          if (!mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1, abort_flag, 1)) break;
          mbar_expect_tx(fb, stage_bytes);
          tma_load_2d(sa + cfg.a_rows * 128, &tmap_w, (kb0 + i) * BK, n0, fb);
        }
        tma_load_2d(sa, &tmap_a, (kb0 + i) * BK, m0, fb);
        if (++s == S) { s = 0; ph ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 9) {
    // ---------------- MMA issuer ----------------
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc<T, BN>();
      bool ok = !kLN || mbar_wait(smem_u32(a_bar), 0, abort_flag, 5);
      int s = 0;
      uint32_t ph = 0;
      for (int i = 0; ok && i < kbn; ++i) {
        if (!mbar_wait(smem_u32(&full_bar[s]), ph, abort_flag, 3)) { ok = false; break; }
        tcgen05_fence_after();
        const uint32_t sa = smem_u32(smem + s * stage_bytes);
        const uint64_t adesc = make_smem_desc(sa), bdesc = make_smem_desc(sa + cfg.a_rows * 128);
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          tcgen05_mma_f16(tmem, adesc + 2 * k, bdesc + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
        if (i + S < kbn) tcgen05_commit(smem_u32(&empty_bar[s]));
        if (++s == S) { s = 0; ph ^= 1; }
      }
      if (ok) tcgen05_commit(smem_u32(tfull_bar));
    }
    __syncwarp();
  } else {
    // per-column vectors (constants) and per-row vectors (written by the kernels before this one) while the tile is computed
    if (p.bias) load8(p.bias, col, p.N, vb);
    if (p.a_stats) load8(p.colsum, col, p.N, vc);
    if (p.res_mode == 2) {
      load8(p.res_gamma, col, p.N, vg);
      load8(p.res_beta, col, p.N, ve);
    }
    grid_dependency_wait();
    if constexpr (kLN) {
      const int row = tid >> 2, q = tid & 3;  // piece c of a row is piece c % 8 of k-block c / 8
      uint4 u[8];
      float mean, rstd;
      // rowv is not used here: no statistics come with a LayerNorm in front
      ln_rows_load<T>(cfg.x, m0 + row, p.M, cfg.group, cfg.eps, reinterpret_cast<float*>(rowv), u, mean, rstd);
      mbar_wait(smem_u32(gb_bar), 0, abort_flag, 6);
      const float* gamma = ln_gb + (row & (cfg.group - 1)) * kLnK;
      const float* beta = gamma + cfg.group * kLnK;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int c = q + 4 * i;
        const uint4 v = ln_piece<T>(u[i], gamma + c * 8, beta + c * 8, mean, rstd);
        st_shared_v4(smem_u32(smem + (c >> 3) * stage_bytes) + row * 128 + (((c & 7) ^ (row & 7)) << 4), v.x, v.y, v.z, v.w);
      }
      fence_async_smem();  // the tensor core reads the rows through the asynchronous proxy
      mbar_arrive(smem_u32(a_bar));
    }
    if (tid < rp && (p.a_stats || p.res_mode == 2)) {
      const int m = m0 + rank * rp + tid;
      float4 v = make_float4(0.f, 1.f, 0.f, 1.f);
      if (m < p.M) {
        if (p.a_stats) mean_rstd(p.a_stats, m, p.a_inv_c, p.a_eps, v.x, v.y);
        if (p.res_mode == 2) mean_rstd(p.res_stats, m, p.res_inv_c, p.res_eps, v.z, v.w);
      }
      rowv[tid] = v;
    }
    mbar_wait(smem_u32(tfull_bar), 0, abort_flag, 4);
    tcgen05_fence_after();
  }
  // The partial tiles overwrite the ring of the CTA that owns them: its MMAs must have read their last stage.
  if (ks > 1) cluster_sync_all();
  if (warp < 8) {
    const int quarter = warp & 3, half = warp >> 2, row = quarter * 32 + lane;
    if (quarter * 32 < cfg.a_rows) {
      constexpr int kCols = BN / 2;  // columns of this warp's half
      constexpr int kStep = kCols < 32 ? 16 : 32;
      const int owner = row / rp, rr = row - owner * rp;
      uint32_t dst = smem_u32(smem) + (uint32_t)((rank * rp + rr) * BN) * 4;
      if (ks > 1) dst = mapa(dst, (uint32_t)owner);
#pragma unroll
      for (int c = 0; c < kCols; c += kStep) {
        uint32_t r[kStep];
        const uint32_t ta = tmem + ((uint32_t)(quarter * 32) << 16) + half * kCols + c;
        if constexpr (kStep == 16) tmem_ld16(ta, r); else tmem_ld32(ta, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < kStep; j += 4) {
          // 16-byte pieces swizzled by the row: the 32 rows of a warp write the same columns
          const uint32_t a = dst + (uint32_t)((((half * kCols + c + j) >> 2) ^ (rr & 7)) << 4);
          if (ks > 1) st_cluster_v4(a, r[j], r[j + 1], r[j + 2], r[j + 3]);
          else st_shared_v4(a, r[j], r[j + 1], r[j + 2], r[j + 3]);
        }
      }
    }
  }
  tcgen05_fence_before();
  if (ks > 1) cluster_sync_all(); else __syncthreads();
  if (warp == 9) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)BN) : "memory");
  }
  if (warp < 8) {
    // lanes of this warp that finish the same row; they go through the loop together
    const uint32_t row_lanes = (kGroups == 32 ? 0xffffffffu : ((1u << kGroups) - 1u)) << (lane & ~(kGroups - 1));
    const float* part = reinterpret_cast<const float*>(smem);
    const bool whole = col + 8 <= p.N;
    const bool second = p.n_split > 0 && col >= p.n_split;
#pragma unroll 1
    for (int r = r0; r < rp; r += kRowStep) {
      const int m = m0 + rank * rp + r;
      if (m >= p.M) break;
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = 0.f;
      for (int j = 0; j < ks; ++j) {
        const float* src = part + (j * rp + r) * BN;
        const float4 a = *reinterpret_cast<const float4*>(src + (((2 * cg) ^ (r & 7)) << 2));
        const float4 b = *reinterpret_cast<const float4*>(src + (((2 * cg + 1) ^ (r & 7)) << 2));
        v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w; v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
      }
      const float4 rv = (p.a_stats || p.res_mode == 2) ? rowv[r] : make_float4(0.f, 1.f, 0.f, 1.f);
      if (p.scale != 1.0f) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] *= p.scale;
      }
      if (p.a_stats) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = rv.y * (v[i] - rv.x * vc[i]);
      }
      if (p.bias) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] += vb[i];
      }
      apply_activation(v, p.act);
      if (p.res_mode) {
        const T* rs = reinterpret_cast<const T*>(p.res) + (long long)m * p.ldres + col;
        float s[8];
        if (whole) {
          const uint4 u = *reinterpret_cast<const uint4*>(rs);
          const T* e = reinterpret_cast<const T*>(&u);
#pragma unroll
          for (int i = 0; i < 8; ++i) s[i] = to_f(e[i]);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) s[i] = col + i < p.N ? to_f(rs[i]) : 0.f;
        }
        if (p.res_mode == 2) {
          const float sh = -rv.z * rv.w;
#pragma unroll
          for (int i = 0; i < 8; ++i) s[i] = fmaf(fmaf(s[i], rv.w, sh), vg[i], ve[i]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = fmaf(p.alpha, v[i], s[i]);
      }
      if (p.out_stats) {
        // Sums of 32 columns (four lanes, one after the other) in fp32, their totals in double: the order of gemm_tc.cu,
        // so that a row's statistics do not depend on which kernel took the product.
        float a = 0.f, q = 0.f;
#pragma unroll
        for (int step = 0; step < 4; ++step) {
          if ((lane & 3) == step) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              if (col + i < p.N) { a += v[i]; q = fmaf(v[i], v[i], q); }
          }
          a = __shfl_sync(row_lanes, a, (lane & ~3) | step);
          q = __shfl_sync(row_lanes, q, (lane & ~3) | step);
        }
        double da = (double)a, dq = (double)q;
#pragma unroll
        for (int off = 4; off < kGroups; off <<= 1) {
          da += __shfl_xor_sync(row_lanes, da, off);
          dq += __shfl_xor_sync(row_lanes, dq, off);
        }
        if (cg == 0) {
          atomicAdd(p.out_stats + 2 * (long long)m, da);
          atomicAdd(p.out_stats + 2 * (long long)m + 1, dq);
        }
      }
      if (col >= p.N) continue;
      if (p.out_f32) {
        float* o = reinterpret_cast<float*>(p.C) + (long long)m * p.ldc + col;
        if (whole && p.vec_c) {
          *reinterpret_cast<float4*>(o) = make_float4(v[0], v[1], v[2], v[3]);
          *reinterpret_cast<float4*>(o + 4) = make_float4(v[4], v[5], v[6], v[7]);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (col + i < p.N) o[i] = v[i];
        }
      } else {
        T* o = second ? reinterpret_cast<T*>(p.C2) + (long long)m * p.ldc2 + (col - p.n_split)
                      : reinterpret_cast<T*>(p.C) + (long long)m * p.ldc + col;
        if (whole && p.vec_c) {
          uint4 u;
          u.x = pack_pair<T>(v[0], v[1]); u.y = pack_pair<T>(v[2], v[3]);
          u.z = pack_pair<T>(v[4], v[5]); u.w = pack_pair<T>(v[6], v[7]);
          *reinterpret_cast<uint4*>(o) = u;
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (col + i < p.N) o[i] = from_f<T>(v[i]);
        }
      }
    }
  }
  if (*abort_flag) {
    // Give copies that may still be in flight time to land before the CTA's shared memory is released.
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    if (tid == 0 && p.status) atomicCAS(p.status, 0, 500 + *abort_flag);
  }
}

// Tile width, cluster size and stages of a product: the least of a cost model in microseconds, fitted to chains of dependent
// launches of this kernel before its issuing lanes were elected (M x N x K; us at columns per tile / CTAs per tile).  A k-block
// took 731 cycles to issue then, 0.39 us, and takes 495 - 527 now: the model still orders the plans it was fitted to, but
// weighs a long K range too heavily against the exchange of a cut one, and has not been fitted again (another plan may cut K
// elsewhere, and results would change).  Tiles of 64 rows also above 64 rows: 10 x 256 attention network 2 / 8 / 16 / 37
// positions 271 / 283 / 307 / 369 -> 225 / 258 / 271 / 332 us, BT4-class 2 / 8 963 / 1057 -> 842 / 1008.
//   1536x1024x1024  32/1 19.5  64/1 11.2  64/2 17.6  128/1 13.9  128/2 12.5    2368x768x256   32/1 10.3  64/1 6.7  128/1 9.2
//   512x1024x1024   32/1 10.0  32/2 7.9   64/1 11.3  64/4 9.1    128/1 13.6    2368x256x256   32/1 5.3   64/1 6.6  128/1 9.0
//   512x1024x1536   32/2 9.5   64/2 10.9  64/4 9.8   128/2 12.7                64x1024x1024   32/4 5.9   64/1 9.8  64/4 6.3
//   1x256x2048      32/1 15.2  32/4 7.1   32/8 5.9   64/4 7.2                  32x4096x256    32/1 4.6   64/1 4.7  128/1 5.5
// A CTA's time grows with its tile's width and its k-blocks, not with a second CTA beside it on the SM: what is waited for is
// the latency of loads and of the epilogue.  Beyond two CTAs per SM the rest runs in another round.
struct SplitPlan { int bn, ks, a_rows, stages; };

SplitPlan split_plan(const GemmParams& g, int sm_count) {
  SplitPlan best{64, 1, 128, 1};
  double best_cost = 1e30;
  const int k_blocks = ceil_div(g.K, BK);
  // of plans that cost the same the one with the taller tiles, which fetch W less often
  for (int a_rows = g.M <= 64 ? 64 : 128; a_rows >= 64; a_rows /= 2) {
    const int m_tiles = ceil_div(g.M, a_rows);
    for (int bn = 32; bn <= 128; bn *= 2) {
      const int n_tiles = ceil_div(g.N, bn);
      for (int ks = 1; ks <= 8; ks *= 2) {
        if (ks > k_blocks || (ks > 1 && !g.split_k)) break;
        const int kb = ceil_div(k_blocks, ks);
        const long long ctas = (long long)n_tiles * m_tiles * ks;
        const int rounds = ceil_div(ctas, 2 * sm_count);
        const double tile = 2.5 + a_rows * bn * (1.0 / 3300), exchange = ks == 1 ? 0.0 : (0.25 + 0.2 * ks) * (a_rows == 64 ? 1.0 : 1.6);
        const double cost = rounds * (tile + 0.39 * kb + exchange + (ctas > sm_count ? 0.5 : 0.0));
        if (cost < best_cost) {
          best_cost = cost;
          best = SplitPlan{bn, ks, a_rows, kb};
        }
      }
    }
  }
  // a ring of at most 96 KB leaves room for a second CTA on the SM: the next tile, or the next kernel fetching its weights
  const int cap = 96 * 1024 / ((best.a_rows + best.bn) * 128);
  if (best.stages > cap) best.stages = cap;
  return best;
}

template <typename T, int BN, bool kLN = false>
cudaError_t launch_split_bn(const GemmParams& g, const SplitPlan& plan, int* status, cudaStream_t s) {
  static std::atomic<unsigned long long> attr_mask{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (!(attr_mask.load() >> (dev & 63) & 1ull)) {
    e = cudaFuncSetAttribute(gemm_split_kernel<T, BN, kLN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kLN ? SplitTile<BN>::bytes(64, kLnK / BK) + SplitTile<BN>::ln_bytes(kLnMaxGroup) : 112 * 1024);
    if (e != cudaSuccess) return e;
    attr_mask.fetch_or(1ull << (dev & 63));
  }
  const int prec = TypeTag<T>::prec;
  CUtensorMap ma, mw;
  if ((e = gemm_tensor_map(g.A, g.lda, g.M, g.K, plan.a_rows, prec, &ma)) != cudaSuccess) return e;
  if ((e = gemm_tensor_map(g.W, g.ldw, g.N, g.K, BN, prec, &mw)) != cudaSuccess) return e;
  TcParams p;
  fill_tc_params(p, g, status);
  const SplitCfg cfg{plan.stages, plan.a_rows, plan.ks, g.A, g.ln_gamma, g.ln_beta, g.ln_group, g.ln_eps};
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(ceil_div(g.N, BN) * plan.ks, ceil_div(g.M, plan.a_rows));
  lc.blockDim = dim3(kSplitThreads);
  lc.dynamicSmemBytes = SplitTile<BN>::bytes(plan.a_rows, plan.stages) + (kLN ? SplitTile<BN>::ln_bytes(g.ln_group) : 0);
  lc.stream = s;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (plan.ks > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = plan.ks;
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
  return cudaLaunchKernelEx(&lc, gemm_split_kernel<T, BN, kLN>, ma, mw, p, cfg);
}

}  // namespace

bool gemm_ln_supported(const GemmParams& g) {
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  return gemm_tc_supported(g) && !g.skip && g.K == kLnK && g.lda == kLnK && g.ln_group >= 1 && g.ln_group <= kLnMaxGroup &&
         (g.ln_group & (g.ln_group - 1)) == 0 && g.M % g.ln_group == 0 && g.ln_gamma && g.ln_beta && al16(g.A) &&
         al16(g.ln_gamma) && al16(g.ln_beta) && !g.a_stats && !g.res && !g.out_stats && g.n_split == 0 && g.conv_cin == 0 &&
         g.batch_rows == 0;
}

template <typename T>
cudaError_t launch_gemm_ln(const GemmParams& g, int* status, cudaStream_t s) {
  if (g.M <= 0 || g.N <= 0) return cudaSuccess;
  if (!gemm_ln_supported(g)) return cudaErrorInvalidValue;
  return launch_split_bn<T, 64, true>(g, SplitPlan{64, 1, 64, kLnK / BK}, status, s);
}
template <typename T>
cudaError_t launch_ln_rows(const T* x, T* out, const float* gamma, const float* beta, int group, float eps, int M, cudaStream_t s) {
  if (M <= 0) return cudaSuccess;
  return launch_dependent(ln_rows_kernel<T>, dim3(ceil_div(M, 64)), dim3(256), 0, s, x, out, gamma, beta, group, eps, M);
}
template cudaError_t launch_ln_rows<__half>(const __half*, __half*, const float*, const float*, int, float, int, cudaStream_t);
template cudaError_t launch_ln_rows<__nv_bfloat16>(const __nv_bfloat16*, __nv_bfloat16*, const float*, const float*, int, float, int,
                                                   cudaStream_t);
template cudaError_t launch_gemm_ln<__half>(const GemmParams&, int*, cudaStream_t);
template cudaError_t launch_gemm_ln<__nv_bfloat16>(const GemmParams&, int*, cudaStream_t);

template <typename T>
cudaError_t launch_gemm_split(const GemmParams& g, int* status, int sm_count, cudaStream_t s) {
  const SplitPlan plan = split_plan(g, sm_count);
  if (plan.bn == 32) return launch_split_bn<T, 32>(g, plan, status, s);
  if (plan.bn == 64) return launch_split_bn<T, 64>(g, plan, status, s);
  return launch_split_bn<T, 128>(g, plan, status, s);
}
template cudaError_t launch_gemm_split<__half>(const GemmParams&, int*, int, cudaStream_t);
template cudaError_t launch_gemm_split<__nv_bfloat16>(const GemmParams&, int*, int, cudaStream_t);

}  // namespace b200
