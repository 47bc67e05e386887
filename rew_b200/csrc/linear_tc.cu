// bf16 Linear on the 5th-generation tensor cores (tcgen05.mma, accumulator in
// tensor memory): y[M,N] = x[M,K] @ W[K,N] (+ b), src/rew/nn/linear.nim:43-49.
//
// Operand roles follow the reference's weight layout.  W is [in,out] row-major,
// i.e. `out` is contiguous, which is an MN-major UMMA operand: W is the A
// operand (UMMA M = 128 output features per CTA), the activations x[token][k]
// (k contiguous, K-major) are the B operand (UMMA N = TN tokens).  The f32
// accumulator D[feature][token] lives in TMEM: lane = output feature, column =
// token.
//
// Roles inside the CTA (320 threads):
//   warp 0   TMA producer: cp.async.bulk.tensor boxes of W (64 k x 64 features,
//            two per stage) and x (64 k x TN tokens), 128-byte swizzle, into a
//            multi-stage mbarrier ring; W loads of weights that no kernel
//            of a step writes (TcArgs::early_w) are issued before
//            griddepcontrol.wait so the ramp overlaps the previous kernel.
//   warp 1   allocates TMEM, then one elected thread (elect.sync: see elect_one
//            in tc.cuh) issues four tcgen05.mma.kind::f16 (K = 16 each) per stage
//            from shared-memory descriptors in one block of code and releases the
//            stage with tcgen05.commit.
//   warps 2-9 epilogue: tcgen05.ld the accumulator (a warp owns 32 lanes),
//            apply bias / SwiGLU, store.
// All waits on barriers are bounded; on a timeout the roles fall through to the
// common exit, where TMEM is released.  tcgen05.alloc, the cluster barriers and
// the stream dependency have no limit of their own: see
// alloc_then_launch_dependents (tc.cuh) and kAllSmem for what ends them.
#include <string.h>

#include "act.cuh"
#include "common.cuh"
#include "ptx.cuh"
#include "tc.cuh"

namespace rewb {
namespace {

constexpr int BM = 128;  // output features per CTA
constexpr int BK = 64;
constexpr int A_BYTES = 2 * BK * 64 * 2;  // two 64x64 boxes
// All the shared memory of an SM.  The kernels that take all of its tensor memory ask for all of this too, whatever their ring
// needs: no CTA of a launch that starts early sits beside them.
constexpr int kAllSmem = 227 * 1024;

struct TcArgs {
  int64_t M, N, K;
  int kb_per_split;
  int epi;
  void* out;
  int64_t ldo;
  int64_t split_stride;
  const float* bias;
  int* status;
  const int* row_offsets;  // grouped launches (persistent kernel): rows of group g = [row_offsets[g], row_offsets[g+1])
  int groups;
  int tn, stages;          // launches that choose their tile and ring
  int ksplit;              // persistent kernel: pieces of a tile along K
  int early_w;             // the weights are final before any step: they may be requested ahead of the stream dependency
  int fuse_qkv;       // cluster kernel: finish q|k|v in the epilogue (bias, RoPE, cache write) instead of one f32 slab
  QkvPostArgs qp;     // what qkv_post_kernel would have been given (partial / nsplit unused)
};

template <int TN>
struct TcCfg {
  // 32 tokens: 5 x 20 KB, 64: 4 x 24 KB, so that two CTAs share an SM (these tiles serve steps with a single token
  // tile, where a launch has only as many CTAs as feature tiles x splits)
  static constexpr int STAGES = TN <= 32 ? 5 : 4;
  static constexpr int B_BYTES = TN * 128;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 + 256;
  static constexpr int TMEM_COLS = TN < 32 ? 32 : TN;
  __device__ __forceinline__ static int tn(const TcArgs&) { return TN; }
  __device__ __forceinline__ static int stages(const TcArgs&) { return STAGES; }
  __device__ __forceinline__ static uint32_t tmem_cols(const TcArgs&) { return TMEM_COLS; }
};
// TN = 0: steps of more than 64 tokens, whose tile (a multiple of 16 tokens) and ring are the launch's choice.  Up to 160
// tokens two CTAs share an SM, with three stages or more each; larger tiles have the SM to themselves.
template <>
struct TcCfg<0> {
  static constexpr int MAX_STAGES = 8;
  static constexpr int FIXED = 1024 + 256;
  static constexpr int stage_bytes(int tn) { return A_BYTES + tn * 128; }
  __device__ __forceinline__ static int tn(const TcArgs& a) { return a.tn; }
  __device__ __forceinline__ static int stages(const TcArgs& a) { return a.stages; }
  __device__ __forceinline__ static uint32_t tmem_cols(const TcArgs& a) { return a.tn <= 128 ? 128u : 256u; }
};

// ---- thread-block cluster pieces of the split-K kernel
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  __syncwarp();  // one arrival a warp: its lanes may come from different branches
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of the same shared-memory location in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t dsmem_addr(uint32_t saddr, uint32_t rank) {
  uint32_t ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(saddr), "r"(rank));
  return ra;
}
__device__ __forceinline__ float ld_dsmem_f32(uint32_t cluster_addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr));
  return v;
}

__device__ __forceinline__ float silu_f(float x) { return x * (1.0f / (1.0f + __expf(-x))); }
// bf16 outputs: the square of relu (EPI_RELU2_BF16), tanh GELU (EPI_GELU_BF16) or the value itself
__device__ __forceinline__ float act_f(float v, int epi) {
  if (epi == EPI_GELU_BF16) return gelu_tanh_fast(v);
  if (epi != EPI_RELU2_BF16) return v;
  v = fmaxf(v, 0.f);
  return v * v;
}

// The way out of an accumulator.  Eight warps share a tile: warp w owns the tensor-memory lanes 32 (w % 4) .. + 31, one feature
// a lane, and every other run of 16 tokens, so that each scheduler has two warps to hide the tensor-memory loads and the
// shuffles of one another.  Values leave straight from the registers: for bf16, two neighbouring lanes trade a token, so that a
// store holds two neighbouring features and a warp writes whole 32-byte sectors.  SwiGLU: gates sit in lanes with
// (lane & 8) == 0, their up partners eight lanes higher; such a pair trades a token the same way, so that both compute.
// With four warps and rows staged through shared memory for 16-byte stores, 32 tokens took 1.2 us of a tile's exposed tail.
constexpr int EPI_WARPS = 8;
constexpr int TC_THREADS = 64 + 32 * EPI_WARPS;

template <int EPI>
__device__ __forceinline__ void store_tokens(const TcArgs& a, uint32_t tmem, void* out, int64_t feat0, int lane, int half, float bias_v, int64_t row0,
                                             int rows, bool any) {
  const bool feat_ok = feat0 + lane < a.N;
  const int64_t ldo = a.ldo;
#pragma unroll 1
  for (int c0 = 16 * half; c0 < rows; c0 += 32) {
    uint32_t r[16];
    if (any) {
      tc::ld16(tmem + (uint32_t)c0, r);
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) r[j] = 0u;
    }
    const int here = feat_ok ? min(16, rows - c0) : 0;
    float v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]) + bias_v;
    if constexpr (EPI == EPI_PARTIAL_F32 || EPI == EPI_BIAS_F32) {
      float* o = reinterpret_cast<float*>(out) + (row0 + c0) * ldo + feat0 + lane;
#pragma unroll
      for (int j = 0; j < 16; ++j, o += ldo)
        if (j < here) *o = v[j];
    } else if constexpr (EPI == EPI_SWIGLU_BF16) {
      const bool up = (lane & 8) != 0, odd = (lane & 1) != 0;
      const int first = (odd ? 2 : 0) + (up ? 1 : 0);   // of every four tokens
      bf16* o = reinterpret_cast<bf16*>(out) + (row0 + c0 + first) * ldo + feat0 / 2 + (lane >> 4) * 8 + (lane & 6);
#pragma unroll
      for (int j = 0; j < 16; j += 4, o += 4 * ldo) {
        float h[2];   // of tokens j + up and j + 2 + up
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float keep = up ? v[j + 2 * i + 1] : v[j + 2 * i];
          const float got = __shfl_xor_sync(0xffffffffu, up ? v[j + 2 * i] : v[j + 2 * i + 1], 8);
          h[i] = silu_f(up ? got : keep) * (up ? keep : got);
        }
        const float got = __shfl_xor_sync(0xffffffffu, odd ? h[0] : h[1], 1);
        if (j + first < here) *reinterpret_cast<uint32_t*>(o) = odd ? pack_bf16(got, h[1]) : pack_bf16(h[0], got);
      }
    } else {
      const bool odd = (lane & 1) != 0;
      const int first = odd ? 1 : 0;                    // of every two tokens
      bf16* o = reinterpret_cast<bf16*>(out) + (row0 + c0 + first) * ldo + feat0 + (lane & 30);
#pragma unroll
      for (int j = 0; j < 16; j += 2, o += 2 * ldo) {
        const float v0 = act_f(v[j], EPI), v1 = act_f(v[j + 1], EPI);
        const float got = __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 1);
        if (j + first < here) *reinterpret_cast<uint32_t*>(o) = odd ? pack_bf16(got, v1) : pack_bf16(v0, got);
      }
    }
  }
}
// tmem: the accumulator's first column at this warp's lanes; row0, rows: the tile's tokens; any: whether anything was accumulated
__device__ __forceinline__ void store_tile(const TcArgs& a, uint32_t tmem, void* out, int64_t feat0, int lane, int half, const float* bias, int64_t row0,
                                           int rows, bool any) {
  const float b = (bias && feat0 + lane < a.N && a.epi != EPI_PARTIAL_F32) ? bias[feat0 + lane] : 0.f;
  switch (a.epi) {
    case EPI_PARTIAL_F32:
    case EPI_BIAS_F32: return store_tokens<EPI_BIAS_F32>(a, tmem, out, feat0, lane, half, b, row0, rows, any);
    case EPI_SWIGLU_BF16: return store_tokens<EPI_SWIGLU_BF16>(a, tmem, out, feat0, lane, half, b, row0, rows, any);
    case EPI_RELU2_BF16: return store_tokens<EPI_RELU2_BF16>(a, tmem, out, feat0, lane, half, b, row0, rows, any);
    case EPI_GELU_BF16: return store_tokens<EPI_GELU_BF16>(a, tmem, out, feat0, lane, half, b, row0, rows, any);
    default: return store_tokens<EPI_BIAS_BF16>(a, tmem, out, feat0, lane, half, b, row0, rows, any);
  }
}

// Second half of the cluster split-K epilogue, run by the four epilogue warps of every CTA after the
// cluster barrier: this CTA finishes tokens [rank * 32/KS, (rank+1) * 32/KS) of the tile.  All loads of
// the peers' tiles are issued before the first add, and the sum runs in split order, so the result
// equals what the slab consumer kernels compute.
template <int KS>
__device__ __forceinline__ void cluster_finish(const TcArgs& a, uint8_t* smem, int q, int lane, int col0, int row0,
                                               bool epi_ok) {
  constexpr int TPR = 32 / KS;  // tokens this CTA finishes
  const uint32_t cr = cluster_ctarank();
  const int64_t feat = (int64_t)col0 + q * 32 + lane;
  const bool feat_ok = feat < a.N;
  const int j0 = (int)cr * TPR;
  const uint32_t soff = smem_u32(smem) + (uint32_t)(j0 * BM + q * 32 + lane) * 4u;
  float v[TPR];
  {
    float t[KS][TPR];
#pragma unroll
    for (int rr = 0; rr < KS; ++rr) {
      const uint32_t ra = dsmem_addr(soff, (uint32_t)rr);
#pragma unroll
      for (int jj = 0; jj < TPR; ++jj) t[rr][jj] = ld_dsmem_f32(ra + (uint32_t)jj * (BM * 4u));
    }
#pragma unroll
    for (int jj = 0; jj < TPR; ++jj) {
      v[jj] = 0.f;
#pragma unroll
      for (int rr = 0; rr < KS; ++rr) v[jj] += t[rr][jj];  // split order
    }
  }
  if (!a.fuse_qkv) {
    if (feat_ok && epi_ok) {
#pragma unroll
      for (int jj = 0; jj < TPR; ++jj) {
        const int64_t grow = (int64_t)row0 + j0 + jj;
        if (grow < a.M) reinterpret_cast<float*>(a.out)[grow * a.ldo + feat] = v[jj];
      }
    }
    return;
  }
  // ---- q|k|v: bias, RoPE on interleaved pairs, q to its buffer, k / v into the cache.
  // Lane t < TPR looks up token t's position and cache row once; everyone reads them by shuffle.
  const QkvPostArgs& p = a.qp;
  const int hd = p.hd, nq = p.nh * hd, nkv = p.kvh * hd;
  int m_rpos = -1;          // RoPE table row, -1: row outside the launch or a bad index
  long long m_crb = 0;      // cache row of kv head 0
  const int64_t head_stride = p.kv.block_table ? p.kv.page : p.kv.contiguous_len;
  if (lane < TPR) {
    const int64_t grow = (int64_t)row0 + j0 + lane;
    if (grow < a.M) {
      const int b = (int)(grow / p.S), sidx = (int)(grow % p.S);
      const int pos = p.pos0[b] + sidx, rpos = pos + p.rope_shift;
      if (pos < 0 || pos >= p.kv_capacity || rpos < 0 || rpos >= p.max_seq) {
        atomicExch(p.status, KS_BAD_INDEX);
      } else {
        m_rpos = rpos;
        if (p.kv.block_table) {
          const int page = p.kv.block_table[(int64_t)b * p.kv.max_pages + pos / p.kv.page];
          m_crb = ((long long)page * p.kvh) * p.kv.page + pos % p.kv.page;
        } else {
          m_crb = ((long long)b * p.kvh) * p.kv.contiguous_len + pos;
        }
      }
    }
  }
  const int col = (int)feat;
  const bool rot = col < nq + nkv;
  const int e = rot ? col % hd : (col - nq - nkv) % hd;
  const int hkv = col < nq ? 0 : (rot ? (col - nq) / hd : (col - nq - nkv) / hd);
  const float bias_v = (p.bias && feat_ok) ? p.bias[feat] : 0.f;
  int rpos[TPR];
  long long crb[TPR];
  float cs[TPR], sn[TPR];
#pragma unroll
  for (int jj = 0; jj < TPR; ++jj) {
    rpos[jj] = __shfl_sync(0xffffffffu, m_rpos, jj);
    crb[jj] = __shfl_sync(0xffffffffu, m_crb, jj);
  }
#pragma unroll
  for (int jj = 0; jj < TPR; ++jj) {
    cs[jj] = 1.f;
    sn[jj] = 0.f;
    if (rot && feat_ok && rpos[jj] >= 0) {
      cs[jj] = p.cosT[(int64_t)rpos[jj] * hd + e];
      sn[jj] = p.sinT[(int64_t)rpos[jj] * hd + e];
    }
  }
#pragma unroll
  for (int jj = 0; jj < TPR; ++jj) {
    const float x = v[jj] + bias_v;
    const float pr = __shfl_xor_sync(0xffffffffu, x, 1);  // the other element of the pair
    if (!feat_ok || !epi_ok || rpos[jj] < 0) continue;
    const int64_t grow = (int64_t)row0 + j0 + jj;
    if (rot) {
      const float r = (e & 1) ? rope_odd(cs[jj], sn[jj], pr, x) : rope_even(cs[jj], sn[jj], x, pr);
      if (col < nq)
        reinterpret_cast<bf16*>(p.q_out)[grow * nq + col] = __float2bfloat16_rn(r);
      else
        reinterpret_cast<bf16*>(p.kv.k)[(crb[jj] + hkv * head_stride) * hd + e] = __float2bfloat16_rn(r);
    } else {
      reinterpret_cast<bf16*>(p.kv.v)[(crb[jj] + hkv * head_stride) * hd + e] = __float2bfloat16_rn(x);
    }
  }
}

// CL = 1 (decode tile only): the CTAs of one feature tile that split K form a thread-block cluster
// along z and sum their accumulators through distributed shared memory, each finishing 32 / ksplit
// of the tile's tokens, so the launch leaves one finished slab (or finished q / k / v) instead of
// ksplit partial slabs for the next kernel to add up.
template <int TN, int CL>
__global__ void __launch_bounds__(TC_THREADS) linear_tc_kernel(const __grid_constant__ CUtensorMap tmW,
                                                         const __grid_constant__ CUtensorMap tmX, TcArgs a) {
  static_assert(CL == 0 || TN == 32, "the cluster reduction is written for the decode tile");
  using C = TcCfg<TN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tn = C::tn(a), stages = C::stages(a), stage_bytes = A_BYTES + tn * 128;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + stages * stage_bytes);
  uint64_t* empty = full + stages;
  uint64_t* tmem_full = empty + stages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_full + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Tile order: with several token tiles the CTAs walk groups of 8 token tiles per feature tile,
  // so a wave touches ~8 x-tiles and ~18 W-tiles instead of one x-tile and every W-tile; without
  // this a weight matrix larger than L2 is re-streamed from HBM once per token tile.
  int tile_n = blockIdx.x, tile_m = blockIdx.y;
  if (gridDim.y > 1) {
    constexpr int GROUP_M = 8;
    const int lin = blockIdx.x + gridDim.x * blockIdx.y;
    const int per_group = GROUP_M * gridDim.x;
    const int group = lin / per_group;
    const int first_m = group * GROUP_M;
    const int group_rows = min(GROUP_M, (int)gridDim.y - first_m);
    const int in_group = lin - group * per_group;
    tile_m = first_m + in_group % group_rows;
    tile_n = in_group / group_rows;
  }
  const int col0 = tile_n * BM;              // first output feature of the tile
  const int row0 = tile_m * tn;              // first token of the tile
  const int split = blockIdx.z;
  const int rows_valid = (int)min((int64_t)tn, a.M - row0);
  const int nkb_total = (int)((a.K + BK - 1) / BK);
  const int kb0 = split * a.kb_per_split;
  const int nkb = max(0, min(a.kb_per_split, nkb_total - kb0));

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tmem_full, 1);
    fence_barrier_init();
  }
  if (warp == 1) tc::alloc_then_launch_dependents(tmem_slot, C::tmem_cols(a));
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem_base = *tmem_slot;

  bool epi_ok = true;
  if (warp == 0) {
    if (tc::elect_one()) {
      tma_prefetch_desc(&tmW);
      tma_prefetch_desc(&tmX);
      const uint64_t pol_w = policy_evict_first();
      const uint64_t pol_x = policy_evict_last();
      const int pre = min(stages, nkb);
      if (!a.early_w) pdl_wait();  // the launch before may be the one that writes them
      for (int kb = 0; kb < pre; ++kb) {
        uint8_t* st = smem + kb * stage_bytes;
        mbar_expect_tx(&full[kb], stage_bytes);
        const int k = (kb0 + kb) * BK;
        tma_load_2d_hint(st, &tmW, &full[kb], col0, k, pol_w);
        tma_load_2d_hint(st + A_BYTES / 2, &tmW, &full[kb], col0 + 64, k, pol_w);
      }
      pdl_wait();
      for (int kb = 0; kb < pre; ++kb)
        tma_load_2d_hint(smem + kb * stage_bytes + A_BYTES, &tmX, &full[kb], (kb0 + kb) * BK, row0, pol_x);
      for (int kb = pre, s = 0, lap = 0; kb < nkb; ++kb) {
        if (!mbar_wait(&empty[s], lap & 1, a.status)) break;
        uint8_t* st = smem + s * stage_bytes;
        mbar_expect_tx(&full[s], stage_bytes);
        const int k = (kb0 + kb) * BK;
        tma_load_2d_hint(st, &tmW, &full[s], col0, k, pol_w);
        tma_load_2d_hint(st + A_BYTES / 2, &tmW, &full[s], col0 + 64, k, pol_w);
        tma_load_2d_hint(st + A_BYTES, &tmX, &full[s], k, row0, pol_x);
        if (++s == stages) s = 0, ++lap;
      }
    }
  } else if (warp == 1) {
    if (nkb > 0 && tc::elect_one()) {
      // instruction descriptor: D f32, A/B bf16, A MN-major, B K-major, N = tn, M = 128
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | ((uint32_t)(tn >> 3) << 17) |
                             ((uint32_t)(BM >> 4) << 24);
      const uint32_t smem_base = smem_u32(smem);
      bool ok = true;
      for (int kb = 0, s = 0, lap = 0; kb < nkb && ok; ++kb) {
        ok = mbar_wait(&full[s], lap & 1, a.status);
        if (!ok) break;
        tc::fence_after();
        const uint32_t sa = smem_base + s * stage_bytes;
        const uint32_t sb = sa + A_BYTES;
        // A: 16 k-rows of 128 bytes = two 8-row swizzle atoms 1024 B apart (SBO); the second
        //    64-feature box is 8192 B further (LBO).  B: rows of 128 B, 8-row atoms 1024 B apart.
        tc::umma4_bf16_ss<tc::MN_MAJOR, tc::K_MAJOR>(tmem_base, tc::desc_lo(sa, A_BYTES / 2), tc::desc_lo(sb, 16), tc::desc_hi(1024), idesc, kb > 0);
        tc::commit(&empty[s]);  // stage is free once these MMAs have read it
        if (++s == stages) s = 0, ++lap;
      }
      if (ok) tc::commit(tmem_full);
    }
  } else {
    // ---------------- epilogue warps 2..9; TMEM lanes 32*(warp%4) .. +31
    const int q = warp & 3, half = (warp - 2) >> 2;
    bool ok = true;
    if (nkb > 0) {
      ok = mbar_wait_warp(tmem_full, 0, a.status);
      tc::fence_after();
    }
    pdl_wait();
    if constexpr (CL == 1) {
      // own partial tile -> shared memory as [token][feature] f32 (the pipeline stages are free by now)
      if (half == 0) {
        uint32_t r[32];
        if (ok && nkb > 0) {
          tc::ld32(tmem_base + ((uint32_t)(q * 32) << 16), r);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = 0u;
        }
        float* stg = reinterpret_cast<float*>(smem);
#pragma unroll
        for (int j = 0; j < 32; ++j) stg[j * BM + q * 32 + lane] = __uint_as_float(r[j]);
      }
      epi_ok = ok;
    } else if (ok) {
      void* out = reinterpret_cast<uint8_t*>(a.out) + (a.epi == EPI_PARTIAL_F32 ? (size_t)split * a.split_stride * 4 : 0);
      store_tile(a, tmem_base + ((uint32_t)(q * 32) << 16), out, (int64_t)col0 + q * 32, lane, half, a.bias, row0, rows_valid, nkb > 0);
    }
  }
  (void)epi_ok;
  if constexpr (CL == 1) {
    (void)rows_valid;
    __syncwarp();
    cluster_sync_all();  // every CTA of the cluster has staged its partial tile
    if (warp >= 2 && warp < 6) {
      const int q = warp & 3;
      switch (gridDim.z) {
        case 2: cluster_finish<2>(a, smem, q, lane, col0, row0, epi_ok); break;
        case 4: cluster_finish<4>(a, smem, q, lane, col0, row0, epi_ok); break;
        default: cluster_finish<8>(a, smem, q, lane, col0, row0, epi_ok); break;
      }
    }
    cluster_sync_all();  // nobody leaves while a peer may still read its tile
  }
  __syncwarp();  // the lanes of a role come back together: what follows is warp-collective
  tc::fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after();
    tc::dealloc(tmem_base, C::tmem_cols(a));
  }
}

// ---- persistent variant for steps of more than 64 tokens ------------------------------------------
// One CTA per SM walks its share of the output tiles (or of their pieces along K).  The accumulator is
// double-buffered in TMEM (2 x 256 columns), so the epilogue warps drain tile j while the MMA warp
// already accumulates tile j + 1 and the TMA ring keeps running across tile boundaries; the per-tile
// cost becomes max(main loop, epilogue) instead of their sum.  What bounds it: up to 256 tokens the
// weights' way from HBM, at equal work of all SMs, so a step is slow when 32 of them have all of it: hence
// the pieces along K, and tiles of the step's own size (a multiple of 16 tokens), which leave room for a deep
// ring.  135 tokens of 4096 x 28672: 42 us (67 us in one-tile CTAs of 256 tokens), of which 35 us are the
// weights' time out of HBM.
struct PersistCfg {
  static constexpr int TN = 256;                          // most tokens of a tile
  static constexpr int MAX_STAGES = 8;
  static constexpr int FIXED = 1024 + 256;
  static constexpr int TMEM_COLS = 512;
  static constexpr int stage_bytes(int tn) { return A_BYTES + tn * 128; }
  static constexpr int stages(int tn) {
    const int n = (SMEM - FIXED) / stage_bytes(tn);
    return n < MAX_STAGES ? n : MAX_STAGES;
  }
  static constexpr int SMEM = kAllSmem;
};

// GROUPED: the weights are `groups` stacked matrices (3-D tensor map, third coordinate = group, e.g. the
// routed experts of a MoE layer) and group g owns the rows [row_offsets[g], row_offsets[g+1]) of x and of the
// output; the offsets are device data from an earlier kernel of the step.  The tile list is then built on
// the device: token tiles are numbered group by group (a group's last tile may be ragged), and a tile loads a
// full box of rows (the surplus belongs to the next group or is out of range) but stores only its own.
constexpr int kMaxGroups = 256;
constexpr int kMaxPersistCtas = 256;
// Per-CTA list "token tiles ahead of each group" of the grouped launches.  The kernel's shared memory is full
// (the stages of its ring), so each CTA keeps its copy in global memory, where it stays in L1.
static __device__ int g_first_tile[kMaxPersistCtas][kMaxGroups + 1];

template <bool GROUPED>
__global__ void __launch_bounds__(TC_THREADS) linear_tc_persist_kernel(const __grid_constant__ CUtensorMap tmW,
                                                                 const __grid_constant__ CUtensorMap tmX, TcArgs a,
                                                                 int tiles_n, int tiles_m) {
  using C = PersistCfg;
  const int TN = GROUPED ? C::TN : a.tn, STAGES = C::stages(TN), stage_bytes = C::stage_bytes(TN);
  int* const s_first_tile = g_first_tile[blockIdx.x % kMaxPersistCtas];  // this CTA's copy (grouped launches only)
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * stage_bytes);
  uint64_t* empty = full + STAGES;
  uint64_t* tmem_full = empty + STAGES;   // [2]
  uint64_t* tmem_empty = tmem_full + 2;      // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nkb_total = (int)((a.K + BK - 1) / BK);
  if constexpr (GROUPED) {
    pdl_wait();  // the row offsets come from an earlier kernel of the step
    if (threadIdx.x == 0) {
      int acc = 0;
      for (int g = 0; g < a.groups; ++g) {
        s_first_tile[g] = acc;
        acc += (a.row_offsets[g + 1] - a.row_offsets[g] + TN - 1) / TN;
      }
      s_first_tile[a.groups] = acc;
      __threadfence_block();
    }
    __syncthreads();
    tiles_m = s_first_tile[a.groups];
  }
  // a tile is cut into a.ksplit pieces along K, whose sums go to slabs of their own; a whole output tile is one piece
  const int plane = tiles_n * tiles_m, total_tiles = GROUPED ? plane : plane * a.ksplit;
  auto k_range = [&](int lin, int& kb0, int& nkb) {
    kb0 = GROUPED ? 0 : lin / plane * a.kb_per_split;
    nkb = GROUPED ? nkb_total : max(0, min(a.kb_per_split, nkb_total - kb0));
  };
  // Dense: same tile order as the one-tile kernel, groups of 8 token tiles per feature tile.  Grouped:
  // feature tiles fastest, so the CTAs of a wave work on a few token tiles of one or two experts.
  // row0 = first row of the tile, rows_valid = rows of it that belong to the output, grp = weight matrix.
  auto tile_coords = [&](int lin, int& tile_n, int& row0, int& rows_valid, int& grp) {
    if constexpr (GROUPED) {
      const int gm = lin / tiles_n;
      tile_n = lin - gm * tiles_n;
      int lo = 0, hi = a.groups;  // the group g with s_first_tile[g] <= gm < s_first_tile[g + 1]
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (s_first_tile[mid] <= gm) lo = mid;
        else hi = mid;
      }
      grp = lo;
      row0 = a.row_offsets[lo] + (gm - s_first_tile[lo]) * TN;
      rows_valid = min(TN, a.row_offsets[lo + 1] - row0);
    } else {
      constexpr int GROUP_M = 8;
      const int per_group = GROUP_M * tiles_n;
      lin %= plane;
      const int group = lin / per_group;
      const int first_m = group * GROUP_M;
      const int group_rows = min(GROUP_M, tiles_m - first_m);
      const int in_group = lin - group * per_group;
      const int tile_m = first_m + in_group % group_rows;
      tile_n = in_group / group_rows;
      row0 = tile_m * TN;
      rows_valid = (int)min((int64_t)TN, a.M - row0);
      grp = 0;
    }
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], 1);
    }
    fence_barrier_init();
  }
  if (warp == 1) tc::alloc_then_launch_dependents(tmem_slot, (uint32_t)C::TMEM_COLS);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (tc::elect_one()) {
      tma_prefetch_desc(&tmW);
      tma_prefetch_desc(&tmX);
      const uint64_t pol_w = policy_evict_first();
      const uint64_t pol_x = policy_evict_last();
      int early = 0;   // stages whose weights were requested ahead of the stream dependency (no kernel of a step writes them)
      if constexpr (!GROUPED) {
        int tile_n, row0, rows_valid, grp, kb0, nkb;
        tile_coords(blockIdx.x, tile_n, row0, rows_valid, grp);
        k_range(blockIdx.x, kb0, nkb);
        early = a.early_w ? min(STAGES, nkb) : 0;
        for (int i = 0; i < early; ++i) {
          uint8_t* st = smem + i * stage_bytes;
          mbar_expect_tx(&full[i], stage_bytes);
          tma_load_2d_hint(st, &tmW, &full[i], tile_n * BM, (kb0 + i) * BK, pol_w);
          tma_load_2d_hint(st + A_BYTES / 2, &tmW, &full[i], tile_n * BM + 64, (kb0 + i) * BK, pol_w);
        }
      }
      pdl_wait();  // the activations come from the previous kernel
      int s = 0, lap = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        int tile_n, row0, rows_valid, grp, kb0, nkb;
        tile_coords(t, tile_n, row0, rows_valid, grp);
        k_range(t, kb0, nkb);
        const int col0 = tile_n * BM;
        for (int kb = 0; kb < nkb; ++kb) {
          if (lap > 0 && !mbar_wait(&empty[s], (lap - 1) & 1, a.status)) {
            ok = false;
            break;
          }
          uint8_t* st = smem + s * stage_bytes;
          const int k = (kb0 + kb) * BK;
          if (early > 0) {
            --early;
          } else {
            mbar_expect_tx(&full[s], stage_bytes);
            if constexpr (GROUPED) {
              tma_load_3d_hint(st, &tmW, &full[s], col0, k, grp, pol_x);  // an expert's weights serve several token tiles: keep them in L2
              tma_load_3d_hint(st + A_BYTES / 2, &tmW, &full[s], col0 + 64, k, grp, pol_x);
            } else {
              tma_load_2d_hint(st, &tmW, &full[s], col0, k, pol_w);
              tma_load_2d_hint(st + A_BYTES / 2, &tmW, &full[s], col0 + 64, k, pol_w);
            }
          }
          tma_load_2d_hint(st + A_BYTES, &tmX, &full[s], k, row0, pol_x);
          if (++s == STAGES) s = 0, ++lap;
        }
      }
    }
  } else if (warp == 1) {
    if (tc::elect_one()) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | ((uint32_t)(TN >> 3) << 17) |
                             ((uint32_t)(BM >> 4) << 24);
      const uint32_t smem_base = smem_u32(smem);
      int s = 0, lap = 0, j = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++j) {
        int kb0, nkb;
        k_range(t, kb0, nkb);
        const int buf = j & 1;
        if (j >= 2) {  // the epilogue must have drained this accumulator (tile j - 2)
          ok = mbar_wait(&tmem_empty[buf], ((j >> 1) - 1) & 1, a.status);
          if (!ok) break;
          tc::fence_after();
        }
        const uint32_t d_tmem = tmem_base + (uint32_t)(buf * C::TN);
        for (int kb = 0; kb < nkb; ++kb) {
          ok = mbar_wait(&full[s], lap & 1, a.status);
          if (!ok) break;
          tc::fence_after();
          const uint32_t sa = smem_base + s * stage_bytes;
          const uint32_t sb = sa + A_BYTES;
          tc::umma4_bf16_ss<tc::MN_MAJOR, tc::K_MAJOR>(d_tmem, tc::desc_lo(sa, A_BYTES / 2), tc::desc_lo(sb, 16), tc::desc_hi(1024), idesc, kb > 0);
          tc::commit(&empty[s]);
          if (++s == STAGES) s = 0, ++lap;
        }
        if (ok) tc::commit(&tmem_full[buf]);
      }
    }
  } else {
    // ---------------- epilogue warps 2..9; TMEM lanes 32*(warp%4) .. +31
    const int q = warp & 3, half = (warp - 2) >> 2;
    pdl_wait();  // the output buffer may still be read by the previous kernel
    int j = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < total_tiles; t += gridDim.x, ++j) {
      int tile_n, row0, rows_valid, grp, kb0, nkb;
      tile_coords(t, tile_n, row0, rows_valid, grp);
      k_range(t, kb0, nkb);
      const int col0 = tile_n * BM;
      const int buf = j & 1;
      if (ok) ok = mbar_wait_warp(&tmem_full[buf], (j >> 1) & 1, a.status);
      tc::fence_after();
      // grouped launches keep one bias row per group: [groups][N]
      void* const out = reinterpret_cast<uint8_t*>(a.out) + (GROUPED || a.epi != EPI_PARTIAL_F32 ? 0 : (size_t)(t / plane) * a.split_stride * 4);
      if (ok)
        store_tile(a, tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * C::TN), out, (int64_t)col0 + q * 32, lane, half,
                   a.bias ? a.bias + (int64_t)grp * a.N : nullptr, row0, rows_valid, nkb > 0);
      // every epilogue warp has read its part of the accumulator: hand the buffer back
      tc::fence_before();
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (warp == 2 && lane == 0) mbar_arrive(&tmem_empty[buf]);
    }
  }
  __syncwarp();  // the lanes of a role come back together: what follows is warp-collective
  tc::fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after();
    tc::dealloc(tmem_base, (uint32_t)C::TMEM_COLS);
  }
}

// ---- two-CTA variant of the persistent kernel (prefill, dense weights) -------------------------------
// A cluster of two CTAs on neighbouring SMs works on one 256-feature x 256-token output tile with
// tcgen05.mma.cta_group::2: each CTA stages its own 128 features of W (A operand) and its own 128 tokens of x
// (half of the B operand), the tensor cores of both SMs read both halves, and each CTA's tensor memory
// receives the accumulator rows of its own 128 features for all 256 tokens.  Per CTA a stage is 32 KB
// instead of 48 KB for the same tensor-core work, which takes the kernel off the shared-memory bandwidth
// limit of the one-CTA tile (48 KB written and read per 512 tensor cycles = 188 B/cycle against 128).
// Protocol: the bulk tensor loads of both CTAs complete on the LEADER's (even CTA's) `full` barrier (the
// cta_group::2 form of the load; no multicast: every CTA loads only what it alone needs); the leader's MMA
// thread issues for both and releases a stage by committing to the `empty` barrier of each CTA; finished
// accumulators are announced to both CTAs' epilogue warps the same way; the leader reuses an accumulator
// buffer once the epilogues of both CTAs have arrived on its `tmem_empty` barrier.
struct PairCfg {
  static constexpr int TN = 256;                          // most tokens per tile (both CTAs together), a multiple of 32
  static constexpr int MAX_STAGES = 10;
  static constexpr int FIXED = 1024 + 256;
  static constexpr int SMEM = kAllSmem;
  static constexpr int TMEM_COLS = 512;
  static constexpr int stage_bytes(int tn) { return A_BYTES + tn * 64; }   // this CTA's tn / 2 tokens x 64 k: 32 KB in all at 256 tokens
  static constexpr int stages(int tn) {
    const int n = (SMEM - FIXED) / stage_bytes(tn);
    return n < MAX_STAGES ? n : MAX_STAGES;
  }
};

constexpr uint32_t kPeerBitMask = 0xFEFFFFFFu;  // clears the bit that tells the two CTAs of a pair apart in a shared::cluster address

__device__ __forceinline__ void tma_load_2d_pair(void* dst, const void* tmap, uint64_t* leader_bar, int x, int y, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%3, %4}], [%2], %5;"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(leader_bar) & kPeerBitMask), "r"(x), "r"(y),
      "l"(policy)
      : "memory");
}
// arrives on the barrier at shared::cluster address `bar_cluster_addr` once every tcgen05 operation this thread
// has issued so far is complete
__device__ __forceinline__ void commit_pair(uint32_t bar_cluster_addr) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_cluster_addr) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_THREADS) linear_tc_pair_kernel(const __grid_constant__ CUtensorMap tmW,
                                                                                        const __grid_constant__ CUtensorMap tmX,
                                                                                        TcArgs a, int tiles_n, int tiles_m) {
  using C = PairCfg;
  const int TN = a.tn, STAGES = C::stages(TN), stage_bytes = C::stage_bytes(TN);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * stage_bytes);
  uint64_t* empty = full + STAGES;
  uint64_t* tmem_full = empty + STAGES;   // [2]
  uint64_t* tmem_empty = tmem_full + 2;      // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();   // 0: leader
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int total_tiles = tiles_n * tiles_m;  // tiles of 256 features x TN tokens
  const int nkb = (int)((a.K + BK - 1) / BK);
  auto tile_coords = [&](int lin, int& tile_n, int& tile_m) {
    constexpr int GROUP_M = 8;
    const int per_group = GROUP_M * tiles_n;
    const int group = lin / per_group;
    const int first_m = group * GROUP_M;
    const int group_rows = min(GROUP_M, tiles_m - first_m);
    const int in_group = lin - group * per_group;
    tile_m = first_m + in_group % group_rows;
    tile_n = in_group / group_rows;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], 2);  // the epilogues of both CTAs
    }
    fence_barrier_init();
  }
  if (warp == 1) tc::alloc_then_launch_dependents<2>(tmem_slot, (uint32_t)C::TMEM_COLS);
  tc::fence_before();
  cluster_sync_all();  // both CTAs' barriers are initialised before any remote arrival, and both allocations are done
  tc::fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (tc::elect_one()) {
      tma_prefetch_desc(&tmW);
      tma_prefetch_desc(&tmX);
      const uint64_t pol_w = policy_evict_first();
      const uint64_t pol_x = policy_evict_last();
      // stages whose weights are requested ahead of the stream dependency (no kernel of a step writes them)
      int early = 0;
      if (a.early_w && pair < total_tiles) {
        int tile_n, tile_m;
        tile_coords(pair, tile_n, tile_m);
        early = min(STAGES, nkb);
        for (int i = 0; i < early; ++i) {
          uint8_t* st = smem + i * stage_bytes;
          if (rank == 0) mbar_expect_tx(&full[i], 2 * stage_bytes);
          tma_load_2d_pair(st, &tmW, &full[i], tile_n * 256 + (int)rank * BM, i * BK, pol_w);
          tma_load_2d_pair(st + A_BYTES / 2, &tmW, &full[i], tile_n * 256 + (int)rank * BM + 64, i * BK, pol_w);
        }
      }
      pdl_wait();  // the activations come from the previous kernel
      int s = 0, lap = 0;
      bool ok = true;
      for (int t = pair; t < total_tiles && ok; t += n_pairs) {
        int tile_n, tile_m;
        tile_coords(t, tile_n, tile_m);
        const int col0 = tile_n * 256 + (int)rank * BM, row0 = tile_m * TN + (int)rank * (TN / 2);
        for (int kb = 0; kb < nkb; ++kb) {
          if (lap > 0 && !mbar_wait(&empty[s], (lap - 1) & 1, a.status)) {
            ok = false;
            break;
          }
          uint8_t* st = smem + s * stage_bytes;
          const int k = kb * BK;
          if (early > 0) {
            --early;
          } else {
            if (rank == 0) mbar_expect_tx(&full[s], 2 * stage_bytes);  // this CTA's stage and the peer's
            tma_load_2d_pair(st, &tmW, &full[s], col0, k, pol_w);
            tma_load_2d_pair(st + A_BYTES / 2, &tmW, &full[s], col0 + 64, k, pol_w);
          }
          tma_load_2d_pair(st + A_BYTES, &tmX, &full[s], k, row0, pol_x);
          if (++s == STAGES) s = 0, ++lap;
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && tc::elect_one()) {
      // D f32, A/B bf16, A MN-major, B K-major, N = TN tokens, M = 256 features over the pair
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
      const uint32_t smem_base = smem_u32(smem);
      int s = 0, lap = 0, j = 0;
      bool ok = true;
      for (int t = pair; t < total_tiles && ok; t += n_pairs, ++j) {
        const int buf = j & 1;
        if (j >= 2) {  // both epilogues must have drained this accumulator (tile j - 2)
          ok = mbar_wait(&tmem_empty[buf], ((j >> 1) - 1) & 1, a.status);
          if (!ok) break;
          tc::fence_after();
        }
        const uint32_t d_tmem = tmem_base + (uint32_t)(buf * C::TN);
        for (int kb = 0; kb < nkb; ++kb) {
          ok = mbar_wait(&full[s], lap & 1, a.status);
          if (!ok) break;
          tc::fence_after();
          const uint32_t sa = smem_base + s * stage_bytes;
          const uint32_t sb = sa + A_BYTES;
          tc::umma4_bf16_ss<tc::MN_MAJOR, tc::K_MAJOR, 2>(d_tmem, tc::desc_lo(sa, A_BYTES / 2), tc::desc_lo(sb, 16), tc::desc_hi(1024), idesc, kb > 0);
          // the stage is free in BOTH CTAs once these MMAs have read it
          commit_pair(smem_u32(&empty[s]));
          commit_pair(dsmem_addr(smem_u32(&empty[s]), 1));
          if (++s == STAGES) s = 0, ++lap;
        }
        if (ok) {
          commit_pair(smem_u32(&tmem_full[buf]));
          commit_pair(dsmem_addr(smem_u32(&tmem_full[buf]), 1));
        }
      }
    }
  } else {
    // ---------------- epilogue warps 2..9 of each CTA; TMEM lanes 32*(warp%4) .. +31 = this CTA's 128 features
    const int q = warp & 3, half = (warp - 2) >> 2;
    const uint32_t leader_tmem_empty0 = dsmem_addr(smem_u32(&tmem_empty[0]), 0);
    pdl_wait();  // the output buffer may still be read by the previous kernel
    int j = 0;
    bool ok = true;
    for (int t = pair; t < total_tiles; t += n_pairs, ++j) {
      int tile_n, tile_m;
      tile_coords(t, tile_n, tile_m);
      const int col0 = tile_n * 256 + (int)rank * BM, row0 = tile_m * TN;
      const int rows_valid = (int)min((int64_t)TN, a.M - row0);
      const int buf = j & 1;
      if (ok) ok = mbar_wait_warp(&tmem_full[buf], (j >> 1) & 1, a.status);
      tc::fence_after();
      if (ok)
        store_tile(a, tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * C::TN), a.out, (int64_t)col0 + q * 32, lane, half,
                   a.bias, row0, rows_valid, true);
      // every epilogue warp of this CTA has read its part of the accumulator: tell the leader
      tc::fence_before();
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (warp == 2 && lane == 0) mbar_arrive_cluster(leader_tmem_empty0 + (uint32_t)buf * 8u);
    }
  }
  __syncwarp();
  tc::fence_before();
  __syncthreads();
  cluster_sync_all();  // nobody leaves (or frees tensor memory) while the peer may still use this CTA's memory or barriers
  if (warp == 1) {
    tc::fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)C::TMEM_COLS) : "memory");
  }
}

template <int TN>
int launch_tn(Ctx* c, const LinearBf16Plan& plan, const CUtensorMap& tmX, const TcArgs& a, dim3 grid) {
  using C = TcCfg<TN>;
  static bool attr_set = false;
  if (!attr_set) {
    RB_CUDA(cudaFuncSetAttribute(linear_tc_kernel<TN, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
    attr_set = true;
  }
  RB_CUDA(launch_k(linear_tc_kernel<TN, 0>, grid, dim3(TC_THREADS), (size_t)C::SMEM, c->stream, c->use_pdl, plan.tmW, tmX, a));
  ++g_launch_total;
  ++g_route_launches[ROUTE_LINEAR_TILE];
  return REWB200_OK;
}

}  // namespace

bool linear_tc_cluster_ok(Ctx* c, const LinearBf16Plan& plan, int64_t M, int ksplit) {
  return c->splitk_cluster != 0 && c->linear_impl == 2 && plan.groups == 0 && M >= 1 && M <= 32 &&
         (ksplit == 2 || ksplit == 4 || ksplit == 8);
}

int linear_tc_cluster_launch(Ctx* c, const LinearBf16Plan& plan, const bf16* x, int64_t ldx, int64_t M, int ksplit,
                             float* out, int64_t ldo, const QkvPostArgs* fuse_qkv) {
  RB_REQUIRE(linear_tc_cluster_ok(c, plan, M, ksplit), "cluster split-K: at most 32 rows and 2, 4 or 8 splits");
  RB_REQUIRE(ldx % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0, "bf16 Linear: activations must be 16-byte aligned rows");
  using C = TcCfg<32>;
  CUtensorMap tmX;
  RB_TRY(make_tmap_2d_bf16(&tmX, x, (uint64_t)plan.K, (uint64_t)M, (uint64_t)ldx * 2, 64, 32));
  TcArgs a;
  memset(&a, 0, sizeof(a));
  a.M = M;
  a.N = plan.N;
  a.K = plan.K;
  const int nkb = (int)((plan.K + BK - 1) / BK);
  a.kb_per_split = (nkb + ksplit - 1) / ksplit;
  a.epi = EPI_PARTIAL_F32;
  a.out = out;
  a.ldo = ldo;
  a.split_stride = 0;
  a.bias = nullptr;
  a.status = c->d_status;
  a.early_w = plan.early_w;
  if (fuse_qkv) {
    RB_REQUIRE(fuse_qkv->act_dtype == REWB200_BF16 && fuse_qkv->hd % 2 == 0 &&
                   (int64_t)(fuse_qkv->nh + 2 * fuse_qkv->kvh) * fuse_qkv->hd == plan.N,
               "fused q|k|v epilogue: bf16 activations and a weight of nq + 2 nkv columns");
    a.fuse_qkv = 1;
    a.qp = *fuse_qkv;
  }
  static bool attr_set = false;
  if (!attr_set) {
    RB_CUDA(cudaFuncSetAttribute(linear_tc_kernel<32, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
    attr_set = true;
  }
  dim3 grid((unsigned)((plan.N + BM - 1) / BM), 1u, (unsigned)ksplit);
  RB_CUDA(launch_k_cluster(linear_tc_kernel<32, 1>, grid, dim3(TC_THREADS), (size_t)C::SMEM, c->stream, c->use_pdl,
                           dim3(1, 1, (unsigned)ksplit), plan.tmW, tmX, a));
  ++g_launch_total;
  return REWB200_OK;
}

// Grouped launch (plan.groups stacked weight matrices, rows of group g = [row_offsets[g], row_offsets[g+1]) of
// x / out, bias [groups][N] or NULL): the persistent kernel with its tile list built on the device.  For
// groups of prefill size (MoE experts with hundreds of rows each); smaller ones stay on the HBM-bound
// mma.sync kernel of linear_bf16.cu.
int linear_tc_grouped_launch(Ctx* c, const LinearBf16Plan& plan, const bf16* x, int64_t ldx, int64_t M, int epi, void* out,
                             int64_t ldo, const float* bias, const int* row_offsets) {
  RB_REQUIRE(plan.groups >= 1 && plan.groups <= kMaxGroups && row_offsets != nullptr, "grouped tcgen05 Linear: 1..256 groups and row offsets");
  RB_REQUIRE(ldx % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0, "bf16 Linear: activations must be 16-byte aligned rows");
  RB_REQUIRE(epi != EPI_PARTIAL_F32, "grouped Linear does not split K");
  RB_REQUIRE(epi != EPI_SWIGLU_BF16 || plan.N % 16 == 0, "SwiGLU epilogue needs interleaved width % 16 == 0");
  if (M == 0) return REWB200_OK;
  CUtensorMap tmX;
  RB_TRY(make_tmap_2d_bf16(&tmX, x, (uint64_t)plan.K, (uint64_t)M, (uint64_t)ldx * 2, 64, PersistCfg::TN));
  TcArgs a;
  memset(&a, 0, sizeof(a));
  a.M = M;
  a.N = plan.N;
  a.K = plan.K;
  a.kb_per_split = (int)((plan.K + BK - 1) / BK);
  a.epi = epi;
  a.out = out;
  a.ldo = ldo;
  a.split_stride = M * ldo;
  a.bias = bias;
  a.status = c->d_status;
  a.row_offsets = row_offsets;
  a.groups = plan.groups;
  a.tn = PersistCfg::TN;
  static bool attr_set = false;
  if (!attr_set) {
    RB_CUDA(cudaFuncSetAttribute(linear_tc_persist_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, PersistCfg::SMEM));
    attr_set = true;
  }
  const int tiles_n = (int)((plan.N + BM - 1) / BM);
  // at most ceil(M / TN) + groups token tiles exist; one CTA per SM walks them
  const int64_t max_tiles = (int64_t)tiles_n * ((M + PersistCfg::TN - 1) / PersistCfg::TN + plan.groups);
  const int ctas = (int)std::min<int64_t>(std::min<int64_t>(max_tiles, c->sm_count), kMaxPersistCtas);
  RB_CUDA(launch_k(linear_tc_persist_kernel<true>, dim3((unsigned)ctas), dim3(TC_THREADS), (size_t)PersistCfg::SMEM, c->stream, c->use_pdl,
                   plan.tmW, tmX, a, tiles_n, 0));
  ++g_launch_total;
  return REWB200_OK;
}

// Loads this file's module on the current device and prepares the decode-size kernel (M <= 32), so that a
// later launch of it neither loads code nor changes function attributes.
int linear_tc_preload() {
  RB_CUDA(cudaFuncSetAttribute(linear_tc_kernel<32, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcCfg<32>::SMEM));
  cudaFuncAttributes fa;
  RB_CUDA(cudaFuncGetAttributes(&fa, linear_tc_kernel<32, 0>));
  return REWB200_OK;
}

// More tiles of up to 160 tokens than SMs: two CTAs an SM, since those of a second wave start as the first ones leave
// (4096 x 28672: 135 tokens 42 us, 48 in the persistent kernel).  Otherwise the persistent kernel.
static bool tc_two_per_sm(Ctx* c, int tn, int64_t tiles) { return tn <= 160 && tiles > c->sm_count; }

// Token tiles of a step of 65 to 1023 rows whose K is not cut: of one CTA (*tn tokens) or of a pair (*pair_tn, else 0).  More tiles
// than the rows need fill SMs that a launch would leave empty and even out its last wave.  What a tile of one, or of a pair, costs
// a block of 64 k: what arrives at an SM (weights and tokens; a pair shares the tokens), 0.2 us from its latency up; measured over
// 4096 x 28672, 4096 x 6144, 4096 x 4096, 14336 x 4096, 2048 x 11264 and 2048 x 2048 at 100 to 900 rows.  Us a launch, before (as few tiles
// of one CTA as hold the rows) / now: 14336 x 4096 at 333 rows 56.4 / 45.5, 512 rows 74.4 / 51.4; 4096 x 4096 at 333 rows 20.1 / 16.0; 4096 x 6144 at
// 333 rows 21.2 / 17.4, 900 rows 45.6 / 34.9; 4096 x 28672 at 256 rows 55.7 / 51.9, 512 rows 103 / 94; 2048 x 11264 at 512 rows 28.1 / 21.1.
// Two CTAs an SM (tc_two_per_sm) cost less than that in one wave or two, where the second CTA of an SM fills the pauses of the first, and
// more than that in three, where every wave begins and ends by itself.  So pairs must be ahead of them by 1.3 % (us, pairs / two an SM:
// 4096 x 28672 at 81 to 96 rows 44.4 / 39.8, at 113 to 128 44.8 / 41.0; 2048 x 11264 at 257 to 288 rows 20.4 / 19.6; 4096 x 5120 at 785 to 896
// rows 35.0 / 32.6), and steps that fewer tiles hold don't go there for a third wave (2048 x 21888, two an SM / tiles of one CTA: 640
// rows 56.5 / 52.3, 700 rows 59.5 / 55.6, 800 rows 62.2 / 60.0).
static void choose_tiles(Ctx* c, int64_t M, int64_t N, bool pairs, int* tn, int* pair_tn) {
  const int64_t fewest = (M + 255) / 256, cols = (N + BM - 1) / BM, sms = c->sm_count;
  auto waves = [](int64_t n, int64_t at_once) { return (double)((n + at_once - 1) / at_once); };
  double best = 0;
  bool best_shared = false;
  for (int64_t t = fewest; t <= fewest + 4; ++t) {
    const int64_t rows = (M + t - 1) / t;
    const int one = (int)((rows + 15) / 16 * 16), two = (int)((rows + 31) / 32 * 32);
    if (t > fewest && one < 64) break;
    const int64_t tiles_one = cols * ((M + one - 1) / one);
    const bool shared = tc_two_per_sm(c, one, tiles_one);   // SMs, by two CTAs each
    const double us = 0.18 + 0.0002 * std::min(one, 144) + 0.0014 * std::max(one - 144, 0);
    const double cost = us * (shared ? 2 * waves(tiles_one, 2 * sms) : waves(tiles_one, sms));
    if (best == 0 || (cost < best && !(shared && tiles_one > 4 * sms))) best = cost, *tn = one, *pair_tn = 0, best_shared = shared;
    if (!pairs) continue;
    const double pair_cost = (0.178 + 0.0002 * std::min(two, 128) + 0.00075 * std::max(two - 128, 0)) * waves(cols / 2 * ((M + two - 1) / two), sms / 2);
    if (pair_cost * (best_shared ? 1.013 : 1) < best) best = pair_cost, *pair_tn = two, best_shared = false;
  }
}

// Same contract as linear_bf16_launch (ungrouped).
int linear_tc_launch(Ctx* c, const LinearBf16Plan& plan, const bf16* x, int64_t ldx, int64_t M, int epi, int ksplit,
                     void* out, int64_t ldo, const float* bias) {
  RB_REQUIRE(plan.groups == 0, "the tcgen05 Linear does not take grouped weights");
  RB_REQUIRE(ldx % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0, "bf16 Linear: activations must be 16-byte aligned rows");
  RB_REQUIRE(ksplit >= 1 && (ksplit == 1 || epi == EPI_PARTIAL_F32), "split-K needs the partial epilogue");
  RB_REQUIRE(epi != EPI_SWIGLU_BF16 || plan.N % 16 == 0, "SwiGLU epilogue needs interleaved width % 16 == 0");
  if (M == 0) return REWB200_OK;
  const bool pairs = c->prefill_persistent && c->prefill_pair && plan.N % 256 == 0 && c->sm_count % 2 == 0 && ksplit == 1;
  const int64_t fewest = (M + 255) / 256;   // token tiles
  int TN = M <= 32 ? 32 : M <= 64 ? 64 : (int)(((M + fewest - 1) / fewest + 15) / 16 * 16), pair_tn = 0;
  if (M >= 1024) {
    // Pairs of CTAs from four tiles an SM on, where their half of the shared-memory traffic counts: 1 to 4 per cent ahead of one CTA
    // a tile (us, pairs / one CTA: 4096 x 28672, 1024 rows 200 / 204; 2048 x 11264, 3072 rows 119 / 122; 14336 x 4096, 6144 rows
    // 616 / 638; 5632 x 2048, 12 288 rows 240 / 249).  With fewer tiles the last wave decides, which is coarser in pairs (4096 x 6144,
    // 2048 rows, 384 tiles 102 / 99; 2048 x 3072, 4096 rows, 384 tiles 57 / 55).
    if (pairs && (plan.N + BM - 1) / BM * fewest >= 4 * (int64_t)c->sm_count) pair_tn = PairCfg::TN;
  } else if (M > 64 && ksplit == 1 && c->prefill_persistent) {
    choose_tiles(c, M, plan.N, pairs, &TN, &pair_tn);
  }
  TcArgs a;
  memset(&a, 0, sizeof(a));
  a.M = M;
  a.N = plan.N;
  a.K = plan.K;
  const int nkb = (int)((plan.K + BK - 1) / BK);
  a.kb_per_split = (nkb + ksplit - 1) / ksplit;
  a.epi = epi;
  a.out = out;
  a.ldo = ldo;
  a.split_stride = M * ldo;
  a.bias = bias;
  a.status = c->d_status;
  a.ksplit = ksplit;
  a.early_w = plan.early_w;
  a.tn = TN;
  dim3 grid((unsigned)((plan.N + BM - 1) / BM), (unsigned)((M + TN - 1) / TN), (unsigned)ksplit);
  if (pair_tn) {
    // two-CTA tiles: 256 features x pair_tn tokens per pair of SMs
    CUtensorMap tmXh;
    RB_TRY(make_tmap_2d_bf16(&tmXh, x, (uint64_t)plan.K, (uint64_t)M, (uint64_t)ldx * 2, 64, pair_tn / 2));
    static bool pair_attr = false;
    if (!pair_attr) {
      RB_CUDA(cudaFuncSetAttribute(linear_tc_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg::SMEM));
      pair_attr = true;
    }
    a.tn = pair_tn;
    const int tiles_n = (int)(plan.N / 256), tiles_m = (int)((M + pair_tn - 1) / pair_tn);
    const int64_t ctas = std::min<int64_t>(2 * (int64_t)tiles_n * tiles_m, c->sm_count);
    RB_CUDA(launch_k(linear_tc_pair_kernel, dim3((unsigned)ctas), dim3(TC_THREADS), (size_t)PairCfg::SMEM, c->stream, c->use_pdl, plan.tmW, tmXh, a,
                     tiles_n, tiles_m));
    ++g_launch_total;
    ++g_route_launches[ROUTE_LINEAR_PAIR];
    return REWB200_OK;
  }
  CUtensorMap tmX;
  RB_TRY(make_tmap_2d_bf16(&tmX, x, (uint64_t)plan.K, (uint64_t)M, (uint64_t)ldx * 2, 64, TN));
  if (M <= 32) return launch_tn<32>(c, plan, tmX, a, grid);
  if (M <= 64) return launch_tn<64>(c, plan, tmX, a, grid);
  const bool two = tc_two_per_sm(c, TN, (int64_t)grid.x * grid.y * grid.z);
  if (c->prefill_persistent && !two) {
    static bool attr_set = false;
    if (!attr_set) {
      RB_CUDA(cudaFuncSetAttribute(linear_tc_persist_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, PersistCfg::SMEM));
      attr_set = true;
    }
    const int ctas = (int)std::min<int64_t>((int64_t)grid.x * grid.y * grid.z, c->sm_count);
    RB_CUDA(launch_k(linear_tc_persist_kernel<false>, dim3((unsigned)ctas), dim3(TC_THREADS), (size_t)PersistCfg::SMEM, c->stream, c->use_pdl, plan.tmW,
                     tmX, a, (int)grid.x, (int)grid.y));
    ++g_launch_total;
    ++g_route_launches[ROUTE_LINEAR_PERSISTENT];
    return REWB200_OK;
  }
  using C = TcCfg<0>;
  a.stages = std::min((int)C::MAX_STAGES, ((TN <= 160 ? 113 * 1024 : kAllSmem) - C::FIXED) / C::stage_bytes(TN));
  static bool attr_set = false;
  if (!attr_set) {
    RB_CUDA(cudaFuncSetAttribute(linear_tc_kernel<0, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAllSmem));
    attr_set = true;
  }
  RB_CUDA(launch_k(linear_tc_kernel<0, 0>, grid, dim3(TC_THREADS), (size_t)(a.stages * C::stage_bytes(TN) + C::FIXED), c->stream, c->use_pdl, plan.tmW, tmX, a));
  ++g_launch_total;
  ++g_route_launches[ROUTE_LINEAR_TILE];
  return REWB200_OK;
}

}  // namespace rewb
