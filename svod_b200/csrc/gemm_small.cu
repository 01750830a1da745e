// tcgen05 GEMM for few tiles: y = epilogue(x . w^T) where 128-row tiles do not fill the
// chip (one query, a handful of paragraphs). Same contract and epilogue order as
// gemm_tc.cu (tk/src/kernels/gemm.rs:605-651).
//
// What bounds such a call: latency. A projection of one 128-row batch is 2-8 MB of
// weights, 0.3-1.3 us at HBM rate, but on the persistent kernel it is 16-64 CTAs that
// each walk the whole k loop and then a chain of accumulator read, staging, TMA store:
// 9-20 us. Here:
//   * the k loop is split over a cluster of S CTAs (1..8), each of which takes K/S of
//     one 128 x BN tile, so that 100-150 CTAs pull the weights at once;
//   * rows are dealt over the cluster's CTAs; every CTA sends each owner its rows' f32
//     partials by one bulk copy into the owner's shared memory (row-by-row stores into
//     a peer's memory measured 5400 cycles for a 128-row tile), and the owner sums its
//     rows' S partials in rank order (bit-equal from run to run) and applies the epilogue
//     with a row's columns across neighbouring lanes: the per-head RMSNorm and the
//     rotation are shuffles, stores are whole 128-byte lines;
//   * no ring is deeper than the slice needs and rows past M are neither loaded nor
//     sent, so that the next launch can mostly come up beside this one;
//   * weights the caller declares constant (`w_static`) are requested before the wait for
//     the previous kernel: they travel while it finishes.
// Measured: figures at `gemm_small_splits`.
//
// CTA roles (192 threads): warp 0 TMA, warp 1 MMA issuer, warps 2-5 accumulator read and
// push; all six reduce. Every mbarrier wait is bounded; the cluster barrier is reached by
// every thread on every path.
#include <cuda.h>
#include <stdio.h>

#include "common.cuh"
#include "gemm_parts.cuh"
#include "kernels.h"
#include "launch.h"
#include "svodb.h"
#include "tensormap.h"

namespace svodb {

namespace {

using namespace gemm_parts;

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int kThreads = 192;
constexpr int kMaxStages = 8;

struct ParamsS {
  int64_t m;
  int n, k;
  int tiles_m;
  int a_box;      // rows of an A box: 64 or 128 (a tile of at most 64 rows loads no more)
  int stages;
  int ring_bytes;  // stages * stage, or the partial tile that takes the ring's place if that is larger
  int gated, act, has_scale;
  float scale;
  const void* bias;
  const void* residual;
  void* c;
  int64_t ldr, ldc;
  int w_static;
  // per-head store: norm weights below norm_q_cols / norm_cols, rotation below rope_width
  int head;       // 0, or the head width (== BN)
  const void* norm_q;
  const void* norm_k;
  int norm_q_cols, norm_cols;
  float norm_eps;
  const void* rope_cos;
  const void* rope_sin;
  int rope_width;
  int64_t rope_seq;
  const int32_t* block_pos;  // packed rows: their blocks' positions, nullable
  uint32_t* status;
};

// Bulk copy from this CTA's shared memory into a peer's, its bytes counted on the peer's barrier.
__device__ __forceinline__ void bulk_to_peer(uint32_t dst, const void* src, uint32_t bytes, uint32_t peer_bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "r"(smem_u32(src)), "r"(bytes), "r"(peer_bar)
               : "memory");
}

template <typename T>
__device__ __forceinline__ void unpack8(uint4 u, float (&f)[8]) {
  const uint32_t uu[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = Elem<T>::unpack(uu[i]);
    f[2 * i] = v.x, f[2 * i + 1] = v.y;
  }
}
template <typename T>
__device__ __forceinline__ void add8(float (&x)[8], uint4 u) {
  float f[8];
  unpack8<T>(u, f);
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] += f[i];
}
__device__ __forceinline__ void act8(float (&x)[8], int act) {
  switch (act) {
    case kActGelu:
#pragma unroll
      for (int i = 0; i < 8; i += 2) gelu2_f(x[i], x[i + 1]);
      break;
    case kActSilu:
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = silu_f(x[i]);
      break;
    case kActGeluTanh:
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = gelu_tanh_f(x[i]);
      break;
    default: break;
  }
}

template <typename T, int BN>
__global__ void __launch_bounds__(kThreads, 2)
    gemm_small_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w,
                      const ParamsS p) {
  constexpr int kPitch = BN + 4;  // floats of a partial row: 16-byte pieces of 32 rows fall in distinct banks
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int a_bytes = p.a_box * 128;
  const int stage_bytes = a_bytes + BN * 128;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + p.ring_bytes);
  uint64_t* full = bars;
  uint64_t* empty = bars + kMaxStages;
  uint64_t* acc_full = bars + 2 * kMaxStages;
  uint64_t* red_full = acc_full + 1;  // the peers' partials of this CTA's rows have arrived
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kMaxStages + 2);
  float* part = reinterpret_cast<float*>(bars + 2 * kMaxStages + 4);  // [S sources][share rows][kPitch]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)cluster_ctarank();
  uint32_t csz;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(csz));
  const int S = (int)csz;
  const int tile = blockIdx.x / S;
  const int mt = tile % p.tiles_m, nt = tile / p.tiles_m;
  const int m0 = mt * BM;
  const int out_bn = p.gated ? BN / 2 : BN;
  const int n0 = nt * out_bn;
  const int live = (int)(p.m - m0 < BM ? p.m - m0 : BM);  // rows of this tile
  const int share = (live + S - 1) / S;                   // rows an owner reduces
  const int first = rank * share;
  const int mine = live - first < share ? live - first : share;  // <= 0: this CTA owns no row
  const int num_kb = (p.k + BK - 1) / BK;
  const int per = (num_kb + S - 1) / S;
  const int kb0 = rank * per < num_kb ? rank * per : num_kb;
  const int nkb = num_kb - kb0 < per ? num_kb - kb0 : per;

  // Stage numbers and phases run along as counters: a division by the stage count per k-block
  // costs the one thread that loads (or issues) 500 cycles, more than the block's MMAs
  // (128 x 1024 x 4096 over 8 CTAs a tile 8.7 -> 7.7 us).
  auto load_w = [&](int i, int s) {
    uint8_t* dst = smem + (size_t)s * stage_bytes + a_bytes;
    mbar_expect_tx(&full[s], (uint32_t)stage_bytes);
    const int x = (kb0 + i) * BK;
    if (p.gated) {
      tma_load_2d(dst, &tmap_w, &full[s], x, n0);
      tma_load_2d(dst + (BN / 2) * 128, &tmap_w, &full[s], x, p.n + n0);
    } else {
      tma_load_2d(dst, &tmap_w, &full[s], x, n0);
    }
  };
  auto load_a = [&](int i, int s) {
    tma_load_2d(smem + (size_t)s * stage_bytes, &tmap_a, &full[s], (kb0 + i) * BK, m0);
  };
  const int ahead = nkb < p.stages ? nkb : p.stages;
  if (tid == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_a);
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(red_full, 1);
    mbar_fence_init();
    if (S > 1 && mine > 0) mbar_expect_tx(red_full, (uint32_t)((S - 1) * mine * kPitch * 4));
    if (p.w_static)
      for (int i = 0; i < ahead; ++i) load_w(i, i);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");  // waited for before the first push
  tc_fence_after();
  pdl_trigger();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      pdl_wait();
      bool ok = true;
      int s = 0;
      uint32_t ph = 1;  // the parity of a stage nobody has used yet
      for (int i = 0; i < nkb; ++i) {
        if (i >= p.stages && !mbar_wait(&empty[s], ph, p.status)) {
          ok = false;
          break;
        }
        if (!p.w_static || i >= ahead) load_w(i, s);
        load_a(i, s);
        if (++s == p.stages) s = 0, ph ^= 1;
      }
      if (!ok)
        for (int i = 0; i < 64; ++i) __nanosleep(1000);  // copies in flight land before the CTA's memory goes
    }
    __syncwarp();
  } else if (warp == 1) {
    constexpr uint32_t idesc = umma_idesc(Elem<T>::kUmmaFormat, BM, BN, 0, 0);
    const bool leader = elect_one();
    const uint64_t desc0 = umma_desc_sw128(smem_u32(smem), 16, 1024);
    bool ok = true;
    int s = 0;
    uint32_t ph = 0;
    for (int i = 0; i < nkb; ++i) {
      if (!mbar_wait(&full[s], ph, p.status)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const uint64_t ad = desc0 + (uint64_t)((s * stage_bytes) >> 4);
      const uint64_t wd = ad + (uint64_t)(a_bytes >> 4);
#pragma unroll
      for (int k4 = 0; k4 < BK / 16; ++k4)
        if (leader) umma_ss(tmem, ad + (uint64_t)(k4 * 2), wd + (uint64_t)(k4 * 2), idesc, (i | k4) != 0 ? 1u : 0u);
      if (leader) tc_commit(&empty[s]);
      if (++s == p.stages) s = 0, ph ^= 1;
    }
    if (ok && leader) tc_commit(acc_full);
    __syncwarp();
  }
  // ---- partial rows: tensor memory -> this CTA's shared memory -> the owners ----
  // The ring is free once every MMA is done: the partial tile [rows][kPitch] takes its place,
  // and an owner's rows of it are one run of bytes, one bulk copy.
  float* own = reinterpret_cast<float*>(smem);
  if (warp >= 2) {
    const bool have = nkb > 0 && mbar_wait(acc_full, 0, p.status);
    tc_fence_after();
    const int quarter = warp & 3;
    if (quarter * 32 < live) {
      float* dst = own + (quarter * 32 + lane) * kPitch;
      const uint32_t t_acc = tmem + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < BN; c += 32) {
        uint32_t x[32];
        if (have) {
          tmem_ld32(t_acc + c, x);
          tmem_ld_wait_for(x);
        } else {  // an empty slice of the k loop (or a wait that ran out) adds zeros
#pragma unroll
          for (int i = 0; i < 32; ++i) x[i] = 0u;
        }
#pragma unroll
        for (int i = 0; i < 32; i += 4) *reinterpret_cast<uint4*>(dst + c + i) = make_uint4(x[i], x[i + 1], x[i + 2], x[i + 3]);
      }
    }
    fence_proxy_async_smem();
    tc_fence_before();
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // every CTA of the cluster has its barriers
  __syncthreads();
  if (tid < S && tid != rank) {
    const int rows = live - tid * share < share ? live - tid * share : share;  // <= 0: that CTA owns no row
    if (rows > 0)
      bulk_to_peer(cluster_map(part + rank * share * kPitch, (uint32_t)tid), own + tid * share * kPitch,
                   (uint32_t)(rows * kPitch * 4), cluster_map(red_full, (uint32_t)tid));
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, BN);
  }
  pdl_wait();  // the residual and the tables may come from the kernel before; y may still be read by it

  // ---- the owner's rows: sum the partials in rank order, epilogue, store ----
  const T* bias = (const T*)p.bias;
  const int sh = p.gated ? (BN == 64 ? 2 : 3) : (BN == 64 ? 3 : 4);  // log2 of the 8-column chunks of a row
  auto sum8 = [&](int row, int col, float (&x)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = 0.f;
    for (int s = 0; s < S; ++s) {
      const float* src = (s == rank ? own + first * kPitch : part + s * share * kPitch) + row * kPitch + col;
      const float4 u = *reinterpret_cast<const float4*>(src);
      const float4 v = *reinterpret_cast<const float4*>(src + 4);
      x[0] += u.x, x[1] += u.y, x[2] += u.z, x[3] += u.w;
      x[4] += v.x, x[5] += v.y, x[6] += v.z, x[7] += v.w;
    }
  };
  const int chunks = mine > 0 ? mine << sh : 0;
  for (int i0 = 0; i0 < chunks; i0 += kThreads) {
    const int i = i0 + tid;
    const int at = i < chunks ? i : chunks - 1;  // idle lanes repeat the last chunk: the shuffles need them
    const int row = at >> sh, ch = at & ((1 << sh) - 1);
    const int col = n0 + ch * 8;
    const int64_t grow = m0 + first + row;
    const bool in_n = col < p.n, in = i < chunks && in_n;
    // What the epilogue reads from memory is on its way while the partials arrive.
    const uint4 zero = make_uint4(0, 0, 0, 0);
    const uint4 b4 = bias != nullptr && in_n ? ldg128(bias + col) : zero;
    const uint4 u4 = bias != nullptr && in_n && p.gated ? ldg128(bias + p.n + col) : zero;
    const uint4 r4 = p.residual != nullptr && in ? ldg128((const T*)p.residual + grow * p.ldr + col) : zero;
    const T* nw = (const T*)(col < p.norm_q_cols ? p.norm_q : (col < p.norm_cols ? p.norm_k : nullptr));
    const uint4 w4 = nw != nullptr ? ldg128(nw + ch * 8) : zero;
    uint4 c4 = zero, s4 = zero;
    const bool turned = col < p.rope_width;
    if (turned) {
      const int64_t tab = table_row((uint32_t)grow, p.rope_seq, p.block_pos) * (BN / 2) + (ch & (BN / 16 - 1)) * 8;
      c4 = ldg128((const T*)p.rope_cos + tab);
      s4 = ldg128((const T*)p.rope_sin + tab);
    }
    if (i0 == 0 && S > 1) mbar_wait(red_full, 0, p.status);
    float x[8];
    sum8(row, ch * 8, x);
    if (bias != nullptr) add8<T>(x, b4);
    if (p.head != 0) {
      constexpr int L = BN / 8;  // lanes of a head
      if (p.norm_cols > 0) {  // some head of this call is normalised: all lanes take the reduction
        float ss = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) ss = fmaf(x[e], x[e], ss);
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (nw != nullptr) {
          const float inv = rsqrtf(ss * (1.0f / BN) + p.norm_eps);
          float w[8];
          unpack8<T>(w4, w);
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = x[e] * inv * w[e];
        }
      }
      if (p.rope_width > 0) {
        float y[8];  // the same elements of the head's other half
#pragma unroll
        for (int e = 0; e < 8; ++e) y[e] = __shfl_xor_sync(0xffffffffu, x[e], L / 2);
        if (turned) {
          float cs[8], sn[8];
          unpack8<T>(c4, cs);
          unpack8<T>(s4, sn);
          const bool second = ch >= L / 2;
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = second ? y[e] * sn[e] + x[e] * cs[e] : x[e] * cs[e] - y[e] * sn[e];
        }
      }
    } else {
      act8(x, p.act);
      if (p.gated) {
        float u[8];
        sum8(row, BN / 2 + ch * 8, u);
        if (bias != nullptr) add8<T>(u, u4);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] *= u[e];
      }
      if (p.has_scale) {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] *= p.scale;
      }
      if (p.residual != nullptr) add8<T>(x, r4);
    }
    if (in)
      stg128((T*)p.c + grow * p.ldc + col, make_uint4(Elem<T>::pack(x[0], x[1]), Elem<T>::pack(x[2], x[3]),
                                                      Elem<T>::pack(x[4], x[5]), Elem<T>::pack(x[6], x[7])));
  }
  // No CTA leaves before its copies have reached every owner: an owner that has waited for
  // its rows has all of them.
  if (S > 1) {
    __syncwarp();
    cluster_sync_all();
  }
}

int sm_count_s() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  return sms;
}

template <typename T, int BN>
int run_s(const GemmArgs& a, int splits, cudaStream_t s, char* cfg, size_t cfg_len) {
  ParamsS p{};
  p.m = a.m, p.n = a.n, p.k = a.k;
  p.gated = a.gated, p.act = a.act, p.has_scale = a.has_scale, p.scale = a.scale;
  p.bias = a.bias, p.residual = a.residual, p.c = a.c;
  p.ldr = a.ldr, p.ldc = a.ldc;
  p.w_static = a.w_static;
  p.status = a.status;
  p.block_pos = a.block_pos;
  const bool per_head = a.rope_cos != nullptr || a.norm_q != nullptr || a.norm_k != nullptr;
  if (per_head) {
    p.head = BN;
    p.norm_q = a.norm_q, p.norm_k = a.norm_k;
    p.norm_q_cols = a.norm_q_heads * BN;
    p.norm_cols = (a.norm_q_heads + a.norm_k_heads) * BN;
    if (a.norm_q == nullptr && a.norm_k == nullptr) p.norm_q_cols = p.norm_cols = 0;
    p.norm_eps = a.norm_eps;
    p.rope_cos = a.rope_cos, p.rope_sin = a.rope_sin;
    p.rope_width = a.rope_cos != nullptr ? a.rope_heads * BN : 0;
    p.rope_seq = a.rope_seq > 0 ? a.rope_seq : 1;
  }
  const int out_bn = a.gated ? BN / 2 : BN;
  p.tiles_m = (int)((a.m + BM - 1) / BM);
  const int tiles_n = (a.n + out_bn - 1) / out_bn;
  p.a_box = a.m <= 64 ? 64 : 128;
  const int kb = (a.k + BK - 1) / BK;
  if (splits > kb) splits = kb;
  const int per = (kb + splits - 1) / splits;
  const int rows = (int)(a.m < BM ? a.m : BM);
  const size_t part = (size_t)((rows + splits - 1) / splits) * splits * (BN + 4) * 4;
  const size_t stage = (size_t)p.a_box * 128 + BN * 128;
  // A ring within half an SM where at most three rounds of it cover the slice: CTAs of this
  // launch and the next then share SMs, and clusters of eight all find a place at once (K 4096
  // over 8 CTAs: 7.3 us with 5 stages, 12.8 with 8 and one CTA an SM). A longer slice through
  // few stages would pay the latency of HBM once per round (16 blocks: 16 us through 3 stages,
  // 9 through 8), so it takes the whole SM.
  const size_t fixed = 1024 + 256 + (splits > 1 ? part : 0);
  const size_t half = 113 * 1024;
  const int fit = fixed < half ? (int)((half - fixed) / stage) : 0;
  p.stages = per < kMaxStages ? per : kMaxStages;
  if (fit * 3 >= per && fit < p.stages) p.stages = fit;
  while (fixed + p.stages * stage > 226 * 1024) --p.stages;
  const size_t tile = (size_t)((rows + 31) / 32 * 32) * (BN + 4) * 4;  // warps write 32 rows at a time
  p.ring_bytes = (int)(p.stages * stage > tile ? p.stages * stage : ((tile + 1023) & ~(size_t)1023));
  // (the MMA reads 128 rows of A whatever was loaded: 64 rows and the W tile behind them are as much)
  const size_t smem = fixed + (size_t)p.ring_bytes;
  CUtensorMap ta, tw;
  if (!make_tmap_2d(&ta, a.a, a.dtype, (uint64_t)a.k, (uint64_t)a.m, (uint64_t)a.lda, BK, (uint32_t)p.a_box)) return -1;
  if (!make_tmap_2d(&tw, a.w, a.dtype, (uint64_t)a.k, (uint64_t)(a.gated ? 2 * a.n : a.n), (uint64_t)a.ldw, BK, out_bn))
    return -1;
  static bool attr_seen[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_seen[dev & 63]) {
    if (cudaFuncSetAttribute(gemm_small_kernel<T, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) !=
        cudaSuccess)
      return -1;
    attr_seen[dev & 63] = true;
  }
  const int grid = p.tiles_m * tiles_n * splits;
  if (launch_pdl(gemm_small_kernel<T, BN>, dim3((unsigned)grid), dim3(kThreads), smem, s, (unsigned)splits, a.m, ta, tw,
                 p) != cudaSuccess)
    return -1;
  if (cfg != nullptr)
    snprintf(cfg, cfg_len, "{bm:%d,bn:%d,bk:%d,stages:%d,gated:%d,grid:%d,cluster:%d}", BM, BN, BK, p.stages, a.gated, grid,
             splits);
  return 0;
}

}  // namespace

// Measured against the persistent kernels, us a launch in a graph, each launch with weights of
// its own (M x N x K, this kernel | the better of the others):
//   32 x 1024 x 1024     3.9 | 8.2       128 x 1024 x 1024    5.8 | 8.5      512 x 1024 x 1024   7.1 | 8.9
//   32 x 1024 x 4096     5.6 | 17.3      128 x 1024 x 4096    7.7 | 18.0     512 x 1024 x 4096  12.3 | 18.3
//   32 x 3072 x 1024     5.2 | 8.0       128 x 3072 x 1024    7.0 | 8.7      256 x 3072 x 1024   8.3 | 8.8
//   32 x 4096 x 1024 with the attention prologue  6.1 | 14.3;  128 rows  10.0 | 16.1;  256 rows  12.3 | 16.1
// Where the lines lie:
//   * up to 64 rows a tile is cheap to send, so it pays up to 100 tiles, two CTAs an SM; slices
//     of four k-blocks (64 x 1152 gated x 768: 4.9 us in three CTAs a tile, 5.4 in five);
//   * a slice of at most nine blocks (three rounds of three stages) leaves room for two CTAs an
//     SM: two CTAs a tile up to 110 tiles (384 x 2304 x 768 rotated 8.2 | 9.1 us, 384 x 3072 x
//     1024 with 144 tiles 9.3 | 8.8);
//   * a longer one takes the whole SM, where clusters of three do not all find a place at once
//     (48 tiles of K 4096: 19 us, in pairs 12.9), and 128-column tiles halve what is read of x:
//     512 x 1024 x 4096 12.3 us in four CTAs a tile against 13.5 in two of 64 columns, 1024 rows
//     16.6 | 18.4; at K 2048 the narrow pairs are ahead (512 x 1024 x 2048 9.8, 10.3 | 11.6);
//   * whole 128-wide heads up to 75 tiles (384 rows x 4096: 17.8 | 16.1).
int gemm_small_splits(const GemmArgs& a) {
  if (!gemm_tc_covers(a)) return 0;
  const bool per_head = a.rope_cos != nullptr || a.norm_q != nullptr || a.norm_k != nullptr;
  if (small_code(a.force_bn)) return a.force_bn - kForceSmall;
  const int bn = per_head ? a.rope_head_dim : 64;
  const int out_bn = a.gated ? bn / 2 : bn;
  const int64_t tiles = ((a.m + BM - 1) / BM) * ((a.n + out_bn - 1) / out_bn);
  const int kb = (a.k + BK - 1) / BK;
  auto fill = [&](int64_t room, int most) {  // CTAs a tile: as many as the chip holds, eight at most
    int64_t s = room / tiles < 8 ? room / tiles : 8;
    if (s > most) s = most;
    return s < 1 ? 1 : (int)s;
  };
  if (a.m <= 64) return tiles <= 100 ? fill(200, bn == 128 ? kb / 2 : (kb + 3) / 4) : 0;
  if (bn == 128) return tiles <= 75 ? fill(sm_count_s(), kb / 2) : 0;
  if (kb <= 18) {
    if (tiles <= 48) return fill(sm_count_s(), kb / 2);
    return tiles <= 110 && a.m < 1024 ? 2 : 0;
  }
  if (tiles <= 18) return 8;
  if (tiles <= 36) return 4;
  if (tiles <= 64) return kb >= 40 && !per_head ? kSmallWide + 4 : 2;
  return tiles <= 128 && kb >= 64 && !per_head ? kSmallWide + 2 : 0;
}

int launch_gemm_small(const GemmArgs& a, int splits, cudaStream_t s, char* cfg, size_t cfg_len) {
  const bool per_head = a.rope_cos != nullptr || a.norm_q != nullptr || a.norm_k != nullptr;
  const bool wide = per_head ? a.rope_head_dim == 128 : (splits & kSmallWide) != 0;
  splits &= kSmallWide - 1;
  if (a.dtype == SVODB_BF16)
    return wide ? run_s<__nv_bfloat16, 128>(a, splits, s, cfg, cfg_len) : run_s<__nv_bfloat16, 64>(a, splits, s, cfg, cfg_len);
  return wide ? run_s<__half, 128>(a, splits, s, cfg, cfg_len) : run_s<__half, 64>(a, splits, s, cfg, cfg_len);
}

}  // namespace svodb
