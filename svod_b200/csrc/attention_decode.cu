// Attention of few query rows against many keys (a decoding step): the keys and
// values of a KV head are read once from HBM for all the query rows that share it.
//
// What bounds it: the cache. B8 x Tk 32768 x 8 KV heads x 128 is 1.03 GB of keys and
// values for 2 query rows each. The 256-row tile kernel (attention_tc_p.cu) spends its
// time on the exponentials of 254 rows nobody asked for (416 us with lengths from 30000);
// here it takes 160 us, 6.46 TB/s of the keys it reads (a plain copy: 6.54). Appended cache
// rows used to go to the exact kernel, on scalar loads (B24, 150..2048 keys + 5, 8 KV heads
// x 64: 1114 us; 19 us here).
//
// How it is laid out for that: keys are the M dimension of both contractions, so
// a 128-key block costs two small MMAs whatever the number of query rows:
//     S^T [128 keys x NQ]  = K [128 x D] . Q^T          (A = K, B = Q rows)
//     O^T [D x 2*NQ]      += V^T [D x 128] . P^T        (A = V, MN-major; B = P rows)
// with NQ = 16 / 32 / 64 columns for the t * (heads / kv_heads) query rows of a KV
// head. A softmax thread owns one key: its scores are NQ columns of one tensor-memory
// lane, so the exponentials are those of real query rows only. The softmax weights go
// to shared memory as two 16-bit halves (value and remainder, 2*NQ rows of B) with an
// accumulator each, so O carries them to 16 bits (bf16) or 22 bits (f16) although the MMA
// is a 16-bit one. f16 has no exponents below 2^-24: its value half is scaled by 2^7 (a
// weight is at most 2^8, see kRescaleAbove) and its remainder by another 2^11, which keeps
// 22 bits of a weight down to 2^-21 and 2^-44 of any smaller one: 32768 keys of weight
// 2.5e-8 beside one of weight 1 keep their 8.2e-4 (unscaled, those in the heavy key's share
// vanished from O, not from the sum).
//
// Work split: a cluster of C CTAs (1..16) takes one (batch lane, KV head); each CTA
// walks an equal share of that lane's VISIBLE key blocks, and the C partial states
// are merged through distributed shared memory: one launch, no workspace, no merge
// kernel. With NQ = 16 an SM holds two CTAs of a 96 KiB ring (three of 48 KiB for D <= 64):
// as many bytes in flight as one CTA could have, and each hides the others' softmax chain
// (about 1.2 us a block: score load, two barriers for the block's maxima, exponentials,
// weights to shared memory).
//
// CTA roles (192 threads): warps 0-3 softmax (one key per thread), warp 4 TMA loader,
// warp 5 MMA issuer. The ring holds single K or V blocks in the order the issuer uses
// them: K0 K1 V0 K2 V1 ... Appended cache rows are one more run of key blocks behind
// the cached ones, with tensor maps of their own.
//
// Semantics: tk/src/kernels/attention.rs:381-450 and `ops::Cache`
// (tk/src/ops/attention.rs:39-55); the lazy rescale of the tile kernels (threshold 8
// in log2 units), zeros for a row without a visible key.
//
// Every mbarrier wait is bounded. A softmax warp whose wait ran out keeps walking the
// named barriers (nothing in between waits without a limit) and the cluster barriers.
#include <cuda.h>
#include <cuda_fp16.h>
#include <math.h>
#include <stdio.h>

#include <type_traits>

#include "attention_parts.cuh"
#include "common.cuh"
#include "kernels.h"
#include "launch.h"
#include "svodb.h"
#include "tensormap.h"

namespace svodb {

namespace {

using namespace fa_parts;

constexpr int kKeys = 128;  // keys per block: the M of both MMAs
constexpr int kThreadsDec = 192;
constexpr int kBox = kKeys * 128;  // bytes of one 64-column box of 128 rows

// Powers of two the halves of a weight are scaled by: value, and the remainder once more.
template <typename T>
constexpr float kValueUp = std::is_same<T, __half>::value ? 128.f : 1.f;
template <typename T>
constexpr float kRestUp = std::is_same<T, __half>::value ? 2048.f : 1.f;

template <int D, int NQ>
struct DecCfg {
  static constexpr int kSlotBytes = kKeys * D * 2;
  // D = 64 keeps one slot less: the V operand (M = 128) then reads 64 rows past a
  // 64-wide block, whatever lies there (those accumulator rows are never read).
  static constexpr int kSlots = D == 128 ? (NQ == 16 ? 3 : NQ == 32 ? 5 : 4) : (NQ == 16 ? 3 : NQ == 32 ? 10 : 8);
  // CTAs an SM holds: the small rings leave room for others, which hide one CTA's softmax chain.
  static constexpr int kPerSm = NQ > 16 ? 1 : D == 128 ? 2 : 3;
  static constexpr int kRing = kSlots * kSlotBytes;
  static constexpr int kQBytes = NQ * D * 2;
  static constexpr int kPBytes = 2 * 2 * NQ * 128;  // two 64-key boxes of 2*NQ rows
  // A second buffer of weights lets a block's exponentials run under the previous block's
  // P.V; the (D 128, 16 rows) ring leaves no room for it and is bound by HBM anyway.
  static constexpr int kPBufs = NQ == 64 || (NQ == 16 && D == 128) ? 1 : 2;
  // Sums per (key, column): registers for one chunk of columns, else shared memory.
  static constexpr int kLBytes = NQ > 16 ? NQ * 128 * 4 : 0;
  static constexpr int kRedBytes = NQ * 4 * 4;      // per-warp maxima (and sums)
  static constexpr int kTail = kQBytes + kPBufs * kPBytes + kLBytes + kRedBytes + 4 * NQ * 4 + 256;
  static constexpr size_t kSmem = 1024 + (size_t)kRing + (kTail > kBox ? kTail : kBox);
  static constexpr int kTmemCols = 4 * NQ;
  static_assert(kSmem <= 232448, "beyond the 227 KiB a CTA may hold");
  static_assert(kPerSm * (kSmem + 1024) <= 233472, "the CTAs of an SM fit its shared memory");
  static_assert(NQ * D * 4 <= kRing, "the partial outputs are laid over the ring");
};

struct DecParams {
  const void* q;
  void* o;
  int64_t q_sb, q_st, q_sh, o_sb, o_st, o_sh;
  int64_t t, tk, batch, kv_rows;
  int heads, kv_heads, group, rows;  // rows = t * group query rows per KV head
  int d_real;
  float scale_log2, inv_scale;
  const int32_t* key_lens;
  const void* key_mask;
  int key_mask_i32;
  const int32_t* row_map;
  int n_app;
  const int32_t* app_lens;
  const void* bias;
  int bias_per_batch;
  float* lse;
  uint32_t* status;
};

__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[16]) {
  tmem_ld16(taddr, r);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 16; ++i) asm volatile("" : "+r"(r[i]));  // no use moves above the wait
}

__device__ __forceinline__ float redux_max(float x) {
  float y;
  asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(y) : "f"(x));
  return y;
}

// Named barrier over the 128 softmax threads that also ORs a predicate over them.
__device__ __forceinline__ bool barrier_or(int id, bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred P, Q;\n\t"
      "setp.ne.u32 P, %1, 0;\n\t"
      "barrier.cta.red.or.pred Q, %2, 128, P;\n\t"
      "selp.u32 %0, 1, 0, Q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)v), "r"(id)
      : "memory");
  return r != 0;
}

__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

// Position of block j's K and V in the ring's order K0 K1 V0 K2 V1 ... K(n-1) V(n-2) V(n-1).
__device__ __forceinline__ uint32_t pos_k(int j) { return j == 0 ? 0u : (uint32_t)(2 * j - 1); }
__device__ __forceinline__ uint32_t pos_v(int j, int n) { return j == n - 1 ? (uint32_t)(2 * n - 1) : (uint32_t)(2 * j + 2); }

// Runs `f` on the first 4, 8 or 16 columns of a chunk: the least that holds `live` of them.
// The columns between are zero query rows: whatever is computed for them is never stored.
template <typename F>
__device__ __forceinline__ void by_width(int live, F&& f) {
  if (live <= 4) f(std::integral_constant<int, 4>{});
  else if (live <= 8) f(std::integral_constant<int, 8>{});
  else f(std::integral_constant<int, 16>{});
}

template <typename T, int D, int NQ>
__global__ void __launch_bounds__(kThreadsDec, (DecCfg<D, NQ>::kPerSm))
    attention_decode_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                            const __grid_constant__ CUtensorMap tmap_ka, const __grid_constant__ CUtensorMap tmap_va,
                            const DecParams p) {
  using C = DecCfg<D, NQ>;
  constexpr int S = C::kSlots;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_s = ring + C::kRing;                                 // [D/64][NQ rows][128 B]
  uint8_t* p_s = q_s + C::kQBytes;                                // [2 key halves][2*NQ rows][128 B]
  float* l_s = reinterpret_cast<float*>(p_s + C::kPBufs * C::kPBytes);  // [NQ][128] (NQ > 16)
  float* red = l_s + C::kLBytes / 4;                              // [NQ][4 warps]
  float* mc = red + NQ * 4;                                       // [2][NQ]: the maximum in use, the rescale factor
  float* ml = mc + 2 * NQ;                                        // [2][NQ]: this CTA's m and l
  uint64_t* bars = reinterpret_cast<uint64_t*>(ml + 2 * NQ);
  uint64_t* full = bars;
  uint64_t* empty = full + S;
  uint64_t* s_full = empty + S;  // [2]
  // [2], as each of a pair of blocks has its own: with two buffers of weights a softmax warp may
  // have arrived for block j + 1 before the issuer looks at block j, which on one barrier would
  // then read as not complete for ever.
  uint64_t* p_full = s_full + 2;
  uint64_t* pv_done = p_full + 2;  // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_done + 2);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 128) {
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
  }
  uint32_t rank, csize;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(csize));
  const int pair = blockIdx.x / csize;
  const int b = pair / p.kv_heads, hk = pair % p.kv_heads;

  pdl_wait();
  // This lane's visible keys and this CTA's share of their blocks.
  int64_t kv_row = p.row_map != nullptr ? (int64_t)p.row_map[b] : b;
  const bool bad_row = kv_row < 0 || kv_row >= p.kv_rows;
  int64_t len64 = p.tk;
  if (p.key_lens != nullptr) {
    const int64_t kl = p.key_lens[b];
    len64 = kl < 0 ? 0 : (kl < len64 ? kl : len64);
  }
  int seen = p.n_app;
  if (p.app_lens != nullptr) {
    const int s = p.app_lens[b];
    seen = s < 0 ? 0 : (s < seen ? s : seen);
  }
  if (bad_row) {  // an entry outside the cache: nothing is read, zeros, and the status word says so
    kv_row = 0, len64 = 0, seen = 0;
    if (tid == 0 && rank == 0) atomicExch(p.status, (uint32_t)kStatusBadIndex);
  }
  const int len = (int)len64;
  const int cached = (len + kKeys - 1) / kKeys;
  const int total = cached + (seen + kKeys - 1) / kKeys;
  const int per = (total + (int)csize - 1) / (int)csize;
  const int g_lo = min((int)rank * per, total);
  const int n = min(per, total - g_lo);  // blocks of this CTA (0: an empty share)

  // The loader's lane sets the barriers up and starts filling the ring before the CTA
  // meets: the first keys travel while the query rows and tensor memory are got ready.
  constexpr int kLoader = 128;
  bool ok = true;
  int at = 0;  // copies issued so far, in the ring's order
  auto load = [&]() {
    const int s = at % S;
    // K0, then K(j+1) and V(j) in turn, V(n-1) last
    const bool is_v = at == 2 * n - 1 || (at > 0 && (at & 1) == 0);
    const int g = g_lo + (at == 2 * n - 1 ? n - 1 : is_v ? at / 2 - 1 : (at + 1) / 2);
    if (at >= S && !mbar_wait(&empty[s], (at / S - 1) & 1, p.status)) {
      ok = false;
      return;
    }
    ++at;
    const bool app = g >= cached;
    const CUtensorMap* m = app ? (is_v ? &tmap_va : &tmap_ka) : (is_v ? &tmap_v : &tmap_k);
    mbar_expect_tx(&full[s], C::kSlotBytes);
    for (int c = 0; c < D / 64; ++c)
      tma_load_4d(ring + s * C::kSlotBytes + c * kBox, m, &full[s], c * 64, hk, (app ? g - cached : g) * kKeys,
                  app ? b : (int)kv_row);
  };
  if (tid == kLoader) {
    for (int i = 0; i < S; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(&s_full[0], 1);
    mbar_init(&s_full[1], 1);
    mbar_init(&p_full[0], 4);
    mbar_init(&p_full[1], 4);
    mbar_init(&pv_done[0], 1);
    mbar_init(&pv_done[1], 1);
    mbar_fence_init();
    while (at < 2 * n && at < S) load();
  }
  if (warp == 5) {
    tmem_alloc(tmem_slot, C::kTmemCols);
    tmem_relinquish();
  }
  // Query rows (zero past `rows` and past the real head dim) and zeroed weights: the
  // columns of dead rows stay zero throughout.
  if (tid < 128) {
    for (int i = tid; i < NQ * (D / 8); i += 128) {
      const int r = i / (D / 8), c = i % (D / 8);
      uint4 u = make_uint4(0, 0, 0, 0);
      if (r < p.rows && c * 8 < p.d_real)
        u = ldg128((const T*)p.q + b * p.q_sb + (r / p.group) * p.q_st + (hk * p.group + r % p.group) * p.q_sh + c * 8);
      *reinterpret_cast<uint4*>(q_s + (c >> 3) * (NQ * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = u;
    }
    for (int i = tid; i < C::kPBufs * C::kPBytes / 16; i += 128) reinterpret_cast<uint4*>(p_s)[i] = make_uint4(0, 0, 0, 0);
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_trigger();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 4) {
    if (tid == kLoader) {
      // the rest of the ring's copies
      while (ok && at < 2 * n) load();
      if (!ok)
        for (int i = 0; i < 64; ++i) __nanosleep(1000);  // copies in flight land before the CTA's memory goes
    }
  } else if (warp == 5) {
    // ---------------- MMA issuer ----------------
    constexpr uint32_t idesc_s = umma_idesc(Elem<T>::kUmmaFormat, 128, NQ, 0, 0);
    constexpr uint32_t idesc_o = umma_idesc(Elem<T>::kUmmaFormat, 128, 2 * NQ, 1, 0);
    const bool leader = elect_one();
    const uint64_t k_desc = umma_desc_sw128(smem_u32(ring), 16, 1024);
    const uint64_t v_desc = umma_desc_sw128(smem_u32(ring), kBox, 1024);
    const uint64_t q_desc = umma_desc_sw128(smem_u32(q_s), 16, 1024);
    const uint64_t p_desc = umma_desc_sw128(smem_u32(p_s), 16, 1024);
    bool ok = true;
    auto scores = [&](int j) {
      const uint32_t pos = pos_k(j);
      const int s = (int)(pos % S);
      if (!mbar_wait(&full[s], (pos / S) & 1, p.status)) {
        ok = false;
        return;
      }
      tc_fence_after();
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks)
        if (leader)
          umma_ss(tmem_base + (uint32_t)((j & 1) * NQ),
                  k_desc + (uint64_t)((s * C::kSlotBytes + (ks >> 2) * kBox) >> 4) + (uint64_t)((ks & 3) * 2),
                  q_desc + (uint64_t)(((ks >> 2) * (NQ * 128)) >> 4) + (uint64_t)((ks & 3) * 2), idesc_s, ks != 0 ? 1u : 0u);
      if (leader) {
        tc_commit(&empty[s]);
        tc_commit(&s_full[j & 1]);
      }
    };
    if (n > 0) scores(0);
    for (int j = 0; j < n && ok; ++j) {
      if (j + 1 < n) scores(j + 1);
      if (!ok || !mbar_wait(&p_full[j & 1], (j >> 1) & 1, p.status)) break;
      const uint32_t pos = pos_v(j, n);
      const int s = (int)(pos % S);
      if (!mbar_wait(&full[s], (pos / S) & 1, p.status)) break;
      tc_fence_after();
#pragma unroll
      for (int ks = 0; ks < kKeys / 16; ++ks)
        if (leader)
          umma_ss(tmem_base + 2 * NQ, v_desc + (uint64_t)((s * C::kSlotBytes) >> 4) + (uint64_t)(ks * (2048 >> 4)),
                  p_desc + (uint64_t)(((j % C::kPBufs) * C::kPBytes + (ks >> 2) * (2 * NQ * 128)) >> 4) + (uint64_t)((ks & 3) * 2), idesc_o,
                  (j | ks) != 0 ? 1u : 0u);
      if (leader) {
        tc_commit(&empty[s]);
        tc_commit(&pv_done[j & 1]);
      }
      __syncwarp();
    }
  } else {
    // ---------------- softmax: thread = key ----------------
    // Columns (query rows) go by chunks of 16. The body is one chunk's straight code: with
    // 64 columns unrolled it no longer fits the instruction cache (16 us a block against 2).
    const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
    const uint32_t o_tmem = tmem_base + 2 * NQ + lane_addr;
    const float sl2 = p.scale_log2;
    float m_run = -INFINITY;  // of column `tid`: thread c keeps the running maximum of column c
    float l_lane[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) l_lane[c] = 0.f;
    if (tid < 2 * NQ) mc[tid] = 0.f;
    if (NQ > 16)
      for (int c = 0; c < NQ; ++c) l_s[c * 128 + tid] = 0.f;
    bool live = true;  // false once a bounded wait ran out: barriers are still walked, nothing is waited for
    uint32_t sr[16];
    for (int j = 0; j < n; ++j) {
      if (live && !mbar_wait(&s_full[j & 1], (j >> 1) & 1, p.status)) live = false;
      tc_fence_after();
      const uint32_t s_tmem = tmem_base + (uint32_t)((j & 1) * NQ) + lane_addr;
      const int g = g_lo + j;
      const bool app = g >= cached;
      const int at = (app ? g - cached : g) * kKeys + tid;  // this thread's key
      const int limit = app ? seen : len;
      bool seen_key = at < limit;
      if (p.key_mask != nullptr && !app && seen_key)
        seen_key = (p.key_mask_i32 ? ((const int32_t*)p.key_mask)[b * p.tk + at]
                                   : (int)((const uint8_t*)p.key_mask)[b * p.tk + at]) != 0;
      auto load_scores = [&](int q0) {
        tmem_ld_cols(s_tmem + q0, sr);
        if (p.bias != nullptr && seen_key) {
          const int64_t keys = p.tk + p.n_app;
          const T* bp = (const T*)p.bias + (int64_t)(p.bias_per_batch ? b : 0) * p.heads * p.t * keys + (app ? p.tk : 0) + at;
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            const int q = q0 + c;
            if (q < p.rows)
              sr[c] = __float_as_uint(fmaf(
                  Elem<T>::to_f(bp[((int64_t)(hk * p.group + q % p.group) * p.t + q / p.group) * keys]), p.inv_scale,
                  __uint_as_float(sr[c])));
          }
        }
        if (!seen_key) {
#pragma unroll
          for (int c = 0; c < 16; ++c) sr[c] = 0xff800000u;
        }
      };
#pragma unroll 1
      for (int q0 = 0; q0 < p.rows; q0 += 16) {
        load_scores(q0);
        float mine = 0.f;
        auto maxima = [&](auto width) {
#pragma unroll
          for (int c = 0; c < decltype(width)::value; ++c) {
            const float wm = redux_max(__uint_as_float(sr[c]));
            if (lane == c) mine = wm;
          }
        };
        by_width(p.rows - q0, maxima);
        if (lane < 16 && q0 + lane < p.rows) red[(q0 + lane) * 4 + warp] = mine;
        if (NQ == 16) break;
      }
      named_barrier(1, 128);
      bool moved = false;
      if (tid < p.rows) {
        const float4 w4 = *reinterpret_cast<const float4*>(red + tid * 4);
        const float mx = fmaxf(fmaxf(w4.x, w4.y), fmaxf(w4.z, w4.w)) * sl2;
        float corr = 1.f;
        if (mx > m_run + kRescaleAbove || m_run == -INFINITY) {
          const float m_new = fmaxf(m_run, mx);
          if (m_new != m_run && m_run != -INFINITY) {
            corr = ex2_approx(m_run - m_new);
            moved = true;
          }
          m_run = m_new;
        }
        mc[tid] = m_run == -INFINITY ? 0.f : m_run;
        mc[NQ + tid] = corr;
      }
      moved = barrier_or(2, moved);
      if (moved) {
        // O holds the blocks before this one: rescale it once the last P.V is complete
        if (live && !mbar_wait(&pv_done[(j - 1) & 1], ((j - 1) >> 1) & 1, p.status)) live = false;
        tc_fence_after();
#pragma unroll 1
        for (int q0 = 0; q0 < p.rows; q0 += 16) {
          float f[16];
#pragma unroll
          for (int c = 0; c < 16; ++c) f[c] = mc[NQ + q0 + c];
#pragma unroll 1
          for (int half = 0; half < 2; ++half) {
            uint32_t orr[16];
            tmem_ld_cols(o_tmem + half * NQ + q0, orr);
#pragma unroll
            for (int c = 0; c < 16; ++c) orr[c] = __float_as_uint(__uint_as_float(orr[c]) * f[c]);
            tmem_st16(o_tmem + half * NQ + q0, orr);
          }
          if (NQ == 16) {
#pragma unroll
            for (int c = 0; c < 16; ++c) l_lane[c] *= f[c];
            break;
          } else {
#pragma unroll
            for (int c = 0; c < 16; ++c) l_s[(q0 + c) * 128 + tid] *= f[c];
          }
        }
        tmem_st_wait();
      }
      // the block that last used this buffer of weights has been multiplied
      if (j >= C::kPBufs && live &&
          !mbar_wait(&pv_done[(j - C::kPBufs) & 1], ((j - C::kPBufs) >> 1) & 1, p.status))
        live = false;
      uint8_t* pbox = p_s + (j % C::kPBufs) * C::kPBytes + (tid >> 6) * (2 * NQ * 128) + (tid & 7) * 2;
      const int chunk = (tid & 63) >> 3;
#pragma unroll 1
      for (int q0 = 0; q0 < p.rows; q0 += 16) {
        if (NQ > 16) load_scores(q0);
        // All loads, then the arithmetic, then all stores: the compiler may not move a load
        // of a maximum or a sum above a store of a weight, and one column after another is
        // a chain of latencies.
        auto weights = [&](auto width) {
          constexpr int W = decltype(width)::value;
          float mu[W], lv[W];
#pragma unroll
          for (int c = 0; c < W; ++c) {
            mu[c] = mc[q0 + c];
            if (NQ > 16) lv[c] = l_s[(q0 + c) * 128 + tid];
          }
          T hi[W], lo[W];
#pragma unroll
          for (int c = 0; c < W; ++c) {
            const float pr = ex2_approx(fmaf(__uint_as_float(sr[c]), sl2, -mu[c]));
            if (NQ > 16) lv[c] += pr;
            else l_lane[c] += pr;
            const float up = pr * kValueUp<T>;
            hi[c] = Elem<T>::from_f(up);
            lo[c] = Elem<T>::from_f((up - Elem<T>::to_f(hi[c])) * kRestUp<T>);
          }
#pragma unroll
          for (int c = 0; c < W; ++c) {
            uint8_t* dst = pbox + (q0 + c) * 128 + ((chunk ^ (c & 7)) << 4);
            *reinterpret_cast<T*>(dst) = hi[c];
            *reinterpret_cast<T*>(dst + NQ * 128) = lo[c];
            if (NQ > 16) l_s[(q0 + c) * 128 + tid] = lv[c];
          }
        };
        by_width(p.rows - q0, weights);
        if (NQ == 16) break;
      }
      if (limit - (at - tid) < kKeys) {
        // The block's rows past the visible keys hold whatever the cache holds there:
        // their weights are zero, and zero values keep 0 * NaN out of the sum.
        const uint32_t pos = pos_v(j, n);
        if (live && !mbar_wait(&full[pos % S], (pos / S) & 1, p.status)) live = false;
        if (at >= limit) {
          uint8_t* vr = ring + (pos % S) * C::kSlotBytes + tid * 128;
#pragma unroll
          for (int c = 0; c < D / 8; ++c)
            *reinterpret_cast<uint4*>(vr + (c >> 3) * kBox + (c & 7) * 16) = make_uint4(0, 0, 0, 0);
        }
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[j & 1]);
    }
    // ---- this CTA's state: m, l, O (f32) into shared memory ----
    if (n > 0) {
      if (live && !mbar_wait(&pv_done[(n - 1) & 1], ((n - 1) >> 1) & 1, p.status)) live = false;
      tc_fence_after();
      float* op = reinterpret_cast<float*>(ring);
#pragma unroll 1
      for (int q0 = 0; q0 < p.rows; q0 += 16) {
        float mine = 0.f;
#pragma unroll
        for (int c = 0; c < 16; ++c)
          if (q0 + c < p.rows) {
            const float s = warp_sum(NQ == 16 ? l_lane[c] : l_s[(q0 + c) * 128 + tid]);
            if (lane == c) mine = s;
          }
        if (lane < 16 && q0 + lane < p.rows) red[(q0 + lane) * 4 + warp] = mine;
        if (warp * 32 < D) {
          uint32_t lo[16];
          tmem_ld_cols(o_tmem + q0, sr);
          tmem_ld_cols(o_tmem + NQ + q0, lo);
#pragma unroll
          for (int c = 0; c < 16; ++c)
            if (q0 + c < p.rows)
              op[(q0 + c) * D + tid] =
                  fmaf(__uint_as_float(lo[c]), 1.f / kRestUp<T>, __uint_as_float(sr[c])) * (1.f / kValueUp<T>);
        }
        if (NQ == 16) break;
      }
      named_barrier(1, 128);
    }
    if (tid < p.rows) {
      float l = 0.f;
      if (n > 0) {
        const float4 w4 = *reinterpret_cast<const float4*>(red + tid * 4);
        l = (w4.x + w4.y) + (w4.z + w4.w);
      }
      ml[tid] = n > 0 ? m_run : -INFINITY;
      ml[NQ + tid] = l;
    }
    tc_fence_before();
  }
  __syncwarp();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
  // ---- merge the cluster's partial states: CTA `rank` takes every csize-th run of columns ----
  cluster_sync_all();
  {
    const int per_row = p.d_real / 8;
    const uint32_t op_addr = smem_u32(ring), ml_addr = smem_u32(ml);
    for (int i = (int)rank * kThreadsDec + tid; i < p.rows * per_row; i += (int)csize * kThreadsDec) {
      const int c = i / per_row, d0 = (i % per_row) * 8;
      auto peer = [&](uint32_t addr, uint32_t r) {
        uint32_t out;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(addr), "r"(r));
        return out;
      };
      float m = -INFINITY;
      for (uint32_t r = 0; r < csize; ++r) m = fmaxf(m, ld_cluster_f32(peer(ml_addr + c * 4, r)));
      float l = 0.f, acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (uint32_t r = 0; r < csize; ++r) {
        const float mr = ld_cluster_f32(peer(ml_addr + c * 4, r));
        const float lr = ld_cluster_f32(peer(ml_addr + (NQ + c) * 4, r));
        if (lr == 0.f) continue;  // the share saw no key (its sum says so: NaN scores leave the maximum at -inf too)
        const float w = mr == -INFINITY ? 1.f : ex2_approx(mr - m);
        l = fmaf(w, lr, l);
        const uint32_t src = peer(op_addr + (c * D + d0) * 4, r);
        const float4 x = ld_cluster_f32x4(src), y = ld_cluster_f32x4(src + 16);
        acc[0] = fmaf(w, x.x, acc[0]), acc[1] = fmaf(w, x.y, acc[1]), acc[2] = fmaf(w, x.z, acc[2]);
        acc[3] = fmaf(w, x.w, acc[3]), acc[4] = fmaf(w, y.x, acc[4]), acc[5] = fmaf(w, y.y, acc[5]);
        acc[6] = fmaf(w, y.z, acc[6]), acc[7] = fmaf(w, y.w, acc[7]);
      }
      const float inv = l == 0.f ? 0.f : 1.0f / l;
      const int64_t tq = c / p.group;
      const int h = hk * p.group + c % p.group;
      stg128((T*)p.o + b * p.o_sb + tq * p.o_st + h * p.o_sh + d0,
             make_uint4(Elem<T>::pack(acc[0] * inv, acc[1] * inv), Elem<T>::pack(acc[2] * inv, acc[3] * inv),
                        Elem<T>::pack(acc[4] * inv, acc[5] * inv), Elem<T>::pack(acc[6] * inv, acc[7] * inv)));
      if (p.lse != nullptr && d0 == 0)
        p.lse[((int64_t)b * p.heads + h) * p.t + tq] = l == 0.f ? -INFINITY : kLn2F * (m + log2f(l));
    }
  }
  cluster_sync_all();  // no CTA leaves while a peer still reads its partial state
}

int sm_count_dec() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  return sms;
}

int64_t dec_blocks(const AttnArgs& a) { return (a.tk + kKeys - 1) / kKeys + (a.n_app + kKeys - 1) / kKeys; }

// Shares per (lane, KV head): as many as bring the grid to the CTAs the chip holds at
// once; a second wave of short shares costs its fixed 5 us again (B10 x 4 heads x 1750
// keys: 12.7 us with 4 shares, 19.9 with 8). Shares that stay at 32 blocks or more hide
// that, and lanes of unequal length then balance better (B16 x 16 heads x 16384 keys,
// lengths from 5000: 68 us with 4 shares, 110 with 1). 16 is the largest cluster.
// A cluster has to find its CTAs' places within one GPC, and large ones do not all find
// them: sixteen CTAs are worth it up to six clusters per CTA an SM holds (24 pairs x 61
// blocks, three an SM: 21.8 us in sixteen, 14.1 in eight; 16 pairs x 126 blocks 16.6 against
// 21.1), eight with one CTA an SM up to twelve (16 pairs x 32 blocks x 32 rows: 41.8 us in
// eight, 31.2 in four; 8 pairs 22.7 against 31.2).
int dec_cluster(int64_t pairs, int64_t blocks, int per_sm) {
  const int64_t room = (int64_t)sm_count_dec() * per_sm;
  int csize = 1;
  while (csize < 16 && csize * 2 <= blocks &&
         (pairs * csize * 2 <= room || (pairs * csize < 4 * room && blocks >= 32 * csize * 2))) {
    if (csize == 8 && pairs > 6 * per_sm) break;
    if (csize == 4 && per_sm == 1 && pairs > 12) break;
    csize *= 2;
  }
  return csize;
}

template <typename T, int D, int NQ>
int run_dec(const AttnArgs& a, cudaStream_t s, char* cfg, size_t cfg_len) {
  using C = DecCfg<D, NQ>;
  const uint32_t box[4] = {64, 1, kKeys, 1};
  CUtensorMap tk, tv, tka, tva;
  {
    const uint64_t dims[4] = {(uint64_t)a.d, (uint64_t)a.kv_heads, (uint64_t)a.tk, (uint64_t)a.kv_rows};
    const uint64_t stk[3] = {(uint64_t)a.k_sh, (uint64_t)a.k_st, (uint64_t)a.k_sb};
    const uint64_t stv[3] = {(uint64_t)a.v_sh, (uint64_t)a.v_st, (uint64_t)a.v_sb};
    if (!make_tmap(&tk, a.k, a.dtype, 4, dims, stk, box)) return -1;
    if (!make_tmap(&tv, a.v, a.dtype, 4, dims, stv, box)) return -1;
  }
  tka = tk, tva = tv;
  if (a.n_app > 0) {
    const uint64_t row = (uint64_t)a.kv_heads * a.d;
    const uint64_t dims[4] = {(uint64_t)a.d, (uint64_t)a.kv_heads, (uint64_t)a.n_app, (uint64_t)a.batch};
    const uint64_t st[3] = {(uint64_t)a.d, row, row * (uint64_t)a.n_app};
    if (!make_tmap(&tka, a.k_app, a.dtype, 4, dims, st, box)) return -1;
    if (!make_tmap(&tva, a.v_app, a.dtype, 4, dims, st, box)) return -1;
  }
  static bool attr_seen[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_seen[dev & 63]) {
    if (cudaFuncSetAttribute(attention_decode_kernel<T, D, NQ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)C::kSmem) != cudaSuccess ||
        cudaFuncSetAttribute(attention_decode_kernel<T, D, NQ>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
            cudaSuccess)
      return -1;
    attr_seen[dev & 63] = true;
  }
  DecParams p{};
  p.q = a.q, p.o = a.o;
  p.q_sb = a.q_sb, p.q_st = a.q_st, p.q_sh = a.q_sh;
  p.o_sb = a.o_sb, p.o_st = a.o_st, p.o_sh = a.o_sh;
  p.t = a.t, p.tk = a.tk, p.batch = a.batch, p.kv_rows = a.kv_rows;
  p.heads = a.heads, p.kv_heads = a.kv_heads, p.group = a.heads / a.kv_heads;
  p.rows = (int)a.t * p.group;
  p.d_real = a.d;
  p.scale_log2 = a.scale * kLog2eF;
  p.inv_scale = 1.0f / a.scale;
  p.key_lens = a.key_lens, p.key_mask = a.key_mask, p.key_mask_i32 = a.key_mask_i32;
  p.row_map = a.row_map;
  p.n_app = a.n_app, p.app_lens = a.app_lens;
  p.bias = a.bias, p.bias_per_batch = a.bias_per_batch;
  p.lse = a.lse, p.status = a.status;
  const int64_t pairs = a.batch * a.kv_heads;
  const int csize = dec_cluster(pairs, dec_blocks(a), C::kPerSm);
  if (launch_pdl(attention_decode_kernel<T, D, NQ>, dim3((unsigned)(pairs * csize)), dim3(kThreadsDec), C::kSmem, s,
                 (unsigned)csize, a.batch * a.t, tk, tv, tka, tva, p) != cudaSuccess)
    return -1;
  if (cfg != nullptr)
    snprintf(cfg, cfg_len, "{rows:%d,bkv:%d,d:%d,stages:%d,splits:1,cluster:%d}", NQ, kKeys, a.d, C::kSlots, csize);
  return 0;
}

template <typename T, int D>
int run_dec_rows(const AttnArgs& a, cudaStream_t s, char* cfg, size_t cfg_len) {
  const int64_t rows = a.t * (a.heads / a.kv_heads);
  if (rows <= 16) return run_dec<T, D, 16>(a, s, cfg, cfg_len);
  if (rows <= 32) return run_dec<T, D, 32>(a, s, cfg, cfg_len);
  return run_dec<T, D, 64>(a, s, cfg, cfg_len);
}

}  // namespace

// No mask that depends on the query row, and up to 16 query rows per KV head: always.
// With 17 to 64 rows a block of 128 keys costs a CTA here 2.6 us (up to 32 rows) or 4.5 us,
// shared by its cluster; the 256-row tile kernels take 1.55 us for it per head (per pair of
// heads once there are more pairs than SMs), whatever the rows, and never share a head's
// keys: the cheaper of the two takes the call (B1 x T4 x 8 heads a KV head, 16000 keys: 34 us
// here, 203 there; B2 x T16 x 4 heads, 20510 keys: 180 | 249; B32 x T16 x 4 heads, 4000
// keys: 435 | 320). Appended rows of up to 64 rows always come here, not to the exact
// kernel (B5 x T16 x 4 x 8, 1111 + 3 keys: 48 us against 1.1 ms). Key splits the caller asked
// for stay with the kernel that leaves them in the caller's workspace, appended rows excepted.
bool attention_decode_covers(const AttnArgs& a) {
  AttnArgs plain = a;
  plain.splits = 1;
  plain.bias = nullptr;
  plain.n_app = 0;
  if (!attention_tc_covers(plain)) return false;
  if (a.causal || a.has_window || a.has_chunk || a.seg_start != nullptr) return false;
  if (a.splits > 1 && a.n_app == 0) return false;
  const int64_t group = a.heads / a.kv_heads, rows = a.t * group;
  if (a.t > 64 || rows > 64) return false;
  const int64_t pairs = a.batch * a.kv_heads;
  if (pairs > (1 << 26)) return false;
  if (a.n_app > 0) return aligned16(a.k_app) && aligned16(a.v_app);
  if (rows <= 16) return true;
  const int64_t sms = sm_count_dec(), blocks = dec_blocks(a);
  const int64_t c = dec_cluster(pairs, blocks, 1);
  const int64_t head_pairs = group % 2 == 0 ? a.batch * a.heads / 2 : 0;
  const int64_t items = head_pairs > sms ? head_pairs : a.batch * a.heads;
  auto up = [](int64_t x, int64_t y) { return (double)((x + y - 1) / y); };
  const double here = 8.0 + (rows <= 32 ? 2.6 : 4.5) * up(blocks, c) * up(pairs * c, sms);
  const double there = 4.0 + 1.55 * (double)blocks * up(items, sms);
  return here < 0.9 * there;
}

int launch_attention_decode(const AttnArgs& a, cudaStream_t s, char* cfg, size_t cfg_len) {
  if (!attention_decode_covers(a)) return 1;
  if (a.dtype == SVODB_BF16)
    return a.d > 64 ? run_dec_rows<__nv_bfloat16, 128>(a, s, cfg, cfg_len) : run_dec_rows<__nv_bfloat16, 64>(a, s, cfg, cfg_len);
  return a.d > 64 ? run_dec_rows<__half, 128>(a, s, cfg, cfg_len) : run_dec_rows<__half, 64>(a, s, cfg, cfg_len);
}

}  // namespace svodb
