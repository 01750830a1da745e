// Exact attention of f32 operands on the CUDA cores, register-tiled: the f32 cases of the
// exact path (attention_generic.cu keeps every other type, head dim, bias, key splits and
// appended rows). f32 products, sums and exponentials throughout, as there.
//
// What bounds it: the FMA pipe (B2 x H8 x 512 x 512 x 64 is 0.27 G multiply-adds in each
// product, 14 us for both at the chip's 37 T a second, 13 for the keys of the case below). The generic kernel read two shared-memory words
// per multiply-add (232 us with key lengths 256..512, 34 here; B4 x H8 x 1024 x 1024 x 128
// 2278 -> 417 us, 31 TFLOP/s; B2 x 20 queries x 1000 keys 378 -> 19 us). Here a thread
// owns 4 query rows x 4 keys of a 64 x 64 score tile and 4 rows x D/16 columns of the output,
// walks the inner dimension four at a time (8 x 16-byte shared loads, most of them broadcast,
// for 64 multiply-adds) and accumulates pairs with packed FMAs, which leaves issue slots for
// the loads.
//
// 256 threads: thread (ty, tx) = (tid / 16, tid % 16) has rows 4*ty .. 4*ty+3 and keys
// tx + 16*c. The 16 lanes of a row group sit in one half-warp, so the row statistics are
// shuffles and the weights pass from the first product to the second through shared memory
// with a warp barrier only. K and V tiles arrive by cp.async, one tile ahead.
#include <math.h>

#include "common.cuh"
#include "kernels.h"
#include "svodb.h"

namespace svodb {

namespace {

constexpr int kTile = 64;
constexpr int kThreadsF = 256;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

template <int D>
struct F32Cfg {
  static constexpr int kPitch = D + 4;      // 16-byte pieces of 8 rows fall in distinct banks
  static constexpr int kPPitch = kTile + 4;
  static constexpr size_t kSmem = sizeof(float) * (size_t)(5 * kTile * kPitch + kTile * kPPitch);
};

__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// A float (or four) of CTA `rank` of this cluster, at the place `p` has in this one.
__device__ __forceinline__ float ld_peer(const float* p, int rank) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_map(p, (uint32_t)rank)) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_peer4(const float* p, int rank) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(cluster_map(p, (uint32_t)rank))
               : "memory");
  return v;
}

__device__ __forceinline__ bool hidden(const AttnArgs& a, int64_t b, int64_t i, int64_t j, int64_t len) {
  if (j >= len) return true;
  if (a.causal && j > i) return true;
  if (a.has_window && (j + a.win_left < i || j > i + a.win_right)) return true;
  if (a.has_chunk) {
    const int64_t cj = j / a.chunk_size, ci = i / a.chunk_size;
    if (cj > ci + a.chunk_right) return true;
    if (a.chunk_left >= 0 && cj + a.chunk_left < ci) return true;
  }
  if (a.key_mask != nullptr) {
    const int64_t at = b * a.tk + j;
    const int m = a.key_mask_i32 ? ((const int32_t*)a.key_mask)[at] : (int)((const uint8_t*)a.key_mask)[at];
    if (m == 0) return true;
  }
  if (a.seg_start != nullptr && j < (int64_t)a.seg_start[b * a.t + i]) return true;
  return false;
}

template <int D>
__global__ void __launch_bounds__(kThreadsF, D == 64 ? 2 : 1) attention_f32_kernel(const AttnArgs a, const int shares) {
  using C = F32Cfg<D>;
  constexpr int PT = C::kPitch, PP = C::kPPitch;
  constexpr int DC = D / 64;  // 4-column groups of the output per thread: columns 64*g + 4*tx
  extern __shared__ __align__(16) float sm[];
  float* q_s = sm;                        // [64][PT]
  float* k_s = q_s + kTile * PT;          // [2][64][PT]
  float* v_s = k_s + 2 * kTile * PT;      // [2][64][PT]
  float* p_s = v_s + 2 * kTile * PT;      // [64][PP]
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int h = blockIdx.y;
  const int64_t b = blockIdx.z;
  const int hk = h / (a.heads / a.kv_heads);
  // heavier (later, under a causal mask) query tiles first
  const int64_t i0 = (int64_t)(gridDim.x / shares - 1 - blockIdx.x / shares) * kTile;
  const int64_t i_last = (i0 + kTile < a.t ? i0 + kTile : a.t) - 1;
  int64_t kv_row = a.row_map != nullptr ? (int64_t)a.row_map[b] : b;
  const bool bad_row = kv_row < 0 || kv_row >= a.kv_rows;
  if (bad_row) {  // an entry outside the cache: nothing is read, the lane sees no key, the status word says so
    kv_row = 0;
    if (tid == 0 && a.status != nullptr) atomicExch(a.status, (uint32_t)kStatusBadIndex);
  }
  const float* q = (const float*)a.q + b * a.q_sb + h * a.q_sh;
  const float* k = (const float*)a.k + kv_row * a.k_sb + hk * a.k_sh;
  const float* v = (const float*)a.v + kv_row * a.v_sb + hk * a.v_sh;
  const float sc = a.scale * kLog2e;
  int64_t len = a.tk;
  if (a.key_lens != nullptr) {
    const int64_t kl = a.key_lens[b];
    len = kl < 0 ? 0 : (kl < len ? kl : len);
  }
  if (bad_row) len = 0;
  // The key tiles any row of this tile can see.
  int64_t j_lo = 0, j_hi = len;
  if (a.causal && i_last + 1 < j_hi) j_hi = i_last + 1;
  if (a.has_window) {
    if (i0 - a.win_left > j_lo) j_lo = i0 - a.win_left;
    if (i_last + a.win_right + 1 < j_hi) j_hi = i_last + a.win_right + 1;
  }
  int64_t t_lo = j_lo / kTile, t_hi = j_hi > j_lo ? (j_hi + kTile - 1) / kTile : j_lo / kTile;
  // this CTA's share of them
  const int rank = (int)cluster_ctarank();
  const int per = (int)((t_hi - t_lo + shares - 1) / shares);
  t_lo = t_lo + rank * per < t_hi ? t_lo + rank * per : t_hi;
  t_hi = t_lo + per < t_hi ? t_lo + per : t_hi;
  const bool masked = a.causal || a.has_window || a.has_chunk || a.key_mask != nullptr || a.seg_start != nullptr;

  auto load_rows = [&](float* dst, const float* src, int64_t stride, int64_t first, int64_t limit) {
    for (int e = tid; e < kTile * (D / 4); e += kThreadsF) {
      const int r = e / (D / 4), c = (e % (D / 4)) * 4;
      const bool ok = first + r < limit && c < a.d;
      cp_async16(dst + r * PT + c, src + (ok ? (first + r) * stride + c : 0), ok);
    }
  };
  load_rows(q_s, q, a.q_st, i0, a.t);
  if (t_lo < t_hi) {
    load_rows(k_s, k, a.k_st, t_lo * kTile, len);
    load_rows(v_s, v, a.v_st, t_lo * kTile, len);
  }
  cp_async_commit();

  float m[4], l[4];
  float2 o[4][2 * DC];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    m[r] = -INFINITY, l[r] = 0.f;
#pragma unroll
    for (int c = 0; c < 2 * DC; ++c) o[r][c] = make_float2(0.f, 0.f);
  }
  for (int64_t t = t_lo; t < t_hi; ++t) {
    const int buf = (int)((t - t_lo) & 1);
    if (t + 1 < t_hi) {
      load_rows(k_s + (buf ^ 1) * kTile * PT, k, a.k_st, (t + 1) * kTile, len);
      load_rows(v_s + (buf ^ 1) * kTile * PT, v, a.v_st, (t + 1) * kTile, len);
      cp_async_commit();
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const float* ks = k_s + buf * kTile * PT;
    const float* vs = v_s + buf * kTile * PT;
    // scores: even and odd inner positions in the two halves of a pair
    float2 acc[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
      float4 qv[4], kv[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) qv[r] = *reinterpret_cast<const float4*>(q_s + (4 * ty + r) * PT + d);
#pragma unroll
      for (int c = 0; c < 4; ++c) kv[c] = *reinterpret_cast<const float4*>(ks + (tx + 16 * c) * PT + d);
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          acc[r][c] = __ffma2_rn(make_float2(qv[r].x, qv[r].y), make_float2(kv[c].x, kv[c].y), acc[r][c]);
          acc[r][c] = __ffma2_rn(make_float2(qv[r].z, qv[r].w), make_float2(kv[c].z, kv[c].w), acc[r][c]);
        }
    }
    const bool check = masked || (t + 1) * kTile > len;
    float s[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        s[r][c] = (acc[r][c].x + acc[r][c].y) * sc;
        if (check && hidden(a, b, i0 + 4 * ty + r < a.t ? i0 + 4 * ty + r : a.t - 1, t * kTile + tx + 16 * c, len))
          s[r][c] = -INFINITY;
      }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      float mx = fmaxf(fmaxf(s[r][0], s[r][1]), fmaxf(s[r][2], s[r][3]));
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
      const float m_new = fmaxf(m[r], mx);
      const float use = m_new == -INFINITY ? 0.f : m_new;
      const float corr = exp2f(m[r] - use);  // 0 for the first visible tile
      float sum = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float p = exp2f(s[r][c] - use);
        sum += p;
        p_s[(4 * ty + r) * PP + tx + 16 * c] = p;
      }
#pragma unroll
      for (int x = 8; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
      l[r] = l[r] * corr + sum;
      m[r] = m_new;
#pragma unroll
      for (int c = 0; c < 2 * DC; ++c) o[r][c].x *= corr, o[r][c].y *= corr;
    }
    __syncwarp();
#pragma unroll 4
    for (int j = 0; j < kTile; j += 4) {
      float4 pv[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) pv[r] = *reinterpret_cast<const float4*>(p_s + (4 * ty + r) * PP + j);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
#pragma unroll
        for (int g = 0; g < DC; ++g) {
          const float4 vv = *reinterpret_cast<const float4*>(vs + (j + e) * PT + g * 64 + tx * 4);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const float p = e == 0 ? pv[r].x : e == 1 ? pv[r].y : e == 2 ? pv[r].z : pv[r].w;
            o[r][2 * g] = __ffma2_rn(make_float2(p, p), make_float2(vv.x, vv.y), o[r][2 * g]);
            o[r][2 * g + 1] = __ffma2_rn(make_float2(p, p), make_float2(vv.z, vv.w), o[r][2 * g + 1]);
          }
        }
      }
    }
    __syncthreads();  // the buffer is read before the tile after next lands in it
  }
  cp_async_wait<0>();
  if (shares > 1) {
    // Merge the cluster's states: every CTA leaves its rows' O (not yet divided), m and l in
    // its shared memory, and CTA `rank` combines every shares-th row.
    float* o_s = k_s;  // [64][PT]: the last tile has been read (the loop ends on a barrier)
    float* ml = p_s;   // [2][64]
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
      for (int g = 0; g < DC; ++g)
        *reinterpret_cast<float4*>(o_s + (4 * ty + r) * PT + g * 64 + tx * 4) =
            make_float4(o[r][2 * g].x, o[r][2 * g].y, o[r][2 * g + 1].x, o[r][2 * g + 1].y);
      if (tx == 0) ml[4 * ty + r] = m[r], ml[kTile + 4 * ty + r] = l[r];
    }
    cluster_sync_all();
    const int cols = a.d / 4, rows = kTile / shares;
    for (int e = tid; e < rows * cols; e += kThreadsF) {
      const int row = (e / cols) * shares + rank, c = (e % cols) * 4;
      const int64_t i = i0 + row;
      if (i >= a.t) continue;
      float mx = -INFINITY;
      for (int r = 0; r < shares; ++r) mx = fmaxf(mx, ld_peer(ml + row, r));
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      float sum = 0.f;
      for (int r = 0; r < shares; ++r) {
        const float mr = ld_peer(ml + row, r);
        const float lr = ld_peer(ml + kTile + row, r);
        if (lr == 0.f) continue;  // the share saw no key (its sum says so: NaN scores leave the maximum at -inf too)
        const float w = mr == -INFINITY ? 1.f : exp2f(mr - mx);
        sum = fmaf(w, lr, sum);
        const float4 x = ld_peer4(o_s + row * PT + c, r);
        acc.x = fmaf(w, x.x, acc.x), acc.y = fmaf(w, x.y, acc.y), acc.z = fmaf(w, x.z, acc.z), acc.w = fmaf(w, x.w, acc.w);
      }
      const float inv = sum == 0.f ? 0.f : 1.0f / sum;
      *reinterpret_cast<float4*>((float*)a.o + b * a.o_sb + i * a.o_st + h * a.o_sh + c) =
          make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
      if (a.lse != nullptr && c == 0)
        a.lse[(b * a.heads + h) * a.t + i] = sum == 0.f ? -INFINITY : kLn2 * (mx + log2f(sum));
    }
    cluster_sync_all();  // no CTA leaves while a peer still reads its state
    return;
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int64_t i = i0 + 4 * ty + r;
    if (i >= a.t) continue;
    const float inv = l[r] == 0.f ? 0.f : 1.0f / l[r];
    float* out = (float*)a.o + b * a.o_sb + i * a.o_st + h * a.o_sh;
#pragma unroll
    for (int g = 0; g < DC; ++g)
      if (g * 64 + tx * 4 < a.d)
        *reinterpret_cast<float4*>(out + g * 64 + tx * 4) =
            make_float4(o[r][2 * g].x * inv, o[r][2 * g].y * inv, o[r][2 * g + 1].x * inv, o[r][2 * g + 1].y * inv);
    if (a.lse != nullptr && tx == 0)
      a.lse[(b * a.heads + h) * a.t + i] = l[r] == 0.f ? -INFINITY : kLn2 * (m[r] + log2f(l[r]));
  }
}

template <int D>
int run_f32(const AttnArgs& a, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(attention_f32_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)F32Cfg<D>::kSmem);
  if (e != cudaSuccess) return (int)e;
  // Query tiles that do not fill the chip (two CTAs an SM at D <= 64) share a lane's keys over
  // a cluster of 2, 4 or 8 CTAs, no share below two key tiles.
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t tiles = (a.t + kTile - 1) / kTile, ctas = tiles * a.heads * a.batch;
  const int64_t room = (int64_t)sms * (D == 64 ? 2 : 1), key_tiles = (a.tk + kTile - 1) / kTile;
  int shares = 1;
  while (shares < 8 && ctas * shares * 2 <= room && key_tiles >= shares * 4) shares *= 2;
  cudaLaunchConfig_t lc{};
  lc.gridDim = dim3((unsigned)(tiles * shares), (unsigned)a.heads, (unsigned)a.batch);
  lc.blockDim = dim3(kThreadsF, 1, 1);
  lc.dynamicSmemBytes = F32Cfg<D>::kSmem;
  lc.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)shares;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  lc.attrs = attr;
  lc.numAttrs = 1;
  if (cudaLaunchKernelEx(&lc, attention_f32_kernel<D>, a, shares) != cudaSuccess) return -1;
  return 0;
}

}  // namespace

// f32 rows on the 16-byte grid (head dim and strides multiples of 4) up to 128 wide; head
// dims below 64 or 128 run zero-padded. One or a few query rows would leave the 64-row tile
// idle: those stay with the generic kernel.
bool attention_f32_covers(const AttnArgs& a) {
  if (a.dtype != SVODB_F32 || a.d > 128 || a.d % 4 != 0) return false;
  if (a.bias != nullptr || a.splits > 1 || a.n_app > 0 || a.t < 16 || a.tk < 1) return false;
  const int64_t strides[] = {a.q_sb, a.q_st, a.q_sh, a.k_sb, a.k_st, a.k_sh, a.v_sb, a.v_st, a.v_sh, a.o_sb, a.o_st, a.o_sh};
  for (int64_t st : strides)
    if (st % 4 != 0) return false;
  return aligned16(a.q) && aligned16(a.k) && aligned16(a.v) && aligned16(a.o);
}

int launch_attention_f32(const AttnArgs& a, cudaStream_t s) { return a.d > 64 ? run_f32<128>(a, s) : run_f32<64>(a, s); }

}  // namespace svodb
