// The row layout of a padded batch: which positions of [B, L] a stack has to compute.
//
// A batch padded to its longest row (and that to a plan's length) spends its GEMMs, norms
// and attention on padding: 64 passages of 64..512 tokens in a [64, 512] plan are 57 % real.
// The layout packs the rows end to end: row b keeps the positions up to its last real token,
// rounded up to whole blocks of kRowBlock. The block is the attention kernel's key block, so
// that no key block holds keys of two rows (a masked key's V still enters the product, and
// 0 * inf is not 0), and half a GEMM tile, so that a tile's rotation-table rows are two runs.
// The lengths live on the device (a captured plan serves every batch of its shape), so the
// kernels read `live` and walk that many rows of tensors that keep their padded capacity.
//
// One block per batch row finds its last real token and writes the mask as bytes; the block
// that finishes last sums up the starts and writes the blocks' (row, position) table.
// Latency-bound: a few us a batch against 0.1 ms and more of a stack. Padded -> packed, whole
// stacks: XLM-R 64 x 512 with rows of 64..512 tokens 22.0 -> 15.1 ms, ModernBERT 16 x 8192 with
// rows of 2048..8192 60.6 -> 42.5 ms, 7 rows of 35..301 1.65 -> 1.47 ms; Qwen3 32 x 4096 without
// padding 157 ms either way.
#include "common.cuh"
#include "kernels.h"
#include "launch.h"

namespace svodb {

namespace {

constexpr int kLayoutThreads = 256;
constexpr int kHeader = 4;  // words before the arrays: rows in all, batch rows done, 2 unused

__global__ void __launch_bounds__(kLayoutThreads) row_layout_kernel(const RowLayoutArgs a, int64_t padded) {
  __shared__ int red[2][kLayoutThreads / 32];
  __shared__ int last_block;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t b = blockIdx.x;
  // First kernel of a stack: the next one comes up only once all before it is done.
  pdl_wait();
  pdl_trigger();
  int32_t* start = a.table + kHeader;
  int32_t* keys = start + a.batch;
  int32_t* rows = keys + a.batch;
  int32_t* holes = rows + a.batch;
  int32_t* block_seq = holes + a.batch;
  int32_t* block_pos = block_seq + a.batch * (padded / kRowBlock);

  int last_set = 0, first_zero = 0x7fffffff;
  if (a.mask != nullptr) {
    const uint8_t* m8 = (const uint8_t*)a.mask + b * a.len;
    uint8_t* out = a.mask_out != nullptr ? a.mask_out + b * padded : nullptr;
    if (!a.mask_i32 && (a.len & 15) == 0 && ((reinterpret_cast<uintptr_t>(a.mask) | reinterpret_cast<uintptr_t>(a.mask_out)) & 15) == 0) {
      for (int c = tid; c < (int)(a.len >> 4); c += kLayoutThreads) {
        const uint4 u = ldg128(m8 + c * 16);
        const uint32_t wd[4] = {u.x, u.y, u.z, u.w};
        uint32_t bits[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t set = __vcmpne4(wd[q], 0u);
          const int at = c * 16 + q * 4;
          if (set != 0u) last_set = max(last_set, at + ((31 - __clz((int)set)) >> 3) + 1);
          if (set != 0xffffffffu) first_zero = min(first_zero, at + ((__ffs((int)~set) - 1) >> 3));
          bits[q] = set & 0x01010101u;
        }
        if (out != nullptr) stg128(out + c * 16, make_uint4(bits[0], bits[1], bits[2], bits[3]));
      }
    } else {
      for (int64_t j = tid; j < a.len; j += kLayoutThreads) {
        const bool set = a.mask_i32 ? ((const int32_t*)a.mask)[b * a.len + j] != 0 : m8[j] != 0;
        if (set) last_set = (int)j + 1;
        else if ((int)j < first_zero) first_zero = (int)j;
        if (out != nullptr) out[j] = set ? 1 : 0;
      }
    }
    if (out != nullptr)
      for (int64_t j = a.len + tid; j < padded; j += kLayoutThreads) out[j] = 0;
  } else {
    const int n = a.lengths[b];
    // a row without tokens pools its first position, which under a causal mask sees itself
    last_set = n < 1 ? 1 : (n < a.len ? n : (int)a.len);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    last_set = max(last_set, __shfl_xor_sync(0xffffffffu, last_set, o));
    first_zero = min(first_zero, __shfl_xor_sync(0xffffffffu, first_zero, o));
  }
  if (lane == 0) red[0][warp] = last_set, red[1][warp] = first_zero;
  __syncthreads();
  if (tid == 0) {
    for (int i = 1; i < kLayoutThreads / 32; ++i) last_set = max(last_set, red[0][i]), first_zero = min(first_zero, red[1][i]);
    keys[b] = last_set;
    // a row with no real token keeps its first block: CLS pooling reads its first position
    rows[b] = (max(last_set, 1) + kRowBlock - 1) / kRowBlock * kRowBlock;
    holes[b] = first_zero < last_set ? 1 : 0;
    __threadfence();
    last_block = atomicAdd(&a.table[1], 1) == (int)a.batch - 1;
  }
  __syncthreads();
  if (!last_block) return;
  __threadfence();
  // The other blocks' counts are read past the L1, which may hold nothing of them anyway.
  if (warp == 0) {
    int at = 0;
    for (int64_t b0 = 0; b0 < a.batch; b0 += 32) {
      const int mine = b0 + lane < a.batch ? __ldcg(rows + b0 + lane) : 0;
      int sum = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += up;
      }
      if (b0 + lane < a.batch) start[b0 + lane] = at + sum - mine;
      at += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) {
      a.table[0] = at;
      a.table[1] = 0;  // as the next launch wants it
    }
  }
  __syncthreads();
  for (int64_t r = warp; r < a.batch; r += kLayoutThreads / 32) {
    const int first = start[r] / kRowBlock, n = __ldcg(rows + r) / kRowBlock;
    for (int i = lane; i < n; i += 32) {
      block_seq[first + i] = (int)r;
      block_pos[first + i] = i * kRowBlock;
    }
  }
}

int64_t padded_len(int64_t len) { return (len + kRowBlock - 1) / kRowBlock * kRowBlock; }

}  // namespace

size_t row_layout_ints(int64_t batch, int64_t len) {
  return (size_t)(kHeader + 4 * batch + 2 * batch * (padded_len(len) / kRowBlock));
}

RowLayout row_layout_of(int64_t batch, int64_t len, const int32_t* table) {
  RowLayout l{};
  l.batch = batch, l.len = padded_len(len);
  l.live = table;
  l.start = table + kHeader;
  l.keys = l.start + batch;
  l.rows = l.keys + batch;
  l.holes = l.rows + batch;
  l.block_seq = l.holes + batch;
  l.block_pos = l.block_seq + batch * (l.len / kRowBlock);
  return l;
}

void launch_row_layout(const RowLayoutArgs& a, cudaStream_t s) {
  launch_pdl(row_layout_kernel, dim3((unsigned)a.batch), dim3(kLayoutThreads), 0, s, 1, a.batch * a.len, a, padded_len(a.len));
}

}  // namespace svodb
