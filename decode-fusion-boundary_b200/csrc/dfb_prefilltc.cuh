// Causal prefill attention on the 5th-generation tensor cores: the reference's flash_attn_varlen_func call
// (causal = True, layers/attention.py:64-70), for both of its cases.  Without a prefix cache K / V are the
// fresh projections of the same tokens; with one they are read from the paged cache through the block tables,
// the keys of a sequence outnumber its queries, and query i attends to keys 0 .. i + (keys - queries).  Two 128-row query
// tiles per CTA, P in tensor memory as the A operand and warps of its own for the rescaling are the published FlashAttention
// method for this architecture.
//
//   * A work item is 128 query rows of the two query heads that share a KV head (an even number of query heads
//     per KV head), or 256 query rows of one head (an odd number): two M = 128 tiles that share every K / V
//     tile.  Persistent CTAs, one per SM, walk the items from the longest to the shortest.
//   * Warp 10 loads the two Q tiles and a ring of eight 16 KB stages (K and V tiles of 64 keys) with TMA boxes
//     (128-byte swizzle), the end of a sequence as 8-row boxes and 16-byte cp.async pieces.
//   * Warps 8 and 9 issue tcgen05.mma, each for one tile: S = Q K^T (K-major operands from shared memory) and O += P V
//     with P as the A operand in tensor memory and V as an MN-major B operand.  Tensor memory holds O of both tiles (128 columns
//     each) and two S buffers per tile (64 columns); P overwrites the first half of its S.  S(j + 1) is computed
//     while the softmax works on S(j), so the softmax never waits for a matrix product.  MMAs of one issuing
//     thread execute in order: S(j + 2) may be issued behind the P V that still reads P(j) from the same columns.
//   * Warps 0-3 and 4-7 are the softmax of tile 0 and 1, one thread per query row: the row of S comes out with
//     two tcgen05.ld, maximum, exp2, bf16, back with tcgen05.st; no shuffles, no shared memory.
//   * Warps 11-14 multiply the rows of O whose maximum has grown, while the softmax warps compute the exponentials
//     of the same key tile; P V of the tile waits for both.  (The split form has no registers left for them: its
//     softmax threads do it themselves behind the store of P.)
//
// Rounding: a probability is rounded to bf16 relative to its row's running maximum, so that the largest one is
// exactly 1, and the row sum adds the rounded values.  Both count: with O rescaled only when a maximum has grown by
// more than 2^8 the error against 64 bits was 2-8 % larger, with a sum over the unrounded values as well 11-24 % (scores
// of four times the usual spread; 1-5 % at the usual one), which was 8-12 % of the time (4 x 2,048 tokens 72.7 us
// against 82.5, the thirteen prompts below 117 against 134, split form 512 tokens 10.5 against 11.0).
//
// What bounds it: per 64 keys the two tiles need 1,250 clocks of MMA (512 for P V, 800 for S, whose N = 64 reads Q
// from shared memory twice as often as N = 128 would; measured with nothing else in the CTA) and 1,024
// clocks of the SM's 16 exponentials per clock; the kernel takes about 2,000: the chain P -> P V and the next S ->
// softmax of the tile after next, and the tensor memory's port, which the rescaling shares with both (for the thirteen
// prompts below the softmax warps doing it cost 6 % more time, eight rescaling warps instead of four 1 %).  Tried before the rescaling
// moved: 128-key tiles with one S buffer each (1,920 against 1,800 clocks per 64 keys: a tile's softmax and its products
// then follow one another), one issuing warp for both tiles (2,400), a quarter to a half of the exponentials as polynomials
// on the FMA pipe (2-5 % slower), the next scores fetched during this tile's exponentials (2 % slower).
// Short batches are bound by the chain of dependent tiles instead: 512 tokens 11.0 us, 1,024 tokens 17.2.
// 4 x 2,048 tokens: 82.5 us = 833 TFLOP/s (mma.sync: 307 us); thirteen prompts of 1 to 2,048 tokens: 134 us (449).
// Every wait is bounded: on expiry the CTA's abort flag is raised, every role drains, status 3 is recorded and
// the tensor memory released.
#pragma once

#include "dfb_attnring.cuh"
#include "dfb_prefill.cuh"
#include "dfb_tcgemv.cuh"

namespace dfb {

constexpr int kKernelPrefill = 9;

struct PrefillArgs {
  const __nv_bfloat16* q;
  const __nv_bfloat16* k;
  const __nv_bfloat16* v;
  __nv_bfloat16* out;
  const int* cu_seqlens;        // [batch + 1] query rows
  const int* cu_seqlens_k;      // [batch + 1] keys; equal to cu_seqlens without a prefix cache
  const int* block_tables;      // null: k / v hold the keys of sequence b at rows cu_seqlens_k[b] ...; else
                                // [batch, bt_stride] physical blocks and k / v are one layer's cache
                                // [num_blocks, block_size] rows
  int bt_stride, block_size, block_shift, num_blocks;   // block_size = 1 << block_shift
  long long q_stride, k_stride, v_stride, out_stride;   // elements between token rows (cache: between slots)
  int batch, q_heads, kv_heads;
  float scale;
  int* status;                  // optional device status word (a block id outside the cache)
  // tiles that lie inside their sequence come by TMA: boxes of 64 columns x box_rows rows, 128-byte swizzle
  int exact;                    // the maps end with the tensors: a box past the last row reads zeros there
  int kv_rows;                  // exact, fresh keys: rows of k and v
  int box_rows;                 // rows of a K / V box: 64, or the block size where that is smaller (a power of two)
  alignas(64) CUtensorMap q_map, k_map, v_map;
  alignas(64) CUtensorMap q_map8, k_map8, v_map8;       // boxes of 8 rows, for the end of a sequence
};

constexpr int kPfRows = 128;                     // query rows of one M tile
constexpr int kPfKeys = 64;                      // keys of one K / V tile
constexpr int kPfQBytes = kPfRows * kHeadDim * 2;         // 32 KB: two 64-column halves of 128-byte rows
constexpr int kPfTileBytes = kPfKeys * kHeadDim * 2;      // 16 KB, the same
constexpr int kPfStages = 8;
constexpr int kPfOutBytes = 8 * 4096;            // output staging of the eight softmax warps: 32 rows x 64 columns each
constexpr int kPfThreads = 352;                  // 8 softmax warps, an MMA issuer per tile, the loader
constexpr int kPfRescaleThreads = 128;           // and, but in the split form, 4 rescaling warps
constexpr int pf_threads(bool split) { return split ? kPfThreads : kPfThreads + kPfRescaleThreads; }
constexpr int kPfSmemBytes = 1024 + 2 * kPfQBytes + kPfStages * kPfTileBytes + kPfOutBytes + 288;

__device__ __forceinline__ void cp_async16_zfill(uint32_t dst, const void* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void st_shared_zero16(uint32_t dst) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(dst), "r"(0u) : "memory");
}
// announces `bytes` of copies to come without arriving
__device__ __forceinline__ void mbar_add_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// true in one lane of the (whole) warp, the same one every time
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
  unsigned long long ra, rb, rd;
  asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(rd) : "l"(ra), "l"(rb));
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(rd));
  return d;
}
__device__ __forceinline__ float2 splat2(float v) { return make_float2(v, v); }
// sum += the two bf16 values of `p` (exact in fp32; the additions take a bf16 operand as it is)
__device__ __forceinline__ void add_bf16x2(float2& sum, uint32_t p) {
  asm("{\n.reg .b16 lo, hi;\nmov.b32 {lo, hi}, %2;\nadd.f32.bf16 %0, lo, %0;\nadd.f32.bf16 %1, hi, %1;\n}"
      : "+f"(sum.x), "+f"(sum.y) : "r"(p));
}
// shared-memory descriptor of an MN-major operand with the 128-byte swizzle: 64-element pieces of the MN
// dimension `mn_bytes` apart, groups of 8 K rows 1024 bytes apart
__device__ __forceinline__ uint64_t tc_smem_desc_mn(uint32_t saddr, uint32_t mn_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(mn_bytes >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// D += A B with A in tensor memory
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
// 32 consecutive columns of this thread's lane (no wait)
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                 "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// the 128 output columns of this thread's row times f (no wait behind the last store)
__device__ __forceinline__ void pf_rescale(uint32_t o_addr, float f) {
#pragma unroll 1
  for (int c = 0; c < kHeadDim; c += 64) {
    float o[64];
    tc_ld32(o_addr + c, o);
    tc_ld32(o_addr + c + 32, o + 32);
    tc_wait_ld();
#pragma unroll
    for (int i = 0; i < 64; i += 2) {
      const float2 y = fmul2(make_float2(o[i], o[i + 1]), splat2(f));
      o[i] = y.x; o[i + 1] = y.y;
    }
    tc_st32(o_addr + c, reinterpret_cast<const uint32_t*>(o));
    tc_st32(o_addr + c + 32, reinterpret_cast<const uint32_t*>(o + 32));
  }
}

// The work items in order of falling length, the same list in every role.  Item rows of one sequence are
// numbered by `level`, its place in units of 128 keys (cached prefix + queries), so one step of the walk
// is one level over all sequences: a ballot per 32 of them.
struct PfItem {
  int seq, q0, head;       // sequence, first query row inside it, head pair (even ratio) or head (odd ratio)
  int seq_start, seq_len, k_start, k_len, shift;
  int n_tiles;             // key tiles
};
template <bool PAIRS, bool SPLIT>
struct PfWalk {
  static constexpr int step = PAIRS || SPLIT ? 1 : 2;      // M tiles along the sequence in one item
  int level, base, heads;
  // lane b's sequence: queries, keys, and their first rows (batches above 32 read them again as they go)
  int q_first, q_len, k_first, k_len;
  __device__ __forceinline__ void load(const PrefillArgs& a, int b) {
    q_first = 0; q_len = 0; k_first = 0; k_len = 0;
    if (b < a.batch) {
      q_first = a.cu_seqlens[b]; q_len = a.cu_seqlens[b + 1] - q_first;
      k_first = a.cu_seqlens_k[b]; k_len = a.cu_seqlens_k[b + 1] - k_first;
    }
  }
  // first level and number of item rows of the loaded sequence
  __device__ __forceinline__ void geometry(int& first, int& blocks) const {
    first = 0; blocks = 0;
    if (q_len > 0 && k_len > 0) {
      blocks = (q_len + step * kPfRows - 1) / (step * kPfRows);
      first = (max(k_len - q_len, 0) + kPfRows - 1) / kPfRows;
    }
  }
  __device__ __forceinline__ void init(const PrefillArgs& a, int lane) {
    heads = PAIRS ? a.q_heads / 2 : a.q_heads;
    int top = -1;
    for (int b = lane; b < a.batch || b == lane; b += 32) {
      int first, blocks;
      load(a, b);
      geometry(first, blocks);
      if (blocks) top = max(top, first + (blocks - 1) * step);
    }
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, m));
    level = top;
    base = 0;
  }
  // item number k (not below the previous call's); false past the end
  __device__ __forceinline__ bool find(const PrefillArgs& a, int k, int lane, PfItem& it) {
    const int row = k / heads;
    for (; level >= 0; --level) {
      int count = 0;
      for (int b0 = 0; b0 < a.batch; b0 += 32) {
        if (a.batch > 32) load(a, b0 + lane);
        int first, blocks;
        geometry(first, blocks);
        const int d = level - first;
        const bool has = d >= 0 && (step == 1 || (d & 1) == 0) && d / step < blocks;
        const unsigned mask = __ballot_sync(0xffffffffu, has);
        const bool mine = has && base + count + __popc(mask & ((1u << lane) - 1u)) == row;
        const unsigned hit = __ballot_sync(0xffffffffu, mine);
        if (hit) {
          const int src = __ffs(hit) - 1;
          it.seq = b0 + src;
          it.head = k % heads;
          it.seq_start = __shfl_sync(0xffffffffu, q_first, src); it.seq_len = __shfl_sync(0xffffffffu, q_len, src);
          it.k_start = __shfl_sync(0xffffffffu, k_first, src); it.k_len = __shfl_sync(0xffffffffu, k_len, src);
          it.shift = max(it.k_len - it.seq_len, 0);
          it.q0 = (level - (it.shift + kPfRows - 1) / kPfRows) * kPfRows;
          const int last = min(it.shift + min(it.q0 + step * kPfRows, it.seq_len), it.k_len);   // one past the last key seen
          it.n_tiles = (last + kPfKeys - 1) / kPfKeys;
          return true;
        }
        count += __popc(mask);
      }
      base += count;
    }
    return false;
  }
};
// item of CTA `cta` in round r: rounds alternate direction, so that nobody always gets the longer one
__device__ __forceinline__ int pf_item_index(int r, int cta, int ctas) { return r * ctas + ((r & 1) ? ctas - 1 - cta : cta); }

// SPLIT (small batches; the rule is where the kernel is launched): an item is 128 query rows of ONE head, and tile t
// takes the key tiles 2 i + t: half as long a chain for the few CTAs of a short batch.  The tiles exchange 64 columns of O each and
// write the columns that they have merged.
template <bool PAGED, bool PAIRS, bool SPLIT = false>
__global__ void __launch_bounds__(pf_threads(SPLIT), 1) prefill_tc_kernel(const __grid_constant__ PrefillArgs a) {
  extern __shared__ unsigned char pf_raw[];
  const uint32_t raw = smem_u32(pf_raw);
  unsigned char* dyn = pf_raw + (((raw + 1023u) & ~1023u) - raw);
  unsigned char* qs = dyn;                                   // two Q tiles
  unsigned char* ring = dyn + 2 * kPfQBytes;                 // K and V tiles
  unsigned char* ostage = ring + kPfStages * kPfTileBytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(ostage + kPfOutBytes);
  uint64_t* empty = full + kPfStages;
  uint64_t* q_full = empty + kPfStages;
  uint64_t* q_empty = q_full + 1;
  uint64_t* s_full = q_empty + 1;                            // [tile][buffer]
  uint64_t* p_full = s_full + 4;                             // [tile][buffer]
  uint64_t* pv_done = p_full + 4;                            // [tile], once per key tile
  uint64_t* o_full = pv_done + 2;                            // [tile], once per item
  uint64_t* f_full = o_full + 2;                             // [tile][buffer]: the rows' factors are there
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(f_full + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 10 && lane < 3) {
    const CUtensorMap* map = lane == 0 ? &a.q_map : lane == 1 ? &a.k_map : &a.v_map;
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
  }
  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < kPfStages; ++s) { mbar_init(&full[s], 32); mbar_init(&empty[s], SPLIT ? 1 : 2); }
    mbar_init(q_full, 32);
    mbar_init(q_empty, 2);
#pragma unroll
    for (int i = 0; i < 4; ++i) { mbar_init(&s_full[i], 1); mbar_init(&p_full[i], SPLIT ? 128 : 132); mbar_init(&f_full[i], 4); }
    mbar_init(&pv_done[0], 1); mbar_init(&pv_done[1], 1);
    mbar_init(&o_full[0], 1); mbar_init(&o_full[1], 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "n"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  pdl_wait();      // nothing above reads what an earlier kernel wrote
  // Behind the wait.  Measured, not explained (us per call, calls queued back to back, trigger before / behind the wait: 512 tokens
  // 11.6 / 11.1, 640 13.9 / 12.4, 400 11.3 / 10.7, 300 + 200 + 100 11.4 / 10.6; large batches even).
  pdl_launch_dependents();
  static_assert(!SPLIT || !PAIRS, "the split form takes one head at a time");
  PfWalk<PAIRS, SPLIT> walk;
  walk.init(a, lane);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);     // O of tile t at column 128 t, S (and P) buffer b of tile t at 256 + 128 t + 64 b
  const int cta = blockIdx.x, ctas = gridDim.x;
  PfItem it;
  bool ok = true;

  if (warp == 8 || warp == 9) {
    // ------------------------------ MMA issuers, one warp per tile ------------------------------
    // The whole warp runs the control flow and one elected lane issues, so that the descriptors stay in
    // uniform registers (issued under `lane == 0` every MMA costs 90-125 clocks instead of its own 50-64); one
    // warp for both tiles still spends 2,400 clocks per 64 keys on waits and issue where the MMAs need 1,330.
    constexpr uint32_t idesc_s = tc_idesc(128, kPfKeys);
    constexpr uint32_t idesc_o = tc_idesc(128, 128) | (1u << 16);    // B (= V) is MN-major
    const int t = __shfl_sync(0xffffffffu, warp - 8, 0);
    const uint64_t qd = tc_smem_desc(smem_u32(qs) + (SPLIT ? 0 : t) * kPfQBytes), kd = tc_smem_desc(smem_u32(ring)),
                   vd = tc_smem_desc_mn(smem_u32(ring), kPfTileBytes / 2);
    const uint32_t o_tmem = tmem + 128 * t, s_tmem = tmem + 256 + 128 * t;
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
      const bool done = __all_sync(0xffffffffu, tc_wait(bar, parity, abort_flag));
      tc_fence_after();
      return done;
    };
    // (the broadcasts tell the compiler that the operands are the same in every lane)
    auto issue_s = [&](int buf, int tile_stage, bool last) {
      const int b = __shfl_sync(0xffffffffu, buf, 0), stage = __shfl_sync(0xffffffffu, tile_stage, 0);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)     // K = 16 is 32 bytes of a 128-byte row; the second 64 columns are the second half of the tile
          tc_mma(s_tmem + 64 * b, qd + ((ks >> 2) * (kPfQBytes / 2) + (ks & 3) * 32) / 16,
                 kd + (uint64_t)(stage * (kPfTileBytes / 16)) + ((ks >> 2) * (kPfTileBytes / 2) + (ks & 3) * 32) / 16, idesc_s, ks ? 1u : 0u);
        tc_commit(&s_full[2 * t + b]);
        tc_commit(&empty[stage]);
        if (last) tc_commit(q_empty);      // the item's last S has been issued
      }
    };
    auto issue_o = [&](int buf, int tile_stage, bool first, bool last) {
      const int b = __shfl_sync(0xffffffffu, buf, 0), stage = __shfl_sync(0xffffffffu, tile_stage, 0);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < kPfKeys / 16; ++ks)    // 16 keys: 8 columns of P, 16 rows of V
          tc_mma_ts(o_tmem, s_tmem + 64 * b + 8 * ks, vd + (uint64_t)(stage * (kPfTileBytes / 16)) + ks * (2048 / 16), idesc_o,
                    ks ? 1u : (first ? 0u : 1u));
        tc_commit(&pv_done[t]);
        if (last) tc_commit(&o_full[t]);
        tc_commit(&empty[stage]);
      }
    };
    int n = 0;                        // ring tiles consumed
    auto place = [&](int e) -> int { return SPLIT ? 2 * e + t : e; };      // ... their place in the loader's order
    int g = 0;                        // key tiles done: buffer g & 1, phase g >> 1
    for (int r = 0; ok && walk.find(a, pf_item_index(r, cta, ctas), lane, it); ++r) {
      const int n_tiles = __shfl_sync(0xffffffffu, SPLIT ? (it.n_tiles + 1) / 2 : it.n_tiles, 0);
      ok = wait(q_full, r & 1);
      for (int j = 0; ok && j < 2 && j < n_tiles; ++j, ++n) {
        ok = wait(&full[place(n) % kPfStages], (place(n) / kPfStages) & 1);
        if (ok) issue_s((g + j) & 1, place(n) % kPfStages, j + 1 == n_tiles);
      }
      for (int j = 0; ok && j < n_tiles; ++j, ++g) {
        const int b = g & 1;
        ok = wait(&full[place(n) % kPfStages], (place(n) / kPfStages) & 1) && wait(&p_full[2 * t + b], (g >> 1) & 1);
        if (!ok) break;
        issue_o(b, place(n) % kPfStages, j == 0, j + 1 == n_tiles);
        ++n;
        if (j + 2 < n_tiles) {
          ok = wait(&full[place(n) % kPfStages], (place(n) / kPfStages) & 1);
          if (!ok) break;
          issue_s(b, place(n) % kPfStages, j + 3 == n_tiles);
          ++n;
        }
      }
    }
    if (!ok) {
      if (lane == 0 && !*abort_flag) report_status(a.status, kStatusCopyTimeout, kKernelPrefill, cta, 1);
      *abort_flag = 1;
    } else if (n > 0) {
      // the last commit has to land before the CTA's shared memory goes away
      tc_wait(&empty[place(n - 1) % kPfStages], (place(n - 1) / kPfStages) & 1, abort_flag);
    }
    __syncwarp();
  } else if (warp == 10) {
    // ------------------------------ loader ------------------------------
    // A tile is one TMA box per 64 columns where it may be fetched whole: inside its sequence, or (Q and K, whose
    // rows past the end change nothing that is stored) inside the tensor, or anywhere when the maps end with the tensor
    // and fill up with zeros (V: only where the sequence ends with it, since another sequence's rows may hold anything).
    // The end of a sequence comes as boxes of 8 rows and, for what is left, as 16-byte pieces; V rows past it are zeros, since they meet
    // probabilities of zero.
    const int piece = lane & 15, row0 = lane >> 4;          // 16-byte piece of a row, even or odd rows
    uint64_t* pend[2] = {nullptr, nullptr};     // barriers of the pieces not yet announced, oldest first
    auto announce = [&](uint64_t* bar) { fence_async_smem(); tc_mbar_arrive(bar); };
    auto drain = [&]() {
      cp_async_wait<0>();
      if (pend[0]) announce(pend[0]);
      if (pend[1]) announce(pend[1]);
      pend[0] = pend[1] = nullptr;
    };
    auto push = [&](uint64_t* bar) {            // the pieces just issued belong to `bar`
      cp_async_commit();
      cp_async_wait<2>();
      if (pend[0]) announce(pend[0]);
      pend[0] = pend[1];
      pend[1] = bar;
    };
    // nothing may stay unannounced while this warp blocks: the consumer could be waiting for it
    auto wait_free = [&](uint64_t* bar, uint32_t parity) -> bool {
      if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
      drain();
      return __all_sync(0xffffffffu, tc_wait(bar, parity, abort_flag));
    };
    auto piece_dst = [&](uint32_t base, int half_bytes, int row) -> uint32_t {
      return base + (piece >> 3) * half_bytes + row * 128 + ((((piece & 7) ^ row) & 7) << 4);
    };
    // the first `rows` of a tile's rows: boxes of 8, then pieces
    auto load_rows = [&](uint32_t base, int tile_rows, int rows, const CUtensorMap* map8, int x, int y, const __nv_bfloat16* src,
                         long long stride, uint64_t* bar) {
      const int boxes = rows >> 3, half_bytes = tile_rows * 128;
      if (lane == 0 && boxes) mbar_add_tx(bar, boxes * 8 * kHeadDim * 2);
      __syncwarp();
      for (int i = lane; i < 2 * boxes; i += 32)
        tma_load_2d(base + (i & 1) * half_bytes + (i >> 1) * 1024, map8, x + 64 * (i & 1), y + 8 * (i >> 1), smem_u32(bar));
      for (int row = 8 * boxes + row0; row < rows; row += 2)
        cp_async16_zfill(piece_dst(base, half_bytes, row), src + (size_t)row * stride + 8 * piece, true);
    };
    int n = 0;
    const int ratio = a.q_heads / a.kv_heads;
    const int all_q = a.cu_seqlens[a.batch], all_k = a.cu_seqlens_k[a.batch];
    auto load_tile = [&](bool is_v, int j, int kvh) -> bool {      // K or V tile j of the item into the next stage
      const int p0 = j * kPfKeys, stage = n % kPfStages;
      const long long stride = is_v ? a.v_stride : a.k_stride;
      if (!wait_free(&empty[stage], ((n / kPfStages) & 1) ^ 1)) return false;
      const uint32_t base = smem_u32(ring) + stage * kPfTileBytes;
      const int rows = min(it.k_len - p0, kPfKeys);
      if (SPLIT && rows <= 0) {       // the last tile of an odd number: no key is visible, V meets zeros
        if (is_v)
          for (int row = row0; row < kPfKeys; row += 2) st_shared_zero16(piece_dst(base, kPfTileBytes / 2, row));
        announce(&full[stage]);
        ++n;
        return true;
      }
      const CUtensorMap* map = is_v ? &a.v_map : &a.k_map;
      // one run of rows: fresh projections, or a cache whose blocks hold whole tiles
      if (!PAGED || a.box_rows == kPfKeys) {
        int y = it.k_start + p0, block = 0;
        if (PAGED) {
          block = a.block_tables[(size_t)it.seq * a.bt_stride + (p0 >> a.block_shift)];
          y = (block << a.block_shift) + (p0 & (a.block_size - 1));
        }
        const bool known = block >= 0 && (!PAGED || block < a.num_blocks);
        if (known && (rows == kPfKeys || (!is_v && (PAGED || a.exact || y + kPfKeys <= all_k)) ||
                      (!PAGED && a.exact && y + rows >= a.kv_rows))) {
          if (lane == 0) mbar_expect_tx(&full[stage], kPfTileBytes);
          else tc_mbar_arrive(&full[stage]);
          __syncwarp();
          if (lane < 2) tma_load_2d(base + lane * (kPfTileBytes / 2), map, kvh * kHeadDim + 64 * lane, y, smem_u32(&full[stage]));
          ++n;
          return true;
        }
        if (known) {
          load_rows(base, kPfKeys, rows, is_v ? &a.v_map8 : &a.k_map8, kvh * kHeadDim, y,
                    (is_v ? a.v : a.k) + (size_t)y * stride + (size_t)kvh * kHeadDim, stride, &full[stage]);
          if (is_v)
            for (int row = rows + row0; row < kPfKeys; row += 2) st_shared_zero16(piece_dst(base, kPfTileBytes / 2, row));
          if (rows & 7) push(&full[stage]);
          else announce(&full[stage]);      // boxes only: nothing of this thread's is in flight
          ++n;
          return true;
        }
      }
      bool boxes = PAGED && rows == kPfKeys && a.box_rows >= 8;   // (a swizzle atom is 8 rows)
      int block = 0;
      if (PAGED && boxes) {
        // lane i looks up the block of box i; a block outside the cache sends the tile to the other path
        const int p = p0 + lane * a.box_rows;
        if (p < p0 + kPfKeys) block = a.block_tables[(size_t)it.seq * a.bt_stride + (p >> a.block_shift)];
        boxes = __all_sync(0xffffffffu, block >= 0 && block < a.num_blocks);
      }
      if (boxes) {
        if (lane == 0) mbar_expect_tx(&full[stage], kPfTileBytes);
        else tc_mbar_arrive(&full[stage]);
        __syncwarp();
        if (lane * a.box_rows < kPfKeys) {                          // lane i requests box i
          const int p = p0 + lane * a.box_rows;
          const int y = (block << a.block_shift) + (p & (a.block_size - 1));
          const uint32_t dst = base + lane * a.box_rows * 128;
          tma_load_2d(dst, map, kvh * kHeadDim, y, smem_u32(&full[stage]));
          tma_load_2d(dst + kPfTileBytes / 2, map, kvh * kHeadDim + 64, y, smem_u32(&full[stage]));
        }
      } else {
        // small blocks at the end of a sequence, or a block outside the cache: row by row
        const __nv_bfloat16* src = (is_v ? a.v : a.k) + (size_t)kvh * kHeadDim + 8 * piece;
#pragma unroll 4
        for (int row = row0; row < kPfKeys; row += 2) {
          const int p = p0 + row;
          bool live = p < it.k_len;
          long long tok = 0;
          if (live) {
            if (PAGED) {
              const int b = a.block_tables[(size_t)it.seq * a.bt_stride + (p >> a.block_shift)];
              if (b >= 0 && b < a.num_blocks) tok = ((long long)b << a.block_shift) + (p & (a.block_size - 1));
              else {
                live = false;     // the row is read as zeros
                if (piece == 0) report_status(a.status, kStatusBadBlock, kKernelPrefill, it.seq, b);
              }
            } else {
              tok = it.k_start + p;
            }
          }
          cp_async16_zfill(piece_dst(base, kPfTileBytes / 2, row), src + tok * stride, live);
        }
        push(&full[stage]);
      }
      ++n;
      return true;
    };
    for (int r = 0; ok && walk.find(a, pf_item_index(r, cta, ctas), lane, it); ++r) {
      const int kvh = PAIRS ? it.head / (ratio / 2) : it.head / ratio;
      if (!wait_free(q_empty, (r & 1) ^ 1)) { ok = false; break; }
      const bool q_boxes = a.exact || it.seq_start + it.q0 + walk.step * kPfRows <= all_q;
      if (q_boxes) {
        if (lane == 0) mbar_expect_tx(q_full, (SPLIT ? 1 : 2) * kPfQBytes);
        else tc_mbar_arrive(q_full);
        __syncwarp();
        if (lane < (SPLIT ? 2 : 4)) {                                     // lane 2 t + h: half h of tile t
          const int t = lane >> 1, h = lane & 1;
          tma_load_2d(smem_u32(qs) + t * kPfQBytes + h * (kPfQBytes / 2), &a.q_map,
                      (PAIRS ? 2 * it.head + t : it.head) * kHeadDim + 64 * h, it.seq_start + it.q0 + (PAIRS ? 0 : t * kPfRows),
                      smem_u32(q_full));
        }
      } else {
        int tail = 0;
#pragma unroll 1
        for (int t = 0; t < (SPLIT ? 1 : 2); ++t) {
          // (rows past the end keep what was there: their results are not stored and touch no other row)
          const int first = it.q0 + (PAIRS ? 0 : t * kPfRows), rows = max(0, min(it.seq_len - first, kPfRows));
          const int x = (PAIRS ? 2 * it.head + t : it.head) * kHeadDim, y = it.seq_start + first;
          tail |= rows & 7;
          load_rows(smem_u32(qs) + t * kPfQBytes, kPfRows, rows, &a.q_map8, x, y, a.q + (size_t)y * a.q_stride + x, a.q_stride, q_full);
        }
        if (tail) push(q_full);
        else announce(q_full);
      }
      // in the order the issuer consumes them: K0 K1 V0 K2 V1 K3 ...
      if constexpr (SPLIT) {
        const int own = (it.n_tiles + 1) / 2;
        auto both = [&](bool is_v, int i) -> bool { return load_tile(is_v, 2 * i, kvh) && load_tile(is_v, 2 * i + 1, kvh); };
        ok = both(false, 0) && (own < 2 || both(false, 1));
        for (int j = 0; ok && j < own; ++j) {
          ok = both(true, j) && (j + 2 >= own || both(false, j + 2));
          if (j == 0) drain();
        }
      } else {
        ok = load_tile(false, 0, kvh) && (it.n_tiles < 2 || load_tile(false, 1, kvh));
        for (int j = 0; ok && j < it.n_tiles; ++j) {
          ok = load_tile(true, j, kvh) && (j + 2 >= it.n_tiles || load_tile(false, j + 2, kvh));
          if (j == 0) drain();      // the item's start waits for nothing further to be issued
        }
      }
    }
    drain();
    if (!ok) *abort_flag = 1;
  } else if (warp < 8) {
    // ------------------------------ softmax: one thread per query row ------------------------------
    const int t = warp >> 2, lrow = 32 * (warp & 3) + lane;
    const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
    const uint32_t s_addr = tmem + lanes + 256 + 128 * t, o_addr = tmem + lanes + 128 * t;
    // scores in units of log2 e; a positive scale is applied behind the maximum, any other one (which turns the order of
    // the scores around, or makes them all equal) to the scores themselves
    const float scale2 = a.scale * 1.4426950408889634f;
    const bool ordered = scale2 > 0.f;
    const float sl2 = ordered ? scale2 : 1.f, pre = ordered ? 1.f : scale2;
    // this row's factor for the rescaling warps, one per S buffer; in the warp's own output staging, which it has read when
    // the next item begins (and the last factor has been read when an item's products are done)
    volatile float* factor = reinterpret_cast<volatile float*>(ostage + warp * 4096) + lane;
    int g = 0;
    for (int r = 0; ok && walk.find(a, pf_item_index(r, cta, ctas), lane, it); ++r) {
      const int row = it.q0 + (PAIRS || SPLIT ? 0 : t * kPfRows) + lrow;               // query row inside the sequence
      const int seen = min(it.shift + row + 1, it.k_len);                     // keys this row attends to
      const int clear = min(it.shift + row - lrow + 1, it.k_len);             // ... that every row of the tile attends to
      float m = 0.f, l = 0.f;
      const int own = SPLIT ? (it.n_tiles + 1) / 2 : it.n_tiles;
      for (int j = 0; j < own; ++j, ++g) {
        const int b = g & 1;
        ok = __all_sync(0xffffffffu, tc_wait(&s_full[2 * t + b], (g >> 1) & 1, abort_flag));
        if (!ok) break;
        tc_fence_after();
        float s[kPfKeys];
        tc_ld32(s_addr + 64 * b, s);
        tc_ld32(s_addr + 64 * b + 32, s + 32);
        tc_wait_ld();
        const int p0 = (SPLIT ? 2 * j + t : j) * kPfKeys;
        if (p0 + kPfKeys > clear || !ordered) {       // the same for every thread of the tile
#pragma unroll
          for (int i = 0; i < kPfKeys; ++i) s[i] = p0 + i < seen ? s[i] * pre : -INFINITY;
        }
        float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
        for (int i = 4; i < kPfKeys; i += 8)
#pragma unroll
          for (int u = 0; u < 4; ++u) mx[u] = i + 4 + u < kPfKeys ? fmax3(mx[u], s[i + u], s[i + 4 + u]) : fmaxf(mx[u], s[i + u]);
        const float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sl2;
        // key 0 is visible to every row: finite (split form, odd tiles: or -inf)
        const float nm = j == 0 ? mt : fmaxf(m, mt);
        const float f = SPLIT && m == -INFINITY ? 0.f : ex2_approx(m - nm);
        const bool rescale = SPLIT && j > 0 && __any_sync(0xffffffffu, nm > m);
        if (!SPLIT) {
          factor[32 * b] = f;
          __syncwarp();
          if (lane == 0) tc_mbar_arrive(&f_full[2 * t + b]);
        }
        m = nm;
        const float ref = SPLIT && m == -INFINITY ? 0.f : m;      // (no key yet: every probability is 0)
        float2 sum[2] = {splat2(0.f), splat2(0.f)};
        uint32_t p[kPfKeys / 2];
#pragma unroll
        for (int i = 0; i < kPfKeys / 2; ++i) {
          const float2 x = ffma2(make_float2(s[2 * i], s[2 * i + 1]), splat2(sl2), splat2(-ref));
          p[i] = pack_bf16(ex2_approx(x.x), ex2_approx(x.y));
          add_bf16x2(sum[i & 1], p[i]);
        }
        tc_st32(s_addr + 64 * b, p);
        if (rescale) {
          // S(g) was issued behind P V of g - 2: at most one phase is missing
          ok = __all_sync(0xffffffffu, tc_wait(&pv_done[t], (g - 1) & 1, abort_flag));
          if (ok) {
            tc_fence_after();
            pf_rescale(o_addr, f);
          }
        }
        tc_wait_st();
        if (!ok) break;
        tc_fence_before();
        tc_mbar_arrive(&p_full[2 * t + b]);
        // the row sum takes the rounded probabilities, the values that multiply V; the product does not wait for it
        sum[0] = fadd2(sum[0], sum[1]);
        l = (j == 0 ? 0.f : l * f) + (sum[0].x + sum[0].y);
      }
      if (!SPLIT && !ok) break;
      ok = ok && __all_sync(0xffffffffu, tc_wait(&o_full[t], r & 1, abort_flag));
      if (SPLIT) ok = named_sync_and(3, 256, ok);      // both tiles' products are done, or both tiles give up
      if (!ok) break;
      tc_fence_after();
      // Out through shared memory, 64 columns at a time: a row per thread in, whole 128-byte lines out (straight
      // from the registers every store instruction would touch 32 lines: 4 us for the CTA).
      unsigned char* stg = ostage + warp * 4096;
      const int wrow = row - lane;                             // first query row of this warp
      __nv_bfloat16* dst = a.out + (size_t)(it.seq_start + wrow) * a.out_stride + (size_t)(PAIRS ? 2 * it.head + t : it.head) * kHeadDim;
      auto write_out = [&](int h, const float* o, float inv) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          uint4 v;
          v.x = pack_bf16(o[8 * i] * inv, o[8 * i + 1] * inv); v.y = pack_bf16(o[8 * i + 2] * inv, o[8 * i + 3] * inv);
          v.z = pack_bf16(o[8 * i + 4] * inv, o[8 * i + 5] * inv); v.w = pack_bf16(o[8 * i + 6] * inv, o[8 * i + 7] * inv);
          *reinterpret_cast<uint4*>(stg + lane * 128 + ((i ^ (lane & 7)) << 4)) = v;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int rr = 4 * i + (lane >> 3), c = lane & 7;
          const uint4 v = *reinterpret_cast<const uint4*>(stg + rr * 128 + ((c ^ (rr & 7)) << 4));
          if (wrow + rr < it.seq_len) *reinterpret_cast<uint4*>(dst + (size_t)rr * a.out_stride + 64 * h + 8 * c) = v;
        }
        __syncwarp();
      };
      if constexpr (SPLIT) {
        // exchanged through the place of the second Q tile, 32 columns at a time ([tile][column][row]), and the output
        // staging ([tile][row] maximum and sum); tile t finishes columns 64 t ... 64 t + 63
        float* xo = reinterpret_cast<float*>(qs + kPfQBytes);
        float2* xm = reinterpret_cast<float2*>(ostage);
        xm[t * kPfRows + lrow] = make_float2(m, l);
        float o[64];
        tc_ld32(o_addr + 64 * t, o);
        tc_ld32(o_addr + 64 * t + 32, o + 32);
        float wa = 0.f, wb = 0.f, sum = 1.f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float x[32];
          tc_ld32(o_addr + 64 * (t ^ 1) + 32 * h, x);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) xo[(t * 32 + i) * kPfRows + lrow] = x[i];
          named_sync(3, 256);
          if (h == 0) {
            const float2 other = xm[(t ^ 1) * kPfRows + lrow];
            const float top = fmaxf(m, other.x);                 // finite: tile 0 holds key 0
            wa = m == -INFINITY ? 0.f : ex2_approx(m - top);
            wb = other.x == -INFINITY ? 0.f : ex2_approx(other.x - top);
            sum = fmaf(wb, other.y, wa * l);
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) o[32 * h + i] = fmaf(wb, xo[((t ^ 1) * 32 + i) * kPfRows + lrow], wa * o[32 * h + i]);
          named_sync(3, 256);
        }
        write_out(t, o, 1.0f / sum);
      } else {
        const float inv = 1.0f / l;
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          float o[64];
          tc_ld32(o_addr + 64 * h, o);
          tc_ld32(o_addr + 64 * h + 32, o + 32);
          tc_wait_ld();
          write_out(h, o, inv);
        }
      }
      tc_fence_before();      // the next item's P arrival orders these reads before the MMA that overwrites O
    }
    if (!ok) *abort_flag = 1;
  } else if (!SPLIT) {
    // ------------------------------ rescaling: four warps, the rows of both tiles ------------------------------
    // O is multiplied while the softmax warps are at the exponentials of the same key tile; P V waits for both.
    const int quarter = warp & 3;                  // the tensor memory lanes this warp may touch
    int g = 0;
    for (int r = 0; ok && walk.find(a, pf_item_index(r, cta, ctas), lane, it); ++r) {
      for (int j = 0; ok && j < it.n_tiles; ++j, ++g) {
#pragma unroll 1
        for (int t = 0; ok && t < 2; ++t) {
          ok = __all_sync(0xffffffffu, tc_wait(&f_full[2 * t + (g & 1)], (g >> 1) & 1, abort_flag));
          if (!ok) break;
          const float f = reinterpret_cast<volatile float*>(ostage + (4 * t + quarter) * 4096)[32 * (g & 1) + lane];
          if (j > 0 && __any_sync(0xffffffffu, f != 1.f)) {
            // S(g) was issued behind P V of g - 2: at most one phase is missing
            ok = __all_sync(0xffffffffu, tc_wait(&pv_done[t], (g - 1) & 1, abort_flag));
            if (!ok) break;
            tc_fence_after();
            pf_rescale(tmem + ((uint32_t)(32 * quarter) << 16) + 128 * t, f);
            tc_wait_st();
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) tc_mbar_arrive(&p_full[2 * t + (g & 1)]);
        }
      }
    }
    if (!ok) *abort_flag = 1;
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
  }
}

}  // namespace dfb
