// Paged GQA decode attention, one thread-block cluster per (batch row, KV head): the same computation as
// paged_attention_kernel (q/k RMSNorm + RoPE + KV-cache write + attention), with the context dealt to the
// cluster's CTAs in equal contiguous pieces instead of fixed chunks of 64 positions.
//
//   * CS CTAs (2, 4 or 8) share one row's context, so the grid is rows x KV heads x CS whatever the contexts are
//     and all CTAs are resident together (two per SM).  A chunked grid of 8 rows x 576 tokens is 640 CTAs: its
//     second wave started 4.7 us after the first.
//   * 16 threads share a position (8 dimensions each, both query heads); a thread holds 8 positions' K and V in
//     registers (128 positions, 64 KB per CTA and pass), those of the first pass requested before the dependency
//     wait, those of the next one as soon as their registers are free.  Every group of 16 threads keeps its own running
//     (maximum, sum, output): no barrier inside the loop.
//   * The 8 positions x 2 heads a thread has partial products of are reduced over the 16 threads with a halving
//     butterfly (15 shuffles instead of 64), which leaves thread (head, i) with the score of ITS position i: one
//     exponential per score instead of sixteen.
//   * One merge: every warp pushes its partial output (256 values) straight into the shared memory of the CTA that
//     will finish those values, CTA r the r-th part of the 256, and its (maximum, sum) to all; one cluster barrier;
//     everything after it is local, so no CTA has to wait for its peers to leave.
//
// At 8 rows it is bound by DRAM while it streams (8 x 2,000 tokens: 16.8 MB per pass in 2.9 us, 5.8 TB/s) and by the
// latency of its first loads where the context fits one pass; half of the CTAs start when the QKV kernel has left
// their SM.  Step time, device, against the chunked kernels: 8 rows x 256 - 2,040 tokens 878 -> 818 us, 8 rows x 1,024
// 820 -> 725, 6 rows x 256 607 -> 564.
#pragma once

#include "dfb_attnring.cuh"
#include "dfb_kernels.cuh"

namespace dfb {

constexpr int kCaThreads = 256, kCaWarps = 8;
constexpr int kCaGroups = 16;                       // positions a pass step covers: 16 threads each
constexpr int kCaIter = 8;                          // positions per thread and pass
constexpr int kCaPass = kCaGroups * kCaIter;        // 128 positions per CTA and pass

__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// address of this CTA's shared variable in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t peer_smem(const void* local, unsigned rank) {
  uint32_t ra;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_u32(local)), "r"(rank));
  return ra;
}
__device__ __forceinline__ void st_peer_f4(uint32_t addr, float a, float b, float c, float d) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
__device__ __forceinline__ void st_peer_f2(uint32_t addr, float a, float b) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1,%2};" ::"r"(addr), "f"(a), "f"(b) : "memory");
}

// grid (CS, KV heads, rows), clusters of CS CTAs along x
template <int CS>
__global__ void __launch_bounds__(kCaThreads, 2) cluster_attention_kernel(const AttnArgs a) {
  constexpr int E = 2 * kHeadDim / CS;              // output values this CTA finishes
  constexpr int kSrc = kCaWarps * E + 4;            // floats of one source CTA's partial results (+ 4: bank offset)
  constexpr float kLog2e = 1.4426950408889634f;
  if (!a.late_trigger) pdl_launch_dependents();
  cluster_arrive_relaxed();                         // completed before the first push: the peers are running by then
  const int rank = blockIdx.x, kvh = blockIdx.y, row = blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int pg = tid >> 4, l16 = tid & 15;
  if (tid == 0) { trace_min(a.trace, 0); trace_max(a.trace, 4); }

  __shared__ __align__(16) float red[CS * kSrc];                     // [source CTA][warp][value]
  __shared__ float2 ml[CS * kCaWarps][2];                            // (maximum, sum) per source warp and head
  __shared__ __align__(16) __nv_bfloat16 qs[2][kHeadDim];            // the two query heads after norm and rotation
  __shared__ __align__(16) __nv_bfloat16 ks[kHeadDim];
  __shared__ __align__(16) __nv_bfloat16 vs[kHeadDim];

  int pos = a.positions[row];
  bool write_ok = true;   // false once any input of this row had to be replaced: its KV slot is then left alone
  if (pos < 0 || pos >= a.max_pos) {
    report_status(a.status, kStatusBadPosition, kKernelAttention, row, pos);
    pos = pos < 0 ? 0 : a.max_pos - 1;
    write_ok = false;
  }
  int ctx = pos + 1;
  if (ctx > a.ctx_limit) {   // the caller's context bound does not cover this row: attend to what it covers
    if (rank == 0) report_status(a.status, kStatusBadGrid, kKernelAttention, row, pos);
    ctx = a.ctx_limit;
    pos = ctx - 1;
    write_ok = false;
  }
  // equal pieces of whole groups of 16 positions (blocks are multiples of 64: a group never crosses one)
  const int piece = (ctx + kCaGroups * CS - 1) / (kCaGroups * CS) * kCaGroups;
  const int start = rank * piece, end = min(ctx, start + piece);

  // ---- K / V of a pass: walks the block table a group at a time (the same for the whole CTA) ----
  int col = start / a.block_size, in_block = start - col * a.block_size, block = -1;
  constexpr unsigned kRow = kHeadDim / 8;           // offsets count 16-byte pieces (8 elements): 32 bits cover 64 GB per layer
  const unsigned stride = (unsigned)a.kv_heads * kRow;
  unsigned new_slot = 0;                            // the new token's row of this head
  auto next_group = [&](int p16) -> unsigned {      // position p16 of this head
    if (block < 0) {
      int c = col;
      bool bad = false;
      if (a.bt_cols > 0 && c >= a.bt_cols) {        // never read a table entry the caller did not fill in
        report_status(a.status, kStatusBadBlock, kKernelAttention, row, -1 - c);
        c = a.bt_cols - 1;
        bad = true;
      }
      block = a.block_tables[row * a.bt_stride + c];
      if (block < 0 || block >= a.num_blocks) {
        report_status(a.status, kStatusBadBlock, kKernelAttention, row, block);
        block = 0;
        bad = true;
      }
      if (bad && pos / a.block_size == col) write_ok = false;
    }
    const unsigned off = (unsigned)(block * a.block_size + in_block) * stride + (unsigned)kvh * kRow;
    if (pos >= p16 && pos < p16 + kCaGroups) new_slot = off + (unsigned)(pos - p16) * stride;
    in_block += kCaGroups;
    if (in_block >= a.block_size) { in_block = 0; ++col; block = -1; }
    return off;
  };
  const unsigned lane_off = (unsigned)pg * stride + (unsigned)l16;
  uint4 kreg[kCaIter], vreg[kCaIter];
  unsigned off[kCaIter];
  auto locate = [&](int base) {
#pragma unroll
    for (int i = 0; i < kCaIter; ++i)
      if (base + kCaGroups * i < end) off[i] = next_group(base + kCaGroups * i) + lane_off;
  };
  auto load = [&](uint4 (&r)[kCaIter], const __nv_bfloat16* cache, int base) {
#pragma unroll
    for (int i = 0; i < kCaIter; ++i) {
      const int p = base + kCaGroups * i + pg;
      r[i] = p < end && p != pos ? ldg_stream(cache + 8 * (size_t)off[i]) : make_uint4(0, 0, 0, 0);
    }
  };
  locate(start);
  load(kreg, a.k_cache, start);
  load(vreg, a.v_cache, start);

  // constants of the new token's norm and rotation: also independent of the predecessor
  uint32_t wlo = 0, whi = 0;
  float2 rc = make_float2(0.f, 0.f), rs = make_float2(0.f, 0.f);
  if (warp < 3) {
    const __nv_bfloat16* nw = warp < 2 ? a.q_norm : a.k_norm;
    const float* cs = a.cos_sin + (size_t)pos * kHeadDim;
    wlo = *reinterpret_cast<const uint32_t*>(nw + 2 * lane);
    whi = *reinterpret_cast<const uint32_t*>(nw + 2 * lane + 64);
    rc = *reinterpret_cast<const float2*>(cs + 2 * lane);
    rs = *reinterpret_cast<const float2*>(cs + 64 + 2 * lane);
  }

  pdl_wait();
  if (tid == 0) { trace_max(a.trace, 1); trace_min(a.trace, 3); }

  // ---- new token: q (2 heads) and k get RMSNorm + RoPE, v is copied ----
  {
    const __nv_bfloat16* src = a.qkv + (size_t)row * a.qkv_stride;
    if (warp < 3) {
      const __nv_bfloat16* vec = warp < 2 ? src + (2 * kvh + warp) * kHeadDim : src + a.q_size + kvh * kHeadDim;
      const int d = 2 * lane;  // handles d, d+1 and their RoPE partners d+64, d+65
      const uint32_t lo = __ldcg(reinterpret_cast<const uint32_t*>(vec + d));
      const uint32_t hi = __ldcg(reinterpret_cast<const uint32_t*>(vec + d + 64));
      float x[4] = {bf_lo(lo), bf_hi(lo), bf_lo(hi), bf_hi(hi)};
      float ss = x[0] * x[0] + x[1] * x[1] + x[2] * x[2] + x[3] * x[3];
#pragma unroll
      for (int m = 16; m >= 1; m >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, m);
      const float rstd = 1.0f / sqrtf(ss / (float)kHeadDim + a.eps);
      const float w[4] = {bf_lo(wlo), bf_hi(wlo), bf_lo(whi), bf_hi(whi)};
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = round_bf16(round_bf16(x[e] * rstd) * w[e]);
      const uint32_t y_lo = pack_bf16(mul_sub_unfused(x[0], rc.x, x[2], rs.x), mul_sub_unfused(x[1], rc.y, x[3], rs.y));
      const uint32_t y_hi = pack_bf16(mul_add_unfused(x[2], rc.x, x[0], rs.x), mul_add_unfused(x[3], rc.y, x[1], rs.y));
      __nv_bfloat16* dst = warp < 2 ? qs[warp] : ks;
      *reinterpret_cast<uint32_t*>(dst + d) = y_lo;
      *reinterpret_cast<uint32_t*>(dst + d + 64) = y_hi;
    } else if (warp == 3) {
      const __nv_bfloat16* vec = src + a.q_size + a.kv_size + kvh * kHeadDim;
      reinterpret_cast<uint2*>(vs)[lane] = __ldcg(reinterpret_cast<const uint2*>(vec) + lane);
    }
  }
  __syncthreads();
  if (a.late_trigger) pdl_launch_dependents();

  float2 q0[4], q1[4];    // this thread's 8 dimensions of the two query heads
  {
    const uint4 u = reinterpret_cast<const uint4*>(qs[0])[l16], v = reinterpret_cast<const uint4*>(qs[1])[l16];
    q0[0] = bf2(u.x); q0[1] = bf2(u.y); q0[2] = bf2(u.z); q0[3] = bf2(u.w);
    q1[0] = bf2(v.x); q1[1] = bf2(v.y); q1[2] = bf2(v.z); q1[3] = bf2(v.w);
  }
  const float scale2 = a.scale * kLog2e;            // scores in powers of two
  const int my_head = l16 >> 3, my_i = l16 & 7;     // the score this thread ends up with
  float m = -INFINITY, l = 0.f;                     // running maximum of the group, this thread's part of the sum (my_head)
  float2 o0[4], o1[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) { o0[e] = make_float2(0.f, 0.f); o1[e] = make_float2(0.f, 0.f); }

#pragma unroll 1
  for (int base = start; base < end; base += kCaPass) {
    if (pos >= base && pos < base + kCaPass && ((pos - base) & (kCaGroups - 1)) == pg && pos < end) {
      // the new token is this group's: its K and V come from shared memory, and go into the cache
      const int i = (pos - base) / kCaGroups;
      const uint4 kn = reinterpret_cast<const uint4*>(ks)[l16], vn = reinterpret_cast<const uint4*>(vs)[l16];
#pragma unroll
      for (int u = 0; u < kCaIter; ++u)
        if (u == i) { kreg[u] = kn; vreg[u] = vn; }
      if (write_ok && (a.row_active == nullptr || a.row_active[row] != 0)) {
        *reinterpret_cast<uint4*>(a.k_cache + 8 * (size_t)(new_slot + l16)) = kn;
        *reinterpret_cast<uint4*>(a.v_cache + 8 * (size_t)(new_slot + l16)) = vn;
      }
    }
    // ---- scores: partial products of 8 dimensions, index = head * 8 + i ----
    float v[2 * kCaIter];
#pragma unroll
    for (int i = 0; i < kCaIter; ++i) {
      v[i] = 0.f;
      v[kCaIter + i] = 0.f;
      if (base + kCaGroups * i < end) {             // the same for the whole CTA
        const float2 k0 = bf2(kreg[i].x), k1 = bf2(kreg[i].y), k2 = bf2(kreg[i].z), k3 = bf2(kreg[i].w);
        const float2 x = ffma2(k3, q0[3], ffma2(k2, q0[2], ffma2(k1, q0[1], fmul2(k0, q0[0]))));
        const float2 y = ffma2(k3, q1[3], ffma2(k2, q1[2], ffma2(k1, q1[1], fmul2(k0, q1[0]))));
        v[i] = x.x + x.y;
        v[kCaIter + i] = y.x + y.y;
      }
    }
    const bool more = base + kCaPass < end;
    if (more) {
      locate(base + kCaPass);
      load(kreg, a.k_cache, base + kCaPass);
    }
    // halving butterfly over the group's 16 threads
#pragma unroll
    for (int n = kCaIter; n >= 1; n >>= 1) {
      const bool up = l16 & n;
#pragma unroll
      for (int j = 0; j < n; ++j) {
        const float keep = up ? v[j + n] : v[j], send = up ? v[j] : v[j + n];
        v[j] = keep + __shfl_xor_sync(0xffffffffu, send, n);
      }
    }
    const bool valid = base + kCaGroups * my_i + pg < end;
    const float s = valid ? v[0] * scale2 : -INFINITY;
    float bm = s;
#pragma unroll
    for (int n = 4; n >= 1; n >>= 1) bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, n));
    const float nm = fmaxf(m, bm), ref = nm == -INFINITY ? 0.f : nm;   // (a group may have no position yet)
    const float corr = exp2f(m - ref), p = exp2f(s - ref);
    m = nm;
    l = l * corr + p;
    if (base > start) {
      const float other = __shfl_xor_sync(0xffffffffu, corr, 8);
      const float c0 = my_head ? other : corr, c1 = my_head ? corr : other;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o0[e] = fmul2(o0[e], make_float2(c0, c0));
        o1[e] = fmul2(o1[e], make_float2(c1, c1));
      }
    }
    // ---- P.V ----
#pragma unroll
    for (int i = 0; i < kCaIter; ++i) {
      if (base + kCaGroups * i < end) {
        const float p0 = __shfl_sync(0xffffffffu, p, (lane & 16) | i), p1 = __shfl_sync(0xffffffffu, p, (lane & 16) | 8 | i);
        const float2 w0 = make_float2(p0, p0), w1 = make_float2(p1, p1);
        const float2 v0 = bf2(vreg[i].x), v1 = bf2(vreg[i].y), v2 = bf2(vreg[i].z), v3 = bf2(vreg[i].w);
        o0[0] = ffma2(w0, v0, o0[0]); o0[1] = ffma2(w0, v1, o0[1]); o0[2] = ffma2(w0, v2, o0[2]); o0[3] = ffma2(w0, v3, o0[3]);
        o1[0] = ffma2(w1, v0, o1[0]); o1[1] = ffma2(w1, v1, o1[1]); o1[2] = ffma2(w1, v2, o1[2]); o1[3] = ffma2(w1, v3, o1[3]);
      }
    }
    if (more) load(vreg, a.v_cache, base + kCaPass);
  }
  if (tid == 0) trace_max(a.trace, 5);

  // ---- the warp's two groups become one; lanes 0-15 go on with head 0, lanes 16-31 with head 1 ----
  {
    const float M = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
    const float w = m == -INFINITY ? 0.f : exp2f(m - M);
    const float other = __shfl_xor_sync(0xffffffffu, w, 8);
    const float w0 = my_head ? other : w, w1 = my_head ? w : other;
    const bool second = lane & 16;
    float r[8];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 a0 = fmul2(o0[e], make_float2(w0, w0)), a1 = fmul2(o1[e], make_float2(w1, w1));
      const float2 keep = second ? a1 : a0, send = second ? a0 : a1;
      r[2 * e] = keep.x + __shfl_xor_sync(0xffffffffu, send.x, 16);
      r[2 * e + 1] = keep.y + __shfl_xor_sync(0xffffffffu, send.y, 16);
    }
    float sum = l * w;
#pragma unroll
    for (int n = 4; n >= 1; n >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, n);
    sum += __shfl_xor_sync(0xffffffffu, sum, 16);
    // (maximum, sum) of head lane & 1 for CTA lane / 2
    const float hm = __shfl_sync(0xffffffffu, M, 8 * (lane & 1)), hs = __shfl_sync(0xffffffffu, sum, 8 * (lane & 1));
    const int idx = (second ? kHeadDim : 0) + 8 * l16;        // of the 256 values
    cluster_wait();
    const uint32_t dst = peer_smem(&red[rank * kSrc + warp * E + idx % E], idx / E);
    st_peer_f4(dst, r[0], r[1], r[2], r[3]);
    st_peer_f4(dst + 16, r[4], r[5], r[6], r[7]);
    if ((lane >> 1) < CS) st_peer_f2(peer_smem(&ml[rank * kCaWarps + warp][lane & 1], lane >> 1), hm, hs);
    cluster_arrive();
    cluster_wait();
  }
  if (tid == 0) trace_max(a.trace, 6);

  // ---- CS threads per value, one per source CTA ----
  {
    const int src = tid % CS, e = tid / CS, h = (rank * E + e) / kHeadDim;
    float wm[kCaWarps], ws[kCaWarps], val[kCaWarps], M = -INFINITY;
#pragma unroll
    for (int w = 0; w < kCaWarps; ++w) {
      const float2 u = ml[src * kCaWarps + w][h];
      wm[w] = u.x; ws[w] = u.y;
      val[w] = red[src * kSrc + w * E + e];
      M = fmaxf(M, u.x);
    }
#pragma unroll
    for (int n = CS / 2; n >= 1; n >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, n));
    float O = 0.f, S = 0.f;
#pragma unroll
    for (int w = 0; w < kCaWarps; ++w) {
      const float c = exp2f(wm[w] - M);             // -inf (no position): 0.  M is finite: the row has a position
      O = fmaf(c, val[w], O);
      S = fmaf(c, ws[w], S);
    }
#pragma unroll
    for (int n = CS / 2; n >= 1; n >>= 1) {
      O += __shfl_xor_sync(0xffffffffu, O, n);
      S += __shfl_xor_sync(0xffffffffu, S, n);
    }
    if (src == 0) a.out[(size_t)row * a.q_size + 2 * kvh * kHeadDim + rank * E + e] = __float2bfloat16_rn(O / S);
  }
  if (tid == 0) trace_max(a.trace, 2);
}

}  // namespace dfb
