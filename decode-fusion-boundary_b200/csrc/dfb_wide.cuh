// Projections of a decode step for 9 to 32 rows (the fixed-slot runtime): NG groups of 8 batch rows share one
// pass over the weights, which is what bounds such a step when it is taken as launches of 8 rows.
//
//   * wide_norm_kernel: QKV, gate / up and the LM head (K = 1024, residual add + RMSNorm in front), the layout of
//     pair_gemv_kernel (16 weight rows on M, 8 batch rows on N, 8 warps splitting K): a weight fragment is read from shared
//     memory once and multiplied with NG groups.  x stays in shared memory (8 NG rows), so that the kernel keeps
//     within 128 registers and, up to 24 rows, its CTAs start beside their predecessor's (gate / up of 32 rows
//     takes 241 KB with o_proj and 257 with down_proj, of the SM's 228; the LM head takes an SM for itself).  Clusters of four CTAs share the
//     norm: each normalises a quarter of the rows and writes them into all four shared memories (every CTA reading
//     all rows of h and of the residual took 14 MB from L2 in a launch; gate / up, 20 rows: 7.3 -> 5.9 us).
//   * wide_store_kernel: o_proj and down_proj.  A cluster of four CTAs shares 32 weight rows, each with a quarter of K: x is
//     by far the larger operand here (24 rows x 6 KB), and splitting K divides what a CTA has to fetch behind its
//     dependency; all of it is in flight at once, in registers.  The parts meet in the shared memory of the CTA that
//     finishes the row (down_proj, 20 rows, two CTAs: 5.1 us, four: 4.2 us).
//
// 20 rows, 5 - 1,500 tokens: 1,022 us per step, of which attention 13.5 us per layer (paged_attention_ring_kernel on a packed
// list of chunks), LM head 80 us.
// Bound by mma.sync's issue rate (one per 38 clocks and sub-partition: 0.3 us per group and gate / up tile of 16 rows) and
// by the latency of the dependent launches.  Rows beyond the live ones are computed and ignored.
#pragma once

#include "dfb_attncluster.cuh"
#include "dfb_attnring.cuh"
#include "dfb_kernels.cuh"
#include "dfb_pairgemv.cuh"

namespace dfb {

constexpr int kWideRows = 32;                        // = DFB_MAX_SLOTS
constexpr int kKernelWide = 8;
constexpr int kWideCluster = 4;                       // CTAs that share the norm (QKV, gate / up) or K (o_proj, down_proj)

template <int NG, int MODE>
struct WideSmem {
  static constexpr int kStages = MODE == kModeNormStore ? 2 : 3;       // tiles of a CTA (LM head: ring)
  static constexpr int kXBytes = 8 * NG * PairSmem::kRowStride;
  static constexpr int kRed = 8 * 128 * NG;                           // floats: partial sums of one tile, [warp][output]
  static constexpr int bytes() {
    return kStages * PairSmem::kStageBytes + kXBytes + (MODE == kModeNormArgmax ? 2 * 4 * kRed : 0) + 8 * kStages + 16;
  }
};

// The noise stream of a wide step is the one of its groups of 8 rows taken one after the other: group j draws with the
// counter advanced by the sampled groups before it.  Called by one warp.
__device__ __forceinline__ int wide_sample_rows(const GemvArgs& a, SampleRow* rows_smem, int lane) {
  if (!a.temps) return 0;
  const float t = a.temps[lane];
  const unsigned hot = __ballot_sync(0xffffffffu, t > 1e-10f);
  int before = 0, all = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int any = (hot >> (8 * j) & 0xffu) ? 1 : 0;
    if (j < lane / 8) before += any;
    all += any;
  }
  SampleRow s{t, 0u};
  if (t > 1e-10f) s.step = *(volatile unsigned int*)a.sample_ctr + (unsigned)before;
  rows_smem[lane] = s;
  return all;
}

template <int NG, int MODE>
__global__ void __launch_bounds__(256, MODE == kModeNormArgmax ? 1 : 2) wide_norm_kernel(const GemvArgs a) {
  using SM = WideSmem<NG, MODE>;
  constexpr int K = PairSmem::kK, STAGES = SM::kStages, kOut = 128 * NG;
  constexpr bool kArgmax = MODE == kModeNormArgmax, kSwiglu = MODE == kModeNormSwiglu;
  constexpr int CL = kArgmax ? 1 : kWideCluster, kOwn = 8 * NG / CL;     // rows that this CTA normalises
  pdl_launch_dependents();
  if (CL > 1) cluster_arrive_relaxed();      // completed before the peers' shared memory is written
  if (threadIdx.x == 0) trace_min(a.trace, 0);
  extern __shared__ __align__(128) unsigned char dyn_smem[];
  unsigned char* stage_base = dyn_smem;
  unsigned char* xsb = dyn_smem + STAGES * PairSmem::kStageBytes;               // [8 NG][kRowStride] bf16 x
  float* red_base = reinterpret_cast<float*>(xsb + SM::kXBytes);                // LM head: two buffers
  uint64_t* full = reinterpret_cast<uint64_t*>(xsb + SM::kXBytes + (kArgmax ? 2 * 4 * SM::kRed : 0));
  __shared__ SampleRow srows[kArgmax ? kWideRows : 1];
  __shared__ ArgmaxPart wpart[kArgmax ? 8 : 1][8 * 2];
  __shared__ int last_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3, kbase = warp * 128 + 8 * t, stride = gridDim.x;

  auto request_tile = [&](int tile, int s) {      // warp 0
    if (lane == 0) mbar_expect_tx(&full[s], 16 * 2 * K);
    __syncwarp();
    if (lane < 16) {
      const int row = kSwiglu ? (lane >= 8 ? a.gate_rows : 0) + tile * 8 + (lane & 7) : tile * 16 + lane;
      bulk_g2s(stage_base + s * PairSmem::kStageBytes + lane * PairSmem::kRowStride, a.w + (size_t)row * K, 2 * K, &full[s]);
    }
  };
  if (warp == 0) {
    if (lane == 0) {
#pragma unroll
      for (int s = 0; s < STAGES; ++s) mbar_init(&full[s], 1);
      fence_mbar_init();
    }
    __syncwarp();
#pragma unroll
    for (int s = 0; s < STAGES; ++s)
      if ((int)blockIdx.x + s * stride < a.n_tiles) request_tile(blockIdx.x + s * stride, s);
  }
  uint4 nw[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) nw[c] = ldg_stream(a.norm_w + 8 * (32 * c + lane));
  __syncthreads();          // the barriers are initialised before anyone polls them
  pdl_wait();
  if (tid == 0) { trace_max(a.trace, 1); trace_min(a.trace, 3); }

  // ---- x = h (+ residual), RMSNorm: a warp per row; the rows are shared out over the cluster ----
  {
    const int first = CL > 1 ? (blockIdx.x & (CL - 1)) * kOwn : 0;
    uint4 hv[4], rv[4];
    auto load = [&](int b) {
      const size_t xrow = a.ids ? (size_t)clamp_token(a.ids[b], a.embed_rows, a.status, b) : (size_t)b;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        hv[c] = ldg_cg(a.x + xrow * K + 8 * (32 * c + lane));
        rv[c] = a.res_in ? ldg_cg(a.res_in + (size_t)b * K + 8 * (32 * c + lane)) : make_uint4(0, 0, 0, 0);
      }
    };
    if (warp < kOwn) load(first + warp);
    if (CL > 1) cluster_wait();
#pragma unroll
    for (int i = 0; i < (kOwn + 7) / 8; ++i) {
      const int b = first + warp + 8 * i;
      if (warp + 8 * i >= kOwn) break;
      float x[4][8], ss = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float hf[8], rf[8];
        unpack8(hv[c], hf);
        unpack8(rv[c], rf);
#pragma unroll
        for (int e = 0; e < 8; ++e) { x[c][e] = hf[e] + rf[e]; ss = fmaf(x[c][e], x[c][e], ss); }
      }
      if (8 * (i + 1) + warp < kOwn) load(b + 8);
      if (a.res_out && (int)blockIdx.x < CL) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          *reinterpret_cast<uint4*>(a.res_out + (size_t)b * K + 8 * (32 * c + lane)) =
              make_uint4(pack_bf16(x[c][0], x[c][1]), pack_bf16(x[c][2], x[c][3]), pack_bf16(x[c][4], x[c][5]), pack_bf16(x[c][6], x[c][7]));
      }
#pragma unroll
      for (int m = 16; m >= 1; m >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, m);
      const float rstd = 1.0f / sqrtf(ss / (float)K + a.eps);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float wf[8], y[8];
        unpack8(nw[c], wf);
#pragma unroll
        for (int e = 0; e < 8; ++e) y[e] = round_bf16(x[c][e] * rstd) * wf[e];
        const uint32_t y0 = pack_bf16(y[0], y[1]), y1 = pack_bf16(y[2], y[3]), y2 = pack_bf16(y[4], y[5]), y3 = pack_bf16(y[6], y[7]);
        unsigned char* dst = xsb + b * PairSmem::kRowStride + 16 * (32 * c + lane);
        if (CL == 1) {
          *reinterpret_cast<uint4*>(dst) = make_uint4(y0, y1, y2, y3);
        } else {
#pragma unroll
          for (int r = 0; r < CL; ++r)
            asm volatile("st.shared::cluster.v4.b32 [%0], {%1,%2,%3,%4};"
                         ::"r"(peer_smem(dst, r)), "r"(y0), "r"(y1), "r"(y2), "r"(y3) : "memory");
        }
      }
    }
  }
  int sampled_groups = 0;
  if (kArgmax && warp == 0) sampled_groups = wide_sample_rows(a, srows, lane);
  if (CL > 1) {
    cluster_arrive();
    cluster_wait();
  } else {
    __syncthreads();
  }
  if (tid == 0) trace_max(a.trace, 4);

  // ---- one tile: this warp's K columns of 16 weight rows x 8 NG batch rows; c = (row g | g + 8, batch 2t, 2t + 1) ----
  const unsigned char* xp = xsb + g * PairSmem::kRowStride + 2 * kbase;
  auto multiply = [&](int s, float (&c)[NG][4]) {
    const unsigned char* w0p = stage_base + s * PairSmem::kStageBytes + g * PairSmem::kRowStride + 2 * kbase;
    const unsigned char* w1p = w0p + 8 * PairSmem::kRowStride;
    float d[NG][4];
#pragma unroll
    for (int n = 0; n < NG; ++n)
#pragma unroll
      for (int q = 0; q < 4; ++q) { c[n][q] = 0.f; d[n][q] = 0.f; }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint4 u = *reinterpret_cast<const uint4*>(w0p + 64 * j), v = *reinterpret_cast<const uint4*>(w1p + 64 * j);
#pragma unroll
      for (int n = 0; n < NG; ++n) {
        const uint4 xb = *reinterpret_cast<const uint4*>(xp + 8 * n * PairSmem::kRowStride + 64 * j);
        mma_bf16_16816_full(c[n], u.x, v.x, u.y, v.y, xb.x, xb.y);
        mma_bf16_16816_full(d[n], u.z, v.z, u.w, v.w, xb.z, xb.w);
      }
    }
#pragma unroll
    for (int n = 0; n < NG; ++n)
#pragma unroll
      for (int q = 0; q < 4; ++q) c[n][q] += d[n][q];
  };
  // partial sums of a tile: output = group x 128 + row x 8 + batch row of the group
  auto park = [&](float* red, const float (&c)[NG][4]) {
    float* r = red + warp * kOut + g * 8 + 2 * t;
#pragma unroll
    for (int n = 0; n < NG; ++n) {
      *reinterpret_cast<float2*>(r + 128 * n) = make_float2(c[n][0], c[n][1]);
      *reinterpret_cast<float2*>(r + 128 * n + 64) = make_float2(c[n][2], c[n][3]);
    }
  };
  auto sum = [&](const float* red, int o) -> float {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) v += red[w * kOut + o];
    return round_bf16(v);
  };
  bool copy_ok = true;

  if constexpr (!kArgmax) {
    // all of the CTA's tiles, then one barrier (the stages become the buffers of the sums) and one epilogue
    float c[STAGES][NG][4];
    int nt = 0;
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      if ((int)blockIdx.x + s * stride < a.n_tiles) {
        if (!mbar_wait_bounded(&full[s], 0)) copy_ok = false;
        multiply(s, c[s]);
        nt = s + 1;
      }
    }
    __syncthreads();
    if (tid == 0) trace_max(a.trace, 5);
#pragma unroll
    for (int s = 0; s < STAGES; ++s)
      if (s < nt) park(reinterpret_cast<float*>(stage_base + s * PairSmem::kStageBytes), c[s]);
    __syncthreads();
    constexpr int kPer = kSwiglu ? kOut / 2 : kOut;      // SwiGLU: the up row of an output is 8 rows (64 outputs) further
    for (int i = tid; i < nt * kPer; i += 256) {
      const int s = i / kPer, p = i - s * kPer, tile = blockIdx.x + s * stride;
      const float* red = reinterpret_cast<const float*>(stage_base + s * PairSmem::kStageBytes);
      if (kSwiglu) {
        const int n = p >> 6, q = p & 63, o = 128 * n + q;
        const float gv = sum(red, o), uv = sum(red, o + 64);
        a.out[(size_t)(8 * n + (q & 7)) * a.out_stride + tile * 8 + (q >> 3)] = __float2bfloat16_rn(gv / (1.0f + expf(-gv)) * uv);
      } else {
        const int n = p >> 7, q = p & 127;
        a.out[(size_t)(8 * n + (q & 7)) * a.out_stride + tile * 16 + (q >> 3)] = __float2bfloat16_rn(sum(red, p));
      }
    }
  } else {
    float best_v[2] = {-INFINITY, -INFINITY};
    int best_i[2] = {0x7fffffff, 0x7fffffff};
    int it = 0;
    for (int tile = blockIdx.x; tile < a.n_tiles; tile += stride, ++it) {
      const int s = it % STAGES;
      if (copy_ok && !mbar_wait_bounded(&full[s], (it / STAGES) & 1)) copy_ok = false;
      float c[NG][4];
      multiply(s, c);
      float* red = red_base + (it & 1) * SM::kRed;
      park(red, c);
      __syncthreads();      // every warp is done with stage s; the sums are there
      if (warp == 0 && copy_ok && tile + STAGES * stride < a.n_tiles) request_tile(tile + STAGES * stride, s);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int o = tid + 256 * h;
        if (o < kOut) {
          const int b = 8 * (o >> 7) + (o & 7), idx = tile * 16 + ((o & 127) >> 3);
          const float v = sum(red, o);
          const float key = a.temps ? sample_key(a.sample_seed, 0, srows + (b & ~7), b & 7, idx, v) : v;
          if (key > best_v[h] || (key == best_v[h] && idx < best_i[h])) { best_v[h] = key; best_i[h] = idx; }
        }
      }
    }
    // lanes with equal batch row (bits 3, 4), then the four warps of a group, then the CTAs
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int m = 8; m <= 16; m <<= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best_v[h], m);
        const int oi = __shfl_xor_sync(0xffffffffu, best_i[h], m);
        if (ov > best_v[h] || (ov == best_v[h] && oi < best_i[h])) { best_v[h] = ov; best_i[h] = oi; }
      }
      if (lane < 8) wpart[warp][8 * h + lane] = ArgmaxPart{best_v[h], best_i[h]};
    }
    __syncthreads();
    if (tid < 8 * NG) {
      const int n = tid >> 3, w0 = 4 * (n & 1), slot = 8 * (n >> 1) + (tid & 7);
      ArgmaxPart p = wpart[w0][slot];
#pragma unroll
      for (int w = 1; w < 4; ++w) {
        const ArgmaxPart q = wpart[w0 + w][slot];
        if (q.value > p.value || (q.value == p.value && q.index < p.index)) p = q;
      }
      a.parts[blockIdx.x * kWideRows + tid] = p;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) last_flag = (atomicAdd(a.ticket, 1u) == gridDim.x - 1) ? 1 : 0;
    __syncthreads();
    if (last_flag) {
      __threadfence();
      for (int b = warp; b < 8 * NG; b += 8) {
        float v = -INFINITY;
        int i = 0x7fffffff;
        for (int c2 = lane; c2 < (int)gridDim.x; c2 += 32) {
          const int2 raw = __ldcg(reinterpret_cast<const int2*>(a.parts + c2 * kWideRows + b));
          const float pv = __int_as_float(raw.x);
          if (pv > v || (pv == v && raw.y < i)) { v = pv; i = raw.y; }
        }
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) {
          const float ov = __shfl_xor_sync(0xffffffffu, v, m);
          const int oi = __shfl_xor_sync(0xffffffffu, i, m);
          if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
        }
        if (lane == 0) a.tokens[b] = i;
      }
      if (tid == 0) {
        *a.ticket = 0u;
        if (sampled_groups) *a.sample_ctr += (unsigned)sampled_groups;
      }
    }
  }
  if (!copy_ok) {   // a bulk copy never completed: record it, give those in flight one more bounded chance to land
    report_status(a.status, kStatusCopyTimeout, kKernelWide, blockIdx.x, MODE);
#pragma unroll 1
    for (int s = 0; s < STAGES; ++s) mbar_wait_bounded(&full[s], 0);
  }
  if (tid == 0) trace_max(a.trace, 2);
}

// out[8 NG, N] = x[8 NG, K] @ W[N, K]^T: clusters of four CTAs, 32 weight rows each cluster, a quarter of K per CTA
template <int K, int NG>
struct WideStoreSmem {
  static constexpr int kPart = K / kWideCluster, kRowStride = 2 * kPart + 64;      // (+ 64: conflict-free fragment reads)
  static constexpr int kOut = 256 * NG;                                           // outputs: group x 256 + row x 8 + batch row
  static constexpr int bytes() { return 32 * kRowStride + 4 * 8 * kOut + 4 * kOut + 16; }
};
template <int K, int NG>
__global__ void __launch_bounds__(256, 2) wide_store_kernel(const GemvArgs a) {
  using SM = WideStoreSmem<K, NG>;
  constexpr int LJ = SM::kPart / 256, kOut = SM::kOut;       // LJ: 32-column blocks of a warp
  pdl_launch_dependents();
  if (threadIdx.x == 0) trace_min(a.trace, 0);
  cluster_arrive_relaxed();      // completed before a peer's shared memory is written: it is running by then
  extern __shared__ __align__(128) unsigned char dyn_smem[];
  float* red = reinterpret_cast<float*>(dyn_smem + 32 * SM::kRowStride);      // [warp][output]
  float* recv = red + 8 * kOut;                              // [source CTA][64 NG]: partial sums of the rows this CTA finishes
  uint64_t* full = reinterpret_cast<uint64_t*>(recv + kOut);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int tile = blockIdx.x / kWideCluster, rank = blockIdx.x % kWideCluster, kbase = warp * (32 * LJ) + 8 * t;
  if (warp == 0) {
    if (lane == 0) {
      mbar_init(full, 1);
      fence_mbar_init();
      mbar_expect_tx(full, 32 * 2 * SM::kPart);
    }
    __syncwarp();
    bulk_g2s(dyn_smem + lane * SM::kRowStride, a.w + (size_t)(tile * 32 + lane) * K + rank * SM::kPart, 2 * SM::kPart, full);
  }
  __syncthreads();
  pdl_wait();
  if (tid == 0) { trace_max(a.trace, 1); trace_min(a.trace, 3); }

  uint4 xb[NG][LJ];
  const __nv_bfloat16* xp = a.x + (size_t)g * K + rank * SM::kPart + kbase;
#pragma unroll
  for (int n = 0; n < NG; ++n)
#pragma unroll
    for (int j = 0; j < LJ; ++j) xb[n][j] = ldg_cg(xp + (size_t)(8 * n) * K + 32 * j);
  const bool copy_ok = mbar_wait_bounded(full, 0);
  float c[2][NG][4];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int n = 0; n < NG; ++n)
#pragma unroll
      for (int q = 0; q < 4; ++q) c[h][n][q] = 0.f;
#pragma unroll
  for (int j = 0; j < LJ; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const unsigned char* wp = dyn_smem + (16 * h + g) * SM::kRowStride + 2 * kbase + 64 * j;
      const uint4 u = *reinterpret_cast<const uint4*>(wp), v = *reinterpret_cast<const uint4*>(wp + 8 * SM::kRowStride);
#pragma unroll
      for (int n = 0; n < NG; ++n) {
        mma_bf16_16816_full(c[h][n], u.x, v.x, u.y, v.y, xb[n][j].x, xb[n][j].y);
        mma_bf16_16816_full(c[h][n], u.z, v.z, u.w, v.w, xb[n][j].z, xb[n][j].w);
      }
    }
  float* r = red + warp * kOut + g * 8 + 2 * t;
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int n = 0; n < NG; ++n) {
      *reinterpret_cast<float2*>(r + 256 * n + 128 * h) = make_float2(c[h][n][0], c[h][n][1]);
      *reinterpret_cast<float2*>(r + 256 * n + 128 * h + 64) = make_float2(c[h][n][2], c[h][n][3]);
    }
  __syncthreads();
  if (tid == 0) trace_max(a.trace, 5);
  cluster_wait();
  // thread: row tid / 8 of the tile, batch row tid % 8 of every group; CTA row / 8 of the cluster finishes it
#pragma unroll
  for (int n = 0; n < NG; ++n) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) v += red[w * kOut + 256 * n + tid];
    asm volatile("st.shared::cluster.f32 [%0], %1;"
                 ::"r"(peer_smem(recv + rank * 64 * NG + 64 * n + (tid & 63), tid >> 6)), "f"(v) : "memory");
  }
  cluster_arrive();
  cluster_wait();
  if (tid < 64 * NG) {
    const int n = tid >> 6, q = tid & 63;
    const float v = (recv[tid] + recv[64 * NG + tid]) + (recv[2 * 64 * NG + tid] + recv[3 * 64 * NG + tid]);
    a.out[(size_t)(8 * n + (q & 7)) * a.out_stride + tile * 32 + 8 * rank + (q >> 3)] = __float2bfloat16_rn(v);
  }
  if (!copy_ok) {   // as above
    report_status(a.status, kStatusCopyTimeout, kKernelWide, blockIdx.x, kModeStore);
    mbar_wait_bounded(full, 0);
  }
  if (tid == 0) trace_max(a.trace, 2);
}

// Tokens and status of a wide step into pinned host memory, followed by the sequence word (see publish_result_kernel).
__global__ void publish_wide_kernel(const int* tokens, const int* status, int* host_out, unsigned int* seq) {
  pdl_wait();
  const int i = threadIdx.x;
  if (i < kWideRows) host_out[i] = tokens[i];
  else if (i < kWideRows + 4) host_out[i] = status[i - kWideRows];
  __threadfence_system();
  __syncthreads();
  if (i == 0) {
    const unsigned int next = *seq + 1u;
    *seq = next;
    *reinterpret_cast<volatile int*>(host_out + kWideRows + 4) = (int)next;
  }
}

}  // namespace dfb
