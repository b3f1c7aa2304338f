// NVFP4 / MX block-scaled GEMM for few output tiles: the weight matrix is the M operand.
//
//   C[m, n] = alpha * sum_k (A[m,k] * SFA) * (B[n,k] * SFB)          (as in gemm_kernel.cuh)
//
// A decode step multiplies a handful of rows of A with a large B.  With A on the tensor core's 128-row side every stage
// carries 128 rows of A for the few that exist, and a 64-wide slice of B leaves half of the instruction idle.  Here a
// tile is 128 rows of B times kTok rows of A: a stage is 16 KB of weights and kTok * 128 bytes of activations.
//
// Such problems have few tiles and long reductions, so the K steps of a tile are dealt to a cluster of CTAs (up to 8).
// Every CTA accumulates its share in tensor memory; then each sends every other one the columns it is responsible for
// through distributed shared memory, adds the shares in rank order (a fixed order: results do not depend on timing),
// scales, rounds once and stores.  No workspace and no second kernel.
//
// What bounds it: the stream of B plus 4 to 5 us of launch, pipeline fill, exchange and drain; a CTA's own K step takes
// 0.3 us, the round trip of a load against five stages, whatever the stage brings -- hence the split, and two CTAs per
// SM.  128 x 64 tiles before, this kernel now: M = 16, N = K = 4096 8.8 -> 5.5 us; N = K = 8192 (38 MB) 17.5 -> 11.1 us;
// M = 64, N = 2048, K = 7168 12.5 -> 7.4 us.
//
// Roles: warp 0 TMA producer, warp 1 MMA issuer (see gemm_kernel.cuh), warps 2-5 carry the scale slabs from shared to
// tensor memory and then are the epilogue.  One tile share per CTA; up to two CTAs live on an SM, so that one's fill and
// drain overlap the other's stream.  All waits are bounded as in gemm_kernel.cuh; no multicast.
#pragma once

#include "gemm_kernel.cuh"

namespace b200fp4 {

constexpr int kStreamThreads = 6 * 32;
constexpr uint32_t kStreamTmemCols = 256;

// kTok: rows of A per tile (the N of the MMA)
struct StreamLayout {
  int stages;
  uint32_t x_bytes, stage_bytes, sf_col, total;
};
__host__ __device__ constexpr StreamLayout stream_layout(int tok) {
  StreamLayout s{};
  s.x_bytes = static_cast<uint32_t>(tok) * 128;
  s.stage_bytes = 16384 + s.x_bytes + 2 * 2048;
  // two CTAs per SM: 113 KB of shared memory and 256 tensor-memory columns each
  s.stages = tok <= 16 ? 5 : (tok <= 64 ? 4 : 3);
  s.sf_col = tok <= 64 ? 64u : 128u;
  s.total = s.stages * s.stage_bytes + 256;
  return s;
}

template <int kTok, typename OutT>
__global__ void __launch_bounds__(kStreamThreads, 2)
nvfp4_gemm_stream_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                         const GemmParams p, OutT* c, const float* alpha) {
  constexpr StreamLayout L = stream_layout(kTok);
  constexpr int kStages = L.stages;
  constexpr uint32_t kSfSetCols = 32;                    // 16 columns of W scales + 16 of X scales per stage
  static_assert(L.sf_col + kStages * kSfSetCols <= kStreamTmemCols, "TMEM budget");

  // 1024-byte aligned for the swizzled tiles; there is no room for slack with two CTAs on an SM
  extern __shared__ __align__(1024) uint8_t smem_gen[];
  const uint32_t smem_base = ptx::smem_u32(smem_gen);
  const uint32_t bar_base = smem_base + kStages * L.stage_bytes;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kStages + s); };
  auto sf_loaded_bar = [&](int s) { return bar_base + 8u * (2 * kStages + s); };
  auto sf_full_bar = [&](int s) { return bar_base + 8u * (3 * kStages + s); };
  const uint32_t acc_full_bar = bar_base + 8u * (4 * kStages);
  uint8_t* tail_gen = smem_gen + kStages * L.stage_bytes + 8 * (4 * kStages + 1);
  volatile uint32_t* tmem_ptr_smem = reinterpret_cast<volatile uint32_t*>(tail_gen);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail_gen + 4);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int splits = p.k_splits;
  const int rank = static_cast<int>(blockIdx.x) % splits;      // = rank in the cluster
  const int n_blk = static_cast<int>(blockIdx.x) / splits;     // 128 rows of B
  const int m0 = static_cast<int>(blockIdx.y) * kTok;          // first row of A
  const int kt0 = rank * p.num_k_tiles / splits, kt1 = (rank + 1) * p.num_k_tiles / splits;       // never empty

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(full_bar(s), 1);
      ptx::mbar_init(empty_bar(s), 1);
      ptx::mbar_init(sf_loaded_bar(s), 1);
      ptx::mbar_init(sf_full_bar(s), 4);
    }
    ptx::mbar_init(acc_full_bar, 1);
    *abort_flag = 0;
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&tmap_w);
    ptx::prefetch_tensormap(&tmap_x);
  }
  if (warp == 0) {
    __syncwarp();
    ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(tmem_ptr_smem)), kStreamTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;
  grid_dependency_wait();

  const int tps = 4 >> p.sf_block32;                     // 512-byte scale tiles per stage
  if (warp == 0) {
    // =============================== TMA producer ===============================
    if (lane == 0) {
      PipeState st;
      const uint8_t* sfw = p.sfb + static_cast<int64_t>(n_blk) * p.rk * 512;
      const uint8_t* sfx = p.sfa + static_cast<int64_t>(m0 >> 7) * p.rk * 512;
      for (int kt = kt0; kt < kt1; ++kt) {
        if (!wait_bounded(empty_bar(st.stage), st.phase ^ 1u, abort_flag)) {
          atomicOr(p.status, kStatusTimeoutProducer);
          break;
        }
        const uint32_t sw = smem_base + st.stage * L.stage_bytes, sx = sw + 16384, ssf = sx + L.x_bytes;
        const uint32_t sf_bytes = static_cast<uint32_t>(min(tps, p.rk - tps * kt)) * 512u;
        const uint32_t sbar = sf_loaded_bar(st.stage), bar = full_bar(st.stage);
        ptx::mbar_expect_tx(sbar, 2 * sf_bytes);
        ptx::bulk_load(ssf, sfw + tps * kt * 512, sf_bytes, sbar);
        ptx::bulk_load(ssf + 2048, sfx + tps * kt * 512, sf_bytes, sbar);
        ptx::mbar_expect_tx(bar, 16384 + L.x_bytes);
        ptx::tma_load_3d(sw, &tmap_w, kt * 128, n_blk * 128, 0, bar);
        ptx::tma_load_2d(sx, &tmap_x, kt * 128, m0, bar);
        st.advance(kStages);
      }
      let_dependents_launch();       // the last loads are under way (16 x 8192 x 8192: 11.0 -> 10.3 us a call)
    }
    __syncwarp();
  } else if (warp == 1) {
    // =============================== MMA issuer ===============================
    PipeState st;
    bool ok = true;
    const uint64_t w_desc0 = ptx::smem_desc_sw128(smem_base);
    const uint64_t x_desc0 = ptx::smem_desc_sw128(smem_base + 16384);
    const int last_kblocks = ((p.k_bytes - (p.num_k_tiles - 1) * 128) + 31) >> 5;
    for (int kt = kt0; kt < kt1; ++kt) {
      if (!wait_bounded(sf_full_bar(st.stage), st.phase, abort_flag) ||
          !wait_bounded(full_bar(st.stage), st.phase, abort_flag)) {
        if (lane == 0) atomicOr(p.status, kStatusTimeoutMma);
        ok = false;
        break;
      }
      ptx::tc_fence_after_sync();
      const uint64_t off = static_cast<uint64_t>(st.stage * (L.stage_bytes >> 4));
      const uint64_t dw = w_desc0 + off, dx = x_desc0 + off;
      const uint32_t sfw_t = tmem_base + L.sf_col + st.stage * kSfSetCols;
      const uint32_t sfx_t = sfw_t + 16;
      const int kblocks = kt + 1 == p.num_k_tiles ? last_kblocks : 4;
      if (ptx::elect_one()) {
        if (p.sf_block32 == 2) {
#pragma unroll
          for (int kb = 0; kb < 4; ++kb) {
            if (kb < kblocks)       // (the A operand of the instruction is B of the product)
              ptx::mma_mxf8_block32(tmem_base, dw + 2 * kb, dx + 2 * kb,
                                    ptx::idesc_mxf8_block32(kTok, p.b_fmt8, p.a_fmt8, kb), sfw_t, sfx_t,
                                    (kt != kt0 || kb != 0) ? 1u : 0u);
          }
        } else if (p.sf_block32 == 1) {
#pragma unroll
          for (int kb = 0; kb < 4; ++kb) {
            if (kb < kblocks)
              ptx::mma_mxf4_block32(tmem_base, dw + 2 * kb, dx + 2 * kb, ptx::idesc_mxf4_block32(kTok, (kb & 1) * 2),
                                    sfw_t + 4 * (kb >> 1), sfx_t + 4 * (kb >> 1), (kt != kt0 || kb != 0) ? 1u : 0u);
          }
        } else {
#pragma unroll
          for (int kb = 0; kb < 4; ++kb) {
            if (kb < kblocks)
              ptx::mma_mxf4nvf4(tmem_base, dw + 2 * kb, dx + 2 * kb, ptx::idesc_mxf4nvf4(kTok), sfw_t + 4 * kb,
                                sfx_t + 4 * kb, (kt != kt0 || kb != 0) ? 1u : 0u);
          }
        }
        ptx::tc_commit(empty_bar(st.stage));
      }
      __syncwarp();
      st.advance(kStages);
    }
    if (ok && ptx::elect_one()) ptx::tc_commit(acc_full_bar);
    __syncwarp();
  } else {
    // =============================== scale-slab movers ===============================
    const int quarter = warp & 3;
    // The words of a slab row are the row groups 0-3 (32 rows each) of the 128-row scale tile; a tile of A that starts in
    // group g gets its groups moved to the front, so that the MMA always reads from the first column of a K block.
    const int first_group = (m0 & 127) >> 5;
    PipeState st;
    for (int kt = kt0; kt < kt1; ++kt) {
      if (!wait_bounded(sf_loaded_bar(st.stage), st.phase, abort_flag)) {
        if (lane == 0) atomicOr(p.status, kStatusTimeoutMma);
        break;
      }
      const uint8_t* slab = smem_gen + st.stage * L.stage_bytes + 16384 + L.x_bytes + lane * 16;
      const uint32_t t_sf = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + L.sf_col + st.stage * kSfSetCols;
      uint32_t r[32];
#pragma unroll
      for (int i = 0; i < 8; ++i) {                      // four K blocks of W scales, then of X scales
        uint4 v = *reinterpret_cast<const uint4*>(slab + 512 * i);
        if (i >= 4 && kTok < 128) {
          if (first_group & 1) v = make_uint4(v.y, v.z, v.w, v.x);
          if (first_group & 2) v = make_uint4(v.z, v.w, v.x, v.y);
        }
        r[4 * i] = v.x, r[4 * i + 1] = v.y, r[4 * i + 2] = v.z, r[4 * i + 3] = v.w;
      }
      ptx::tmem_st_32x32(t_sf, r);
      ptx::tmem_st_wait();
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(sf_full_bar(st.stage));
      st.advance(kStages);
    }
  }

  // =============================== epilogue ===============================
  // warps 2-5: thread = one row of B (channel), the accumulator's columns are rows of A
  const int quarter = warp & 3;
  const int channel = quarter * 32 + lane;
  const int n = n_blk * 128 + channel;
  const float scale = alpha == nullptr ? 1.0f : ld_word(alpha);
  const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
  auto store = [&](int col, float v) {
    const int m = m0 + col;
    if (n < p.n_cols && m < p.m_rows) {
      const float s = v * scale;
      if constexpr (sizeof(OutT) == 4) c[static_cast<int64_t>(m) * p.n_cols + n] = s;
      else c[static_cast<int64_t>(m) * p.n_cols + n] = to_out<OutT>(s);
    }
  };
  if (warp >= 2) {
    if (!wait_bounded<32>(acc_full_bar, 0, abort_flag) && lane == 0) atomicOr(p.status, kStatusTimeoutEpilogue);
    __syncwarp();
    ptx::tc_fence_after_sync();
  }
  if (splits == 1) {
    if (warp >= 2) {
#pragma unroll 1
      for (int c0 = 0; c0 < kTok; c0 += 16) {
        uint32_t r[16];
        ptx::tmem_ld_32x16(t_acc + c0, r);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) store(c0 + i, __uint_as_float(r[i]));
      }
    }
  } else {
    // every CTA of the cluster is past its loads and MMAs: the stages can take the partial sums
    ptx::cluster_sync();
    const int cols = kTok / splits, shift = __ffs(cols) - 1;       // columns this CTA is responsible for (a power of two)
    if (warp >= 2) {
#pragma unroll 1
      for (int c0 = 0; c0 < kTok; c0 += 16) {
        uint32_t r[16];
        ptx::tmem_ld_32x16(t_acc + c0, r);
        ptx::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i += 4) {        // groups of four columns: [source rank][group][channel][4]
          const int col = c0 + i;
          const uint32_t at = smem_base + ((rank * cols + (col & (cols - 1))) * 128 + 4 * channel) * 4;
          ptx::st_cluster_v4(ptx::map_to_rank(at, col >> shift), r[i], r[i + 1], r[i + 2], r[i + 3]);
        }
      }
    }
    ptx::cluster_sync();
    if (warp >= 2) {
      const float4* part = reinterpret_cast<const float4*>(smem_gen) + channel;
      for (int j = 0; j < cols; j += 4) {
        float4 sum = part[j * 32];
        for (int s = 1; s < splits; ++s) {
          const float4 v = part[(s * cols + j) * 32];
          sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
        }
        store(rank * cols + j, sum.x);
        store(rank * cols + j + 1, sum.y);
        store(rank * cols + j + 2, sum.z);
        store(rank * cols + j + 3, sum.w);
      }
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    if (*abort_flag) {
      for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    __syncwarp();
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem_base, kStreamTmemCols);
  }
}

}  // namespace b200fp4
