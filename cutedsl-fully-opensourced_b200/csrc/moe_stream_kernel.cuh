// Grouped NVFP4 GEMMs of the MoE for few rows per expert: the weights are the M operand (as in gemm_stream_kernel.cuh).
//
// With the tokens on the tensor core's 128-row side an expert that was named by two tokens multiplies 126 rows of padding
// -- the padding costs no time while the step waits for its weights, but it costs power: a 64-token step of the large
// decode configuration ran at 1.3 GHz under the power cap, and slower DRAM traffic with it.  Here a tile is 256 rows of an
// expert's weights (two instructions of 128) times the rows of one block of tokens, at most kTok, with the instruction's
// N set to the rows the block has (rounded up to 16).  Rows of a block lie kTok apart from the next block's, so nothing
// is padded to 128 in memory either, and the scale bytes of tokens and activations are plain rows.
//
//   FC1: the two pieces are up rows j..j+127 and gate rows j..j+127: a lane (channel) holds both of every token.
//        silu(gate) * up -> bf16 goes through shared memory, where a thread picks up 16 adjacent channels of a token
//        and quantises them (same arithmetic as EpilogueSwiglu in gemm_kernel.cuh).
//   FC2: the two pieces are 256 adjacent output columns; rows leave through shared memory as whole lines.
//
// Roles as in gemm_kernel.cuh: warp 0 TMA producer, warp 1 MMA issuer, warps 2-9 epilogue, warps 10-13 scale-slab movers;
// persistent over (block, column block), row block outermost; two accumulators; all waits bounded; no multicast.
//
// What bounds it: the stream of the weights.  Steps of hidden 7168, 256 experts, intermediate 2048, top-8, 128-row kernels
// before and these: 64 tokens 943 -> 829 us (5.5 GB: 6.65 TB/s), one token 58 -> 51 us; hidden 2048, 128 experts,
// intermediate 768, 333 tokens 102 -> 91 us.
#pragma once

#include "gemm_kernel.cuh"

namespace b200fp4 {

constexpr int kMoeStreamThreads = 14 * 32;

struct MoeStreamLayout {
  int stages;
  int park_rows;               // rows parked at a time: FC1 all of a tile, FC2 of either piece
  uint32_t x_bytes, sfx_bytes, stage_bytes, park_bytes, total;
};
__host__ __device__ constexpr MoeStreamLayout moe_stream_layout(int tok, int park_elem, bool swiglu) {
  MoeStreamLayout s{};
  s.x_bytes = static_cast<uint32_t>(tok) * 128;
  s.sfx_bytes = 1024;                                    // kTok rows of 16 bytes
  s.stage_bytes = 2 * 16384 + s.x_bytes + 2 * 2048 + s.sfx_bytes;
  s.park_rows = swiglu ? tok : (park_elem == 4 || tok < 32 ? 16 : 32);
  s.park_bytes = static_cast<uint32_t>(swiglu ? tok : 2 * s.park_rows) * 128 * park_elem;
  s.stages = tok <= 32 ? 5 : 4;
  s.total = s.stages * s.stage_bytes + 1024 + 512 + s.park_bytes;
  return s;
}

struct MoeStreamFc1 {          // swiglu + re-quantisation
  static constexpr bool kSwiglu = true;
  static constexpr int kParkElem = 2;                    // bf16 activations [token][128 channels]
  uint8_t* act_codes;          // [rows][inter / 2]
  uint8_t* act_sf;             // [rows][sf_pitch]
  const float* w1_alpha;
  const float* fc2_input_scale;
  int inter, sf_pitch;
};
template <typename RowT>
struct MoeStreamFc2 {          // per-slot output rows
  using Row = RowT;
  static constexpr bool kSwiglu = false;
  static constexpr int kParkElem = sizeof(RowT);         // [token][128 columns], one piece at a time
  RowT* rows;                  // [rows][hidden]
  const float* w2_alpha;
  int hidden;
};

template <int kTok, typename Epi>
__global__ void __launch_bounds__(kMoeStreamThreads, 1)
moe_stream_gemm_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                       const __grid_constant__ CUtensorMap tmap_sfx, const GemmParams p, const Epi epi) {
  constexpr MoeStreamLayout L = moe_stream_layout(kTok, Epi::kParkElem, Epi::kSwiglu);
  constexpr int kStages = L.stages;
  constexpr uint32_t kAccCols = 2 * kTok;                // two pieces
  constexpr uint32_t kSfaCol = 2 * kAccCols;             // two accumulators first
  constexpr uint32_t kSfSetCols = 48;                    // scales of piece 0, piece 1 and X: 16 columns each
  static_assert(kSfaCol + kStages * kSfSetCols <= kTmemCols, "TMEM budget");

  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + kStages * L.stage_bytes;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kStages + s); };
  auto sf_loaded_bar = [&](int s) { return bar_base + 8u * (2 * kStages + s); };
  auto sf_full_bar = [&](int s) { return bar_base + 8u * (3 * kStages + s); };
  auto acc_full_bar = [&](int s) { return bar_base + 8u * (4 * kStages + s); };
  auto acc_empty_bar = [&](int s) { return bar_base + 8u * (4 * kStages + 2 + s); };
  uint8_t* tail_gen = smem_gen + kStages * L.stage_bytes + 8 * (4 * kStages + 4);
  volatile uint32_t* tmem_ptr_smem = reinterpret_cast<volatile uint32_t*>(tail_gen);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail_gen + 4);
  volatile int* early_blocks = reinterpret_cast<volatile int*>(tail_gen + 8);
  uint8_t* park = smem_gen + kStages * L.stage_bytes + 512;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (p.early_b && threadIdx.x == 32) *early_blocks = ld_early_word(p.num_m_blocks_dev);    // one read per CTA: past L1 they add up
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(full_bar(s), 1);
      ptx::mbar_init(empty_bar(s), 1);
      ptx::mbar_init(sf_loaded_bar(s), 1);
      ptx::mbar_init(sf_full_bar(s), 4);
    }
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(acc_full_bar(s), 1);
      ptx::mbar_init(acc_empty_bar(s), 8);
    }
    *abort_flag = 0;
    ptx::fence_mbar_init();
    ptx::prefetch_tensormap(&tmap_w);
    ptx::prefetch_tensormap(&tmap_x);
    ptx::prefetch_tensormap(&tmap_sfx);
  }
  if (warp == 0) {
    __syncwarp();
    ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(tmem_ptr_smem)), kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr_smem;
  if (!p.early_b) grid_dependency_wait();

  // block counts read from device memory are never trusted beyond the table size
  const int num_blocks = max(0, min(p.early_b ? *early_blocks : ld_word(p.num_m_blocks_dev), p.num_m_blocks));
  const int num_tiles = num_blocks * p.num_n_blocks;
  auto rows_of = [&](int blk) { return max(0, min(ld_word(p.m_block_rows + blk), kTok)); };

  if (warp == 0) {
    // =============================== TMA producer ===============================
    if (lane == 0) {
      PipeState st;
      bool ok = true;
      int blk = 0, group = 0, w_row[2];
      const uint8_t* sfw[2];
      auto begin_tile = [&](int tile, auto before_wait) {
        blk = tile / p.num_n_blocks;
        const int n_blk = tile - blk * p.num_n_blocks;
        const int* g = p.m_block_group + blk;
        group = max(0, min(decltype(before_wait)::value ? ld_early_word(g) : ld_word(g), p.num_groups - 1));
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          w_row[i] = Epi::kSwiglu ? n_blk * 128 + i * p.gate_row_offset : n_blk * 256 + i * 128;
          // the last 256-wide column block of an odd number of 128-row tiles: its second half does not exist
          const int t = min(w_row[i] >> 7, p.b_row_tiles - 1);
          sfw[i] = p.sfb + (static_cast<int64_t>(group) * p.b_row_tiles + t) * p.rk * 512;
        }
      };
      auto issue = [&](int kt, int stage, auto x_part, auto w_part) {
        constexpr bool kX = decltype(x_part)::value, kW = decltype(w_part)::value;
        const uint32_t sw = smem_base + stage * L.stage_bytes, sx = sw + 32768;
        const uint32_t ssfw = sx + L.x_bytes, ssfx = ssfw + 4096;
        const uint32_t sf_bytes = static_cast<uint32_t>(min(4, p.rk - 4 * kt)) * 512u;
        const uint32_t sbar = sf_loaded_bar(stage), bar = full_bar(stage);
        if constexpr (kW) {
          ptx::mbar_expect_tx(sbar, 2 * sf_bytes + kTok * 16);
          ptx::bulk_load(ssfw, sfw[0] + kt * 2048, sf_bytes, sbar);
          ptx::bulk_load(ssfw + 2048, sfw[1] + kt * 2048, sf_bytes, sbar);
        }
        if constexpr (kX) ptx::tma_load_2d(ssfx, &tmap_sfx, kt * 16, blk * kTok, sbar);
        if constexpr (kW) {
          ptx::mbar_expect_tx(bar, 32768 + L.x_bytes);
          ptx::tma_load_3d(sw, &tmap_w, kt * 128, w_row[0], group, bar);
          ptx::tma_load_3d(sw + 16384, &tmap_w, kt * 128, w_row[1], group, bar);
        }
        if constexpr (kX) ptx::tma_load_2d(sx, &tmap_x, kt * 128, blk * kTok, bar);
      };
      int primed = 0;                    // stages whose weights are under way
      if (p.early_b) {
        for (int tile = blockIdx.x; tile < num_tiles && primed < kStages; tile += gridDim.x) {
          begin_tile(tile, std::true_type{});
          for (int kt = 0; kt < p.num_k_tiles && primed < kStages; ++kt) issue(kt, primed++, std::false_type{}, std::true_type{});
        }
        grid_dependency_wait();
      }
      if (p.early_trigger) let_dependents_launch();
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        begin_tile(tile, std::false_type{});
        for (int kt = 0; kt < p.num_k_tiles; ++kt) {
          if (!wait_bounded(empty_bar(st.stage), st.phase ^ 1u, abort_flag)) {
            atomicOr(p.status, kStatusTimeoutProducer);
            ok = false;
            break;
          }
          if (primed > 0) {
            --primed;
            issue(kt, st.stage, std::true_type{}, std::false_type{});
          } else {
            issue(kt, st.stage, std::true_type{}, std::true_type{});
          }
          st.advance(kStages);
        }
      }
    }
  } else if (warp == 1) {
    // =============================== MMA issuer ===============================
    PipeState st, acc;
    bool ok = true;
    const uint64_t w_desc0 = ptx::smem_desc_sw128(smem_base);
    const uint64_t x_desc0 = ptx::smem_desc_sw128(smem_base + 32768);
    const int last_kblocks = ((p.k_bytes - (p.num_k_tiles - 1) * 128) + 31) >> 5;
    if (p.early_b) grid_dependency_wait();               // nothing can be multiplied before the rows are there anyway
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
      // N of the instructions: the rows of the block, rounded up to 16
      const int n = kTok == 16 ? 16 : max(16, (rows_of(tile / p.num_n_blocks) + 15) & ~15);
      const uint32_t idesc = ptx::idesc_mxf4nvf4(n);
      if (!wait_bounded(acc_empty_bar(acc.stage), acc.phase ^ 1u, abort_flag)) {
        if (lane == 0) atomicOr(p.status, kStatusTimeoutMma);
        break;
      }
      ptx::tc_fence_after_sync();
      const uint32_t d = tmem_base + acc.stage * kAccCols;
      for (int kt = 0; kt < p.num_k_tiles; ++kt) {
        if (!wait_bounded(sf_full_bar(st.stage), st.phase, abort_flag) ||
            !wait_bounded(full_bar(st.stage), st.phase, abort_flag)) {
          if (lane == 0) atomicOr(p.status, kStatusTimeoutMma);
          ok = false;
          break;
        }
        ptx::tc_fence_after_sync();
        const uint64_t off = static_cast<uint64_t>(st.stage * (L.stage_bytes >> 4));
        const uint64_t dw = w_desc0 + off, dx = x_desc0 + off;
        const uint32_t sf = tmem_base + kSfaCol + st.stage * kSfSetCols;
        const int kblocks = kt + 1 == p.num_k_tiles ? last_kblocks : 4;
        if (ptx::elect_one()) {
#pragma unroll
          for (int kb = 0; kb < 4; ++kb) {
            if (kb < kblocks) {
              const uint32_t on = (kt != 0 || kb != 0) ? 1u : 0u;
              ptx::mma_mxf4nvf4(d, dw + 2 * kb, dx + 2 * kb, idesc, sf + 4 * kb, sf + 32 + 4 * kb, on);
              ptx::mma_mxf4nvf4(d + kTok, dw + 1024 + 2 * kb, dx + 2 * kb, idesc, sf + 16 + 4 * kb, sf + 32 + 4 * kb, on);
            }
          }
          ptx::tc_commit(empty_bar(st.stage));
        }
        __syncwarp();
        st.advance(kStages);
      }
      if (ok && ptx::elect_one()) ptx::tc_commit(acc_full_bar(acc.stage));
      __syncwarp();
      acc.advance(2);
    }
  } else if (warp >= 10) {
    // =============================== scale-slab movers ===============================
    const int quarter = warp & 3;
    PipeState st;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
      for (int kt = 0; kt < p.num_k_tiles; ++kt) {
        if (!wait_bounded(sf_loaded_bar(st.stage), st.phase, abort_flag)) {
          if (lane == 0) atomicOr(p.status, kStatusTimeoutMma);
          ok = false;
          break;
        }
        const uint8_t* slab = smem_gen + st.stage * L.stage_bytes + 32768 + L.x_bytes + lane * 16;
        const uint32_t t_sf = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + kSfaCol + st.stage * kSfSetCols;
        uint32_t r[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {                    // four K blocks of piece 0, then of piece 1
          const uint4 v = *reinterpret_cast<const uint4*>(slab + 512 * i);
          r[4 * i] = v.x, r[4 * i + 1] = v.y, r[4 * i + 2] = v.z, r[4 * i + 3] = v.w;
        }
        ptx::tmem_st_32x32(t_sf, r);
        // plain rows: the words of row 32 c + lane are K blocks 0..3 of row group c
        uint32_t x[16];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint4 v = make_uint4(0u, 0u, 0u, 0u);
          if (32 * c < kTok && (kTok >= 32 || lane < kTok)) v = *reinterpret_cast<const uint4*>(slab + 4096 + 512 * c);
          x[c] = v.x, x[4 + c] = v.y, x[8 + c] = v.z, x[12 + c] = v.w;
        }
        ptx::tmem_st_32x16(t_sf + 32, x);
        ptx::tmem_st_wait();
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(sf_full_bar(st.stage));
        st.advance(kStages);
      }
    }
  } else {
    // =============================== epilogue ===============================
    // Two groups of four warps, one warp of each per quarter of tensor memory.  FC1: the groups take the rows by sixteens in
    // turn; FC2: a piece each.
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int channel = quarter * 32 + lane;
    const int tid = threadIdx.x - 64;                    // 0..255
    if (p.early_b) grid_dependency_wait();
    // what a tile needs from the tables is read one tile ahead: behind the accumulator's barrier the two dependent loads
    // would be on the path of every tile
    struct Tile {
      int blk, n_blk, rows, group;
      float alpha;
    };
    auto look_up = [&](int tile) {
      Tile t{};
      if (tile < num_tiles) {
        t.blk = tile / p.num_n_blocks;
        t.n_blk = tile - t.blk * p.num_n_blocks;
        t.rows = rows_of(t.blk);
        t.group = max(0, min(ld_word(p.m_block_group + t.blk), p.num_groups - 1));
        const float* alpha;
        if constexpr (Epi::kSwiglu) alpha = epi.w1_alpha;
        else alpha = epi.w2_alpha;
        t.alpha = alpha == nullptr ? 1.0f : ld_word(alpha + t.group);
      }
      return t;
    };
    float gs = 1.0f;
    if constexpr (Epi::kSwiglu) {
      if (epi.fc2_input_scale != nullptr) gs = ld_word(epi.fc2_input_scale);
    }
    const bool gs_pow2 = is_power_of_two(gs);
    PipeState acc;
    Tile next = look_up(blockIdx.x);
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      const Tile now = next;
      next = look_up(tile + gridDim.x);
      const int rows = now.rows, n_blk = now.n_blk;
      const int64_t row0 = static_cast<int64_t>(now.blk) * kTok;
      const bool ready = wait_bounded<64>(acc_full_bar(acc.stage), acc.phase, abort_flag);
      // the eight warps go on or give up together: they meet at barriers below
      if (!ptx::bar_all(1, 256, ready)) {
        if (lane == 0) atomicOr(p.status, kStatusTimeoutEpilogue);
        break;
      }
      ptx::tc_fence_after_sync();
      const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc.stage * kAccCols;
      auto release = [&] {                               // once per warp and tile, after its last read of the accumulator
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(acc_empty_bar(acc.stage));
      };
      if constexpr (Epi::kSwiglu) {
        __nv_bfloat16* act = reinterpret_cast<__nv_bfloat16*>(park);
        if (16 * half >= rows) release();
#pragma unroll 1
        for (int c0 = 16 * half; c0 < rows; c0 += 32) {
          uint32_t up[16], gate[16];
          ptx::tmem_ld_32x16(t_acc + c0, up);
          ptx::tmem_ld_32x16(t_acc + kTok + c0, gate);
          ptx::tmem_ld_wait();
          if (c0 + 32 >= rows) release();
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float u = __fmul_rn(__uint_as_float(up[i]), now.alpha), g = __fmul_rn(__uint_as_float(gate[i]), now.alpha);
            const float s = __fdividef(g, __fadd_rn(1.0f, __expf(-g)));
            act[(c0 + i) * 128 + channel] = __float2bfloat16_rn(__fmul_rn(s, u));
          }
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        // item: 16 adjacent channels of one token; eight lanes hold the 128 channels of a token
        for (int item = tid; item < ((rows + 15) & ~15) * 8; item += 256) {
          const int t = item >> 3, b = item & 7;
          const uint4* src = reinterpret_cast<const uint4*>(act + t * 128 + b * 16);
          const uint4 q0 = src[0], q1 = src[1];
          const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
          const Block16Codes q = quantize_bf16x16(w, gs, gs_pow2);
          uint32_t sf = q.sf;
          sf |= __shfl_down_sync(0xffffffffu, sf, 1) << 8;
          sf |= __shfl_down_sync(0xffffffffu, sf, 2) << 16;
          if (t < rows) {
            *reinterpret_cast<uint2*>(epi.act_codes + (row0 + t) * (epi.inter >> 1) + n_blk * 64 + b * 8) = make_uint2(q.lo, q.hi);
            if ((b & 3) == 0) *reinterpret_cast<uint32_t*>(epi.act_sf + (row0 + t) * epi.sf_pitch + n_blk * 8 + b) = sf;
          }
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");   // the parking space is free again
      } else {
        using Row = typename Epi::Row;
        constexpr int kParkRows = L.park_rows;
        Row* out = reinterpret_cast<Row*>(park) + half * kParkRows * 128;
        auto meet = [&] { asm volatile("bar.sync %0, 128;" ::"r"(2 + half) : "memory"); };      // the piece's four warps
        if (rows == 0) release();
#pragma unroll 1
        for (int t0 = 0; t0 < rows; t0 += kParkRows) {
          const int t1 = min(rows, t0 + kParkRows);
#pragma unroll 1
          for (int c0 = t0; c0 < t1; c0 += 16) {
            uint32_t r[16];
            ptx::tmem_ld_32x16(t_acc + half * kTok + c0, r);
            ptx::tmem_ld_wait();
            if (c0 + 16 >= rows) release();
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float v = __fmul_rn(__uint_as_float(r[i]), now.alpha);
              if constexpr (sizeof(Row) == 4) out[(c0 - t0 + i) * 128 + channel] = v;
              else out[(c0 - t0 + i) * 128 + channel] = to_out<Row>(v);
            }
          }
          meet();
          // rows leave as 16-byte pieces, 128 columns of a row side by side
          constexpr int kPer = 16 / sizeof(Row), kChunks = 128 / kPer;
          const int col0 = n_blk * 256 + half * 128;
          for (int i = tid & 127; i < (t1 - t0) * kChunks; i += 128) {
            const int t = i / kChunks, c = i % kChunks;
            if (col0 + c * kPer < epi.hidden)
              *reinterpret_cast<uint4*>(epi.rows + (row0 + t0 + t) * epi.hidden + col0 + c * kPer) =
                  *reinterpret_cast<const uint4*>(out + t * 128 + c * kPer);
          }
          meet();
        }
      }
      acc.advance(2);
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
    ptx::tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace b200fp4
