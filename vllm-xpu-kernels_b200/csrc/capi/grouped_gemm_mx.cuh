// Block-scaled grouped GEMM: microscaling (MX) operands on tcgen05.mma
// kind::mxf8f6f4.block_scale.  Included by grouped_gemm.cu inside its namespace.
//
//   A  [R, K]      e4m3, rows grouped by expert, with e8m0 scales per 32 of K
//                  (row-major bytes [R, a_sf_pitch]);
//   B  [E, N, K/2] e2m1 pairs (the MXFP4 weight layout of the operator), read by a
//                  tensor map of the "16 x 4 bit, 16-byte aligned" type, which
//                  expands every element to a byte container on the way into shared
//                  memory -- HBM and L2 carry 4 bits per weight, the tensor core
//                  sees the element layout kind::mxf8f6f4 wants;
//   SFB            the weight scales, rearranged once per layer by
//                  mx_prepare_weight_scales_kernel into 512-byte pieces per
//                  (expert, 128 of K, 128 rows of N) in tensor-memory order.
//
// The scales never touch the accumulators: tcgen05.cp moves them from shared memory
// into tensor memory and the MMA applies them, so a tile is one uninterrupted chain
// of MMAs into one accumulator buffer, and the reader warps only run epilogues
// (bias, SwigluOAI, MXFP8 quantisation of the result for the second GEMM).
//
// Roles (one persistent CTA per SM): warp 0 TMA producer (A and B), warp 1 MMA issuer,
// warp 2 scale loader, warps 4.. accumulator readers.  Scales travel in groups of four
// K blocks through a ring of their own: the tile's 128 rows start at an arbitrary row, so
// their scale words are fetched with plain loads, transposed into the tensor-memory
// order in shared memory and published with one proxy fence per group; the weight
// scales of the group are two bulk copies.  (On the operand ring they cost the loader a fence
// and two barrier waits, and the producer a third load, per K block.)  What bounds it: with many
// rows the tensor pipe (384 cycles of MMAs per K block) and the issue loop that feeds it; with
// few, the same loop at the clock that streaming from HBM leaves (128 experts, one row each,
// N = 5760: 272 -> 248 us, 4.55 TB/s).  K need not be a multiple of 128: the last stage is loaded at
// K-128 and only its new 32-wide sub-blocks are issued.

constexpr int kMxBK = 128;            // elements of K per stage (128 bytes per row for both operands)
constexpr int kMxSfaBytes = 512;      // one scale word per row of the A tile
constexpr int kMxAtomBytes = 512;     // scales of 128 rows of B for one stage
constexpr int kMxGroup = 4;           // K blocks per scale group
constexpr int kMxSfGroups = 2;        // scale groups in flight
constexpr int kMxSfaCol = 448;        // tensor-memory columns of the scale words
constexpr int kMxSfbCol = 456;

struct MxParams {
  const uint8_t* a_sf;
  int64_t a_sf_pitch;
  const uint8_t* b_sf;  // prepared layout
  int b_atoms;          // 128-row pieces per expert in b_sf
  const void* bias;
  int bias_dtype;
  void* D;
  int d_dtype;
  int64_t ldd;          // row pitch of D in elements
  uint8_t* d_sf;
  int64_t d_sf_pitch;
  const int32_t* rows_per_expert;
  int64_t R;
  int N, K, E;
  float alpha, limit;
};

template <int BN_, int EPI_, int STAGES_>
struct MxConfig {
  static constexpr int BN = BN_;
  static constexpr int EPI = EPI_;
  static constexpr int STAGES = STAGES_;
  static constexpr int A_BYTES = BM * kStageRowBytes;
  static constexpr int B_BYTES = BN * kStageRowBytes;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int B_ATOMS = (BN + 127) / 128;           // pieces copied per stage
  static constexpr int SF_GROUP_BYTES = kMxGroup * (kMxSfaBytes + B_ATOMS * kMxAtomBytes);
  static constexpr int COL_GROUPS = BN / 64;                 // reader warps per lane quadrant
  static constexpr int EPI_WARPS = 4 * COL_GROUPS;
  static constexpr int THREADS = 128 + EPI_WARPS * 32;
  static constexpr int ACC_STRIDE = 256;                     // tensor-memory columns between the two accumulators
  static constexpr int TMEM_COLS = 512;
  static constexpr size_t SMEM_BYTES =
      1024 + static_cast<size_t>(STAGES) * STAGE_BYTES + kMxSfGroups * SF_GROUP_BYTES;
  static_assert(BN % 64 == 0 && BN <= 192, "two accumulators and the scale words share 512 columns");
  static_assert(STAGE_BYTES % 1024 == 0, "swizzled tiles start on 1 KiB boundaries");
};

struct alignas(8) MxBarriers {
  uint64_t full[8];
  uint64_t empty[8];
  uint64_t tfull[2];
  uint64_t tempty[2];
  uint64_t sffull[kMxSfGroups];
  uint64_t sfempty[kMxSfGroups];
};

// e8m0 byte of the smallest power of two >= max(amax, eps) / 448, floored like
// per_token_group_fp8_quant floors its scale, and that power of two.
__device__ __forceinline__ uint32_t mx_scale_byte(float amax, float* scale) {
  float s = fmaxf(fmaxf(amax, 1e-10f) * (1.0f / 448.0f), 1.0f / (448.0f * 512.0f));
  uint32_t bits = __float_as_uint(s);
  uint32_t e = bits >> 23;
  if (bits & 0x7FFFFFu) ++e;
  *scale = __uint_as_float(e << 23);
  return e;
}

// The reader warps only run epilogues here (the scales are applied inside the MMA), one tile
// behind the tensor pipe, so a row's results leave with plain 16-byte stores from the thread
// that owns the row: no shared-memory staging, which leaves room for a fifth operand stage.
template <typename C>
__device__ __forceinline__ void mx_tile_epilogue(const MxParams& p, const TileCoord& tc, int g,
                                                 bool row_ok, int64_t grow, float (&acc)[64]) {
  const int col0 = tc.n_tile * C::BN + g * 64;  // first accumulator column of this thread
  if (col0 >= p.N) return;
  if (p.bias) add_bias_run<64>(p.bias, p.bias_dtype, static_cast<int64_t>(tc.expert) * p.N + col0, p.N - col0, acc);
  if constexpr (C::EPI == B200MOE_EPI_STORE) {
    if (row_ok) store_row16<64>(p.D, p.d_dtype, grow * p.ldd + col0, acc, p.N - col0);
  } else {  // SWIGLU_OAI: (gate, up) pairs are adjacent columns -> 32 results
    float o[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) o[j] = swiglu_oai_f32(acc[2 * j], acc[2 * j + 1], p.alpha, p.limit);
    const int ocol0 = col0 / 2;
    const int n_valid = (p.N - col0) / 2;
    if (p.d_dtype == B200MOE_E4M3) {
      // the 32 results are one MX group of the second GEMM's A operand
      float amax = 0.f;
#pragma unroll
      for (int j = 0; j < 32; ++j) amax = fmaxf(amax, j < n_valid ? fabsf(o[j]) : 0.f);
      float s;
      const uint32_t sbyte = mx_scale_byte(amax, &s);
      const float inv_s = 1.0f / s;  // exact: s is a power of two
      if (row_ok) {
        p.d_sf[grow * p.d_sf_pitch + (ocol0 >> 5)] = static_cast<uint8_t>(sbyte);
        uint8_t* dst = reinterpret_cast<uint8_t*>(p.D) + grow * p.ldd + ocol0;
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float v0 = fmaxf(-448.0f, fminf(o[4 * i + 0] * inv_s, 448.0f));
          const float v1 = fmaxf(-448.0f, fminf(o[4 * i + 1] * inv_s, 448.0f));
          const float v2 = fmaxf(-448.0f, fminf(o[4 * i + 2] * inv_s, 448.0f));
          const float v3 = fmaxf(-448.0f, fminf(o[4 * i + 3] * inv_s, 448.0f));
          const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v0, v1), __NV_SATFINITE, __NV_E4M3);
          const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v2, v3), __NV_SATFINITE, __NV_E4M3);
          w[i] = lo | (hi << 16);
        }
        if (n_valid >= 32) {
          *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
          *reinterpret_cast<uint4*>(dst + 16) = make_uint4(w[4], w[5], w[6], w[7]);
        } else {
          const uint8_t* b = reinterpret_cast<const uint8_t*>(w);
          for (int j = 0; j < n_valid; ++j) dst[j] = b[j];
        }
      }
    } else if (row_ok) {
      store_row16<32>(p.D, p.d_dtype, grow * p.ldd + ocol0, o, n_valid);
    }
  }
}

template <typename C>
__global__ void __launch_bounds__(C::THREADS, 1)
grouped_gemm_mx_kernel(const __grid_constant__ CUtensorMap map_a,
                       const __grid_constant__ CUtensorMap map_a_small,
                       const __grid_constant__ CUtensorMap map_b,
                       const __grid_constant__ CUtensorMap map_b_tail, MxParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ Schedule sched;
  __shared__ MxBarriers bars;
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
  // per scale group: four K blocks of row scales, then four of each piece of weight scales
  uint8_t* sf_smem = tiles + C::STAGES * C::STAGE_BYTES;
  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const int n_tiles = (p.N + C::BN - 1) / C::BN;
  const int num_kb = (p.K + kMxBK - 1) / kMxBK;
  // K % 128 != 0: the last stage covers [K-128, K) and repeats `tail_skip` 32-wide
  // sub-blocks of the stage before it, which are not issued again.
  const int tail_skip = (p.K % kMxBK) ? (kMxBK - p.K % kMxBK) / 32 : 0;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(&bars.full[s], 1);
      mbar_init(&bars.empty[s], 1);
    }
    for (int g = 0; g < kMxSfGroups; ++g) {
      mbar_init(&bars.sffull[g], 1);
      mbar_init(&bars.sfempty[g], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&bars.tfull[b], 1);
      mbar_init(&bars.tempty[b], C::EPI_WARPS);
    }
    mbar_fence_init();
    prefetch_tensormap(&map_a);
    prefetch_tensormap(&map_a_small);
    prefetch_tensormap(&map_b);
    prefetch_tensormap(&map_b_tail);
  }
  pdl_wait();
  build_schedule(sched, p.rows_per_expert, p.E, p.R, n_tiles, BM);
  if (warp == 1) {
    tmem_alloc(&tmem_base_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  const int num_tiles = total_tiles(sched);
  volatile int* abort_p = &abort_flag;
  const int sched_id = blockIdx.x, sched_stride = gridDim.x;

  if (warp == 0) {
    // ---------------- TMA producer (warp-uniform loop, one elected lane issues) ----------------
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = sched_id; t < num_tiles && ok; t += sched_stride) {
      const TileCoord tc = decode_tile(sched, t);
      const int n0 = tc.n_tile * C::BN;
      const int small = small_boxes(tc.rows_valid);
      // the barrier counts what TMA read: the packed 4-bit source, half of what lands in shared memory
      const uint32_t stage_tx = (small ? small * (kSmallBox * kStageRowBytes) : C::A_BYTES) + C::B_BYTES / 2;
      for (int kb = 0; kb < num_kb && ok; ++kb) {
        ok = mbar_wait_warp(&bars.empty[stage], phase ^ 1u, abort_p);
        if (!ok) break;
        const bool tail = tail_skip && kb == num_kb - 1;
        uint8_t* a_dst = tiles + stage * C::STAGE_BYTES;
        if (elect_one()) {
          mbar_arrive_expect_tx(&bars.full[stage], stage_tx);
          const int ak = tail ? p.K - kMxBK : kb * kMxBK;
          if (!small) tma_load_2d(a_dst, &map_a, &bars.full[stage], ak, tc.row_start);
          else
            for (int i = 0; i < small; ++i)
              tma_load_2d(a_dst + i * (kSmallBox * kStageRowBytes), &map_a_small, &bars.full[stage], ak,
                          tc.row_start + i * kSmallBox);
          if (tail) tma_load_3d(a_dst + C::A_BYTES, &map_b_tail, &bars.full[stage], 0, n0, tc.expert);
          else tma_load_3d(a_dst + C::A_BYTES, &map_b, &bars.full[stage], kb * kMxBK, n0, tc.expert);
        }
        __syncwarp();
        if (++stage == C::STAGES) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    // The 384 cycles of MMAs per K block (the scale copies hide behind them) leave no room for a
    // slow issue loop: a plain loop whose descriptors are base + stage * constant, on values the
    // compiler knows to be warp-uniform.  (Unrolled over the ring, with the tensor-memory base
    // as a per-lane value out of shared memory, issuing alone took 520 of 620 cycles.)
    // Whole blocks of straight-line issues, chosen by a uniform branch, are kept: a
    // per-instruction guard between MMAs once issued wrong sub-blocks.
    const uint32_t a0 = smem_u32(tiles);
    const uint32_t sw_hi = (1024u >> 4) | (1u << 14) | (2u << 29);  // SBO 1024, version, 128-byte swizzle
    const uint32_t sf_hi = (128u >> 4) | (1u << 14);                // SBO 128, version, no swizzle
    const uint32_t a_lo0 = ((a0 & 0x3FFFFu) >> 4) | ((16u >> 4) << 16);
    const uint32_t sf_lo0 = (smem_u32(sf_smem) & 0x3FFFFu) >> 4;
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
    const uint32_t sfa_t = tmem + kMxSfaCol;
    auto desc = [](uint32_t lo, uint32_t hi) { return (static_cast<uint64_t>(hi) << 32) | lo; };
    uint32_t stage = 0, phase = 0;
    uint32_t buf = 0, buf_phase = 0;
    uint32_t sg = 0, sg_phase = 0;   // scale group in use
    bool ok = true;
    for (int t = sched_id; t < num_tiles && ok; t += sched_stride) {
      // a tile that starts inside a 128-row piece of the scales (192-column tiles: every odd one
      // starts at row 64) reads its scale columns from that offset on
      const int n_tile = __shfl_sync(0xffffffffu, decode_tile(sched, t).n_tile, 0);
      const uint32_t sfb_t = tmem + kMxSfbCol + ((n_tile * C::BN) % 128) / 32;
      ok = mbar_wait_warp(&bars.tempty[buf], buf_phase ^ 1u, abort_p);
      if (!ok) break;
      const uint32_t d_tmem = tmem + buf * C::ACC_STRIDE;
      uint32_t accum = 0;
      for (int kb = 0; kb < num_kb && ok; ++kb) {
        const uint32_t j = static_cast<uint32_t>(kb) % kMxGroup;
        const bool last = kb == num_kb - 1;
        if (j == 0) {
          ok = mbar_wait_warp(&bars.sffull[sg], sg_phase, abort_p);
          if (!ok) break;
        }
        ok = mbar_wait_warp(&bars.full[stage], phase, abort_p);
        if (!ok) break;
        tc_fence_after();
        const uint32_t sf_lo = sf_lo0 + (sg * C::SF_GROUP_BYTES + j * kMxSfaBytes) / 16;
        const uint32_t a_lo = a_lo0 + stage * (C::STAGE_BYTES >> 4);
        const uint32_t b_lo = a_lo + (C::A_BYTES >> 4);
        if (elect_one()) {
          tmem_cp_32x128b_x4(sfa_t, desc(sf_lo, sf_hi));
#pragma unroll
          for (int a = 0; a < C::B_ATOMS; ++a)
            tmem_cp_32x128b_x4(tmem + kMxSfbCol + 4 * a, desc(sf_lo + (1 + a) * (kMxGroup * kMxAtomBytes / 16), sf_hi));
          if (tail_skip && last) {
            // K % 128 == 64 (rows of packed 4-bit weights have a 32-byte pitch, so K is a
            // multiple of 64): the stage was loaded at K-128 and its first two sub-blocks were
            // issued with the stage before
            mma_mxf8f6f4(d_tmem, desc(a_lo + 4, sw_hi), desc(b_lo + 4, sw_hi),
                         make_idesc_mx(0u, 5u, 0u, BM, C::BN, 2, 2), sfa_t, sfb_t, accum);
            mma_mxf8f6f4(d_tmem, desc(a_lo + 6, sw_hi), desc(b_lo + 6, sw_hi),
                         make_idesc_mx(0u, 5u, 0u, BM, C::BN, 3, 3), sfa_t, sfb_t, 1u);
          } else {
            mma_mxf8f6f4(d_tmem, desc(a_lo, sw_hi), desc(b_lo, sw_hi),
                         make_idesc_mx(0u, 5u, 0u, BM, C::BN, 0, 0), sfa_t, sfb_t, accum);
#pragma unroll
            for (int kk = 1; kk < 4; ++kk)
              mma_mxf8f6f4(d_tmem, desc(a_lo + kk * 2, sw_hi), desc(b_lo + kk * 2, sw_hi),
                           make_idesc_mx(0u, 5u, 0u, BM, C::BN, kk, kk), sfa_t, sfb_t, 1u);
          }
          mma_commit(&bars.empty[stage]);
          if (last) mma_commit(&bars.tfull[buf]);
          if (last || j == kMxGroup - 1) mma_commit(&bars.sfempty[sg]);   // the group has been copied
        }
        __syncwarp();
        accum = 1;
        if (last || j == kMxGroup - 1) {
          if (++sg == kMxSfGroups) { sg = 0; sg_phase ^= 1u; }
        }
        if (++stage == C::STAGES) { stage = 0; phase ^= 1u; }
      }
      if (++buf == 2) { buf = 0; buf_phase ^= 1u; }
    }
  } else if (warp == 2) {
    // ---------------- scale loader ----------------
    // Lane l owns rows l, 32+l, 64+l, 96+l of the tile.  One 16-byte load per row brings
    // the scale words of a group; they are fetched one group ahead.
    uint32_t sg = 0, sg_phase = 1;
    bool ok = true;
    const int groups = (num_kb + kMxGroup - 1) / kMxGroup;
    auto load_group = [&](const TileCoord& tc, int grp, uint4 (&w)[4]) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        int64_t row = static_cast<int64_t>(tc.row_start) + c * 32 + lane;
        if (row >= p.R) row = p.R - 1;  // rows past the end are never stored
        w[c] = *reinterpret_cast<const uint4*>(p.a_sf + row * p.a_sf_pitch + grp * 16);
      }
    };
    auto word = [](const uint4& v, int j) { return j == 0 ? v.x : (j == 1 ? v.y : (j == 2 ? v.z : v.w)); };
    uint4 cur[4], nxt[4];
    uint32_t prev_last[4] = {0u, 0u, 0u, 0u};
    int t = sched_id;
    TileCoord tc{}, tc_next{};
    if (t < num_tiles) {
      tc_next = decode_tile(sched, t);
      load_group(tc_next, 0, nxt);
    }
    for (; t < num_tiles && ok; t += sched_stride) {
      tc = tc_next;
      if (t + sched_stride < num_tiles) tc_next = decode_tile(sched, t + sched_stride);
      const uint8_t* sfb = p.b_sf + (static_cast<int64_t>(tc.expert) * p.b_atoms + tc.n_tile * C::BN / 128) *
                                        num_kb * kMxAtomBytes;
      for (int grp = 0; grp < groups && ok; ++grp) {
#pragma unroll
        for (int c = 0; c < 4; ++c) cur[c] = nxt[c];
        if (grp + 1 < groups) load_group(tc, grp + 1, nxt);
        else if (t + sched_stride < num_tiles) load_group(tc_next, 0, nxt);
        ok = mbar_wait_warp(&bars.sfempty[sg], sg_phase, abort_p);
        if (!ok) break;
        uint8_t* dst = sf_smem + sg * C::SF_GROUP_BYTES;
        const int n = num_kb - grp * kMxGroup < kMxGroup ? num_kb - grp * kMxGroup : kMxGroup;
#pragma unroll
        for (int j = 0; j < kMxGroup; ++j) {
          uint4 o;
          uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t v = word(cur[c], j);
            if (tail_skip && grp * kMxGroup + j == num_kb - 1) {
              // bytes of sub-blocks [K/32 - 4, K/32): the last (4 - tail_skip) bytes of the
              // previous word followed by the first tail_skip... of this one
              const uint32_t before = j > 0 ? word(cur[c], j - 1) : prev_last[c];
              v = __funnelshift_r(before, v, 8 * (4 - tail_skip));
            }
            ow[c] = v;
          }
          if (j < n) *reinterpret_cast<uint4*>(dst + j * kMxSfaBytes + lane * 16) = o;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) prev_last[c] = cur[c].w;
        fence_proxy_async_smem();
        __syncwarp();
        if (elect_one()) {
          mbar_arrive_expect_tx(&bars.sffull[sg], C::B_ATOMS * n * kMxAtomBytes);
#pragma unroll
          for (int a = 0; a < C::B_ATOMS; ++a)
            bulk_load(dst + (1 + a) * (kMxGroup * kMxAtomBytes),
                      sfb + (static_cast<int64_t>(a) * num_kb + grp * kMxGroup) * kMxAtomBytes, n * kMxAtomBytes,
                      &bars.sffull[sg]);
        }
        __syncwarp();
        if (++sg == kMxSfGroups) { sg = 0; sg_phase ^= 1u; }
      }
    }
  } else if (warp >= 4) {
    // ---------------- accumulator readers / epilogue ----------------
    const int quad = warp & 3;
    const int g = (warp - 4) >> 2;
    const int row_in_tile = quad * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    int buf = 0;
    uint32_t buf_phase = 0;
    bool ok = true;
    for (int t = sched_id; t < num_tiles && ok; t += sched_stride) {
      const TileCoord tc = decode_tile(sched, t);
      const bool row_ok = row_in_tile < tc.rows_valid;
      const int64_t grow = static_cast<int64_t>(tc.row_start) + row_in_tile;
      float acc[64];
      ok = mbar_wait(&bars.tfull[buf], buf_phase, abort_p);
      if (!ok) break;
      tc_fence_after();
      const uint32_t src = tmem_base + lane_addr + buf * C::ACC_STRIDE + g * 64;
      tmem_ld_32x32(src, *reinterpret_cast<float(*)[32]>(acc));
      tmem_ld_32x32(src + 32, *reinterpret_cast<float(*)[32]>(acc + 32));
      tmem_ld_wait_on2(*reinterpret_cast<float(*)[32]>(acc), *reinterpret_cast<float(*)[32]>(acc + 32));
      // the accumulator is in registers: the MMA warp may start the tile after next
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.tempty[buf]);
      if (++buf == 2) { buf = 0; buf_phase ^= 1u; }
      mx_tile_epilogue<C>(p, tc, g, row_ok, grow, acc);
    }
  }

  pdl_trigger();
  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (abort_flag) {
    if (threadIdx.x == 0) atomicExch(&g_device_status, B200MOE_TIMEOUT);
    for (int i = 0; i < 64; ++i) __nanosleep(10000);  // copies in flight land before smem is released
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
}

// Tensor map over packed e2m1 pairs, [batch, rows, cols] with `cols` 4-bit elements per
// row (a multiple of 128), box 128 x box_rows; elements arrive in shared memory one per
// byte container (16 elements = 8 bytes of data + 8 bytes of padding), 128-byte swizzle.
inline int make_map_fp4(CUtensorMap* map, const void* base, uint64_t cols, uint64_t row_pitch_bytes,
                        uint64_t rows, uint64_t batch, uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return B200MOE_CUDA_ERROR;
  cuuint64_t dims[3] = {cols, rows, batch};
  cuuint64_t strides[2] = {row_pitch_bytes, row_pitch_bytes * rows};
  cuuint32_t box[3] = {128, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, 3, const_cast<void*>(base), dims,
                  strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_last_error("cuTensorMapEncodeTiled (packed 4-bit)", cudaErrorInvalidValue);
    return B200MOE_CUDA_ERROR;
  }
  return B200MOE_OK;
}

template <typename C>
int launch_mx(const b200moe_mx_gemm_args& a, cudaStream_t st) {
  CUtensorMap map_a, map_a_small, map_b, map_b_tail;
  int rc = make_map(&map_a, B200MOE_E4M3, a.A, a.K, a.R, 0, kMxBK, BM);
  if (rc == B200MOE_OK) rc = make_map(&map_a_small, B200MOE_E4M3, a.A, a.K, a.R, 0, kMxBK, kSmallBox);
  if (rc != B200MOE_OK) return rc;
  const uint64_t pitch = static_cast<uint64_t>(a.K) / 2;
  const uint64_t k_main = static_cast<uint64_t>(a.K / kMxBK) * kMxBK;
  rc = make_map_fp4(&map_b, a.B, k_main, pitch, a.N, a.E, C::BN);
  if (rc != B200MOE_OK) return rc;
  // the last 128 elements of every row, for a K that is not a multiple of 128
  rc = make_map_fp4(&map_b_tail, reinterpret_cast<const uint8_t*>(a.B) + (a.K - kMxBK) / 2, kMxBK,
                    pitch, a.N, a.E, C::BN);
  if (rc != B200MOE_OK) return rc;

  MxParams p;
  p.a_sf = a.a_sf;
  p.a_sf_pitch = a.a_sf_pitch;
  p.b_sf = a.b_sf;
  p.b_atoms = (a.N + 127) / 128 + 1;
  p.bias = a.bias;
  p.bias_dtype = a.bias_dtype;
  p.D = a.D;
  p.d_dtype = a.d_dtype;
  p.ldd = a.epilogue == B200MOE_EPI_STORE ? a.N : a.N / 2;
  p.d_sf = a.d_sf;
  p.d_sf_pitch = a.d_sf_pitch;
  p.rows_per_expert = a.rows_per_expert;
  p.R = a.R;
  p.N = a.N;
  p.K = a.K;
  p.E = a.E;
  p.alpha = a.alpha;
  p.limit = a.limit;
  rc = ensure_dynamic_smem<C>(grouped_gemm_mx_kernel<C>, C::SMEM_BYTES, "cudaFuncSetAttribute (mx)");
  if (rc != B200MOE_OK) return rc;
  const int n_tiles = (a.N + C::BN - 1) / C::BN;
  int64_t grid = ((a.R + BM - 1) / BM + a.E) * n_tiles;
  if (grid > kNumSMs) grid = kNumSMs;
  if (grid < 1) grid = 1;
  return launch_pdl("grouped_gemm_mx_kernel", grouped_gemm_mx_kernel<C>, dim3(static_cast<unsigned>(grid)),
                    dim3(C::THREADS), C::SMEM_BYTES, st, 1, a.R, map_a, map_a_small,
                    map_b, map_b_tail, p);
}

// Weight scales [E, N, K/32] (e8m0 bytes) -> [E, ceil(N/128)+1, ceil(K/128), 512]: per
// (expert, 128 rows, K block) the 512 bytes tcgen05.cp wants, byte (n%32)*16 + (n%128/32)*4 + j
// holding the scale of row n and sub-block j of that K block.  A last K block that starts at
// K-128 gets the sub-blocks it really covers.  Rows past N and the extra piece hold 1.0.
__global__ void mx_prepare_weight_scales_kernel(const uint8_t* __restrict__ s, uint8_t* __restrict__ out,
                                                int E, int N, int K, int64_t total_words) {
  const int num_kb = (K + kMxBK - 1) / kMxBK;
  const int atoms = (N + 127) / 128 + 1;
  const int sub_total = K / 32;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total_words;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int in_atom = static_cast<int>(i % 128);  // word index: lane * 4 + column
    int64_t rest = i / 128;
    const int kb = static_cast<int>(rest % num_kb);
    rest /= num_kb;
    const int atom = static_cast<int>(rest % atoms);
    const int e = static_cast<int>(rest / atoms);
    const int n = atom * 128 + (in_atom & 3) * 32 + (in_atom >> 2);
    const int sub0 = (kb == num_kb - 1 && (K % kMxBK)) ? sub_total - 4 : kb * 4;
    uint32_t w = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t b = 127;
      if (n < N && sub0 + j < sub_total)
        b = s[(static_cast<int64_t>(e) * N + n) * sub_total + sub0 + j];
      w |= b << (8 * j);
    }
    reinterpret_cast<uint32_t*>(out)[i] = w;
  }
}
