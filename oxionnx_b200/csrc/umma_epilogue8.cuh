// Epilogues of the persistent integer kernel for whole groups of 64 output channels with a fragment of the accumulator per
// thread instead of a row of it: requantisation, alone or joined with a quantised residual (epilogue_bytes), and the
// dequantisation of a dynamically quantised linear (epilogue_floats).
//
// The general epilogue (epilogue_role) reads one output pixel per thread and 32 channels a run, so every thread loads all
// 32 channels' parameters (sixteen 16-byte loads a run, 8 KB of register writes a warp) and its code is one straight body
// of 32 outputs.  Both bound it where K is short: on 1x1 64 -> 256 at M = 3211264 a run of 32 x 32 outputs took 315
// instructions of which 121 were the requantisation, on 1x1 128 -> 512 with a join 626 whose first stall was instruction
// fetch.  Here a warp takes 64 channels of 32 pixels in two halves of sixteen pixels (tcgen05.ld.16x256b: of every eight
// columns a thread gets two, for two rows).  The weights' rows are brought into shared memory in an order that makes a
// thread's sixteen columns sixteen consecutive channels (a five-dimensional tensor map, see b_perm): a thread's parameters
// are read once for two rows, its output is one 16-byte piece per row that goes straight to memory (four threads fill a
// 64-byte run of a row), and the body in the loop is 32 outputs with nothing but their arithmetic.
//
// Measured, general epilogue -> this one: 1x1 64 -> 256 at M = 3211264 340 -> 224 us (4.6 TB/s), 1x1 128 -> 512 at
// M = 802816 175 -> 130 us, the same with a join 355 -> 249 us (3.7 TB/s), 1x1 256 -> 1024 at M = 200704 with a join
// 194 -> 145 us; 1x1 256 -> 64 and 3x3 64 -> 64 the same within 2 %.  Stores by TMA from staged rows, and the residual by
// TMA, were 1x1 64 -> 256 234 us and the join of 128 -> 512 316 us; parameters held in registers spilled (311 us).
#pragma once

#include "umma_kernel.cuh"

namespace oxb {
namespace k {
namespace umma {

// Sixteen TMEM lanes x 64 columns: r[4 g + 2 s + e] is row lane / 4 + 8 s, column 8 g + 2 (lane % 4) + e.
__device__ __forceinline__ void tmem_ld_frag64(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
        "=r"(r[31])
      : "r"(taddr));
}

// Sixteen TMEM lanes x 16 N columns in the same fragments: r[4 g + 2 s + e], g < 2 N.
template <int N>
__device__ __forceinline__ void tmem_ld_frag16(uint32_t taddr, uint32_t (&r)[8 * N]) {
  static_assert(N == 1 || N == 2, "8 or 16 registers");
  if constexpr (N == 1)
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
  else
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
                   "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}
// The wait for it, naming the registers it lands in (see tmem_ld_wait_for).
template <int N>
__device__ __forceinline__ void tmem_ld_frag16_wait(uint32_t (&r)[8 * N]) {
  if constexpr (N == 1)
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]) :);
  else
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :);
}
__device__ __forceinline__ void lds_v4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ float fma_sat(float x, float y, float z) {
  float r;
  asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(x), "f"(y), "f"(z));
  return r;
}

// Forms: requantisation with any bounds or with a lower bound of 0, the join with any bounds or with a lower bound of 0.
constexpr uint32_t B8_RES_BYTES = 32 * 64;  // a warp's part of the residual of one tile
constexpr uint32_t FRAG_PARAM_BYTES = 768;  // ... and its channels' parameters: two or three vectors of 64
enum { B8_REQUANT = 0, B8_REQUANT_RELU = 1, B8_JOIN = 2, B8_JOIN_RELU = 3 };

// Four channels of one row.  Requantisation: math_requant_packed's operations.  Join: the requantised lane is clamped to the
// full range of its type by a saturating fma that also scales it to [0, 1] (join_d is 1 / 255 rounded up to 21 bits, so that
// its product with 1.5 * 2^23 is exact and 255 goes to 1), two minima and maxima on the slower pipe less; then math_join's
// operations with constants for that scale, which the host has checked for every pair of inputs (residual_join_constants).
template <int FORM>
__device__ __forceinline__ uint32_t bytes_word(const KParams& p, uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3, const uint32_t (&b)[4], const uint32_t (&c)[4],
                                               float magic_zp, uint32_t lo2, uint32_t hi2, uint32_t rw) {
  float a0 = __int2float_rn((int32_t)v0), a1 = __int2float_rn((int32_t)v1), a2 = __int2float_rn((int32_t)v2), a3 = __int2float_rn((int32_t)v3);
  add2(a0, a1, __uint_as_float(b[0]), __uint_as_float(b[1]));
  add2(a2, a3, __uint_as_float(b[2]), __uint_as_float(b[3]));
  fma2(a0, a1, __uint_as_float(c[0]), __uint_as_float(c[1]), magic_zp);
  fma2(a2, a3, __uint_as_float(c[2]), __uint_as_float(c[3]), magic_zp);
  if constexpr (FORM >= B8_JOIN) {
    const float magic = 12582912.0f, d = p.join_d, dm = -12582912.0f * d;
    const float b_off = p.join_flip ? -8388736.0f : -8388608.0f;
    a0 = fma_sat(a0, d, dm), a1 = fma_sat(a1, d, dm), a2 = fma_sat(a2, d, dm), a3 = fma_sat(a3, d, dm);
    const uint32_t r = rw ^ (p.join_flip ? 0x80808080u : 0u);
    float b0 = __uint_as_float(__byte_perm(r, 0x4B000000u, 0x7440)), b1 = __uint_as_float(__byte_perm(r, 0x4B000000u, 0x7441));
    float b2 = __uint_as_float(__byte_perm(r, 0x4B000000u, 0x7442)), b3 = __uint_as_float(__byte_perm(r, 0x4B000000u, 0x7443));
    add2(b0, b1, b_off, b_off);
    add2(b2, b3, b_off, b_off);
    fma2(b0, b1, p.join_b8, p.join_b8, p.join_c8);
    fma2(b2, b3, p.join_b8, p.join_b8, p.join_c8);
    fma2v(a0, a1, p.join_a8, b0, b1);
    fma2v(a2, a3, p.join_a8, b2, b3);
    add2(a0, a1, magic, magic);
    add2(a2, a3, magic, magic);
  }
  uint32_t p01 = __byte_perm(__float_as_uint(a0), __float_as_uint(a1), 0x5410), p23 = __byte_perm(__float_as_uint(a2), __float_as_uint(a3), 0x5410);
  if constexpr (FORM == B8_REQUANT_RELU || FORM == B8_JOIN_RELU) {
    p01 = __vimin_s16x2_relu(p01, hi2);
    p23 = __vimin_s16x2_relu(p23, hi2);
  } else {
    p01 = __vmins2(__vmaxs2(p01, lo2), hi2);
    p23 = __vmins2(__vmaxs2(p23, lo2), hi2);
  }
  return __byte_perm(p01, p23, 0x6420);
}

template <int BN, bool PAIR, int FORM>
__device__ __forceinline__ void epilogue_bytes(const KParams& p, int warp, int lane, uint32_t tmem_base, uint64_t* bar_acc_full, uint64_t* bar_acc_empty,
                                               uint32_t res_addr, volatile int* abortp, int total_tiles, int tile0, int tile_step, int pair_rank) {
  using ES = EpiShape<BN, epi_warps(KIND_I8)>;
  static_assert(ES::CPW == 2, "a warp takes 64 channels of a tile");
  constexpr bool JOIN = FORM >= B8_JOIN;
  constexpr int M_STEP = PAIR ? 2 * BLOCK_M : BLOCK_M;
  const int quarter = warp & 3, slot = (warp - 2) >> 2, group = slot / ES::WPQ, col0 = (slot % ES::WPQ) * 64;
  const int row = (PAIR ? pair_rank * BLOCK_M : 0) + quarter * 32 + (lane >> 2);  // of the tile; this thread's others are 8, 16 and 24 further on
  const int chan = col0 + 16 * (lane & 3);                                        // the first of this thread's sixteen channels of the tile
  const uint32_t row8 = (uint32_t)p.OC * 8u;
  const float magic_zp = 12582912.0f + (float)(JOIN ? p.y_zp - p.lo : p.y_zp);
  const int lo = JOIN ? p.join_lo : p.lo, hi = JOIN ? p.join_hi : p.hi;
  const uint32_t lo2 = ((uint32_t)lo & 0xffffu) * 0x00010001u, hi2 = ((uint32_t)hi & 0xffffu) * 0x00010001u;
  // This warp's 64 biases and 64 scales in shared memory, [k][q][4] for thread q's channels 4 k .. 4 k + 3: the eight loads
  // of a half tile are broadcasts, and 32 registers less stay alive than with the thread's own channels held in them
  // (which spilled).
  const uint32_t params = res_addr + (JOIN ? (uint32_t)p.res_bufs * B8_RES_BYTES : 0u);
  int have_oc = -1;
  // tile number i of this warp is tile number group + i * NG of the CTA
  const int step = tile_step * ES::NG;
  int t = tile0 + group * tile_step;
  TileWalk walk(t, step, p.n_tiles);
  // The residual's pieces are copied ahead into shared memory, each by the thread that will use it: res_bufs tiles of
  // this warp, [tile][row 0, 8, 16, 24][lane], so that its own wait is all it needs.
  const int nb = JOIN ? p.res_bufs : 1;
  TileWalk ahead = walk;
  int ahead_t = t;
  res_addr += (uint32_t)lane * 16u;
  auto fetch = [&](uint32_t dst) {
    if (ahead_t < total_tiles && ahead.n * BN + col0 < p.OC) {
      const int m = ahead.m * M_STEP + row;
      const uint8_t* src = (const uint8_t*)p.residual + ((size_t)m * p.OC + ahead.n * BN + chan);
#pragma unroll
      for (int j = 0; j < 4; ++j, src += row8)
        if (m + 8 * j < p.M) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 512u * j), "l"(src) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    ahead_t += step;
    ahead.next();
  };
  uint32_t res_at = res_addr;
  if (JOIN)
    for (int i = 0; i < nb; ++i) fetch(res_addr + (uint32_t)i * B8_RES_BYTES);
  uint32_t turn = 0;  // counts this warp's tiles: accumulator group + NG * (turn & 1), phase turn / 2
  for (; t < total_tiles; t += step, ++turn, walk.next()) {
    const uint32_t buf = (uint32_t)group + (uint32_t)ES::NG * (turn & 1u);
    const int oc = walk.n * BN;
    const bool mine = oc + col0 < p.OC;  // not in a ragged last channel tile
    if (mine && oc != have_oc) {
      have_oc = oc;
      __syncwarp();  // every thread has read the ones before
      const float4 f = __ldg(reinterpret_cast<const float4*>((lane < 16 ? p.bias_if : p.combined) + oc + col0) + (lane & 15));
      asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(params + (uint32_t)((lane >> 4) * 256 + (lane & 3) * 64 + ((lane >> 2) & 3) * 16)), "f"(f.x), "f"(f.y), "f"(f.z), "f"(f.w) : "memory");
      __syncwarp();
    }
    bool ok = mbar_wait(smem_u32(&bar_acc_full[buf]), (turn >> 1) & 1u, abortp);
    if (!ok && !*abortp) {
      *abortp = 1;
      atomicExch(p.err_flag, 3);
    }
    if (!__all_sync(0xffffffffu, ok)) break;
    tc_fence_after();
    if (JOIN) {  // all but the newest nb - 1 copies have landed
      if (nb == 2) asm volatile("cp.async.wait_group 1;" ::: "memory");
      else if (nb == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
      else asm volatile("cp.async.wait_group 3;" ::: "memory");
    }
    const int m = walk.m * M_STEP + row;
    uint8_t* dst = (uint8_t*)p.out + ((size_t)m * p.OC + oc + chan);
    int rows = mine ? p.M - m : 0;  // rows 0, 8, .. of this thread below this bound are written
    uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * (uint32_t)BN + (uint32_t)col0;
    uint32_t res = res_at;
#pragma unroll 1
    for (int h = mine ? 0 : 1; h < 2; ++h, taddr += 16u << 16, res += 1024u) {
      uint32_t v[32];
      tmem_ld_frag64(taddr, v);
      tmem_ld_wait_for(v);
      if (h == 1) {  // every TMEM read of this warp for this tile has landed
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (PAIR) mbar_arrive_cluster(mapa(smem_u32(&bar_acc_empty[buf]), 0));
          else mbar_arrive(smem_u32(&bar_acc_empty[buf]));
        }
      }
      uint32_t rv[2][4] = {}, w[2][4];
      if (JOIN) {
#pragma unroll
        for (int s = 0; s < 2; ++s) lds_v4(res + 512u * s, rv[s]);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t b[4], c[4];
        lds_v4(params + (uint32_t)((lane & 3) * 16 + k * 64), b);
        lds_v4(params + (uint32_t)((lane & 3) * 16 + k * 64 + 256), c);
#pragma unroll
        for (int s = 0; s < 2; ++s)
          w[s][k] = bytes_word<FORM>(p, v[8 * k + 2 * s], v[8 * k + 2 * s + 1], v[8 * k + 4 + 2 * s], v[8 * k + 5 + 2 * s], b, c, magic_zp, lo2, hi2, rv[s][k]);
      }
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (rows > 0) *reinterpret_cast<uint4*>(dst) = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
        rows -= 8;
        dst += row8;
      }
    }
    if (JOIN) {
      // this thread has read its pieces: their place is the next tile's to be fetched
      fetch(res_at);
      res_at = res_at == res_addr + (uint32_t)(nb - 1) * B8_RES_BYTES ? res_addr : res_at + B8_RES_BYTES;
    }
  }
  if (JOIN) asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The dequantising epilogue of a dynamically quantised linear (math_dequant's operations, lane for lane) over the same
// fragments, with the weights' rows reordered in groups of sixteen channels: a thread's four columns of a group are four
// consecutive channels, one 16-byte piece of f32 lanes per row.  The zero point's share of the bias and the product of the
// two scales are formed once per channel tile instead of once per output.  GELU: the exact Gelu follows; its body is kept to
// eight outputs so that the loop stays in the instruction cache (sixteen: 1 % slower over an encoder).
// Measured, general epilogue -> this one: M = 8192, N = 768, K = 768 22.6 -> 16.5 us, with extrema 24.9 -> 18.5 us, K = 3072
// 43.2 -> 31.0 us; N = 3072, K = 768 with Gelu 70.1 -> 59.8 us; an encoder of 64x128 tokens 3480 -> 2949 us.
template <int BN, bool PAIR, bool DYN, bool GELU, bool TRANSPOSED>
__device__ __forceinline__ void epilogue_floats(const KParams& p, int warp, int lane, uint32_t tmem_base, uint64_t* bar_acc_full, uint64_t* bar_acc_empty,
                                                uint32_t params, volatile int* abortp, int total_tiles, int tile0, int tile_step, int pair_rank) {
  using ES = EpiShape<BN, epi_warps(KIND_I8)>;
  static_assert(ES::CPW == 2, "a warp takes 64 channels of a tile");
  constexpr int M_STEP = PAIR ? 2 * BLOCK_M : BLOCK_M;
  constexpr int GROUPS = GELU ? 1 : 2;  // groups of sixteen channels of a body
  const int quarter = warp & 3, slot = (warp - 2) >> 2, group = slot / ES::WPQ, col0 = (slot % ES::WPQ) * 64;
  const int row = (PAIR ? pair_rank * BLOCK_M : 0) + quarter * 32 + (lane >> 2);
  const int xz = DYN ? __float2int_rn(*p.x_zp_dev) : 0;
  const float xs = *p.dq_x_scale;
  const uint64_t neg_zero = p.neg_zero2;
  const bool track = p.minmax_keys != nullptr, round = p.round_tf32 != 0;
  float seen_min = INFINITY, seen_max = -INFINITY;
  int have_oc = -1;
  const int step = tile_step * ES::NG;
  int t = tile0 + group * tile_step;
  TileWalk walk(t, step, p.n_tiles);
  uint32_t turn = 0;
  for (; t < total_tiles; t += step, ++turn, walk.next()) {
    const uint32_t buf = (uint32_t)group + (uint32_t)ES::NG * (turn & 1u);
    const int oc = walk.n * BN + col0;
    const bool mine = oc < p.OC;  // not in a ragged last channel tile
    if (mine && oc != have_oc) {
      have_oc = oc;
      __syncwarp();  // every thread has read the ones before
      const int2 bi = __ldg(reinterpret_cast<const int2*>(p.bias_i + oc) + lane);
      const int2 ws = DYN ? __ldg(reinterpret_cast<const int2*>(p.wsum + oc) + lane) : make_int2(0, 0);
      const float2 sc = __ldg(reinterpret_cast<const float2*>(p.dq_w_scale + oc) + lane), bf = __ldg(reinterpret_cast<const float2*>(p.dq_bias + oc) + lane);
      const uint32_t at = params + (uint32_t)lane * 8u;
      asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(bi.x - xz * ws.x), "r"(bi.y - xz * ws.y) : "memory");
      asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(at + 256u), "f"(__fmul_rn(xs, sc.x)), "f"(__fmul_rn(xs, sc.y)) : "memory");
      asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(at + 512u), "f"(bf.x), "f"(bf.y) : "memory");
      __syncwarp();
    }
    bool ok = mbar_wait(smem_u32(&bar_acc_full[buf]), (turn >> 1) & 1u, abortp);
    if (!ok && !*abortp) {
      *abortp = 1;
      atomicExch(p.err_flag, 3);
    }
    if (!__all_sync(0xffffffffu, ok)) break;
    tc_fence_after();
    const int m = walk.m * M_STEP + row;
    float* const out = (float*)p.out + ((size_t)m * p.OC + oc + 4 * (lane & 3));
    float* out_t = nullptr;  // transposed: a warp's 32 rows are in one sequence, eight rows of a channel are 32 contiguous bytes
    if (TRANSPOSED) out_t = (float*)p.out + (((size_t)(m / p.out_seq) * p.OC + oc + 4 * (lane & 3)) * p.out_seq + m % p.out_seq);
    const int rows = mine ? p.M - m : 0;  // of this thread's rows 0, 8, 16 and 24 those below this bound are written
    const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * (uint32_t)BN + (uint32_t)col0;
    constexpr int STEPS = 4 / GROUPS;  // bodies of a half
#pragma unroll 1
    for (int i = mine ? 0 : 2 * STEPS - 1; i < 2 * STEPS; ++i) {
      const int h = i / STEPS, g0 = (i % STEPS) * GROUPS;
      uint32_t v[8 * GROUPS];
      tmem_ld_frag16<GROUPS>(taddr + ((uint32_t)(16 * h) << 16) + (uint32_t)(16 * g0), v);
      tmem_ld_frag16_wait<GROUPS>(v);
      if (i == 2 * STEPS - 1) {  // every TMEM read of this warp for this tile has landed
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (PAIR) mbar_arrive_cluster(mapa(smem_u32(&bar_acc_empty[buf]), 0));
          else mbar_arrive(smem_u32(&bar_acc_empty[buf]));
        }
      }
#pragma unroll
      for (int g = 0; g < GROUPS; ++g) {
        uint32_t bb[4], cc[4], ff[4];
        const uint32_t at = params + (uint32_t)((g0 + g) * 64 + (lane & 3) * 16);
        lds_v4(at, bb);
        lds_v4(at + 256u, cc);
        lds_v4(at + 512u, ff);
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          float y[4];
#pragma unroll
          for (int e = 0; e < 2; ++e) {  // channels 2 e and 2 e + 1 of the four
            const uint32_t* a = v + 8 * g + 4 * e + 2 * s;
            const uint64_t acc = pack2(__int2float_rn((int32_t)(a[0] + bb[2 * e])), __int2float_rn((int32_t)(a[1] + bb[2 * e + 1])));
            const uint64_t c2 = pack2(__uint_as_float(cc[2 * e]), __uint_as_float(cc[2 * e + 1])), f2 = pack2(__uint_as_float(ff[2 * e]), __uint_as_float(ff[2 * e + 1]));
            uint64_t y2 = addp(fmap(acc, c2, neg_zero), f2);
            if (GELU) y2 = gelu_erf2(y2, neg_zero);
            unpack2(y2, y[2 * e], y[2 * e + 1]);
          }
          if (round) {  // the lanes feed a TF32 product
#pragma unroll
            for (int j = 0; j < 4; ++j) y[j] = round_tf32(y[j]);
          }
          const int r = 16 * h + 8 * s;
          if (r < rows) {
            if (TRANSPOSED) {
#pragma unroll
              for (int j = 0; j < 4; ++j) out_t[(size_t)(16 * (g0 + g) + j) * p.out_seq + r] = y[j];
            } else {
              *reinterpret_cast<float4*>(out + (size_t)r * p.OC + 16 * (g0 + g)) = make_float4(y[0], y[1], y[2], y[3]);
            }
            if (track) {
              seen_min = fminf(seen_min, fminf(fminf(y[0], y[1]), fminf(y[2], y[3])));
              seen_max = fmaxf(seen_max, fmaxf(fmaxf(y[0], y[1]), fmaxf(y[2], y[3])));
            }
          }
        }
      }
    }
  }
  if (track) merge_extrema(p, lane, seen_min, seen_max);
}

}  // namespace umma
}  // namespace k
}  // namespace oxb
