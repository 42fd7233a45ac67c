// tcgen05 contraction for problems that leave most of the chip idle: one output tile per CTA, the K range of a tile
// split over the CTAs of a cluster.
//
// The persistent kernel (umma_kernel.cuh) is built for throughput; at a batch of one a layer of a residual network
// is 16 to 100 of its tiles, and its time is latency: measured on 196 x 256 x 1024 (i8) from the release of the
// predecessor, 1.6 us to the first operand block, 2.0 us to pull 160 KB of operands through one SM (an SM keeps about
// 100 KB of ring in flight and a ring slot's round trip is near 2 us), 0.6 us of MMAs, 1.1 us of epilogue math of
// which 0.7 us is waiting for instructions and per-channel parameters.  Here
//
//  * the K range is cut into up to eight slices, each on its own SM.  The slices' accumulators meet in distributed
//    shared memory: a unit (32 rows x 32 channels) of the tile belongs to one CTA of the cluster, the others send
//    their accumulators to it with st.async, which counts the bytes on the owner's mbarrier, so nobody polls and
//    there is one one-way trip (through L2 and arrival counters the same step cost about 10 us).  The owner adds the
//    slices in the order 0 .. splits-1, whatever the arrival order;
//  * everything that does not depend on the predecessor happens before griddepcontrol.wait: barriers, TMEM, the
//    tensor maps' prefetch, the first ring of WEIGHT blocks, one dry pass through the epilogue's code (which brings its
//    instructions and the unit's parameters into the caches).  The shared memory is kept below half an SM's where
//    that suffices, so that this prologue runs beside the predecessor;
//  * a role is one elected thread: a warp-wide vote per step costs more than the step.  A TMA instruction occupies its
//    thread for 120 cycles whatever its size, so the weight blocks of a ring stage (and, without im2col, its
//    activation blocks) are one three-dimensional box;
//  * the activation box has no more rows than the problem (MMA rows beyond it read whatever the shared memory
//    holds; they belong to no output);
//  * results leave by plain 16-byte stores: a TMA store's round trip is longer than the tile is large.
//
// Measured, microseconds per layer in a chain of equal layers under a graph, persistent kernel -> this one: i8 1x1
// 1024 <-> 256 at 14x14 5.5 -> 4.1, 3x3 256 at 14x14 9.6 -> 5.4, 3x3 512 at 7x7 15.4 -> 5.9, 1x1 64 <-> 256 at 56x56
// 6.3 -> 3.2; TF32 1x1 1024 <-> 256 at 14x14 9.8 -> 6.0, 3x3 128 at 28x28 14.9 -> 7.2.
//
// Warps: 0 TMA producer, 1 MMA issuer and TMEM owner, 2..5 epilogue (one per TMEM lane quarter).
#pragma once

#include <mutex>

#include "umma_kernel.cuh"

namespace oxb {
namespace k {
namespace umma {

// Six warps: with 168 registers a thread two CTAs still share an SM (the next layer's prologue runs under this one).
constexpr int SMALL_THREADS = 64 + 32 * 4;
constexpr int SMALL_MAX_STAGES = 16;
constexpr int SMALL_UNIT_BYTES = 32 * 32 * 4;  // one slice's accumulators of one unit

__device__ __forceinline__ void st_async_v4(uint32_t addr, uint32_t bar, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%2, %3, %4, %5}, [%1];" ::"r"(addr), "r"(bar), "r"(a), "r"(b),
               "r"(c), "r"(d)
               : "memory");
}
// The bounded wait (see mbar_wait) without the suspend hint: nothing else here needs the issue slots.
__device__ __forceinline__ bool mbar_spin(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long start = clock64();
  while (true) {
#pragma unroll 1
    for (int attempt = 0; attempt < 64; ++attempt)
      if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
    if (clock64() - start > WAIT_CYCLES) return false;
  }
}
// The same with the acquire at cluster scope that data sent by another CTA needs.
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  const long long start = clock64();
  while (true) {
#pragma unroll 1
    for (int attempt = 0; attempt < 64; ++attempt) {
      uint32_t ok;
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(ok)
          : "r"(bar), "r"(parity)
          : "memory");
      if (ok) return true;
    }
    if (*abort_flag) return false;
    if (clock64() - start > WAIT_CYCLES) return false;
  }
}
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* m) { asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)m) : "memory"); }
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
               "l"((uint64_t)map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void small_lds_v4(uint32_t addr, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(addr) : "memory");
}

// Finishes one unit: fused epilogue of 32 rows x 32 channels, extrema, store.
template <int KIND, int VARIANT>
__device__ __forceinline__ void small_finish(const KParams& p, const uint32_t (&acc)[32], long long m, int oc, int xz, float xs, size_t esz,
                                             float& seen_min, float& seen_max) {
  const bool row_ok = m < p.M;
  uint32_t w[32];
  uint4 rv[8];
  load_residual<VARIANT>(p, m, oc, row_ok, rv);
  epilogue_chunk<KIND, VARIANT>(p, acc, xz, xs, oc, esz, rv, w);
  const int valid = min(32, p.OC - oc);
  if (!row_ok) return;
  if (p.minmax_keys != nullptr && esz == 4 && (VARIANT < V_REQUANT || VARIANT >= V_DEQUANT)) {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < valid) {
        seen_min = fminf(seen_min, __uint_as_float(w[j]));
        seen_max = fmaxf(seen_max, __uint_as_float(w[j]));
      }
  }
  store_direct(w, (uint8_t*)p.out + ((size_t)m * p.OC + oc) * esz, esz, valid);
}

template <int KIND, int VARIANT>
__device__ __forceinline__ void small_epilogue(const KParams& p, int warp, int lane, uint32_t tmem_base, uint32_t bar_acc, uint32_t bar_recv, uint32_t recv,
                                               volatile int* abortp, int slice, int rank0, int m0, int oc0) {
  const int quarter = warp & 3;
  const int runs = p.small_bn / 32, splits = p.splits;
  const long long m = (long long)m0 + quarter * 32 + lane;
  const size_t esz = (p.out_dt == (int)DT::F32 || p.out_dt == (int)DT::I32) ? 4 : ((p.out_dt == (int)DT::I16 || p.out_dt == (int)DT::F16 || p.out_dt == (int)DT::BF16) ? 2 : 1);
  const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16);
  const bool rows_here = m0 + quarter * 32 < p.M;
  float seen_min = INFINITY, seen_max = -INFINITY;
  uint32_t v[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = 0;
  int xz = 0;
  float xs = 0.f;
  // Pass 0 runs the code that finishes a unit on zeros and stores nothing: its instructions and the first unit's
  // per-channel parameters are then in the caches when the real accumulators arrive (0.5 us of the critical path
  // otherwise).  It reads nothing that the predecessor writes.
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    if (pass == 1) {
      // the predecessor may still read what this grid overwrites, and write what the lines below read
      asm volatile("griddepcontrol.wait;" ::: "memory");
      if (p.x_zp_dev) xz = __float2int_rn(*p.x_zp_dev);
      if (VARIANT >= V_DEQUANT) xs = *p.dq_x_scale;
      bool ok = mbar_spin(bar_acc, 0u, abortp);
      if (!ok && !*abortp) {
        *abortp = 1;
        atomicExch(p.err_flag, 3);
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      // every unit's accumulators to its owner (an own unit into the same place in this CTA's memory)
      if (splits > 1 && rows_here) {
        for (int r = 0; r < runs; ++r) {
          const int u = quarter * runs + r, owner = u % splits;
          if (oc0 + r * 32 >= p.OC) break;
          tmem_ld32_nowait(taddr + (uint32_t)r * 32u, v);
          tmem_ld_wait_for(v);
          const uint32_t place = recv + (uint32_t)((u / splits) * splits + slice) * SMALL_UNIT_BYTES + (uint32_t)lane * 16u;
          if (owner == slice) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(place + (uint32_t)j * 512u), "r"(v[4 * j]), "r"(v[4 * j + 1]), "r"(v[4 * j + 2]), "r"(v[4 * j + 3]) : "memory");
          } else {
            const uint32_t dst = mapa(place, (uint32_t)(rank0 + owner)), bar = mapa(bar_recv, (uint32_t)(rank0 + owner));
#pragma unroll
            for (int j = 0; j < 8; ++j) st_async_v4(dst + (uint32_t)j * 512u, bar, v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          }
        }
      }
    }
    bool waited = splits == 1;
    for (int r = 0; r < runs && rows_here; ++r) {
      const int u = quarter * runs + r, oc = oc0 + r * 32;
      if (oc >= p.OC) break;
      if (u % splits != slice) continue;
      if (pass == 1) {
        if (!waited) {
          waited = true;
          bool ok = mbar_wait_cluster(bar_recv, 0u, abortp);
          if (!ok && !*abortp) {
            *abortp = 1;
            atomicExch(p.err_flag, 6);
          }
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
        }
        if (splits == 1) {
          tmem_ld32_nowait(taddr + (uint32_t)r * 32u, v);
          tmem_ld_wait_for(v);
        } else {
          constexpr bool kFloatAcc = VARIANT < V_REQUANT;
          uint32_t src = recv + (uint32_t)((u / splits) * splits) * SMALL_UNIT_BYTES + (uint32_t)lane * 16u;
#pragma unroll
          for (int j = 0; j < 8; ++j) small_lds_v4(src + (uint32_t)j * 512u, v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
#pragma unroll 1
          for (int sl = 1; sl < splits; ++sl) {
            src += SMALL_UNIT_BYTES;
            uint32_t x[32];
#pragma unroll
            for (int j = 0; j < 8; ++j) small_lds_v4(src + (uint32_t)j * 512u, x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = kFloatAcc ? __float_as_uint(__fadd_rn(__uint_as_float(v[j]), __uint_as_float(x[j]))) : v[j] + x[j];
          }
        }
      }
      small_finish<KIND, VARIANT>(p, v, pass == 0 ? (long long)p.M : m, oc, xz, xs, esz, seen_min, seen_max);
      if (pass == 0) break;  // one unit warms the code; the parameters of the others are few
    }
  }
  if (p.minmax_keys != nullptr) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      seen_min = fminf(seen_min, __shfl_xor_sync(0xffffffffu, seen_min, off));
      seen_max = fmaxf(seen_max, __shfl_xor_sync(0xffffffffu, seen_max, off));
    }
    if (lane == 0) {
      if (seen_min != INFINITY) atomicMin(p.minmax_keys, float_order_key(seen_min));
      if (seen_max != -INFINITY) atomicMax(p.minmax_keys + 1, float_order_key(seen_max));
    }
  }
}

// CTA `cta` of a problem whose launch has clusters of `width` CTAs: a cluster holds width / splits tiles, the slices of a
// tile side by side; the CTAs that the last cluster has too many do nothing.
template <int KIND>
__device__ __forceinline__ void small_tile(const KParams& p, int cta, int width) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_full[SMALL_MAX_STAGES];
  __shared__ __align__(8) uint64_t bar_empty[SMALL_MAX_STAGES];
  __shared__ __align__(8) uint64_t bar_acc;
  __shared__ __align__(8) uint64_t bar_recv;
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int swz = p.swizzle_bytes, bn = p.small_bn, splits = p.splits;
  // a ring stage holds kpb K blocks: their activation rows, then their weight rows
  const uint32_t a_bytes = (uint32_t)p.a_rows * swz, b_bytes = (uint32_t)bn * swz, kpb = (uint32_t)p.kpb;
  const uint32_t stage_bytes = kpb * (a_bytes + b_bytes);
  const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t recv = ring + p.stage_off;
  const int tile = cta / splits, slice = splits > 1 ? cta - tile * splits : 0;
  const int rank0 = splits < width ? cta % width - slice : 0;  // the cluster rank of the tile's first slice
  if (tile >= p.m_tiles * p.n_tiles) {
    if (splits > 1) cluster_sync_all();
    return;
  }
  const int tile_m = tile / p.n_tiles, tile_n = tile - tile_m * p.n_tiles;
  const int m0 = tile_m * BLOCK_M, oc0 = tile_n * bn;
  const int it_begin = slice * p.k_per, it_end = min(p.taps * p.cblocks, it_begin + p.k_per);
  const uint32_t tmem_cols = bn < 32 ? 32u : (uint32_t)bn;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(smem_u32(&bar_full[i]), 1);
      mbar_init(smem_u32(&bar_empty[i]), 1);
    }
    mbar_init(smem_u32(&bar_acc), 1);
    mbar_init(smem_u32(&bar_recv), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (splits > 1) {  // what the other slices will send here
      const int runs = bn / 32;
      int owned = 0;
      for (int u = slice; u < 4 * runs; u += splits) owned += (m0 + (u / runs) * 32 < p.M && oc0 + (u % runs) * 32 < p.OC) ? 1 : 0;
      mbar_expect_tx(smem_u32(&bar_recv), (uint32_t)(owned * (splits - 1)) * SMALL_UNIT_BYTES);
    }
  }
  if (warp == 0 && lane < 2) prefetch_tensormap(lane == 0 ? &p.tmA : &p.tmB);
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (splits > 1) cluster_sync_all();  // every owner's barrier exists before anything is sent to it
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  volatile int* abortp = &abort_flag;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == 0) {
    // ---------------- TMA producer: weights of the first ring, then the wait, then everything else ----------------
    // A box that runs past the slice brings blocks that nobody multiplies.
    const int chunks = (it_end - it_begin + p.kpb - 1) / p.kpb;
    int q0 = 0, p0 = 0, n0 = 0;
    if (p.a_im2col) {
      q0 = m0 % p.Q;
      const int rest = m0 / p.Q;
      p0 = rest % p.P;
      n0 = rest / p.P;
    }
    const int w_base = q0 * p.sw - p.pl, h_base = p0 * p.sh - p.pt;
    int cb = it_begin % p.cblocks, sx = (it_begin / p.cblocks) % p.S, r = (it_begin / p.cblocks) / p.S;
    auto expect = [&](int chunk) -> uint32_t {
      const int valid = min(p.kpb, it_end - it_begin - chunk * p.kpb);
      return kpb * b_bytes + (p.a_im2col ? (uint32_t)valid : kpb) * a_bytes;
    };
    if (elect_one()) {
      for (int i = 0; i < min(p.stages, chunks); ++i) {
        mbar_expect_tx(smem_u32(&bar_full[i]), expect(i));
        tma_load_3d(ring + (uint32_t)i * stage_bytes + kpb * a_bytes, &p.tmB, smem_u32(&bar_full[i]), 0, oc0, it_begin + i * p.kpb);
      }
      asm volatile("griddepcontrol.wait;" ::: "memory");
      uint32_t stage = 0, phase = 0;
      for (int c = 0, it = it_begin; c < chunks; ++c, it += p.kpb) {
        const uint32_t full = smem_u32(&bar_full[stage]), dst = ring + stage * stage_bytes;
        if (c >= p.stages) {  // this stage has held an earlier chunk
          if (!mbar_spin(smem_u32(&bar_empty[stage]), phase ^ 1u, abortp)) {
            if (!*abortp) {
              *abortp = 1;
              atomicExch(p.err_flag, 1);
            }
            break;
          }
          mbar_expect_tx(full, expect(c));
          tma_load_3d(dst + kpb * a_bytes, &p.tmB, full, 0, oc0, it);
        }
        if (p.a_im2col) {
          const int valid = min(p.kpb, it_end - it);
          for (int g = 0; g < valid; ++g) {
            tma_load_im2col_4d(dst + (uint32_t)g * a_bytes, &p.tmA, full, cb * p.cb_elems, w_base, h_base, n0, (uint16_t)(sx * p.dw), (uint16_t)(r * p.dh));
            if (++cb == p.cblocks) {
              cb = 0;
              if (++sx == p.S) {
                sx = 0;
                ++r;
              }
            }
          }
        } else {
          tma_load_3d(dst, &p.tmA, full, 0, m0, it);
        }
        if (++stage == (uint32_t)p.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (elect_one()) {
      asm volatile("griddepcontrol.wait;" ::: "memory");  // the bounded waits below must not time the predecessor
      const uint64_t desc = make_smem_desc(0, swz);
      uint32_t stage = 0, phase = 0;
      for (int it = it_begin; it < it_end; it += p.kpb) {
        if (!mbar_spin(smem_u32(&bar_full[stage]), phase, abortp)) {
          if (!*abortp) {
            *abortp = 1;
            atomicExch(p.err_flag, 2);
          }
          break;
        }
        tc_fence_after();
        uint32_t a16 = (ring + stage * stage_bytes) >> 4, b16 = a16 + ((kpb * a_bytes) >> 4);
        const int valid = min(p.kpb, it_end - it);
        for (int g = 0; g < valid; ++g, a16 += a_bytes >> 4, b16 += b_bytes >> 4) {
          // descriptors differ between blocks only in the 16-byte granular start address
          const uint64_t da = desc | (a16 & 0x3fffu), db = desc | (b16 & 0x3fffu);
          tc_mma_one<KIND>(tmem_base, da, db, p.idesc, (it + g) > it_begin ? 1u : 0u);
          if (swz >= 64) tc_mma_one<KIND>(tmem_base, da + 2, db + 2, p.idesc, 1u);
          if (swz == 128) {
            tc_mma_one<KIND>(tmem_base, da + 4, db + 4, p.idesc, 1u);
            tc_mma_one<KIND>(tmem_base, da + 6, db + 6, p.idesc, 1u);
          }
        }
        if (it + p.kpb >= it_end) tc_commit<false>(smem_u32(&bar_acc));
        else if (it + p.stages * p.kpb < it_end) tc_commit<false>(smem_u32(&bar_empty[stage]));  // somebody waits for this stage
        if (++stage == (uint32_t)p.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    __syncwarp();
  } else {
    // ---------------- epilogue ----------------
#define OXB_SMALL(V)                                                                                                                                   \
  case V: small_epilogue<KIND, V>(p, warp, lane, tmem_base, smem_u32(&bar_acc), smem_u32(&bar_recv), recv, abortp, slice, rank0, m0, oc0); break;
    if constexpr (KIND == KIND_I8) {
      switch (p.variant) {
        OXB_SMALL(V_REQUANT)
        OXB_SMALL(V_REQUANT_DYN)
        OXB_SMALL(V_INT32)
        OXB_SMALL(V_INT32_DYN)
        OXB_SMALL(V_REQUANT_FMA)
        OXB_SMALL(V_REQUANT_FMA_DYN)
        OXB_SMALL(V_REQUANT_LEAN)
        OXB_SMALL(V_REQUANT_LEAN_DYN)
        OXB_SMALL(V_REQUANT_FBIAS)
        OXB_SMALL(V_REQUANT_PACKED)
        OXB_SMALL(30)
        OXB_SMALL(31)
        OXB_SMALL(32)
        OXB_SMALL(33)
        OXB_SMALL(34)
        OXB_SMALL(35)
        OXB_SMALL(V_JOIN)
        default: break;
      }
    } else {
      switch (p.variant) {
        OXB_SMALL(0)
        OXB_SMALL(1)
        OXB_SMALL(2)
        OXB_SMALL(3)
        OXB_SMALL(4)
        OXB_SMALL(5)
        OXB_SMALL(6)
        OXB_SMALL(7)
        OXB_SMALL(8)
        OXB_SMALL(9)
        OXB_SMALL(10)
        OXB_SMALL(11)
        OXB_SMALL(12)
        OXB_SMALL(13)
        OXB_SMALL(14)
        OXB_SMALL(15)
        OXB_SMALL(16)
        OXB_SMALL(17)
        OXB_SMALL(18)
        OXB_SMALL(19)
        default: break;
      }
    }
#undef OXB_SMALL
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (abort_flag && threadIdx.x == 0) {
    // copies of this CTA may still be in flight, and a slice that has not given up yet may still send to it: every
    // wait of a slice ends within WAIT_CYCLES, and one that gave up sends nothing
    const long long start = clock64();
    while (clock64() - start < 2 * WAIT_CYCLES) {
    }
  }
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
}

// Independent problems side by side (the Q, K and V products of an attention layer, a residual block's first convolution
// and its shortcut): each leaves most of the chip idle, and one after the other each would wait for the one before.  In
// one grid they share one griddepcontrol.wait, which orders every member behind everything before the grid.  A lone
// problem is a group of one: a kernel of its own for groups would evict this one's instructions and find its own cold
// (encoder of 2x77 tokens 1048 us with two kernels, 1016 us with one).  The cluster is the widest that a member's slices
// need, also where the members together are more than are resident at once (INT8 frame: 303 us, against 308 us when such
// members are launched one after the other).
template <int KIND>
__global__ void __launch_bounds__(SMALL_THREADS, 2) umma_small_kernel(const __grid_constant__ SmallGroup g) {
  int i = 0;
#pragma unroll
  for (int j = 1; j < GROUP_MAX; ++j) i += (int)blockIdx.x >= g.first[j] ? 1 : 0;
  small_tile<KIND>(g.m[i], (int)blockIdx.x - g.first[i], g.width);
}

// The opt-in for more than 48 KB of dynamic shared memory, per kernel and device (see ensure_smem_attr).  The split
// between L1 and shared memory is fixed too: it must not keep the second CTA off an SM, nor change between layers.
template <int KIND>
void ensure_small_attr(int device) {
  static std::mutex mu;
  static bool have[kMaxDevices] = {};
  const int d = (device >= 0 && device < kMaxDevices) ? device : 0;
  std::lock_guard<std::mutex> lock(mu);
  if (have[d]) return;
  OXB_CUDA(cudaFuncSetAttribute(umma_small_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMALL_SMEM_MAX));
  OXB_CUDA(cudaFuncSetAttribute(umma_small_kernel<KIND>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
  have[d] = true;
}

template <int KIND>
void launch_small_kind(const SmallGroup& g, int grid, size_t smem, int device, cudaStream_t s) {
  ensure_small_attr<KIND>(device);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(SMALL_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)g.width;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g.width > 1 ? 2 : 1;
  OXB_CUDA(cudaLaunchKernelEx(&cfg, umma_small_kernel<KIND>, g));
}

}  // namespace umma
}  // namespace k
}  // namespace oxb
