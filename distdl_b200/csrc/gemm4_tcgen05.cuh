// bf16 GEMM on CTA pairs with 512x256 tiles: the form for large outputs.
//
// What bounds a large product here is power, not cycles: the 256x256 tiles of gemm2_tcgen05.cuh keep the tensor cores
// as busy as the library's kernels do, but bring 8.6 GB through L2 for an 8192^3 product where 6.4 are enough, and the
// clock falls in proportion.  So a pair takes two 256-row blocks of the same 256 columns at once: per 64-deep k-block
// a CTA stages 128x64 of A for either block (32 KB) and its 128x64 half of B (16 KB), four stages of 48 KB, and the
// two accumulators (256 columns each) fill tensor memory.
//
// With both accumulators in use there is none to spare while a tile is stored.  Two sets of epilogue warps drain them
// side by side (an accumulator is given back after its last tcgen05.ld, before its stores), and the MMA issuer starts
// the next tile on accumulator 0 alone, up to STAGES k-blocks ahead, until accumulator 1 is free as well.
//
// Work items: the first `full` tiles (whole waves of the pairs) are taken as 512x256; the tiles of a last, partial
// wave are taken as their two 256x256 blocks where that shortens it.
//
// Roles per CTA: warp 0 TMA producer, warp 1 MMA issuer (leader CTA only), warps 2..5 / 6..9 epilogue of accumulator
// 0 / 1.  All waits are bounded.
#pragma once

#include "gemm2_tcgen05.cuh"

namespace dd {
namespace gemm4 {

using gemm::Params;
using gemm2::cluster_ctarank;
using gemm2::cluster_sync;
using gemm2::mapa;
using gemm2::mbar_arrive_cluster;
using gemm2::tma_load_3d_pair;
using gemm2::umma_commit_pair;
using gemm2::umma_f16_pair;

constexpr int BLK = 256;                       // rows of a block of a pair (128 per CTA)
constexpr int BN = 256;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int STAGES = 4;
constexpr int SLICE = 128 * BK * 2;            // 16 KB: 128 rows of an operand, one k-block
constexpr int STAGE_BYTES = 3 * SLICE;         // A of block 0, A of block 1, B
constexpr int NUM_EPI_WARPS = 8;
constexpr int NUM_THREADS = 64 + 32 * NUM_EPI_WARPS;
constexpr int OUT_BOX = 32 * 128;              // one box of 32 rows x 128 bytes per epilogue warp
constexpr int SMEM = 1024 + STAGES * STAGE_BYTES + NUM_EPI_WARPS * OUT_BOX + 256;
static_assert(SMEM <= 232448, "shared memory of an SM");

struct SharedStorage {
  uint64_t full[STAGES];
  uint64_t empty[STAGES];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  volatile int abort_flag;
};

__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred P;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// One work item of a pair: `blocks` (0, 1 or 2) row blocks from block `rb` on; zero: nothing is multiplied for it.
struct Item {
  int rb, tn, tb, blocks;
  bool zero;
};

struct Plan {
  int tiles_m, tiles_n, row_blocks, full, items;
};

// full: the tiles of whole waves, or all of them where the rest is more than half a wave.
inline Plan make_plan(int M, int N, int batch, int pairs) {
  Plan w;
  w.row_blocks = (M + BLK - 1) / BLK;
  w.tiles_m = (w.row_blocks + 1) / 2;
  w.tiles_n = (N + BN - 1) / BN;
  const int tiles = w.tiles_m * w.tiles_n * batch, rest = tiles % pairs;
  w.full = rest * 2 > pairs && tiles > pairs ? tiles : tiles - rest;
  w.items = w.full + 2 * (tiles - w.full);
  return w;
}

// The items of one pair in order, for each of its roles.
//
// Batched products with rows[b] live rows (see Params): only blocks with live rows are dealt out, in slots of two blocks
// (a tile, or the last, odd block of two neighbouring columns), so that every pair gets as many; the blocks without live
// rows follow, whose zeros the epilogue writes.  In us back to back, against 256-row tiles dealt out with the empty ones: eight
// experts of about 256 rows in 320, 28672 x 4096 622 -> 489, 14336 x 4096 356 -> 333.
struct Walk {
  int at, sub = 0, tb = 0, base = 0;
  bool dead = false;

  __device__ explicit Walk(int pair) : at(pair) {}

  __device__ __forceinline__ bool next(Item& it, const Params& p, const Plan& w, int num_pairs) {
    if (p.rows == nullptr) {
      if (at >= w.items) return false;
      const int rest = at - w.full;
      const int t = rest < 0 ? at : w.full + (rest >> 1);
      int tm;
      gemm::tile_coords(t, w.tiles_m, w.tiles_n, p.group_m, tm, it.tn, it.tb);
      it.rb = 2 * tm + (rest < 0 ? 0 : (rest & 1));
      it.blocks = min(rest < 0 ? 2 : 1, max(0, w.row_blocks - it.rb));
      it.zero = false;
      at += num_pairs;
      return true;
    }
    while (true) {
      if (tb == p.batch) {
        if (dead) return false;
        dead = true;
        tb = 0;
      }
      const int live = min(w.row_blocks, max(0, (p.rows[tb] + BLK - 1) / BLK));
      const int half = live >> 1, odd = live & 1, per = 2 * half + odd;      // slots of two columns
      const int n = dead ? (w.row_blocks - live) * w.tiles_n : per * ((w.tiles_n + 1) >> 1);
      if (at >= base + n) {
        base += n;
        ++tb;
        continue;
      }
      const int s = at - base;
      it.tb = tb;
      it.zero = dead;
      if (dead) {
        it.tn = s / (w.row_blocks - live);
        it.rb = live + s - it.tn * (w.row_blocks - live);
        it.blocks = 1;
        at += num_pairs;
        return true;
      }
      const int q = s / per, r = s - q * per;
      if (r < 2 * half) {
        it.tn = 2 * q + (r >= half ? 1 : 0);
        it.rb = 2 * (r >= half ? r - half : r);
        it.blocks = 2;
      } else {
        it.tn = 2 * q + sub;
        it.rb = 2 * half;
        it.blocks = 1;
        sub ^= 1;
      }
      if (it.tn >= w.tiles_n) it.blocks = 0;
      if (sub == 0) at += num_pairs;
      return true;
    }
  }
};

// Adds bias[col0 .. col0 + 31] to a chunk of 32 columns (columns past N are never stored).
__device__ __forceinline__ void add_bias(const Params& q, int col0, uint32_t (&r)[32]) {
  const int nv = min(32, q.N - col0);
  if (q.flags & gemm::F_BIAS_F32) {
    const float* bp = reinterpret_cast<const float*>(q.bias) + col0;
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (i < nv) r[i] = __float_as_uint(__uint_as_float(r[i]) + bp[i]);
    return;
  }
  const __nv_bfloat16* bp = reinterpret_cast<const __nv_bfloat16*>(q.bias) + col0;
  if (nv == 32 && (reinterpret_cast<uintptr_t>(bp) & 15) == 0) {
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const uint4 u = reinterpret_cast<const uint4*>(bp)[g];
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 f = unpack_bf16x2(w[i]);
        r[8 * g + 2 * i] = __float_as_uint(__uint_as_float(r[8 * g + 2 * i]) + f.x);
        r[8 * g + 2 * i + 1] = __float_as_uint(__uint_as_float(r[8 * g + 2 * i + 1]) + f.y);
      }
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 32; ++i)
    if (i < nv) r[i] = __float_as_uint(__uint_as_float(r[i]) + __bfloat162float(bp[i]));
}

// 128 bytes per row (w[0 .. 31] of lane = row) through the warp's box to columns col0 .. of D.
__device__ __forceinline__ void store_box(const CUtensorMap* map, uint8_t* box, int lane, const uint32_t* w, bool add,
                                          int col0, int row0, int tb) {
  if (lane == 0) tma_store_wait_read();
  __syncwarp();
#pragma unroll
  for (int g = 0; g < 8; ++g)
    *reinterpret_cast<uint4*>(box + lane * 128 + ((g ^ (lane & 7)) << 4)) =
        make_uint4(w[4 * g], w[4 * g + 1], w[4 * g + 2], w[4 * g + 3]);
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) {
    if (add) tma_reduce_add_3d(map, box, col0, row0, tb);
    else     tma_store_3d(map, box, col0, row0, tb);
    tma_store_commit();
  }
}

// One epilogue warp: 32 rows x 256 columns of the accumulator at `taddr`.  The MMA issuer waits for the accumulator, so
// its first columns go through the box as they are read, the last 192 (bf16, packed) or 96 (fp32) are first taken into
// registers, and it is given back through the barrier `release` before these are stored.  zero: nothing was multiplied.
// 8192 x 28672 x 4096: 5 200 clocks without products per tile when all columns were stored as they were read, 4 300 so.
template <bool F32>
__device__ __forceinline__ void store_block(const Params& q, const CUtensorMap* map, uint32_t taddr, uint8_t* box,
                                            int lane, int col_tile0, int row0, int tb, bool zero, uint32_t release) {
  const bool add = (q.flags & gemm::F_ACCUMULATE) != 0, bias = (q.flags & gemm::F_BIAS) != 0;
  auto chunk = [&](int c, uint32_t (&r)[32]) {
    if (!zero) {
      tmem_ld_32x32(taddr + c * 32, r);
      tmem_ld_wait();
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) r[i] = 0u;
    }
    if (bias) add_bias(q, col_tile0 + c * 32, r);
  };
  auto packed = [&](int c, uint32_t* w) {              // 64 columns from 64 c on as 32 words
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t r[32];
      chunk(2 * c + h, r);
#pragma unroll
      for (int i = 0; i < 16; ++i)
        w[16 * h + i] = pack_bf16x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
    }
  };
  constexpr int WIDTH = F32 ? 32 : 64, DIRECT = BN / WIDTH - 3;
#pragma unroll 1
  for (int c = 0; c < DIRECT; ++c) {
    uint32_t r[32];
    if (F32) chunk(c, r);
    else     packed(c, r);
    if (col_tile0 + c * WIDTH < q.N) store_box(map, box, lane, r, add, col_tile0 + c * WIDTH, row0, tb);
  }
  uint32_t hold[3][32];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (F32) chunk(DIRECT + c, hold[c]);
    else     packed(DIRECT + c, hold[c]);
  }
  if (!zero) {
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive_cluster(release);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int col0 = col_tile0 + (DIRECT + c) * WIDTH;
    if (col0 < q.N) store_box(map, box, lane, hold[c], add, col0, row0, tb);
  }
}

template <bool A_MN, bool B_MN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
gemm4_bf16_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                  const __grid_constant__ CUtensorMap tmap_d, const Params p, const Plan plan) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* boxes = tiles + STAGES * STAGE_BYTES;
  SharedStorage* ss = reinterpret_cast<SharedStorage*>(boxes + NUM_EPI_WARPS * OUT_BOX);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();          // 0 = leader
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int num_k = (p.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&ss->full[s], 1); mbar_init(&ss->empty[s], 1); }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&ss->tmem_full[a], 1);
      mbar_init(&ss->tmem_empty[a], 2 * (NUM_EPI_WARPS / 2));   // this accumulator's epilogue warps of both CTAs
    }
    ss->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { gemm2::tmem_alloc_pair(&ss->tmem_base, 2 * BN); gemm2::tmem_relinquish_pair(); }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                   // barriers of both CTAs are initialised
  tc_fence_after();
  const uint32_t tmem_base = ss->tmem_base;
  if (!(p.flags & gemm::F_ALONE)) grid_dependency_launch();
  grid_dependency_wait();

  if (warp == 0) {
    // ------------------- TMA producer (both CTAs, own slices) -------------------
    if (elect_one()) {
      tma_prefetch_desc(&tmap_a);
      tma_prefetch_desc(&tmap_b);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      Walk walk(pair);
      Item it;
      while (ok && walk.next(it, p, plan, num_pairs) && !it.zero) {
        if (it.blocks == 0) continue;
        const int n0 = it.tn * BN + rank * 128;
        for (int k = 0; k < num_k; ++k) {
          ok = mbar_wait(&ss->empty[stage], phase ^ 1, &ss->abort_flag, p.status, 311);
          if (!ok) break;
          uint8_t* sa = tiles + stage * STAGE_BYTES;
          uint8_t* sb = sa + 2 * SLICE;
          const uint32_t full_leader = mapa(smem_u32(&ss->full[stage]), 0);
          if (rank == 0) mbar_expect_tx(&ss->full[stage], 2 * (it.blocks + 1) * SLICE);
          for (int h = 0; h < it.blocks; ++h) {
            const int m0 = (it.rb + h) * BLK + rank * 128;
            if (A_MN) {
#pragma unroll
              for (int i = 0; i < 2; ++i)
                tma_load_3d_pair(sa + h * SLICE + i * (SLICE / 2), &tmap_a, full_leader, m0 + i * 64, k * BK, it.tb);
            } else {
              tma_load_3d_pair(sa + h * SLICE, &tmap_a, full_leader, k * BK, m0, it.tb);
            }
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) {                 // boxes of 64 rows or columns
            if (B_MN) tma_load_3d_pair(sb + i * (SLICE / 2), &tmap_b, full_leader, n0 + i * 64, k * BK, it.tb);
            else      tma_load_3d_pair(sb + i * (SLICE / 2), &tmap_b, full_leader, k * BK, n0 + i * 64, it.tb);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 1000000ull) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ---------------------------- MMA issuer (leader) ---------------------------
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(BLK, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
      int stage = 0, sel = 0;
      uint32_t phase = 0, acc_phase = 0;              // acc_phase: one bit per accumulator
      bool ok = true;
      auto product = [&](int s, int slot, int acc, bool first) {
        const uint32_t sa = smem_u32(tiles + s * STAGE_BYTES) + slot * SLICE;
        const uint32_t sb = smem_u32(tiles + s * STAGE_BYTES) + 2 * SLICE;
#pragma unroll
        for (int kk = 0; kk < BK / UMMA_K; ++kk) {
          const uint64_t adesc = A_MN ? make_smem_desc_sw128(sa + kk * (UMMA_K * 128), 64 * BK * 2, 1024)
                                      : make_smem_desc_sw128(sa + kk * (UMMA_K * 2), 16, 1024);
          const uint64_t bdesc = B_MN ? make_smem_desc_sw128(sb + kk * (UMMA_K * 128), 64 * BK * 2, 1024)
                                      : make_smem_desc_sw128(sb + kk * (UMMA_K * 2), 16, 1024);
          umma_f16_pair(tmem_base + acc * BN, adesc, bdesc, idesc, (first && kk == 0) ? 0u : 1u);
        }
      };
      Walk walk(pair);
      Item it;
      while (ok && walk.next(it, p, plan, num_pairs) && !it.zero) {
        const int acc = it.blocks == 1 ? sel : 0;
        if (it.blocks == 1) sel ^= 1;
        if (it.blocks == 0) continue;
        ok = mbar_wait(&ss->tmem_empty[acc], ((acc_phase >> acc) & 1) ^ 1, &ss->abort_flag, p.status, 312);
        if (!ok) break;
        tc_fence_after();
        int k = 0;
        if (it.blocks == 2) {
          // accumulator 0 alone while the epilogue still reads accumulator 1
          int s = stage;
          uint32_t ph = phase;
          const int ahead = min(num_k, STAGES);
          bool free1 = mbar_test(&ss->tmem_empty[1], (acc_phase >> 1) ^ 1);
          while (!free1 && k < ahead) {
            ok = mbar_wait(&ss->full[s], ph, &ss->abort_flag, p.status, 313);
            if (!ok) break;
            tc_fence_after();
            product(s, 0, 0, k == 0);
            ++k;
            if (++s == STAGES) { s = 0; ph ^= 1; }
            free1 = mbar_test(&ss->tmem_empty[1], (acc_phase >> 1) ^ 1);
          }
          if (!ok) break;
          ok = mbar_wait(&ss->tmem_empty[1], (acc_phase >> 1) ^ 1, &ss->abort_flag, p.status, 314);
          if (!ok) break;
          tc_fence_after();
          if (k == num_k) umma_commit_pair(&ss->tmem_full[0]);
          for (int i = 0; i < k; ++i) {
            product(stage, 1, 1, i == 0);
            umma_commit_pair(&ss->empty[stage]);
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
          }
        }
        for (; k < num_k; ++k) {
          ok = mbar_wait(&ss->full[stage], phase, &ss->abort_flag, p.status, 315);
          if (!ok) break;
          tc_fence_after();
          product(stage, 0, acc, k == 0);
          if (it.blocks == 2) {
            if (k == num_k - 1) umma_commit_pair(&ss->tmem_full[0]);
            product(stage, 1, 1, k == 0);
          }
          umma_commit_pair(&ss->empty[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        if (it.blocks == 2) {
          umma_commit_pair(&ss->tmem_full[1]);
          acc_phase ^= 3;
        } else {
          umma_commit_pair(&ss->tmem_full[acc]);
          acc_phase ^= 1u << acc;
        }
      }
    }
  } else {
    // --------------- epilogue (both CTAs, own rows; one set of warps per accumulator) ---------------
    const int quarter = warp & 3, set = (warp - 2) >> 2;
    uint8_t* box = boxes + (warp - 2) * OUT_BOX;
    const uint32_t taddr = tmem_base + set * BN + ((uint32_t)(quarter * 32) << 16);
    const uint32_t release = mapa(smem_u32(&ss->tmem_empty[set]), 0);
    int sel = 0;
    uint32_t acc_phase = 0;
    Walk walk(pair);
    Item it;
    while (walk.next(it, p, plan, num_pairs)) {
      int h = set;                                     // this set's block of the item
      if (it.blocks == 1) {
        h = set == sel ? 0 : 2;
        sel ^= 1;
      }
      if (h >= it.blocks) continue;
      if (!it.zero) {
        if (!mbar_wait(&ss->tmem_full[set], acc_phase, &ss->abort_flag, p.status, 316)) break;
        tc_fence_after();
        acc_phase ^= 1;
      }
      const int row0 = (it.rb + h) * BLK + rank * 128 + quarter * 32;
      if (p.flags & gemm::F_OUT_F32)
        store_block<true>(p, &tmap_d, taddr, box, lane, it.tn * BN, row0, it.tb, it.zero, release);
      else
        store_block<false>(p, &tmap_d, taddr, box, lane, it.tn * BN, row0, it.tb, it.zero, release);
    }
    if (lane == 0) tma_store_wait_all();
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync();               // nobody leaves while the peer may still touch its barriers / TMEM
  if (warp == 1) { tc_fence_after(); gemm2::tmem_dealloc_pair(tmem_base, 2 * BN); }
}

}  // namespace gemm4
}  // namespace dd
