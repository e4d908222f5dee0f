// Flash attention backward for sm_100a (head dimension DD_HEAD_DIM = 128 or 64; this file is included once per
// head dimension by attention_bwd3.cu, inside namespace DD_BWD3_NS).  Any sequence length.
//
// One CTA per key tile (and kv head, sequence, see bwd3_split) sweeps the query tiles of the heads of its group and forms
// all three gradients from ONE recomputation of the scores: five products per tile pair instead of the seven of a
// dK / dV kernel followed by a dQ kernel, and one exponential per score instead of two.  Per tile pair:
//
//   S^T = K Q^T, dP^T = V dO^T   key rows in the tensor-memory lanes, queries in the columns
//   P^T  -> bf16 in tensor memory, A operand of dV += P^T dO
//   dS^T -> bf16 in shared memory: read K-major it is the A operand of dK += dS^T Q, read MN-major that of dQ = dS K
//   dQ   -> tensor memory -> registers -> shared memory -> added in fp32 to a workspace by bulk reductions
//
// The result is deterministic: the partial dQ tiles of a query tile are added in the order of the key tiles.  A
// counter per query tile says how many have been added; key tile j adds its part when it says j.  The first one stores
// (nothing has to be cleared), the last one adds what is there to its own part, scales and writes bf16.  CTAs take
// their key tile from a ticket, in the order of the counters, so that whoever is waited for has started before; every
// CTA sweeps the query tiles in the same (descending) order, so that the CTAs of a head follow one another at the distance
// of one hand-over.  Causal sweeps grow shorter by a tile from one CTA to the next, which hides most of it; full ones do not:
// 8 heads of 128, 4, 8 and 16 key tiles that start together, each call alone: causal 34, 54 and 87 us, full 60, 114 and 214.
//
// Every wait is bounded; a time-out records a status, tells the CTAs that would wait in turn, and falls through to
// the release of the tensor memory.
namespace DD_BWD3_NS {

constexpr int BT = 128;                // tile edge for queries and keys
constexpr int D = DD_HEAD_DIM;         // head dimension
constexpr int DCH = D / 64;            // 64-element (128-byte) chunks per row
constexpr int T_BYTES = BT * D * 2;    // one [128 x D] bf16 tile
constexpr int DS_BYTES = BT * BT * 2;  // one dS^T tile
constexpr float kLog2e = 1.4426950408889634f;

// The two head dimensions differ in what bounds them.
//   64: shared-memory bandwidth (about 2 700 clocks of operands, tiles, dS, dQ and statistics per tile pair; 2 900
//       measured) before the softmax (16 384 exponentials: 1 024 clocks) and the five products (1 550).  Tensor
//       memory has room for S | dP | dV | dK | dQ | P side by side, so that S of the next tile pair is formed as soon as
//       the softmax warps have S in registers, and dP as soon as dS is written: sixteen of them, 32 queries each, never
//       wait for the tensor cores.  Q has three stages (needed early in an iteration, given back late), dS two.
//  128: shared-memory bandwidth (operands of the products 2 300 clocks, tiles coming in 512, dS 256, dQ going out 1 024:
//       4 100 per tile pair, 4 500 measured) and its size.  S | dP | dV | dK fill tensor memory: P lies over S, and dQ takes the columns of dP between the moment dS
//       is in shared memory and the next dP.  Eight softmax warps of 64 queries; dO has one stage (dV(n) is multiplied
//       first in an iteration, dP(n + 1) last, the load lies between).
// Issue order per tile pair: 64: S(n+1), dV(n), dP(n+1), dQ(n), dK(n); 128: dV(n), S(n+1), dQ(n), dK(n), dP(n+1).
constexpr bool ROOMY = D == 64;
constexpr int SOFTMAX_WARPS = ROOMY ? 16 : 8, DRAIN_WARPS = 4;
constexpr int COLS = BT / (SOFTMAX_WARPS / 4);      // queries per softmax thread
constexpr int NUM_THREADS = 128 + 32 * (SOFTMAX_WARPS + DRAIN_WARPS);
// Registers: the warpgroups (issuing warps, softmax, drain) share out what the launch gets, 80 or 128 a thread, so that
// a softmax thread keeps its probabilities and a drain thread its row of dQ without spilling.
constexpr int REGS_LAUNCH = ROOMY ? 80 : 128;
constexpr int REGS_ISSUE = ROOMY ? 64 : 72, REGS_SOFTMAX = ROOMY ? 80 : 136, REGS_DRAIN = ROOMY ? 96 : 168;
static_assert(REGS_ISSUE + SOFTMAX_WARPS / 4 * REGS_SOFTMAX + REGS_DRAIN <= REGS_LAUNCH * (NUM_THREADS / 128),
              "the split may not exceed what the launch gets");
constexpr int Q_STAGES = ROOMY ? 3 : 2, DO_STAGES = ROOMY ? 2 : 1, DS_BUFS = ROOMY ? 2 : 1;
// dQ leaves in chunks of 32 columns through two buffers in shared memory, as bulk reductions: the TMA unit does them
// beside the softmax warps' accesses, where 16-byte reductions from registers took 3 200 clocks a tile at D = 128 and
// held up every other access of the SM (at 1 x 16384, 32 / 8 heads of 128, causal, 6 900 us where bulk reductions took 5 780,
// both in one run on a card below its power limit; the kernel as it is now takes 6 440 back to back, at the limit).
constexpr int CHUNK_BYTES = BT * 32 * 4, CHUNKS = D / 32;
static_assert(CHUNKS % 2 == 0, "a tile starts with the first buffer");

struct BwdParams {
  const float* lse2;    // [batch][Hq][nT * 128]  log-sum-exp of the scaled scores, in base 2 (+inf behind the sequence)
  const float* delta;   // [batch][Hq][nT * 128]  rowsum(O * dO)
  float* dq_sum;        // [batch][Hq][nT][D / 4][128][4]  nT > 1 only
  int* dq_turn;         // [batch][Hq][nT]  key tiles added so far
  float* kv_sum;        // [batch][Hkv][nT][dV, dK][D / 4][128][4]  split > 1 only
  int* kv_turn;         // [batch][Hkv][nT]  parts of the group added so far
  int* ticket;          // next CTA's place in the order; ticket[1]: somebody gave up
  __nv_bfloat16* dq; long long dq_row, dq_head;
  __nv_bfloat16* dk; long long dk_row, dk_head;
  __nv_bfloat16* dv; long long dv_row, dv_head;
  int S, Hq, Hkv, batch, causal, split;
  float scale;
  StatusRecord* status;
};

// Untiled bulk copy global -> shared of this CTA (both addresses 16-byte aligned, size a
// multiple of 16 bytes), completion on an mbarrier.
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(smem_dst)), "l"(gsrc), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// One chunk of fp32 values, shared -> global: stored, or added to what is there.
__device__ __forceinline__ void bulk_put(float* dst, uint32_t src, bool add) {
  if (add)
    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;"
                 ::"l"(dst), "r"(src), "n"(CHUNK_BYTES) : "memory");
  else
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                 ::"l"(dst), "r"(src), "n"(CHUNK_BYTES) : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async;" ::: "memory"); }

// Eight fp32 values times `mul`, plus what was added before, as bf16
__device__ __forceinline__ uint4 pack8(const uint32_t* r, float mul, float4 a, float4 e) {
  uint4 v;
  v.x = pack_bf16x2((a.x + __uint_as_float(r[0])) * mul, (a.y + __uint_as_float(r[1])) * mul);
  v.y = pack_bf16x2((a.z + __uint_as_float(r[2])) * mul, (a.w + __uint_as_float(r[3])) * mul);
  v.z = pack_bf16x2((e.x + __uint_as_float(r[4])) * mul, (e.y + __uint_as_float(r[5])) * mul);
  v.w = pack_bf16x2((e.z + __uint_as_float(r[6])) * mul, (e.w + __uint_as_float(r[7])) * mul);
  return v;
}

// Column ch .. ch + 32 of this thread's row of dV or dK: stored as bf16 (times `mul`) by the last of the group's parts,
// which adds what the earlier ones left in `sum` ([D / 4][128][4], already offset to the row); those store or add.
__device__ __forceinline__ void put_cols32(uint32_t taddr, __nv_bfloat16* dst, float* sum, int ch, float mul, bool first,
                                           bool last, bool live) {
  uint32_t r[32];
  __syncwarp();             // (after the stores of the rows that exist: the read is one of the whole warp)
  tmem_ld_32x32(taddr + ch, r);
  tmem_ld_wait();
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    float* at = sum + (size_t)(ch / 4 + 2 * g) * (BT * 4);
    if (last) {
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f), e = a;
      if (!first) {
        a = __ldcg(reinterpret_cast<const float4*>(at));
        e = __ldcg(reinterpret_cast<const float4*>(at + BT * 4));
      }
      if (live) *reinterpret_cast<uint4*>(dst + ch + 8 * g) = pack8(r + 8 * g, mul, a, e);
    } else if (first) {
      *reinterpret_cast<uint4*>(at) = make_uint4(r[8 * g], r[8 * g + 1], r[8 * g + 2], r[8 * g + 3]);
      *reinterpret_cast<uint4*>(at + BT * 4) = make_uint4(r[8 * g + 4], r[8 * g + 5], r[8 * g + 6], r[8 * g + 7]);
    } else {
#pragma unroll
      for (int u = 0; u < 2; ++u)
        asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
                     ::"l"(at + u * (BT * 4)), "f"(__uint_as_float(r[8 * g + 4 * u])),
                       "f"(__uint_as_float(r[8 * g + 4 * u + 1])), "f"(__uint_as_float(r[8 * g + 4 * u + 2])),
                       "f"(__uint_as_float(r[8 * g + 4 * u + 3])) : "memory");
    }
  }
}

// Descriptors of the operands: made once, then stepped (an address of shared memory never carries into the upper fields).
__device__ __forceinline__ uint64_t kmajor(uint32_t addr) { return make_smem_desc_sw128(addr, 16, 1024); }
// keeps the compiler from holding the stepped descriptors of all products in registers
__device__ __forceinline__ void here(uint64_t& a, uint64_t& b) { asm volatile("" : "+l"(a), "+l"(b)); }
constexpr uint64_t MN = (uint64_t)((BT * 128 >> 4) - 1) << 16;      // what makes it the same tile read MN-major
__device__ __forceinline__ constexpr uint64_t kstep(int kk) { return ((kk / 4) * (BT * 128) + (kk % 4) * 32) >> 4; }
__device__ __forceinline__ constexpr uint64_t mnstep(int kk) { return (kk * (16 * 128)) >> 4; }

// S^T or dP^T: D[128 x 128] = A[128 x D] B[128 x D]^T, both operands K-major tiles in shared memory
__device__ __forceinline__ void issue_kmajor(uint32_t tmem_d, uint64_t a, uint64_t b) {
  constexpr uint32_t idesc = make_idesc_bf16(BT, BT, 0, 0);
  here(a, b);
#pragma unroll
  for (int kk = 0; kk < D / 16; ++kk) umma_f16(tmem_d, a + kstep(kk), b + kstep(kk), idesc, kk > 0 ? 1u : 0u);
}

// dV: D[128 x D] (+)= A[128 x 128] B[128 x D], A = bf16 pairs in tensor memory, B MN-major.  The 16 queries of step kk
// are 8 columns; where P lies over S, every softmax warp leaves its COLS / 2 columns at the start of its COLS.
__device__ __forceinline__ void issue_dv(uint32_t tmem_d, uint32_t tmem_a, uint64_t b, bool accumulate) {
  constexpr uint32_t idesc = make_idesc_bf16(BT, D, 0, 1);
  constexpr int GROUP = COLS / 16;      // steps per softmax warp
  asm volatile("" : "+l"(b));
#pragma unroll
  for (int kk = 0; kk < BT / 16; ++kk)
    umma_f16_ts(tmem_d, tmem_a + (ROOMY ? kk * 8 : kk / GROUP * COLS + kk % GROUP * 8), b + mnstep(kk), idesc,
                (accumulate || kk > 0) ? 1u : 0u);
}

// dK: D[128 x D] (+)= dS^T[128 x 128] Q[128 x D], dS^T K-major (rows = keys, contraction over the queries)
__device__ __forceinline__ void issue_dk(uint32_t tmem_d, uint64_t ds, uint64_t b, bool accumulate) {
  constexpr uint32_t idesc = make_idesc_bf16(BT, D, 0, 1);
  here(ds, b);
#pragma unroll
  for (int kk = 0; kk < BT / 16; ++kk)
    umma_f16(tmem_d, ds + kstep(kk), b + mnstep(kk), idesc, (accumulate || kk > 0) ? 1u : 0u);
}

// dQ: D[128 x D] = dS[128 x 128] K[128 x D]: the same dS^T tile as MN-major A operand (contraction over its rows, the keys)
__device__ __forceinline__ void issue_dq(uint32_t tmem_d, uint64_t ds, uint64_t b) {
  constexpr uint32_t idesc = make_idesc_bf16(BT, D, 1, 1);
  here(ds, b);
#pragma unroll
  for (int kk = 0; kk < BT / 16; ++kk) umma_f16(tmem_d, ds + mnstep(kk), b + mnstep(kk), idesc, kk > 0 ? 1u : 0u);
}

// Waits until `want` parts have been added to a tile.
__device__ __forceinline__ bool wait_turn(const int* turn, int want, const int* given_up, volatile int* abort_flag,
                                          StatusRecord* st) {
  auto read = [&] {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(turn) : "memory");
    return v;
  };
  if (read() == want) return true;
  const uint64_t t0 = globaltimer_ns();
  for (uint32_t it = 1;; ++it) {
    if (read() == want) return true;
    if ((it & 0x3f) == 0) {
      if (*abort_flag || *reinterpret_cast<const volatile int*>(given_up)) return false;
      if (globaltimer_ns() - t0 > kSpinLimitNs) {
        report_timeout(st, 170, want, read());
        return false;
      }
    }
  }
}
__device__ __forceinline__ void pass_turn(int* turn, int value) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(turn), "r"(value) : "memory");
}

// ---------------------------------------------------------------------------
// pre-pass: delta = rowsum(O * dO), lse2 = lse * log2(e), counters and ticket cleared.  Bound by the read of O and dO:
// a CTA takes 64 tokens of one head, D / 8 lanes with 16 bytes each per row and all rows of a warp in flight, and
// writes its statistics as one run (they lie token by token, the rows head by head).  4096 tokens x 25 x 64:
// 19.3 -> 5.2 us, 8192 x 32 x 128: 53.6 -> 24.5 us (one row and 4 or 8 bytes per lane per warp, single words scattered).
// The statistics of a sequence are padded to whole tiles: +inf as log-sum-exp makes the probabilities there zero.
// WIDE: O is 16-byte aligned (dO always is, its tensor map asks for it); otherwise 4-byte aligned.
// ---------------------------------------------------------------------------
constexpr int PRE_TOKENS = 64, PRE_WARPS = 8, PRE_PER_TILE = BT / PRE_TOKENS;
template <bool WIDE>
__device__ __forceinline__ uint4 prepass_load(const __nv_bfloat16* p) {
  if (WIDE) return __ldg(reinterpret_cast<const uint4*>(p));
  const uint32_t* w = reinterpret_cast<const uint32_t*>(p);
  return make_uint4(__ldg(w), __ldg(w + 1), __ldg(w + 2), __ldg(w + 3));
}
template <bool WIDE>
__global__ void __launch_bounds__(32 * PRE_WARPS)
attn_prepass_kernel(const __nv_bfloat16* __restrict__ O, const __nv_bfloat16* __restrict__ dO,
                    const float* __restrict__ lse, float* __restrict__ delta, float* __restrict__ lse2,
                    int* __restrict__ dq_turn, int* __restrict__ kv_turn, int* __restrict__ ticket, int S, int Hq, int Hkv) {
  constexpr int LANES = D / 8, ROWS = 32 / LANES, ITERS = PRE_TOKENS / (PRE_WARPS * ROWS);
  __shared__ float s_delta[PRE_TOKENS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // a flat grid (tokens, then heads, then sequences): any number of sequences and heads, as in the kernel that follows
  const int nT = (S + BT - 1) / BT, slices = nT * PRE_PER_TILE, slice = (int)(blockIdx.x % (unsigned)slices);
  const int row = (int)(blockIdx.x / (unsigned)slices), b = row / Hq, h = row - b * Hq;
  const long long first = (long long)b * S + slice * PRE_TOKENS;
  const int live = S - slice * PRE_TOKENS;            // tokens of this slice that exist (may be none)
  const int mine = warp * ROWS * ITERS + lane / LANES;
  uint4 a[ITERS], g[ITERS];
#pragma unroll
  for (int i = 0; i < ITERS; ++i) {
    a[i] = g[i] = make_uint4(0, 0, 0, 0);
    if (mine + i * ROWS < live) {
      const long long at = ((first + mine + i * ROWS) * Hq + h) * D + (lane % LANES) * 8;
      a[i] = prepass_load<WIDE>(O + at);
      g[i] = prepass_load<true>(dO + at);
    }
  }
#pragma unroll
  for (int i = 0; i < ITERS; ++i) {
    float acc = 0.f;
    const uint32_t au[4] = {a[i].x, a[i].y, a[i].z, a[i].w}, gu[4] = {g[i].x, g[i].y, g[i].z, g[i].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 x = unpack_bf16x2(au[j]), y = unpack_bf16x2(gu[j]);
      acc += x.x * y.x + x.y * y.y;
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane % LANES == 0) s_delta[mine + i * ROWS] = acc;
  }
  __syncthreads();
  if (threadIdx.x < PRE_TOKENS) {
    const size_t o = ((size_t)row * slices + slice) * PRE_TOKENS + threadIdx.x;
    delta[o] = s_delta[threadIdx.x];
    lse2[o] = (int)threadIdx.x < live ? lse[(size_t)row * S + slice * PRE_TOKENS + threadIdx.x] * kLog2e : INFINITY;
  } else if (threadIdx.x == PRE_TOKENS && slice % PRE_PER_TILE == 0) {
    dq_turn[(size_t)row * nT + slice / PRE_PER_TILE] = 0;
    if (h < Hkv) kv_turn[((size_t)b * Hkv + h) * nT + slice / PRE_PER_TILE] = 0;
    if (blockIdx.x == 0) ticket[0] = ticket[1] = 0;
  }
}

// ---------------------------------------------------------------------------
struct Smem {
  static constexpr int TILE_BYTES = (2 + Q_STAGES + DO_STAGES) * T_BYTES;      // K, V, Q, dO
  static constexpr int STAT_BYTES = Q_STAGES * 2 * BT * 4;                     // (lse2, delta) per stage of Q
  static constexpr int TOTAL = TILE_BYTES + DS_BUFS * DS_BYTES + 2 * CHUNK_BYTES + STAT_BYTES + 256;
};
static_assert(Smem::TOTAL <= 227 * 1024, "shared memory of one CTA");
struct Barriers {
  uint64_t kv_full, q_full[Q_STAGES], q_empty[Q_STAGES], do_full[DO_STAGES], do_empty[DO_STAGES];
  uint64_t s_full, s_read, p_full, dp_full, ds_full, dq_full, dq_empty, acc_done;
  uint64_t chunk_full[2][2], chunk_empty[2];     // chunk_full: per adding warp and buffer
  uint32_t tmem_base;
  int place;
  volatile int abort_flag;
};
static_assert(sizeof(Barriers) <= 256, "barriers");

template <bool POLY>
__global__ void __launch_bounds__(NUM_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                const BwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* sK = smem_raw;
  uint8_t* sV = sK + T_BYTES;
  uint8_t* sQ = sV + T_BYTES;
  uint8_t* sdO = sQ + Q_STAGES * T_BYTES;
  uint8_t* sdS = smem_raw + Smem::TILE_BYTES;
  uint8_t* sChunk = sdS + DS_BUFS * DS_BYTES;
  float* stats = reinterpret_cast<float*>(sChunk + 2 * CHUNK_BYTES);   // [stage][lse2 128 | delta 128]
  Barriers* bar = reinterpret_cast<Barriers*>(sChunk + 2 * CHUNK_BYTES + Smem::STAT_BYTES);
  if (smem_u32(smem_raw) & 1023) {        // the swizzled tiles count on it (there is no static shared memory before them)
    if (threadIdx.x == 0) report_timeout(p.status, 171, 0, (int)smem_u32(smem_raw));
    return;
  }

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    bar->place = atomicAdd(p.ticket, 1);
    mbar_init(&bar->kv_full, 1);
    for (int s = 0; s < Q_STAGES; ++s) { mbar_init(&bar->q_full[s], 1); mbar_init(&bar->q_empty[s], 1); }
    for (int s = 0; s < DO_STAGES; ++s) { mbar_init(&bar->do_full[s], 1); mbar_init(&bar->do_empty[s], 1); }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bar->chunk_full[0][s], DRAIN_WARPS); mbar_init(&bar->chunk_full[1][s], DRAIN_WARPS);
      mbar_init(&bar->chunk_empty[s], 1);
    }
    mbar_init(&bar->s_full, 1); mbar_init(&bar->s_read, SOFTMAX_WARPS); mbar_init(&bar->p_full, SOFTMAX_WARPS);
    mbar_init(&bar->dp_full, 1); mbar_init(&bar->ds_full, SOFTMAX_WARPS);
    mbar_init(&bar->dq_full, 1); mbar_init(&bar->dq_empty, DRAIN_WARPS);
    mbar_init(&bar->acc_done, 1);
    bar->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(&bar->tmem_base, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bar->tmem_base;
  const uint32_t tS = tmem_base, tdP = tmem_base + 128, tdV = tmem_base + 256, tdK = tmem_base + 256 + D;
  const uint32_t tdQ = ROOMY ? tmem_base + 256 + 2 * D : tdP, tP = ROOMY ? tmem_base + 256 + 3 * D : tS;

  const int nT = (p.S + BT - 1) / BT;
  // small j first: the long sweeps of a causal call, and the order of the counters
  int place = bar->place;
  const int hb = place % (p.Hkv * p.batch);
  place /= p.Hkv * p.batch;
  const int part = place % p.split, j = place / p.split;
  const int hkv = hb % p.Hkv, b = hb / p.Hkv;
  const int heads = p.Hq / p.Hkv / p.split;                  // query heads of this CTA
  const int h0 = (hkv * p.split + part) * heads;
  const int per_head = p.causal ? nT - j : nT;
  const int iters = heads * per_head;
  // iteration it: query tile nT - 1 - it % per_head of head h0 + it / per_head

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_ISSUE));
    if (warp == 0) {
      // ------------------------------ TMA producer ------------------------------
      if (elect_one()) {
        tma_prefetch_desc(&tmap_q); tma_prefetch_desc(&tmap_k); tma_prefetch_desc(&tmap_v); tma_prefetch_desc(&tmap_do);
        mbar_expect_tx(&bar->kv_full, 2 * T_BYTES);
#pragma unroll
        for (int c = 0; c < DCH; ++c) {
          tma_load_4d(sK + c * (BT * 128), &tmap_k, &bar->kv_full, c * 64, j * BT, hkv, b);
          tma_load_4d(sV + c * (BT * 128), &tmap_v, &bar->kv_full, c * 64, j * BT, hkv, b);
        }
        bool ok = true;
        for (int it = 0; it < iters && ok; ++it) {
          const int h = h0 + it / per_head;
          const int i = nT - 1 - it % per_head;
          const int st = it % Q_STAGES, ot = it % DO_STAGES;
          ok = mbar_wait(&bar->q_empty[st], ((it / Q_STAGES) & 1) ^ 1, &bar->abort_flag, p.status, 131);
          if (!ok) break;
          mbar_expect_tx(&bar->q_full[st], T_BYTES + 2 * BT * 4);
#pragma unroll
          for (int c = 0; c < DCH; ++c)
            tma_load_4d(sQ + st * T_BYTES + c * (BT * 128), &tmap_q, &bar->q_full[st], c * 64, i * BT, h, b);
          const size_t stat = (((size_t)b * p.Hq + h) * nT + i) * BT;
          bulk_load(stats + st * 2 * BT, p.lse2 + stat, BT * 4, &bar->q_full[st]);
          bulk_load(stats + st * 2 * BT + BT, p.delta + stat, BT * 4, &bar->q_full[st]);
          ok = mbar_wait(&bar->do_empty[ot], ((it / DO_STAGES) & 1) ^ 1, &bar->abort_flag, p.status, 132);
          if (!ok) break;
          mbar_expect_tx(&bar->do_full[ot], T_BYTES);
#pragma unroll
          for (int c = 0; c < DCH; ++c)
            tma_load_4d(sdO + ot * T_BYTES + c * (BT * 128), &tmap_do, &bar->do_full[ot], c * 64, i * BT, h, b);
        }
        if (!ok) {
          const uint64_t t0 = globaltimer_ns();
          while (globaltimer_ns() - t0 < 1000000ull) __nanosleep(1000);
        }
      }
    } else if (warp == 1) {
      // ------------------------------- MMA issuer -------------------------------
      if (elect_one()) {
        const uint64_t kK = kmajor(smem_u32(sK)), kV = kmajor(smem_u32(sV)), kQ = kmajor(smem_u32(sQ)),
                       kdO = kmajor(smem_u32(sdO)), kdS = kmajor(smem_u32(sdS));
        auto s_of = [&](int it) -> bool {                              // S^T(it)
          const int st = it % Q_STAGES;
          if (!mbar_wait(&bar->q_full[st], (it / Q_STAGES) & 1, &bar->abort_flag, p.status, 137)) return false;
          tc_fence_after();
          issue_kmajor(tS, kK, kQ + st * (T_BYTES >> 4));
          umma_commit(&bar->s_full);
          return true;
        };
        auto dp_of = [&](int it) -> bool {                             // dP^T(it)
          const int ot = it % DO_STAGES;
          if (!mbar_wait(&bar->do_full[ot], (it / DO_STAGES) & 1, &bar->abort_flag, p.status, 139)) return false;
          tc_fence_after();
          issue_kmajor(tdP, kV, kdO + ot * (T_BYTES >> 4));
          umma_commit(&bar->dp_full);
          return true;
        };
        bool ok = mbar_wait(&bar->kv_full, 0, &bar->abort_flag, p.status, 133);
        if (ok) ok = s_of(0);
        if (ok) ok = dp_of(0);
        for (int it = 0; it < iters && ok; ++it) {
          const int st = it % Q_STAGES, ot = it % DO_STAGES, ds = (it % DS_BUFS) * (DS_BYTES >> 4);
          const bool more = it + 1 < iters;
          if (ROOMY && more) {
            // S has been read: the next one at once
            ok = mbar_wait(&bar->s_read, it & 1, &bar->abort_flag, p.status, 135);
            if (ok) ok = s_of(it + 1);
            if (!ok) break;
          }
          ok = mbar_wait(&bar->p_full, it & 1, &bar->abort_flag, p.status, 136);
          if (!ok) break;
          tc_fence_after();
          issue_dv(tdV, tP, kdO + MN + ot * (T_BYTES >> 4), it > 0);        // dV += P^T dO
          umma_commit(&bar->do_empty[ot]);
          if (!ROOMY && more) {
            ok = s_of(it + 1);                                         // over P, which dV has been issued to read
            if (!ok) break;
          }
          ok = mbar_wait(&bar->ds_full, it & 1, &bar->abort_flag, p.status, 138);
          if (!ok) break;
          if (ROOMY) {
            // dP has been read (dS is written): the next one first, the softmax warps wait for it
            if (more) ok = dp_of(it + 1);
            if (ok && it > 0) ok = mbar_wait(&bar->dq_empty, (it - 1) & 1, &bar->abort_flag, p.status, 144);
            if (!ok) break;
          }
          tc_fence_after();
          issue_dq(tdQ, kdS + MN + ds, kK + MN);                                 // dQ = dS K
          umma_commit(&bar->dq_full);
          issue_dk(tdK, kdS + ds, kQ + MN + st * (T_BYTES >> 4), it > 0);   // dK += dS^T Q
          umma_commit(&bar->q_empty[st]);
          if (!ROOMY && more) {
            ok = mbar_wait(&bar->dq_empty, it & 1, &bar->abort_flag, p.status, 144);
            if (ok) ok = dp_of(it + 1);
          }
        }
        if (ok) umma_commit(&bar->acc_done);
      }
    } else {
      // ---------------------- adds the dQ tiles, one warp the even ones, one the odd ones ----------------------
      if (elect_one()) {
        bool ok = true;
        int phase = 0;                                          // of either of this warp's two barriers
        for (int it = warp - 2; it < iters && ok; it += 2) {
          const int i = nT - 1 - it % per_head;
          const size_t tile = ((size_t)b * p.Hq + h0 + it / per_head) * nT + i;
          if (p.causal ? i == j : j == nT - 1) continue;        // the drain warps finish it themselves
          if (j > 0) {
            ok = wait_turn(p.dq_turn + tile, j, p.ticket + 1, &bar->abort_flag, p.status);
            if (!ok) { bar->abort_flag = 1; break; }
            fence_proxy_async();           // the sums it now adds to were written by another CTA's bulk copies
          }
          for (int ch = 0; ch < CHUNKS; ++ch) {
            ok = mbar_wait(&bar->chunk_full[it & 1][ch & 1], (phase + (ch >> 1)) & 1, &bar->abort_flag, p.status, 146);
            if (!ok) break;
            bulk_put(p.dq_sum + tile * (BT * D) + ch * (BT * 32), smem_u32(sChunk) + (ch & 1) * CHUNK_BYTES, j > 0);
            tma_store_commit();
            if (ch > 0) {
              asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
              mbar_arrive(&bar->chunk_empty[(ch - 1) & 1]);
            }
          }
          phase += CHUNKS / 2;
          tma_store_wait_read();
          if (ok) mbar_arrive(&bar->chunk_empty[(CHUNKS - 1) & 1]);
          tma_store_wait_all();
          if (ok) pass_turn(p.dq_turn + tile, j + 1);
        }
      }
    }
  } else if (warp < 4 + SOFTMAX_WARPS) {
    // -------------------------------- softmax --------------------------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_SOFTMAX));
    const int quarter = warp & 3;                   // tensor-memory lane quarter this warp may access
    const int cg = (warp - 4) >> 2;                 // its COLS queries
    const int row = quarter * 32 + lane;            // key row inside the tile
    const bool live = j * BT + row < p.S;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const uint32_t myS = tS + lane_off + cg * COLS, mydP = tdP + lane_off + cg * COLS;
    const uint32_t myP = tP + lane_off + cg * (ROOMY ? COLS / 2 : COLS);
    // row of the dS^T tile: 64 queries are 128 bytes, their 16-byte units swizzled
    const uint32_t ds_row = smem_u32(sdS) + cg * COLS / 64 * (BT * 128) + row * 128;
    const int unit0 = cg * COLS % 64 / 8;
    const float c = p.scale * kLog2e;
    const uint64_t nc2 = pack_f32x2(-c, -c);
    bool ok = true;
    for (int it = 0; it < iters && ok; ++it) {
      const int st = it % Q_STAGES;
      const bool diag = p.causal && it % per_head == per_head - 1;
      ok = mbar_wait(&bar->q_full[st], (it / Q_STAGES) & 1, &bar->abort_flag, p.status, 140);   // statistics
      if (!ok) break;
      ok = mbar_wait(&bar->s_full, it & 1, &bar->abort_flag, p.status, 141);
      if (!ok) break;
      tc_fence_after();
      float pr[COLS];
      {
        uint32_t s[COLS];
#pragma unroll
        for (int ch = 0; ch < COLS; ch += 32) tmem_ld_32x32(myS + ch, *reinterpret_cast<uint32_t(*)[32]>(s + ch));
        const float4* L4 = reinterpret_cast<const float4*>(stats + st * 2 * BT + cg * COLS);
        tmem_ld_wait();
        if (ROOMY) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar->s_read);
        }
#pragma unroll
        for (int g = 0; g < COLS / 4; ++g) {
          const float4 l = L4[g];
          // (two values per instruction, of l - s c: its negation comes with the exponential)
          const float2 x = unpack_f32x2(fma_f32x2(pack_u32x2(s[4 * g], s[4 * g + 1]), nc2, pack_f32x2(l.x, l.y)));
          const float2 z = unpack_f32x2(fma_f32x2(pack_u32x2(s[4 * g + 2], s[4 * g + 3]), nc2, pack_f32x2(l.z, l.w)));
          pr[4 * g] = exp2_mixed<POLY>(-x.x, 4 * g);
          pr[4 * g + 1] = exp2_mixed<POLY>(-x.y, 4 * g + 1);
          pr[4 * g + 2] = exp2_mixed<POLY>(-z.x, 4 * g + 2);
          pr[4 * g + 3] = exp2_mixed<POLY>(-z.y, 4 * g + 3);
        }
      }
      if (diag) {
        // query cg * COLS + k sees key `row` only if it is not earlier than the key
#pragma unroll
        for (int k = 0; k < COLS; ++k)
          if (cg * COLS + k < row) pr[k] = 0.f;
      }
      if (j * BT + BT > p.S) {
        if (!live) {
#pragma unroll
          for (int k = 0; k < COLS; ++k) pr[k] = 0.f;
        }
        __syncwarp();             // (what follows is of the whole warp)
      }
      if (ROOMY && it > 0) {     // dV of the iteration before has read P
        ok = mbar_wait(&bar->do_empty[(it - 1) % DO_STAGES], ((it - 1) / DO_STAGES) & 1, &bar->abort_flag, p.status, 149);
        if (!ok) break;
        tc_fence_after();
      }
#pragma unroll
      for (int part32 = 0; part32 < COLS; part32 += 32) {
        uint32_t packed[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) packed[k] = pack_bf16x2(pr[part32 + 2 * k], pr[part32 + 2 * k + 1]);
        tmem_st_32x16(myP + part32 / 2, packed);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->p_full);
      // this also says that dQ and dK of the iteration DS_BUFS before have been multiplied: their dS tile is free
      ok = mbar_wait(&bar->dp_full, it & 1, &bar->abort_flag, p.status, 142);
      if (!ok) break;
      tc_fence_after();
      const uint32_t out = ds_row + (it % DS_BUFS) * DS_BYTES;
      const float4* D4 = reinterpret_cast<const float4*>(stats + st * 2 * BT + BT + cg * COLS);
#pragma unroll
      for (int ch = 0; ch < COLS; ch += 32) {
        uint32_t dp[32];
        tmem_ld_32x32(mydP + ch, dp);
        tmem_ld_wait();
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const float4 l = D4[ch / 4 + 2 * g], l2 = D4[ch / 4 + 2 * g + 1];
          const float* q = pr + ch + 8 * g;
          const uint32_t* d = dp + 8 * g;
          const uint32_t w0 = scaled_diff_bf16x2(q[0], q[1], d[0], d[1], l.x, l.y);
          const uint32_t w1 = scaled_diff_bf16x2(q[2], q[3], d[2], d[3], l.z, l.w);
          const uint32_t w2 = scaled_diff_bf16x2(q[4], q[5], d[4], d[5], l2.x, l2.y);
          const uint32_t w3 = scaled_diff_bf16x2(q[6], q[7], d[6], d[7], l2.z, l2.w);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                       ::"r"(out + (((unit0 + ch / 8 + g) ^ (row & 7)) << 4)), "r"(w0), "r"(w1), "r"(w2), "r"(w3)
                       : "memory");
        }
      }
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->ds_full);
    }
    if (ok) ok = mbar_wait(&bar->acc_done, 0, &bar->abort_flag, p.status, 143);
    const size_t kv_tile = ((size_t)b * p.Hkv + hkv) * nT + j;
    if (part > 0) {
      if (ok && lane == 0) ok = wait_turn(p.kv_turn + kv_tile, part, p.ticket + 1, &bar->abort_flag, p.status);
      ok = __all_sync(0xffffffffu, ok);
      __syncwarp();             // orders the other lanes' accesses after lane 0's acquire, as the vote does not
      if (!ok) bar->abort_flag = 1;
    }
    if (ok) {
      tc_fence_after();
      const long long t = (long long)b * p.S + j * BT + row;
      __nv_bfloat16* dv = p.dv + t * p.dv_row + (long long)hkv * p.dv_head;
      __nv_bfloat16* dk = p.dk + t * p.dk_row + (long long)hkv * p.dk_head;
      float* sum = p.kv_sum + kv_tile * (2 * BT * D) + row * 4;
      // sixteen warps: half of the columns of dV or of dK each; eight: half of both
#pragma unroll
      for (int ch = 0; ch < D / 2; ch += 32) {
        const int at = cg % 2 * (D / 2) + ch;
        if (!ROOMY || cg < 2) put_cols32(tdV + lane_off, dv, sum, at, 1.f, part == 0, part == p.split - 1, live);
        if (!ROOMY || cg >= 2)
          put_cols32(tdK + lane_off, dk, sum + BT * D, at, p.scale, part == 0, part == p.split - 1, live);
      }
    }
    if (p.split > 1 && part < p.split - 1) {
      asm volatile("barrier.cta.sync 1, %0;" ::"n"(32 * SOFTMAX_WARPS) : "memory");
      if (threadIdx.x == 128 && !bar->abort_flag) pass_turn(p.kv_turn + kv_tile, part + 1);
    }
  } else {
    // ------------------------------- dQ drain --------------------------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_DRAIN));
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;            // query row inside the tile
    const uint32_t src = tdQ + ((uint32_t)(quarter * 32) << 16);
    bool ok = true;
    int chunk = 0;                                  // chunks written so far: buffer and phase
    for (int it = 0; it < iters && ok; ++it) {
      const int h = h0 + it / per_head;
      const int i = nT - 1 - it % per_head;
      const size_t tile = ((size_t)b * p.Hq + h) * nT + i;
      const bool last = p.causal ? i == j : j == nT - 1;
      uint32_t r[D];
      ok = mbar_wait(&bar->dq_full, it & 1, &bar->abort_flag, p.status, 145);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int ch = 0; ch < D; ch += 32) tmem_ld_32x32(src + ch, *reinterpret_cast<uint32_t(*)[32]>(r + ch));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->dq_empty);
      if (!last) {
#pragma unroll
        for (int ch = 0; ch < CHUNKS; ++ch, ++chunk) {
          ok = mbar_wait(&bar->chunk_empty[ch & 1], ((chunk >> 1) & 1) ^ 1, &bar->abort_flag, p.status, 147);
          if (!ok) break;
          uint4* at = reinterpret_cast<uint4*>(sChunk + (ch & 1) * CHUNK_BYTES) + row;
#pragma unroll
          for (int g = 0; g < 8; ++g)
            at[g * BT] = make_uint4(r[32 * ch + 4 * g], r[32 * ch + 4 * g + 1], r[32 * ch + 4 * g + 2], r[32 * ch + 4 * g + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar->chunk_full[it & 1][ch & 1]);
        }
        continue;
      }
      if (j > 0) {
        if (lane == 0) ok = wait_turn(p.dq_turn + tile, j, p.ticket + 1, &bar->abort_flag, p.status);
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) { bar->abort_flag = 1; break; }
        __syncwarp();           // orders the other lanes' reads after lane 0's acquire, as the shuffle does not
        fence_proxy_async();
      }
      if (i * BT + row < p.S) {
        const float* at = p.dq_sum + tile * (BT * D) + row * 4;
        __nv_bfloat16* dq = p.dq + ((long long)b * p.S + i * BT + row) * p.dq_row + (long long)h * p.dq_head;
#pragma unroll
        for (int g = 0; g < D / 8; ++g) {
          float4 a = make_float4(0.f, 0.f, 0.f, 0.f), e = a;
          if (j > 0) {
            a = __ldcg(reinterpret_cast<const float4*>(at + 2 * g * (BT * 4)));
            e = __ldcg(reinterpret_cast<const float4*>(at + (2 * g + 1) * (BT * 4)));
          }
          *reinterpret_cast<uint4*>(dq + 8 * g) = pack8(r + 8 * g, p.scale, a, e);
        }
      }
      __syncwarp();               // (the next tile is read by the whole warp)
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && bar->abort_flag) p.ticket[1] = 1;
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

int run(const void* q, long long q_row, long long q_head, const void* k, long long k_row, long long k_head,
        const void* v, long long v_row, long long v_head, const void* out, const void* dout, const float* lse,
        float* scratch, long long words, void* dq, long long dq_row, long long dq_head, void* dk, long long dk_row,
        long long dk_head, void* dv, long long dv_row, long long dv_head, int batch, int S, int Hq, int Hkv, int causal,
        float scale, void* stream) {
  if (S <= 0 || batch <= 0 || Hkv <= 0 || Hq <= 0 || Hq % Hkv != 0) return DD_ERR_BAD_ARG;
  if ((dq_row | dq_head | dk_row | dk_head | dv_row | dv_head) % 8) return DD_ERR_ALIGN;
  if ((reinterpret_cast<uintptr_t>(dq) | reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv) |
       reinterpret_cast<uintptr_t>(scratch)) & 15)
    return DD_ERR_ALIGN;
  if ((reinterpret_cast<uintptr_t>(dout) & 15) || (reinterpret_cast<uintptr_t>(out) & 3)) return DD_ERR_ALIGN;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const int nT = S / BT + (S % BT != 0);
  const long long tiles = (long long)batch * Hq * nT, kv_tiles = (long long)batch * Hkv * nT;
  if (tiles * PRE_PER_TILE > 0x7fffffffLL) return DD_ERR_TOO_LARGE;
  const int split = bwd3_split(batch, nT, Hq, Hkv, causal);
  // scratch: delta and lse2, then ticket (4 words) and counters, then the sums, at a multiple of 4 words
  BwdParams p;
  float* delta = scratch;
  float* lse2 = delta + tiles * BT;
  p.ticket = reinterpret_cast<int*>(lse2 + tiles * BT);
  p.dq_turn = p.ticket + 4;
  p.kv_turn = p.dq_turn + tiles;
  p.dq_sum = reinterpret_cast<float*>(p.dq_turn + (2 * tiles + 3) / 4 * 4);
  p.kv_sum = p.dq_sum + (nT > 1 ? tiles * (BT * D) : 0);
  if (bwd3_words(batch, S, Hq, Hkv, D, causal) > words) return DD_ERR_TOO_LARGE;
  CUtensorMap tq, tk, tv, tdo;
  int r = get_tensor_map_bf16_4d(&tq, q, D, S, Hq, batch, q_row * 2, q_head * 2, (uint64_t)S * q_row * 2, 64, BT);
  if (!r) r = get_tensor_map_bf16_4d(&tk, k, D, S, Hkv, batch, k_row * 2, k_head * 2, (uint64_t)S * k_row * 2, 64, BT);
  if (!r) r = get_tensor_map_bf16_4d(&tv, v, D, S, Hkv, batch, v_row * 2, v_head * 2, (uint64_t)S * v_row * 2, 64, BT);
  if (!r)
    r = get_tensor_map_bf16_4d(&tdo, dout, D, S, Hq, batch, (uint64_t)Hq * D * 2, (uint64_t)D * 2, (uint64_t)S * Hq * D * 2,
                               64, BT);
  if (r) return r;
  int err = 0;
  p.lse2 = lse2; p.delta = delta;
  p.dq = reinterpret_cast<__nv_bfloat16*>(dq); p.dq_row = dq_row; p.dq_head = dq_head;
  p.dk = reinterpret_cast<__nv_bfloat16*>(dk); p.dk_row = dk_row; p.dk_head = dk_head;
  p.dv = reinterpret_cast<__nv_bfloat16*>(dv); p.dv_row = dv_row; p.dv_head = dv_head;
  p.S = S; p.Hq = Hq; p.Hkv = Hkv; p.batch = batch; p.causal = causal; p.split = split; p.scale = scale;
  p.status = device_status(&err);
  if (err) return err;
  // DISTDL_ATTN_EXP_POLY=1: a third of the exponentials on the FMA pipe (see exp2_fma)
  static const bool poly = [] { const char* e = getenv("DISTDL_ATTN_EXP_POLY"); return e != nullptr && e[0] == '1'; }();
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(attn_bwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem::TOTAL);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(attn_bwd_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem::TOTAL);
    if (e != cudaSuccess) return (int)e;
    configured[dev & 63] = true;
  }
  auto prepass = (reinterpret_cast<uintptr_t>(out) & 15) == 0 ? attn_prepass_kernel<true> : attn_prepass_kernel<false>;
  prepass<<<(unsigned)(tiles * PRE_PER_TILE), 32 * PRE_WARPS, 0, s>>>(
      reinterpret_cast<const __nv_bfloat16*>(out), reinterpret_cast<const __nv_bfloat16*>(dout), lse, delta, lse2,
      p.dq_turn, p.kv_turn, p.ticket, S, Hq, Hkv);
  r = (int)cudaGetLastError();
  if (r) return r;
  (poly ? attn_bwd_kernel<true> : attn_bwd_kernel<false>)<<<(unsigned)(kv_tiles * split), NUM_THREADS, Smem::TOTAL, s>>>(
      tq, tk, tv, tdo, p);
  return (int)cudaGetLastError();
}

}  // namespace DD_BWD3_NS
