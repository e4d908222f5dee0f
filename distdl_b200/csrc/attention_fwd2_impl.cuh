// Flash attention forward, two query tiles per CTA ("ping-pong"); head dim DD_HEAD_DIM (128 or 64:
// this file is included once per head dimension by attention_fwd2.cu, inside namespace DD_FWD2_NS).
//
// One CTA handles 256 query rows of one (batch, head) as two 128-row tiles:
//   warp 0        TMA producer: both Q tiles once, then K_j / V_j (2-stage rings)
//   warp 1        MMA issuer:   S_t = Q_t K_j^T and O_t += P_t V_j for t = 0, 1
//   warps 2..5    softmax of tile 0 (one thread per query row)
//   warps 6..9    softmax of tile 1
// Tensor memory (512 columns): S_0 | S_1 | O_0 | O_1, 128 fp32 columns each (O_t uses the first
// DD_HEAD_DIM of its 128).  The
// probabilities never touch shared memory: a softmax thread reads its row of S_t
// into registers, and writes P_t (bf16 pairs) back over the first 64 columns of
// S_t with tcgen05.st; the second product takes its A operand from tensor memory.
// O_t stays in tensor memory for the whole row of blocks; it is rescaled only when
// the running maximum has grown by more than 2^8 since the last rescale (the
// probabilities then exceed 1 by at most that factor, which fp32 sums and bf16
// probabilities absorb), and the final 1 / l scaling happens on the way out.
// While tile 0's softmax runs, the tensor cores work on tile 1, and vice versa.
//
// Issue order per KV block j:  PV_0(j), S_0(j+1), PV_1(j), S_1(j+1); products of
// one thread execute in order, so S_t(j+1) may overwrite P_t(j) right after PV_t(j)
// was issued (head dim 64: S_0(j+1), S_1(j+1), PV_0(j), PV_1(j)).  Causal: tile t of query pair qp sees blocks 0 .. 2 qp + t.
// Any sequence length: rows behind the end of a sequence are read as zeros (the tensor maps end there), keys there are
// masked in the last block, queries there are not stored, and a pair's second tile may not exist at all.
// What bounds it: a tile's softmax (1 900 clocks a block, of which the exponentials alone 1 024) and its two products
// (1 030) follow one another, and two tiles do not fill the tensor cores (56 % active at head dim 128).  So the chain is
// kept short: the maximum in four chains, two values per fma / add instruction, and P_t V_j starts on three quarters of P_t.
// Causal 1 x 16384, 32 / 8 heads of 128: 2 083 -> 1 947 us, full 1 x 4096, 16 heads 145 -> 136.
// At head dim 64 P_t has columns of its own (OWN_P), and S_t(j + 1) is formed before P_t(j) V_j: full 1 x 16384, 16 heads
// 1 609 -> 1 439 us, 8 x 1536 158 -> 142, causal 4 x 1024, 25 heads 43.0 -> 37.7.
// All waits are bounded; a timeout drains and frees tensor memory.
namespace DD_FWD2_NS {

constexpr int BQ = 128;
constexpr int BKV = 128;
constexpr int D = DD_HEAD_DIM;
constexpr int KV_STAGES = 2;
// Head dim 64 leaves half of O_t's columns to P_t, so that S_t(j + 1) need not wait for P_t(j) V_j: the tensor cores form it
// while the softmax threads work on block j.
constexpr bool OWN_P = D == 64;
constexpr int P_COL = OWN_P ? 256 + 64 : 0;       // first column of P_0; P_1 128 further
constexpr int P_SPLIT = 96;               // P_t V starts when this many columns of P_t are written
constexpr int NUM_THREADS = 320;
constexpr int Q_BYTES = BQ * D * 2;       // one query tile
constexpr int KV_BYTES = BKV * D * 2;
constexpr int TILE_BYTES = 2 * Q_BYTES + 2 * KV_STAGES * KV_BYTES;
constexpr int SMEM_TOTAL = 1024 + TILE_BYTES + 256;

struct Barriers {
  uint64_t q_full;
  uint64_t k_full[KV_STAGES], k_empty[KV_STAGES];
  uint64_t v_full[KV_STAGES], v_empty[KV_STAGES];
  uint64_t s_full[2];      // S_t complete (tensor core -> softmax)
  uint64_t s_free[2];      // S_t read into registers (softmax -> tensor core), 4 warps arrive; where P_t has columns of its own
  uint64_t p_most[2];      // the first P_SPLIT columns of P_t written, S_t consumed (softmax -> tensor core), 4 warps arrive
  uint64_t p_full[2];      // all of P_t written, 4 warps arrive
  uint64_t pv_done[2];     // O_t += P_t V complete
  uint32_t tmem_base;
  volatile int abort_flag;
};

struct Params2 {
  __nv_bfloat16* O;     // [tokens][Hq][D]
  float* lse;           // [batch][Hq][S]
  int S, Hq, Hkv, batch;
  int causal;
  float scale;
  StatusRecord* status;
};

// PAIRS: the sequence is whole pairs of tiles, so that nothing is masked but the diagonal.  The softmax threads are short of
// registers; the general form spills a third more (head dim 64, causal, 32 / 8 heads, us, one form for all lengths -> PAIRS:
// 8 x 1024 100.4 -> 94.3, 1 x 1024 22.5 -> 20.5, 1 x 16384 1 733 -> 1 644).
template <bool POLY, bool PAIRS>
__global__ void __launch_bounds__(NUM_THREADS, 1)
attn_fwd2_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                 const __grid_constant__ CUtensorMap tmap_v, const Params2 p) {
  constexpr int DCH = D / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = tiles;                          // two tiles back to back
  uint8_t* sK = sQ + 2 * Q_BYTES;
  uint8_t* sV = sK + KV_STAGES * KV_BYTES;
  Barriers* bar = reinterpret_cast<Barriers*>(tiles + TILE_BYTES);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nkv = (p.S + BKV - 1) / BKV;
  const int nQP = (nkv + 1) / 2;
  // heaviest query pairs first; heads vary fastest (kv heads shared through L2)
  const int id = blockIdx.x;
  const int hb = id % (p.Hq * p.batch);
  const int qp = nQP - 1 - id / (p.Hq * p.batch);
  const int h = hb % p.Hq, b = hb / p.Hq;
  const int hkv = h / (p.Hq / p.Hkv);
  const int n0 = p.causal ? 2 * qp + 1 : nkv;      // blocks seen by tile 0
  const int n1 = !PAIRS && 2 * qp + 1 >= nkv ? 0 : p.causal ? 2 * qp + 2 : nkv;      // blocks seen by tile 1 (>= n0, or none)
  const int blocks = PAIRS || n1 > n0 ? n1 : n0;
  const int q_row0 = qp * 2 * BQ;                  // of this sequence

  if (threadIdx.x == 0) {
    mbar_init(&bar->q_full, 1);
    for (int s = 0; s < KV_STAGES; ++s) {
      mbar_init(&bar->k_full[s], 1); mbar_init(&bar->k_empty[s], 1);
      mbar_init(&bar->v_full[s], 1); mbar_init(&bar->v_empty[s], 1);
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(&bar->s_full[t], 1);
      mbar_init(&bar->s_free[t], 4);
      mbar_init(&bar->p_most[t], 4);
      mbar_init(&bar->p_full[t], 4);
      mbar_init(&bar->pv_done[t], 1);
    }
    bar->abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 1) { tmem_alloc(&bar->tmem_base, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bar->tmem_base;
  grid_dependency_launch();

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (elect_one()) {
      tma_prefetch_desc(&tmap_q); tma_prefetch_desc(&tmap_k); tma_prefetch_desc(&tmap_v);
      mbar_expect_tx(&bar->q_full, 2 * Q_BYTES);
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int c = 0; c < DCH; ++c)
          tma_load_4d(sQ + t * Q_BYTES + c * (BQ * 128), &tmap_q, &bar->q_full, c * 64, q_row0 + t * BQ, h, b);
      bool ok = true;
      for (int j = 0; j < blocks && ok; ++j) {
        const int st = j % KV_STAGES;
        const uint32_t ph = (j / KV_STAGES) & 1;
        ok = mbar_wait(&bar->k_empty[st], ph ^ 1, &bar->abort_flag, p.status, 31);
        if (!ok) break;
        mbar_expect_tx(&bar->k_full[st], KV_BYTES);
#pragma unroll
        for (int c = 0; c < DCH; ++c)
          tma_load_4d(sK + st * KV_BYTES + c * (BKV * 128), &tmap_k, &bar->k_full[st], c * 64, j * BKV, hkv, b);
        ok = mbar_wait(&bar->v_empty[st], ph ^ 1, &bar->abort_flag, p.status, 32);
        if (!ok) break;
        mbar_expect_tx(&bar->v_full[st], KV_BYTES);
#pragma unroll
        for (int c = 0; c < DCH; ++c)
          tma_load_4d(sV + st * KV_BYTES + c * (BKV * 128), &tmap_v, &bar->v_full[st], c * 64, j * BKV, hkv, b);
      }
      if (!ok) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 1000000ull) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------- MMA issuer -------------------------------
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc_bf16(BQ, BKV, 0, 0);   // Q, K both K-major
      constexpr uint32_t idesc_pv = make_idesc_bf16(BQ, D, 0, 1);    // P (tensor memory), V MN-major
      bool ok = mbar_wait(&bar->q_full, 0, &bar->abort_flag, p.status, 33);
      // S_t(j) = Q_t K_j^T; the caller has made sure that K_j is in shared memory
      auto issue_S = [&](int t, int j) {
        const int st = j % KV_STAGES;
        const uint32_t q_addr = smem_u32(sQ + t * Q_BYTES), k_addr = smem_u32(sK + st * KV_BYTES);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (kk / 4) * (BQ * 128) + (kk % 4) * 32;
          umma_f16(tmem_base + t * 128, make_smem_desc_sw128(q_addr + off, 16, 1024),
                   make_smem_desc_sw128(k_addr + off, 16, 1024), idesc_s, kk > 0 ? 1u : 0u);
        }
        umma_commit(&bar->s_full[t]);
      };
      auto issue_PV = [&](int t, int j, int from, int to) {
        const int st = j % KV_STAGES;
        const uint32_t v_addr = smem_u32(sV + st * KV_BYTES);
#pragma unroll
        for (int kk = from / 16; kk < to / 16; ++kk)      // 16 kv rows = 8 columns of packed P
          umma_f16_ts(tmem_base + 256 + t * 128, tmem_base + P_COL + t * 128 + kk * 8,
                      make_smem_desc_sw128(v_addr + kk * (16 * 128), BKV * 128, 1024), idesc_pv,
                      (j > 0 || kk > 0) ? 1u : 0u);
      };
      if (ok) ok = mbar_wait(&bar->k_full[0], 0, &bar->abort_flag, p.status, 34);
      if (ok) {
        tc_fence_after();
        issue_S(0, 0);
        if (PAIRS || n1 > 0) issue_S(1, 0);
        if (OWN_P) umma_commit(&bar->k_empty[0]);
      }
      for (int j = 0; j < blocks && ok; ++j) {
        const int st = j % KV_STAGES;
        const uint32_t ph = (j / KV_STAGES) & 1;
        const int stn = (j + 1) % KV_STAGES;
        const uint32_t phn = ((j + 1) / KV_STAGES) & 1;
        bool k_next_ready = false;
        if (OWN_P && j + 1 < blocks) {
          for (int t = 0; t < 2 && ok; ++t) {
            if (j + 1 >= (t == 0 ? n0 : n1)) continue;
            if (!k_next_ready) ok = mbar_wait(&bar->k_full[stn], phn, &bar->abort_flag, p.status, 37);
            k_next_ready = true;
            if (ok) ok = mbar_wait(&bar->s_free[t], j & 1, &bar->abort_flag, p.status, 43);
            if (!ok) break;
            tc_fence_after();
            issue_S(t, j + 1);
          }
          if (!ok) break;
          umma_commit(&bar->k_empty[stn]);
        }
        ok = mbar_wait(&bar->v_full[st], ph, &bar->abort_flag, p.status, 35);
        if (!ok) break;
        for (int t = 0; t < 2 && ok; ++t) {
          const int nt = t == 0 ? n0 : n1;
          if (j >= nt) continue;
          ok = mbar_wait(&bar->p_most[t], j & 1, &bar->abort_flag, p.status, 36);
          if (!ok) break;
          tc_fence_after();
          issue_PV(t, j, 0, P_SPLIT);
          ok = mbar_wait(&bar->p_full[t], j & 1, &bar->abort_flag, p.status, 41);
          if (!ok) break;
          tc_fence_after();
          issue_PV(t, j, P_SPLIT, BKV);
          umma_commit(&bar->pv_done[t]);
          if (!OWN_P && j + 1 < nt) {
            if (!k_next_ready) {
              ok = mbar_wait(&bar->k_full[stn], phn, &bar->abort_flag, p.status, 37);
              if (!ok) break;
              tc_fence_after();
              k_next_ready = true;
            }
            issue_S(t, j + 1);
          }
        }
        if (!ok) break;
        // V_j is free once the products of both tiles are through; K_j was last read by
        // the S products of block j, which precede these commits in issue order
        umma_commit(&bar->v_empty[st]);
        if (!OWN_P) umma_commit(&bar->k_empty[st]);
      }
    }
  } else {
    // -------------------------------- softmax --------------------------------
    const int t = (warp - 2) >> 2;                  // query tile of this warpgroup
    const int quarter = warp & 3;                   // tensor-memory lane quarter this warp may access
    const int row = quarter * 32 + lane;            // row inside the tile
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const uint32_t tS = tmem_base + t * 128 + lane_off;
    const uint32_t tP = tmem_base + P_COL + t * 128 + lane_off;
    const uint32_t tO = tmem_base + 256 + t * 128 + lane_off;
    const int nt = t == 0 ? n0 : n1;
    const float c = p.scale * 1.4426950408889634f;  // scores are exponentiated base 2
    float m_ref = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < nt && ok; ++j) {
      ok = mbar_wait(&bar->s_full[t], j & 1, &bar->abort_flag, p.status, 38);
      if (!ok) break;
      tc_fence_after();
      uint32_t s[128];
      tmem_ld_32x32(tS, *reinterpret_cast<uint32_t(*)[32]>(s));
      tmem_ld_32x32(tS + 32, *reinterpret_cast<uint32_t(*)[32]>(s + 32));
      tmem_ld_32x32(tS + 64, *reinterpret_cast<uint32_t(*)[32]>(s + 64));
      tmem_ld_32x32(tS + 96, *reinterpret_cast<uint32_t(*)[32]>(s + 96));
      tmem_ld_wait();
      if (OWN_P) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar->s_free[t]);
      }
      float top[4] = {m_ref, -INFINITY, -INFINITY, -INFINITY};      // four chains: one of 128 steps waits for itself
      const bool diag = p.causal && j == 2 * qp + t;
      if (diag || (!PAIRS && (j + 1) * BKV > p.S)) {
        // last key of this block that counts: up to the query itself, none behind the end of the sequence
        const int seen = PAIRS ? row : min(diag ? row : BKV - 1, p.S - 1 - j * BKV);
#pragma unroll
        for (int i = 0; i < 128; ++i)
          if (i > seen) s[i] = 0xff800000u;          // -inf
      }
#pragma unroll
      for (int i = 0; i < 128; i += 2)
        top[(i >> 1) & 3] = fmax3(top[(i >> 1) & 3], __uint_as_float(s[i]), __uint_as_float(s[i + 1]));
      const float mx = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
      // rescale O only when the maximum moved by more than 2^8 (whole warp together:
      // the tensor-memory accesses are warp-wide)
      const bool grow = (j > 0) && ((mx - m_ref) * c > 8.f);
      if (j == 0) m_ref = mx;
      if (__any_sync(0xffffffffu, grow)) {
        const float alpha = grow ? exp2f((m_ref - mx) * c) : 1.f;
        if (grow) { m_ref = mx; l *= alpha; }
        ok = mbar_wait(&bar->pv_done[t], (j - 1) & 1, &bar->abort_flag, p.status, 39);
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int ch = 0; ch < D / 32; ++ch) {
          uint32_t r[32];
          tmem_ld_32x32(tO + ch * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
          tmem_st_32x32(tO + ch * 32, r);
        }
        tmem_st_wait();
      }
      const uint64_t c2 = pack_f32x2(c, c), mc2 = pack_f32x2(-m_ref * c, -m_ref * c);
      uint64_t sum2[2] = {0, 0};
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        uint32_t packed[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float2 x = unpack_f32x2(fma_f32x2(pack_u32x2(s[ch * 32 + 2 * i], s[ch * 32 + 2 * i + 1]), c2, mc2));
          const float p0 = exp2_mixed<POLY>(x.x, 2 * i), p1 = exp2_mixed<POLY>(x.y, 2 * i + 1);
          sum2[i & 1] = add_f32x2(sum2[i & 1], pack_f32x2(p0, p1));
          packed[i] = pack_bf16x2(p0, p1);
        }
        if (OWN_P && ch == 0 && j > 0) {              // P_t(j - 1) has been read
          ok = mbar_wait(&bar->pv_done[t], (j - 1) & 1, &bar->abort_flag, p.status, 44);
          if (!ok) break;
          tc_fence_after();
        }
        tmem_st_32x16(tP + ch * 16, packed);
        if (ch == P_SPLIT / 32 - 1) {
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar->p_most[t]);
        }
      }
      if (!ok) break;
      const float2 sums = unpack_f32x2(add_f32x2(sum2[0], sum2[1]));
      const float lsum = sums.x + sums.y;
      l += lsum;
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->p_full[t]);
    }
    if (ok && (PAIRS || nt > 0)) {
      ok = mbar_wait(&bar->pv_done[t], (nt - 1) & 1, &bar->abort_flag, p.status, 40);
      if (ok) {
        tc_fence_after();
        const float inv = 1.f / l;
        int place = blockIdx.x;                  // the head once more, instead of registers held over the loop
        asm volatile("" : "+r"(place));
        const int bh = place % (p.Hq * p.batch);
        const int q_row = q_row0 + t * BQ + row;             // of this sequence
        __nv_bfloat16* orow = p.O + (((size_t)(bh / p.Hq) * p.S + q_row) * p.Hq + bh % p.Hq) * D;
#pragma unroll 1
        for (int ch = 0; ch < D / 32; ++ch) {
          uint32_t r[32];
          tmem_ld_32x32(tO + ch * 32, r);
          tmem_ld_wait();
          uint4* dst = reinterpret_cast<uint4*>(orow + ch * 32);
          if (PAIRS || q_row < p.S) {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              uint4 v;
              v.x = pack_bf16x2(__uint_as_float(r[8 * g]) * inv, __uint_as_float(r[8 * g + 1]) * inv);
              v.y = pack_bf16x2(__uint_as_float(r[8 * g + 2]) * inv, __uint_as_float(r[8 * g + 3]) * inv);
              v.z = pack_bf16x2(__uint_as_float(r[8 * g + 4]) * inv, __uint_as_float(r[8 * g + 5]) * inv);
              v.w = pack_bf16x2(__uint_as_float(r[8 * g + 6]) * inv, __uint_as_float(r[8 * g + 7]) * inv);
              dst[g] = v;
            }
          }
          if (!PAIRS) __syncwarp();         // the lanes of rows behind the sequence take part in the next (aligned) read
        }
        if (p.lse != nullptr && (PAIRS || q_row < p.S))
          p.lse[(size_t)bh * p.S + q_row] = m_ref * p.scale + logf(l);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

int run(const void* q, long long q_row_stride, long long q_head_stride, const void* k,
                        long long k_row_stride, long long k_head_stride, const void* v, long long v_row_stride,
                        long long v_head_stride, void* out, float* lse, int batch, int S, int Hq, int Hkv, int Dh,
                        int causal, float scale, void* stream) {
  if (S <= 0 || Dh != D || Hkv <= 0 || Hq <= 0 || Hq % Hkv != 0 || batch <= 0) return DD_ERR_BAD_ARG;
  CUtensorMap tq, tk, tv;
  int r = get_tensor_map_bf16_4d(&tq, q, D, S, Hq, batch, q_row_stride * 2, q_head_stride * 2,
                                 (uint64_t)S * q_row_stride * 2, 64, BQ);
  if (r) return r;
  r = get_tensor_map_bf16_4d(&tk, k, D, S, Hkv, batch, k_row_stride * 2, k_head_stride * 2,
                             (uint64_t)S * k_row_stride * 2, 64, BKV);
  if (r) return r;
  r = get_tensor_map_bf16_4d(&tv, v, D, S, Hkv, batch, v_row_stride * 2, v_head_stride * 2,
                             (uint64_t)S * v_row_stride * 2, 64, BKV);
  if (r) return r;
  int err = 0;
  Params2 p;
  p.O = reinterpret_cast<__nv_bfloat16*>(out);
  p.lse = lse;
  p.S = S; p.Hq = Hq; p.Hkv = Hkv; p.batch = batch; p.causal = causal; p.scale = scale;
  p.status = device_status(&err);
  if (err) return err;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  // DISTDL_ATTN_EXP_POLY=1: a third of the exponentials on the FMA pipe (exp2_fma in common.cuh)
  static const bool poly = [] { const char* e = getenv("DISTDL_ATTN_EXP_POLY"); return e != nullptr && e[0] == '1'; }();
  using Kernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, Params2);
  const Kernel kernels[4] = {attn_fwd2_kernel<false, false>, attn_fwd2_kernel<false, true>, attn_fwd2_kernel<true, false>,
                             attn_fwd2_kernel<true, true>};
  if (!configured[dev & 63]) {
    for (Kernel k : kernels) {
      const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_TOTAL);
      if (e != cudaSuccess) return (int)e;
    }
    configured[dev & 63] = true;
  }
  const long long grid = (S / (2 * BQ) + (S % (2 * BQ) != 0)) * (long long)Hq * batch;
  if (grid > 0x7fffffffLL) return DD_ERR_TOO_LARGE;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  kernels[(poly ? 2 : 0) + (S % (2 * BQ) == 0 ? 1 : 0)]<<<(unsigned)grid, NUM_THREADS, SMEM_TOTAL, st>>>(tq, tk, tv, p);
  return (int)cudaGetLastError();
}

}  // namespace DD_FWD2_NS
