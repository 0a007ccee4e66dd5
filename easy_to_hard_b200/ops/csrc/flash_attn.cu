// Causal flash attention (forward and backward) on tcgen05 tensor cores, head_dim 128 or 64.
//
// Tiles are stored as D/64 column halves of [rows x 64] bf16, each half 128-byte swizzled (what a TMA box
// {64, rows} produces).
//
// Masking follows the reference model (models/model.py:221-228, 338-344): key j is visible to
// query i when j <= i + (Sk - Sq) and j >= left_pad[b], or when j is the diagonal; with
// left_pad == nullptr this is plain causal attention (training, scoring, reward models).
// Layouts are given by strides, so Q/K/V may be views into the fused qkv activation or the
// static KV cache ([B, Hkv, Smax, D]).
//
// All mbarrier waits are bounded; a time-out sets the status word and the CTA still reaches
// every barrier and frees its tensor memory.
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <float.h>
#include <limits.h>
#include <string.h>

#include "flash_common.cuh"
#include "launch.cuh"
#include "ptx.cuh"

namespace e2h {

constexpr int kBQ = 128;   // queries per CTA
constexpr int kBK = 128;   // keys per tile

struct FlashParams {
  int B, H, Hkv, Sq, Sk, D;
  float scale;              // 1/sqrt(D)
  const int* left_pad;      // [B] or nullptr
  __nv_bfloat16* out;       // [B, Sq, H, D] with strides o_sb, o_ss, o_sh (elements)
  long long o_sb, o_ss, o_sh;
  float* lse;               // [B, H, Sq] or nullptr
  int* status;
};

constexpr int kBwdThreads = 320;
constexpr float kRescaleThreshold = 8.f;   // log2 units: P stays below 2^8 between rescales

// Forward: one CTA per SM stays and takes work items, an item being two tiles of 128 queries that share
// their keys: two query heads of one kv head where heads are grouped in even numbers, else two blocks
// of 128 consecutive queries of one head. The items with the most key tiles come first.
//
// Roles (352 threads):
//   warps 0-3, 4-7  softmax of query tile 0 and of tile 1: thread r owns query row r of its tile (no exchange
//                   between threads for maximum and sum), takes the row's 64 scores from tensor memory in
//                   one trip and writes P = exp2(S - m) in bf16 over their columns, where it is the
//                   tensor-memory A operand of P V: probabilities never touch shared memory;
//   warp 8          TMA producer: the query tiles, then K and V tiles of 64 keys through one ring;
//   warps 9, 10     UMMA issuers of tile 0 and of tile 1. The scores of a key tile go to one of two buffers, and
//                   are issued before P V of the tile before: while the softmax works on one buffer, the
//                   other one is filled, and neither query tile waits for the other but by the ring. "Next"
//                   crosses from one item to the following one, so that the first scores of an item are
//                   there when the outputs of the one before have been written.
// Tensor memory (512 columns): two buffers of S of 64 for either tile, O0, O1 of 128.
// O stays in tensor memory for the whole key loop. The running maximum is only raised -- and O multiplied
// by exp2(m_old - m_new) in place -- when some row of the warp would otherwise exceed 2^8; otherwise the
// stale maximum keeps being used, which is exact after the final division by the row sum. Score tiles
// that lie entirely below the diagonal and right of the left-pad boundary skip the visibility tests.
//
// What bounds it: a pair step, 64 keys of both query tiles, has 1280 cycles of products (of each tile Q K^T at
// N = 64 takes 384, bound by its operands' 6 KB of shared memory, and P V 256) beside 1024 of exponentials
// (16 per cycle and SM). Measured about 1950 a step in long rows (1 x 16000: 0.56 of the burst rate), the rest being
// hand-overs between the roles. Beside its steps an item costs 6000 to 7000: its queries, first scores, last
// products and outputs wait for one another, and only the other query tile fills in. At 768 tokens, 8 steps
// an item, that makes 2750 a step (profiles/flash_fwd_b4_s768_h32_d128.md; 0.37 to 0.39 of the burst rate).
// us per launch, one 128-query tile per CTA with two threads per row and P through shared memory -> this:
//   64 sequences x 768, 32 heads             849 -> 482          16 x 768, 32 heads              225 -> 133
//   32 x 701, 64 query and 8 kv heads        834 -> 423          5 x 1003, 40 heads              142 -> 91
//   4 x 4000, 32 heads, left pads            547 -> 370          1 x 4000, 32 heads              206 -> 166
//   2 x 8000, 32 heads                      1232 -> 1074         64 x 61, 32 heads                93 -> 60
// Launch after launch it runs into the power cap (1.5 to 1.9 GHz, the older form 1.7 to 1.97), and the gain is
// smaller: 64 x 768 858 -> 508, 16 x 768 225 -> 161, 1 x 4000 216 -> 207, 2 x 8000 1390 -> 1260. Head size 64, the
// same way: 64 x 768 749 -> 446, 16 x 768 193 -> 116, 32 x 701 726 -> 378, 4 x 4000 602 -> 387, 2 x 8000 1192 -> 888,
// 64 x 61 78 -> 46.
// Tried: key tiles of 128 with one buffer of scores (the tile's softmax and products wait for each other: 64 x
// 768 646 us with a thread per row, 567 with two), a vote after each barrier wait of the issuers (546).
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// two fp32 operations in one instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n.reg .b64 ra, rb, rc, rd;\nmov.b64 ra, {%2, %3};\nmov.b64 rb, {%4, %5};\nmov.b64 rc, {%6, %7};\n"
      "fma.rn.f32x2 rd, ra, rb, rc;\nmov.b64 {%0, %1}, rd;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 d;
  asm("{\n.reg .b64 ra, rb, rd;\nmov.b64 ra, {%2, %3};\nmov.b64 rb, {%4, %5};\n"
      "add.rn.f32x2 rd, ra, rb;\nmov.b64 {%0, %1}, rd;\n}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

// Raises four running maxima over 64 scores; of those the columns lo .. hi are visible.
template <bool ALL>
__device__ __forceinline__ void row_max(const float* sv, int lo, int hi, float* mx) {
  if (ALL) {
#pragma unroll
    for (int i = 0; i < 64; i += 8)
#pragma unroll
      for (int u = 0; u < 4; ++u) mx[u] = max3(mx[u], sv[i + u], sv[i + u + 4]);
  } else {
#pragma unroll
    for (int i = 0; i < 64; ++i) mx[i & 3] = fmaxf(mx[i & 3], i >= lo && i <= hi ? sv[i] : -INFINITY);
  }
}
// 64 probabilities exp2(s * sl2 - m) of one row: into the row sum, and as bf16 into 32 columns of tensor
// memory. A result of the special function unit is used four steps after it was asked for.
template <bool ALL>
__device__ __forceinline__ void row_probs(float* sv, int lo, int hi, float sl2, float m, float2* rs,
                                          uint32_t dst) {
#pragma unroll
  for (int c = 0; c < 64; c += 32) {
    float2 x[16];
    uint32_t packed[16];
#pragma unroll
    for (int e = 0; e < 16; ++e)
      x[e] = fma2(make_float2(sv[c + 2 * e], sv[c + 2 * e + 1]), make_float2(sl2, sl2),
                  make_float2(-m, -m));
    constexpr int kLag = 4;
#pragma unroll
    for (int e = 0; e < 16 + kLag; ++e) {
      if (e < 16) {
        x[e].x = ex2_approx(x[e].x);
        x[e].y = ex2_approx(x[e].y);
      }
      if (e >= kLag) {
        const int d = e - kLag, i = c + 2 * d;
        if (!ALL) {
          x[d].x = i >= lo && i <= hi ? x[d].x : 0.f;
          x[d].y = i + 1 >= lo && i + 1 <= hi ? x[d].y : 0.f;
        }
        rs[d & 1] = add2(rs[d & 1], x[d]);
        const __nv_bfloat162 pk = __floats2bfloat162_rn(x[d].x, x[d].y);
        packed[d] = *reinterpret_cast<const uint32_t*>(&pk);
      }
    }
    tmem_st_x16(dst + c / 2, packed);
  }
}

// Lane j of four neighbours gives o[i] of its own to lane i and gets o[j] of that one as its o[i].
__device__ __forceinline__ void transpose4(uint32_t (&o)[4][4], int lane) {
#pragma unroll
  for (int s = 1; s < 4; s *= 2) {
    const bool up = lane & s;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i & s) continue;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t give = up ? o[i][e] : o[i | s][e];
        const uint32_t got = __shfl_xor_sync(0xffffffffu, give, s);
        o[i][e] = up ? got : o[i][e];
        o[i | s][e] = up ? o[i | s][e] : got;
      }
    }
  }
}

struct FwdParams : FlashParams {
  int pair_heads, n_qb;
  int nh, heads;           // heads or pairs of them: of a sequence, of all
  unsigned long long m_heads, m_nh, m_group;   // for fast_div
};
// n / d for 0 <= n < 2^31 with m = floor((2^64 - 1) / d) + 1, d > 1, or m = 0 for d = 1
__device__ __forceinline__ int fast_div(int n, unsigned long long m) {
  return m == 0 ? n : (int)__umul64hi((unsigned long long)n, m);
}
inline unsigned long long fast_div_of(int d) { return d == 1 ? 0 : ~0ull / d + 1; }

constexpr int kFK = 64;     // keys per tile of the forward

struct FwdTile {
  int h, q0, jb, je;      // query head, first query, key tiles jb .. je - 1
};
struct FwdItem {
  int b, hk, first, last; // first, last: key tiles of both query tiles
  FwdTile t0, t1;
};

__device__ __forceinline__ FwdTile fwd_tile(const FwdParams& p, int hx, int qb, int lp, int g) {
  FwdTile t;
  t.h = p.pair_heads ? 2 * hx + g : hx;
  t.q0 = (p.pair_heads ? qb : 2 * qb + g) * kBQ;
  // from the left-pad boundary (or the tile's own diagonal when the whole tile is padding) to the diagonal of
  // its last row
  const int off = p.Sk - p.Sq;
  const int last_key = min(p.Sk - 1, t.q0 + kBQ - 1 + off);
  const int first_key = max(0, min(lp, t.q0 + off));
  t.jb = first_key / kFK;
  t.je = t.q0 >= p.Sq || last_key < 0 ? 0 : last_key / kFK + 1;
  if (t.je < t.jb) t.je = t.jb;
  return t;
}
// The items of one CTA, the same for all of its roles. An item is a (sequence, head or pair of heads, query
// block); the blocks with the most keys of all heads come first and are dealt out in turn, so that the loads
// are even to within the smallest block. (Head after head, so that the keys of a few heads stay in L2, was
// slower: 64 x 768 tokens, 32 heads 546 -> 687 us; 4 x 4000 350 -> 390.)
struct FwdWalk {
  int b = 0, hx = 0, qb = 0;
  int at = -1;
  __device__ __forceinline__ bool next(const FwdParams& p) {
    at = at < 0 ? (int)blockIdx.x : at + (int)gridDim.x;
    if (at >= p.heads * p.n_qb) return false;
    const int r = fast_div(at, p.m_heads);
    qb = p.n_qb - 1 - r;
    const int rest = at - r * p.heads;
    b = fast_div(rest, p.m_nh);
    hx = rest - b * p.nh;
    return true;
  }
};

// The next item with key tiles, or false.
__device__ __forceinline__ bool fwd_item(const FwdParams& p, FwdWalk& walk, FwdItem& w) {
  while (walk.next(p)) {
    w.b = walk.b;
    const int lp = p.left_pad ? p.left_pad[w.b] : 0;
    w.t0 = fwd_tile(p, walk.hx, walk.qb, lp, 0);
    w.t1 = fwd_tile(p, walk.hx, walk.qb, lp, 1);
    const bool a0 = w.t0.je > w.t0.jb, a1 = w.t1.je > w.t1.jb;
    w.first = a0 ? (a1 ? min(w.t0.jb, w.t1.jb) : w.t0.jb) : w.t1.jb;
    w.last = a0 ? (a1 ? max(w.t0.je, w.t1.je) : w.t0.je) : w.t1.je;
    w.hk = fast_div(w.t0.h, p.m_group);
    if (a0 || a1) return true;
  }
  return false;
}

constexpr int kFwdThreads = 352;
constexpr int kFwdSlots = 5;      // key tiles in flight: K and V together
struct FwdCtrl {
  uint64_t full[kFwdSlots], empty[kFwdSlots];
  uint64_t q_full[2], q_empty[2], s_full[4], p_full[4];   // S, P: 2 tile + buffer
  // O: a key tile added (waited for before O is rescaled; by then only the last one can be under way), the
  // item's last one added, outputs read
  uint64_t o_full[2], o_done[2], o_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

template <int D>
__global__ void __launch_bounds__(kFwdThreads, 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const FwdParams p) {
  constexpr int NH = D / 64;                 // 64-wide halves of the head dimension
  constexpr int kQHalf = 128 * 128, kKvHalf = kFK * 128;   // [rows x 64] bf16
  constexpr int kQBytes = NH * kQHalf, kKvBytes = NH * kKvHalf;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  FwdCtrl* ctrl = reinterpret_cast<FwdCtrl*>(smem);
  uint8_t* q_s = smem + 1024;                // 2 tiles
  uint8_t* kv_s = q_s + 2 * kQBytes;         // kFwdSlots pairs of a K and a V tile
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* abort_flag = &ctrl->abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kFwdSlots; ++s) {
      mbar_init(smem_u32(&ctrl->full[s]), 1);
      mbar_init(smem_u32(&ctrl->empty[s]), 2);      // one arrival per issuer
    }
    for (int g = 0; g < 2; ++g) {
      mbar_init(smem_u32(&ctrl->q_full[g]), 1);
      mbar_init(smem_u32(&ctrl->q_empty[g]), 1);
      for (int u = 0; u < 2; ++u) {
        mbar_init(smem_u32(&ctrl->s_full[2 * g + u]), 1);
        mbar_init(smem_u32(&ctrl->p_full[2 * g + u]), 4);   // one arrival per softmax warp of the tile
      }
      mbar_init(smem_u32(&ctrl->o_full[g]), 1);
      mbar_init(smem_u32(&ctrl->o_done[g]), 1);
      mbar_init(smem_u32(&ctrl->o_empty[g]), 4);
    }
    ctrl->abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == 9) {
    tmem_alloc(smem_u32(&ctrl->tmem_base), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem0 = ctrl->tmem_base;
  const uint32_t full0 = smem_u32(&ctrl->full[0]), empty0 = smem_u32(&ctrl->empty[0]);

  if (warp == 8) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int slot = 0, armed = 0;
      uint32_t ph = 0, qph[2] = {0, 0};
      bool ok = true;
      FwdWalk walk;
      FwdItem w;
      while (ok && fwd_item(p, walk, w)) {
        for (int j = w.first; j < w.last && ok; ++j) {
          ok = ok && mbar_wait(empty0 + 8 * slot, ph ^ 1, abort_flag, p.status, kStatusTimeoutEmpty);
          if (!ok) break;
          mbar_expect_tx(full0 + 8 * slot, 2 * kKvBytes);
#pragma unroll
          for (int kv = 0; kv < 2; ++kv)
#pragma unroll
            for (int hf = 0; hf < NH; ++hf)
              tma_load_4d(smem_u32(kv_s + (2 * slot + kv) * kKvBytes + hf * kKvHalf), kv ? &tmV : &tmK,
                          hf * 64, j * kFK, w.hk, w.b, full0 + 8 * slot);
          ++armed;
          if (++slot == kFwdSlots) {
            slot = 0;
            ph ^= 1;
          }
          // an item's query tiles come in the order in which their places come free: tile 0 is through with the
          // item before earlier
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const FwdTile t = g ? w.t1 : w.t0;
            if (j > w.first || t.je <= t.jb || !ok) continue;
            ok = mbar_wait(smem_u32(&ctrl->q_empty[g]), qph[g] ^ 1, abort_flag, p.status,
                           kStatusTimeoutEmpty);
            if (!ok) continue;
            qph[g] ^= 1;
            mbar_expect_tx(smem_u32(&ctrl->q_full[g]), kQBytes);
#pragma unroll
            for (int hf = 0; hf < NH; ++hf)
              tma_load_4d(smem_u32(q_s + g * kQBytes + hf * kQHalf), &tmQ, hf * 64, t.q0, t.h, w.b,
                          smem_u32(&ctrl->q_full[g]));
          }
        }
      }
      if (*abort_flag) {   // bounded wait for the copies still in flight into this CTA's smem
        auto drain = [&](uint32_t bar, uint32_t parity) {
          const long long tq = clock64();
          while (!mbar_try_wait(bar, parity))
            if (clock64() - tq > kWaitLimitCycles / 8) break;
        };
        for (int it = armed > kFwdSlots ? armed - kFwdSlots : 0; it < armed; ++it)
          drain(full0 + 8 * (it % kFwdSlots), (it / kFwdSlots) & 1);
        for (int g = 0; g < 2; ++g) drain(smem_u32(&ctrl->q_full[g]), qph[g] ^ 1);
      }
    }
  } else if (warp >= 9) {
    // ---------------- UMMA issuer of tile g (the whole warp walks, one lane issues) ----------------
    const int g = warp - 9;
    const bool lead = elect_one();
    // S = Q K^T, both K-major; with a negative scale -Q K^T (bit 13), so that the maximum is one
    const uint32_t idesc_s = make_idesc_bf16(128, kFK, 0, 0) | (p.scale < 0.f ? 1u << 13 : 0u);
    const uint32_t idesc_o = make_idesc_bf16(128, D, 0, 1);     // O = P V, V is MN-major
    const uint32_t d_hi = sw128_desc_hi(1024);
    const uint32_t t_s = __shfl_sync(0xffffffffu, tmem0 + g * 128, 0);
    const uint32_t tmem_o = t_s + 256;
    const uint32_t q_lo = sw128_desc_lo(smem_u32(q_s + g * kQBytes), 16);
    const uint32_t k_lo = sw128_desc_lo(smem_u32(kv_s), 16);
    const uint32_t v_lo = sw128_desc_lo(smem_u32(kv_s + kKvBytes), kKvHalf);
    const uint32_t q_bar = smem_u32(&ctrl->q_full[g]), qe_bar = smem_u32(&ctrl->q_empty[g]);
    const uint32_t s_bar = smem_u32(&ctrl->s_full[2 * g]), o_bar = smem_u32(&ctrl->o_full[g]);
    const uint32_t p_bar = smem_u32(&ctrl->p_full[2 * g]), oe_bar = smem_u32(&ctrl->o_empty[g]);
    const uint32_t od_bar = smem_u32(&ctrl->o_done[g]);
    uint32_t n_s = 0, n_pv = 0;            // tiles whose scores, and whose products with V are issued
    uint32_t n_q = 0, n_o = 0;             // items begun: scores, outputs
    uint32_t s_slot = 0, s_ph = 0, o_slot = 0;   // place in the ring: of the scores, of the outputs
    bool ok = true;
    // (no vote after each wait: it costs more than the wait. A lane whose wait ran out goes on with what is in
    // memory until the warp looks, at the end of a key tile)
    auto wait = [&](uint32_t bar, uint32_t parity, int code) {
      if (!mbar_wait(bar, parity, abort_flag, p.status, code)) ok = false;
    };
    // scores of key tile j. (A tile that is not this one's is waited for all the same, so that the slots' phases
    // stay in step.)
    auto scores = [&](int j, int jb, int je) {
      wait(full0 + 8 * s_slot, s_ph, kStatusTimeoutFull);
      if (j >= jb && j < je) {
        if (j == jb) wait(q_bar, n_q++ & 1, kStatusTimeoutFull);
        tc_fence_after();
        // the buffer's last P V was issued by this thread: it is read before this product writes
        const uint32_t buf = n_s & 1;
        ++n_s;
        if (lead) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk)
            umma_f16_lohi(t_s + buf * 64, q_lo + (((kk / 4) * kQHalf + (kk % 4) * 32) >> 4), d_hi,
                          k_lo + s_slot * (kKvBytes >> 3) + (((kk / 4) * kKvHalf + (kk % 4) * 32) >> 4),
                          d_hi, idesc_s, kk > 0 ? 1u : 0u);
          umma_commit(s_bar + 8 * buf);
          if (j == je - 1) umma_commit(qe_bar);
        }
      }
      if (++s_slot == kFwdSlots) {
        s_slot = 0;
        s_ph ^= 1;
      }
    };
    auto outputs = [&](int j, int jb, int je) {
      if (j >= jb && j < je) {
        const bool first = j == jb;
        const uint32_t buf = n_pv & 1;
        // the outputs of the item before have been read
        if (first) wait(oe_bar, (n_o++ & 1) ^ 1, kStatusTimeoutTmemEmpty);
        wait(p_bar + 8 * buf, n_pv >> 1 & 1, kStatusTimeoutFull);
        ++n_pv;
        tc_fence_after();
        if (lead) {
#pragma unroll
          for (int kk = 0; kk < kFK / 16; ++kk)
            umma_f16_ts(tmem_o, t_s + buf * 64 + kk * 8, v_lo + o_slot * (kKvBytes >> 3) + (kk * 2048 >> 4),
                        d_hi, idesc_o, (!first || kk > 0) ? 1u : 0u);
          umma_commit(o_bar);
          if (j == je - 1) umma_commit(od_bar);
        }
      }
      if (lead) umma_commit(empty0 + 8 * o_slot);
      if (++o_slot == kFwdSlots) o_slot = 0;
    };
    // scores run one tile ahead of outputs, but into a new item the outputs come first: its queries are still on
    // their way
    FwdWalk walk;
    FwdItem w;
    int j_last = 0, jb_last = 0, je_last = 0;      // the tile whose outputs are due
    bool due = false;
    while (ok && fwd_item(p, walk, w)) {
      const int jb = g ? w.t1.jb : w.t0.jb, je = g ? w.t1.je : w.t0.je;
      if (due) outputs(j_last, jb_last, je_last);
      scores(w.first, jb, je);
      for (int j = w.first + 1; j < w.last && ok; ++j) {
        scores(j, jb, je);
        outputs(j - 1, jb, je);
        ok = __all_sync(0xffffffffu, ok);
      }
      ok = __all_sync(0xffffffffu, ok);
      due = true;
      j_last = w.last - 1;
      jb_last = jb;
      je_last = je;
    }
    if (ok && due) outputs(j_last, jb_last, je_last);
    __syncwarp();
  } else {
    // ---------------- softmax / output warps ----------------
    const int g = warp >> 2;
    const int qrt = warp & 3;
    const int row = qrt * 32 + lane;                  // query row within the tile = TMEM lane
    const uint32_t tmem_s = tmem0 + g * 128 + (static_cast<uint32_t>(qrt * 32) << 16);
    const uint32_t tmem_o = tmem_s + 256;
    const float sl2 = fabsf(p.scale) * 1.4426950408889634f;  // scale * log2(e); its sign is in S
    const uint32_t s_bar = smem_u32(&ctrl->s_full[2 * g]), p_bar = smem_u32(&ctrl->p_full[2 * g]);
    const uint32_t o_bar = smem_u32(&ctrl->o_full[g]), oe_bar = smem_u32(&ctrl->o_empty[g]);
    const uint32_t od_bar = smem_u32(&ctrl->o_done[g]);
    const int off = p.Sk - p.Sq;
    uint32_t tile = 0;                                // key tiles so far: phases of s_full and o_full
    uint32_t n_done = 0;                              // items so far: phase of o_done
    bool ok = true;
    FwdWalk walk;
    while (walk.next(p)) {
      const int b = walk.b;
      const int lp = p.left_pad ? p.left_pad[b] : 0;
      const FwdTile w = fwd_tile(p, walk.hx, walk.qb, lp, g);
      const int q0 = w.q0, jb = w.jb, je = w.je;
      if (q0 >= p.Sq) continue;
      const int qi = q0 + row;                        // query index
      const int qpos = qi + off;                      // its key position (diagonal)
      // visible keys of the row: from the boundary (or the diagonal, left of it) to the diagonal
      const int lo = min(lp, qpos), hi = min(qpos, p.Sk - 1);
      float m = -FLT_MAX, l = 0.f;
      for (int j = jb; j < je; ++j, ++tile) {
        const uint32_t buf = tile & 1, cols = tmem_s + 64 * buf;
        // columns of the tile that the row sees; most tiles are seen in full by all rows of the warp, and of the
        // last two some by none
        const int l_rel = lo - j * kFK, h_rel = hi - j * kFK;
        const bool all = __all_sync(0xffffffffu, l_rel <= 0 && h_rel >= kFK - 1);
        const bool none = __all_sync(0xffffffffu, l_rel >= kFK || h_rel < 0 || h_rel < l_rel);
        ok = ok && mbar_wait(s_bar + 8 * buf, tile >> 1 & 1, abort_flag, p.status, kStatusTimeoutTmemFull);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        if (none) {
          uint32_t z[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) z[i] = 0u;
          tmem_st_x16(cols, z);
          tmem_st_x16(cols + 16, z);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(p_bar + 8 * buf);
          continue;
        }
        float sv[kFK];
        tmem_ld_x32(cols, sv);
        tmem_ld_x32(cols + 32, sv + 32);
        tmem_ld_wait();
        float mx4[4] = {-FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX};
        if (all) row_max<true>(sv, 0, 0, mx4);
        else row_max<false>(sv, l_rel, h_rel, mx4);
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        // in log2 units from here on (the factor keeps the order)
        const float m_new = fmaxf(m, mx == -FLT_MAX ? mx : mx * sl2);
        const bool need = (j > jb) && (m != -FLT_MAX) && (m_new - m > kRescaleThreshold);
        if (__any_sync(0xffffffffu, need)) {
          // raise the maximum of all 32 rows of this warp: O *= exp2(m_old - m_new) in place
          const float alpha = (m == -FLT_MAX) ? 1.f : ex2_approx(m - m_new);
          ok = mbar_wait(o_bar, (tile - 1) & 1, abort_flag, p.status, kStatusTimeoutTmemFull);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < D; c += 16) {       // (few columns at a time: the scores stay in registers)
            float ov[16];
            tmem_ld_x16(tmem_o + c, ov);
            tmem_ld_wait();
            uint32_t r[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(ov[i] * alpha);
            tmem_st_x16(tmem_o + c, r);
          }
          l *= alpha;
          m = m_new;
        } else if (m == -FLT_MAX) {
          m = m_new;                                  // no history yet: nothing to rescale
        }
        const float msafe = (m == -FLT_MAX) ? 0.f : m;
        float2 rs[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        if (all) row_probs<true>(sv, 0, 0, sl2, msafe, rs, cols);
        else row_probs<false>(sv, l_rel, h_rel, sl2, msafe, rs, cols);
        l += (rs[0].x + rs[0].y) + (rs[1].x + rs[1].y);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_bar + 8 * buf);
      }
      if (!ok) break;
      // ---- epilogue: O / l ----
      const bool any = je > jb;
      if (any && ok) {
        ok = mbar_wait(od_bar, n_done++ & 1, abort_flag, p.status, kStatusTimeoutTmemFull);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
      }
      if (!ok) break;
      const float inv = l > 0.f ? 1.f / l : 0.f;
      // A thread holds a row, but a store instruction of 32 rows touches 32 lines (4000 cycles a tile): four
      // lanes exchange their 16-byte pieces of 32 columns, so that they write 64 bytes of one row each time
      __nv_bfloat16* obase = p.out + (long long)b * p.o_sb + (long long)w.h * p.o_sh + 8 * (lane & 3);
      const int r0 = q0 + qrt * 32 + (lane & ~3);
#pragma unroll
      for (int c = 0; c < D; c += 32) {
        float ov[32];
        if (any) tmem_ld_x32(tmem_o + c, ov);
        tmem_ld_wait();
        if (c + 32 == D && any) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(oe_bar);         // the next item's outputs may come
        }
        uint32_t o[4][4];                             // [piece][word]
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float a0 = any ? ov[8 * u + 2 * e] * inv : 0.f;
            const float a1 = any ? ov[8 * u + 2 * e + 1] * inv : 0.f;
            const __nv_bfloat162 pk = __floats2bfloat162_rn(a0, a1);
            o[u][e] = *reinterpret_cast<const uint32_t*>(&pk);
          }
        transpose4(o, lane);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (r0 + i < p.Sq)
            *reinterpret_cast<uint4*>(obase + (long long)(r0 + i) * p.o_ss + c) =
                make_uint4(o[i][0], o[i][1], o[i][2], o[i][3]);
        __syncwarp();
      }
      const bool store = qi < p.Sq;
      if (store && p.lse)
        p.lse[((long long)b * p.H + w.h) * p.Sq + qi] =
            (l > 0.f) ? (m * 0.6931471805599453f + logf(l)) : -FLT_MAX;
    }
    tc_fence_before();
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem0, 512);
}

// =============================================================================================
// Backward pass. Two kernels recompute the probabilities from (Q, K, lse):
//   flash_bwd_dkdv_kernel : one CTA per (batch, kv head, 128-key block); loops over the query
//                           blocks (and the query heads of the group) that see those keys;
//                           dV += P^T dO and dK += dS^T Q accumulate in tensor memory.
//   flash_bwd_dq_kernel   : one CTA per (batch, head, 128-query block); loops over key blocks;
//                           dQ += dS K accumulates in tensor memory.
// with P = exp(S*scale - lse), dP = dO V^T, dS = P o (dP - delta) * scale and
// delta = rowsum(dO o O) from flash_delta_kernel. Splitting the work this way recomputes S and
// dP twice but needs no atomics and is deterministic.
// Shared-memory tiles are [128 rows x 64] bf16 halves with the 128-byte swizzle, so the same
// tile serves as a K-major operand (contraction along the row) or an MN-major operand
// (contraction across rows): P / dS are written once and used both ways.
// =============================================================================================

struct FlashBwdParams {
  int B, H, Hkv, Sq, Sk, D;
  float scale;
  const int* left_pad;
  const float* lse;      // [B, H, Sq]
  const float* delta;    // [B, H, Sq]
  __nv_bfloat16* dq;     // like q   (strides q_sb, q_ss, q_sh)
  __nv_bfloat16* dk;     // like k/v (strides k_sb, k_ss, k_sh)
  __nv_bfloat16* dv;
  long long q_sb, q_ss, q_sh, k_sb, k_ss, k_sh;
  int* status;
};

struct BwdCtrl {
  uint64_t once_full, it_full, it_empty, sdp_full, pds_full, done;
  uint32_t tmem_base;
  int abort_flag;
};

// delta[b, h, i] = sum_d O[b,i,h,d] * dO[b,i,h,d]
__global__ void flash_delta_kernel(const __nv_bfloat16* __restrict__ o,
                                   const __nv_bfloat16* __restrict__ d_o, float* __restrict__ delta,
                                   long long sb, long long ss, long long sh, long long dsb,
                                   long long dss, long long dsh, int H, int Sq, int D) {
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int total = gridDim.y * H * Sq;  // gridDim.y = B
  (void)total;
  const int b = blockIdx.y;
  if (warp_global >= H * Sq) return;
  const int h = warp_global / Sq, i = warp_global - h * Sq;
  const __nv_bfloat16* po = o + b * sb + (long long)i * ss + (long long)h * sh;
  const __nv_bfloat16* pd = d_o + b * dsb + (long long)i * dss + (long long)h * dsh;
  float acc = 0.f;
  for (int d = lane; d < D; d += 32) acc += __bfloat162float(po[d]) * __bfloat162float(pd[d]);
  acc = warp_sum(acc);
  if (lane == 0) delta[((long long)b * H + h) * Sq + i] = acc;
}

// bf16 row of 32 values -> swizzled [128 x 64] halves (row-major, 16-byte chunk c at c ^ (row&7))
__device__ __forceinline__ void store_row32(uint8_t* tile, int row, int col0, const float* v) {
#pragma unroll
  for (int c8 = 0; c8 < 4; ++c8) {
    uint32_t packed[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const __nv_bfloat162 pk = __floats2bfloat162_rn(v[c8 * 8 + 2 * e], v[c8 * 8 + 2 * e + 1]);
      packed[e] = *reinterpret_cast<const uint32_t*>(&pk);
    }
    const int col8 = (col0 >> 3) + c8;
    const int half = col8 >> 3, chunk = col8 & 7;
    *reinterpret_cast<uint4*>(tile + half * (128 * 128) + row * 128 +
                              ((chunk ^ (row & 7)) << 4)) =
        make_uint4(packed[0], packed[1], packed[2], packed[3]);
  }
}

template <int D>
__global__ void __launch_bounds__(kBwdThreads, 1)
flash_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                      const FlashBwdParams p) {
  constexpr int NH = D / 64;
  constexpr int kHalf = 128 * 128;
  constexpr int kTile = NH * kHalf;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  BwdCtrl* ctrl = reinterpret_cast<BwdCtrl*>(smem);
  uint8_t* k_s = smem + 1024;
  uint8_t* v_s = k_s + kTile;
  uint8_t* q_s = v_s + kTile;
  uint8_t* do_s = q_s + kTile;
  uint8_t* p_s = do_s + kTile;          // [128 q x 128 keys]
  uint8_t* ds_s = p_s + 2 * kHalf;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int jb = blockIdx.x, hk = blockIdx.y, b = blockIdx.z;
  const int G = p.H / p.Hkv;
  const int key0 = jb * kBK;
  const int off = p.Sk - p.Sq;
  const int lp = p.left_pad ? p.left_pad[b] : 0;
  const int i_begin = max(0, key0 - off) / kBQ;
  const int n_q = (p.Sq + kBQ - 1) / kBQ;
  const int n_i = max(0, n_q - i_begin);
  const int n_it = n_i * G;
  volatile int* abort_flag = &ctrl->abort_flag;

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&ctrl->once_full), 1);
    mbar_init(smem_u32(&ctrl->it_full), 1);
    mbar_init(smem_u32(&ctrl->it_empty), 1);
    mbar_init(smem_u32(&ctrl->sdp_full), 1);
    mbar_init(smem_u32(&ctrl->pds_full), 8);   // one arrival per compute warp
    mbar_init(smem_u32(&ctrl->done), 1);
    ctrl->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&ctrl->tmem_base), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm_s = ctrl->tmem_base, tm_dp = tm_s + 128, tm_dv = tm_s + 256, tm_dk = tm_s + 384;

  if (warp == 0 && lane == 0) {
    mbar_expect_tx(smem_u32(&ctrl->once_full), 2 * kTile);
#pragma unroll
    for (int hf = 0; hf < NH; ++hf) {
      tma_load_4d(smem_u32(k_s + hf * kHalf), &tmK, hf * 64, key0, hk, b, smem_u32(&ctrl->once_full));
      tma_load_4d(smem_u32(v_s + hf * kHalf), &tmV, hf * 64, key0, hk, b, smem_u32(&ctrl->once_full));
    }
    for (int it = 0; it < n_it; ++it) {
      const int g = it / n_i, i = i_begin + it % n_i;
      const int h = hk * G + g;
      if (!mbar_wait(smem_u32(&ctrl->it_empty), (it & 1) ^ 1, abort_flag, p.status,
                     kStatusTimeoutEmpty))
        break;
      mbar_expect_tx(smem_u32(&ctrl->it_full), 2 * kTile);
#pragma unroll
      for (int hf = 0; hf < NH; ++hf) {
        tma_load_4d(smem_u32(q_s + hf * kHalf), &tmQ, hf * 64, i * kBQ, h, b, smem_u32(&ctrl->it_full));
        tma_load_4d(smem_u32(do_s + hf * kHalf), &tmDO, hf * 64, i * kBQ, h, b, smem_u32(&ctrl->it_full));
      }
    }
  } else if (warp == 1 && lane == 0) {
    const uint32_t id_kk = make_idesc_bf16(128, 128, 0, 0);   // S, dP: both operands K-major
    const uint32_t id_mm = make_idesc_bf16(128, D, 1, 1);     // dV, dK: both MN-major
    bool ok = mbar_wait(smem_u32(&ctrl->once_full), 0, abort_flag, p.status, kStatusTimeoutFull);
    for (int it = 0; it < n_it && ok; ++it) {
      ok = mbar_wait(smem_u32(&ctrl->it_full), it & 1, abort_flag, p.status, kStatusTimeoutFull);
      if (!ok) break;
      tc_fence_after();
      const uint32_t qa = smem_u32(q_s), ka = smem_u32(k_s), va = smem_u32(v_s), da = smem_u32(do_s);
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t o = (kk / 4) * kHalf + (kk % 4) * 32;
        umma_f16_lohi(tm_s, sw128_desc_lo(qa, 16) + ((o) >> 4), sw128_desc_hi(1024),
                      sw128_desc_lo(ka, 16) + ((o) >> 4), sw128_desc_hi(1024), id_kk,
                 kk > 0 ? 1u : 0u);
      }
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t o = (kk / 4) * kHalf + (kk % 4) * 32;
        umma_f16_lohi(tm_dp, sw128_desc_lo(da, 16) + ((o) >> 4), sw128_desc_hi(1024),
                      sw128_desc_lo(va, 16) + ((o) >> 4), sw128_desc_hi(1024), id_kk,
                 kk > 0 ? 1u : 0u);
      }
      umma_commit(smem_u32(&ctrl->sdp_full));
      ok = mbar_wait(smem_u32(&ctrl->pds_full), it & 1, abort_flag, p.status, kStatusTimeoutFull);
      if (!ok) break;
      tc_fence_after();
      const uint32_t pa = smem_u32(p_s), sa = smem_u32(ds_s);
#pragma unroll
      for (int kk = 0; kk < kBQ / 16; ++kk) {   // contraction over the 128 queries
        const uint32_t acc = (it > 0 || kk > 0) ? 1u : 0u;
        umma_f16_lohi(tm_dv, sw128_desc_lo(pa, kHalf) + ((kk * 2048) >> 4), sw128_desc_hi(1024),
                      sw128_desc_lo(da, kHalf) + ((kk * 2048) >> 4), sw128_desc_hi(1024), id_mm, acc);
        umma_f16_lohi(tm_dk, sw128_desc_lo(sa, kHalf) + ((kk * 2048) >> 4), sw128_desc_hi(1024),
                      sw128_desc_lo(qa, kHalf) + ((kk * 2048) >> 4), sw128_desc_hi(1024), id_mm, acc);
      }
      umma_commit(smem_u32(&ctrl->it_empty));
    }
    umma_commit(smem_u32(&ctrl->done));
  }

  if (warp >= 2) {
    const int qrt = warp & 3;
    const int ch = (warp - 2) >> 2;   // 64-column half handled by this thread of the row pair
    const int row = qrt * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(qrt * 32) << 16;
    const float sl2 = p.scale * 1.4426950408889634f;
    bool ok = true;
    for (int it = 0; it < n_it; ++it) {
      const int g = it / n_i, i = i_begin + it % n_i;
      const int h = hk * G + g;
      const int qi = i * kBQ + row;
      const int qpos = qi + off;
      const bool q_ok = qi < p.Sq;
      const float lse2 = q_ok ? p.lse[((long long)b * p.H + h) * p.Sq + qi] * 1.4426950408889634f : 0.f;
      const float dl = q_ok ? p.delta[((long long)b * p.H + h) * p.Sq + qi] : 0.f;
      if (ok) ok = mbar_wait(smem_u32(&ctrl->sdp_full), it & 1, abort_flag, p.status,
                             kStatusTimeoutTmemFull);
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after();
      // interior tiles (all 128 x 128 pairs visible) skip the per-element visibility test
      const bool full_tile = (key0 + kBK - 1 <= i * kBQ + off) && (key0 >= lp) &&
                             (key0 + kBK <= p.Sk) && (i * kBQ + kBQ <= p.Sq);
#pragma unroll
      for (int cc = 0; cc < 64; cc += 32) {
        const int c = ch * 64 + cc;
        float sv[32], dp[32];
        if (ok) {
          tmem_ld_x32(tm_s + lane_off + c, sv);
          tmem_ld_x32(tm_dp + lane_off + c, dp);
        }
        tmem_ld_wait();
        if (full_tile) {
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const float pr = ex2_approx(sv[e] * sl2 - lse2);
            sv[e] = pr;
            dp[e] = pr * (dp[e] - dl) * p.scale;
          }
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const int j = key0 + c + e;
            const bool vis = q_ok && (((j <= qpos) && (j >= lp)) || (j == qpos)) && j < p.Sk;
            const float pr = vis ? ex2_approx(sv[e] * sl2 - lse2) : 0.f;
            sv[e] = pr;
            dp[e] = pr * (dp[e] - dl) * p.scale;
          }
        }
        store_row32(p_s, row, c, sv);
        store_row32(ds_s, row, c, dp);
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctrl->pds_full));
    }
    if (ok) ok = mbar_wait(smem_u32(&ctrl->done), 0, abort_flag, p.status, kStatusTimeoutTmemFull);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    const int kj = key0 + row;
    if (ok) {
      __nv_bfloat16* dkrow = p.dk + (long long)b * p.k_sb + (long long)kj * p.k_ss + (long long)hk * p.k_sh;
      __nv_bfloat16* dvrow = p.dv + (long long)b * p.k_sb + (long long)kj * p.k_ss + (long long)hk * p.k_sh;
#pragma unroll
      for (int cc = 0; cc < D / 2; cc += 32) {
        const int c = ch * (D / 2) + cc;
        float a[32], bq[32];
        if (n_it > 0) {
          tmem_ld_x32(tm_dv + lane_off + c, a);
          tmem_ld_x32(tm_dk + lane_off + c, bq);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) a[e] = bq[e] = 0.f;
        }
        if (kj < p.Sk) {
#pragma unroll
          for (int e = 0; e < 32; e += 8) {
            uint32_t pv[4], pk[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const __nv_bfloat162 x = __floats2bfloat162_rn(a[e + 2 * u], a[e + 2 * u + 1]);
              const __nv_bfloat162 y = __floats2bfloat162_rn(bq[e + 2 * u], bq[e + 2 * u + 1]);
              pv[u] = *reinterpret_cast<const uint32_t*>(&x);
              pk[u] = *reinterpret_cast<const uint32_t*>(&y);
            }
            *reinterpret_cast<uint4*>(dvrow + c + e) = make_uint4(pv[0], pv[1], pv[2], pv[3]);
            *reinterpret_cast<uint4*>(dkrow + c + e) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(ctrl->tmem_base, 512);
}

template <int D>
__global__ void __launch_bounds__(kBwdThreads, 1)
flash_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                    const FlashBwdParams p) {
  constexpr int NH = D / 64;
  constexpr int kHalf = 128 * 128;
  constexpr int kTile = NH * kHalf;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  BwdCtrl* ctrl = reinterpret_cast<BwdCtrl*>(smem);
  uint8_t* q_s = smem + 1024;
  uint8_t* do_s = q_s + kTile;
  uint8_t* k_s = do_s + kTile;
  uint8_t* v_s = k_s + kTile;
  uint8_t* ds_s = v_s + kTile;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the last query tiles meet the most key tiles: launch them first (longest work first)
  const int qb = gridDim.x - 1 - blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int hk = h / (p.H / p.Hkv);
  const int q0 = qb * kBQ;
  const int off = p.Sk - p.Sq;
  const int lp = p.left_pad ? p.left_pad[b] : 0;
  const int last_key = min(p.Sk - 1, q0 + kBQ - 1 + off);
  const int first_key = max(0, min(lp, q0 + off));
  const int j_begin = first_key / kBK;
  const int n_it = last_key / kBK + 1 - j_begin;
  volatile int* abort_flag = &ctrl->abort_flag;

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&ctrl->once_full), 1);
    mbar_init(smem_u32(&ctrl->it_full), 1);
    mbar_init(smem_u32(&ctrl->it_empty), 1);
    mbar_init(smem_u32(&ctrl->sdp_full), 1);
    mbar_init(smem_u32(&ctrl->pds_full), 8);   // one arrival per compute warp
    mbar_init(smem_u32(&ctrl->done), 1);
    ctrl->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&ctrl->tmem_base), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm_s = ctrl->tmem_base, tm_dp = tm_s + 128, tm_dq = tm_s + 256;

  if (warp == 0 && lane == 0) {
    mbar_expect_tx(smem_u32(&ctrl->once_full), 2 * kTile);
#pragma unroll
    for (int hf = 0; hf < NH; ++hf) {
      tma_load_4d(smem_u32(q_s + hf * kHalf), &tmQ, hf * 64, q0, h, b, smem_u32(&ctrl->once_full));
      tma_load_4d(smem_u32(do_s + hf * kHalf), &tmDO, hf * 64, q0, h, b, smem_u32(&ctrl->once_full));
    }
    for (int it = 0; it < n_it; ++it) {
      const int k0 = (j_begin + it) * kBK;
      if (!mbar_wait(smem_u32(&ctrl->it_empty), (it & 1) ^ 1, abort_flag, p.status,
                     kStatusTimeoutEmpty))
        break;
      mbar_expect_tx(smem_u32(&ctrl->it_full), 2 * kTile);
#pragma unroll
      for (int hf = 0; hf < NH; ++hf) {
        tma_load_4d(smem_u32(k_s + hf * kHalf), &tmK, hf * 64, k0, hk, b, smem_u32(&ctrl->it_full));
        tma_load_4d(smem_u32(v_s + hf * kHalf), &tmV, hf * 64, k0, hk, b, smem_u32(&ctrl->it_full));
      }
    }
  } else if (warp == 1 && lane == 0) {
    const uint32_t id_kk = make_idesc_bf16(128, 128, 0, 0);
    const uint32_t id_dq = make_idesc_bf16(128, D, 0, 1);     // dQ = dS K: K tile is MN-major
    bool ok = mbar_wait(smem_u32(&ctrl->once_full), 0, abort_flag, p.status, kStatusTimeoutFull);
    for (int it = 0; it < n_it && ok; ++it) {
      ok = mbar_wait(smem_u32(&ctrl->it_full), it & 1, abort_flag, p.status, kStatusTimeoutFull);
      if (!ok) break;
      tc_fence_after();
      const uint32_t qa = smem_u32(q_s), ka = smem_u32(k_s), va = smem_u32(v_s), da = smem_u32(do_s);
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t o = (kk / 4) * kHalf + (kk % 4) * 32;
        umma_f16_lohi(tm_s, sw128_desc_lo(qa, 16) + ((o) >> 4), sw128_desc_hi(1024),
                      sw128_desc_lo(ka, 16) + ((o) >> 4), sw128_desc_hi(1024), id_kk,
                 kk > 0 ? 1u : 0u);
      }
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        const uint32_t o = (kk / 4) * kHalf + (kk % 4) * 32;
        umma_f16_lohi(tm_dp, sw128_desc_lo(da, 16) + ((o) >> 4), sw128_desc_hi(1024),
                      sw128_desc_lo(va, 16) + ((o) >> 4), sw128_desc_hi(1024), id_kk,
                 kk > 0 ? 1u : 0u);
      }
      umma_commit(smem_u32(&ctrl->sdp_full));
      ok = mbar_wait(smem_u32(&ctrl->pds_full), it & 1, abort_flag, p.status, kStatusTimeoutFull);
      if (!ok) break;
      tc_fence_after();
      const uint32_t sa = smem_u32(ds_s);
#pragma unroll
      for (int kk = 0; kk < kBK / 16; ++kk) {   // contraction over the 128 keys
        umma_f16_lohi(tm_dq, sw128_desc_lo(sa, 16) + (((kk / 4) * kHalf + (kk % 4) * 32) >> 4), sw128_desc_hi(1024),
                      sw128_desc_lo(ka, kHalf) + ((kk * 2048) >> 4), sw128_desc_hi(1024), id_dq, (it > 0 || kk > 0) ? 1u : 0u);
      }
      umma_commit(smem_u32(&ctrl->it_empty));
    }
    umma_commit(smem_u32(&ctrl->done));
  }

  if (warp >= 2) {
    const int qrt = warp & 3;
    const int ch = (warp - 2) >> 2;   // 64-column half handled by this thread of the row pair
    const int row = qrt * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(qrt * 32) << 16;
    const float sl2 = p.scale * 1.4426950408889634f;
    const int qi = q0 + row, qpos = qi + off;
    const bool q_ok = qi < p.Sq;
    const float lse2 = q_ok ? p.lse[((long long)b * p.H + h) * p.Sq + qi] * 1.4426950408889634f : 0.f;
    const float dl = q_ok ? p.delta[((long long)b * p.H + h) * p.Sq + qi] : 0.f;
    bool ok = true;
    for (int it = 0; it < n_it; ++it) {
      const int key0 = (j_begin + it) * kBK;
      if (ok) ok = mbar_wait(smem_u32(&ctrl->sdp_full), it & 1, abort_flag, p.status,
                             kStatusTimeoutTmemFull);
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after();
      const bool full_tile = (key0 + kBK - 1 <= q0 + off) && (key0 >= lp) &&
                             (key0 + kBK <= p.Sk) && (q0 + kBQ <= p.Sq);
#pragma unroll
      for (int cc = 0; cc < 64; cc += 32) {
        const int c = ch * 64 + cc;
        float sv[32], dp[32];
        if (ok) {
          tmem_ld_x32(tm_s + lane_off + c, sv);
          tmem_ld_x32(tm_dp + lane_off + c, dp);
        }
        tmem_ld_wait();
        if (full_tile) {
#pragma unroll
          for (int e = 0; e < 32; ++e)
            dp[e] = ex2_approx(sv[e] * sl2 - lse2) * (dp[e] - dl) * p.scale;
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const int j = key0 + c + e;
            const bool vis = q_ok && (((j <= qpos) && (j >= lp)) || (j == qpos)) && j < p.Sk;
            const float pr = vis ? ex2_approx(sv[e] * sl2 - lse2) : 0.f;
            dp[e] = pr * (dp[e] - dl) * p.scale;
          }
        }
        store_row32(ds_s, row, c, dp);
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctrl->pds_full));
    }
    if (ok) ok = mbar_wait(smem_u32(&ctrl->done), 0, abort_flag, p.status, kStatusTimeoutTmemFull);
    ok = __all_sync(0xffffffffu, ok);
    tc_fence_after();
    if (ok) {   // warp-uniform: the TMEM loads are warp-collective, only the stores are per row
      __nv_bfloat16* dqrow = p.dq + (long long)b * p.q_sb + (long long)qi * p.q_ss + (long long)h * p.q_sh;
#pragma unroll
      for (int cc = 0; cc < D / 2; cc += 32) {
        const int c = ch * (D / 2) + cc;
        float a[32];
        if (n_it > 0) {
          tmem_ld_x32(tm_dq + lane_off + c, a);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e) a[e] = 0.f;
        }
        if (!q_ok) continue;
#pragma unroll
        for (int e = 0; e < 32; e += 8) {
          uint32_t pk[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const __nv_bfloat162 x = __floats2bfloat162_rn(a[e + 2 * u], a[e + 2 * u + 1]);
            pk[u] = *reinterpret_cast<const uint32_t*>(&x);
          }
          *reinterpret_cast<uint4*>(dqrow + c + e) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(ctrl->tmem_base, 512);
}

}  // namespace e2h

// q: [B, Sq, H, D] view (strides q_sb, q_ss, q_sh); k, v: [B, Sk, Hkv, D] views; out like q.
extern "C" int e2h_flash_fwd(const void* q, long long q_sb, long long q_ss, long long q_sh,
                             const void* k, const void* v, long long k_sb, long long k_ss,
                             long long k_sh, void* out, long long o_sb, long long o_ss,
                             long long o_sh, float* lse, const int* left_pad, int B, int H,
                             int Hkv, int Sq, int Sk, int D, float scale, int* status,
                             void* stream) {
  using namespace e2h;
  if (D != 128 && D != 64) return -1;
  if (H % Hkv) return -2;
  if ((q_ss % 8) || (q_sh % 8) || (q_sb % 8) || (k_ss % 8) || (k_sh % 8) || (k_sb % 8)) return -3;
  CUtensorMap tq, tk, tv;
  int r = make_map4d(&tq, q, D, Sq, H, B, q_sb, q_ss, q_sh, kBQ);
  if (r) return r;
  r = make_map4d(&tk, k, D, Sk, Hkv, B, k_sb, k_ss, k_sh, kFK);
  if (r) return r;
  r = make_map4d(&tv, v, D, Sk, Hkv, B, k_sb, k_ss, k_sh, kFK);
  if (r) return r;
  FwdParams p;
  p.B = B; p.H = H; p.Hkv = Hkv; p.Sq = Sq; p.Sk = Sk; p.D = D;
  p.scale = scale; p.left_pad = left_pad;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.o_sb = o_sb; p.o_ss = o_ss; p.o_sh = o_sh;
  p.lse = lse; p.status = status;
  if (Sq <= 0 || B <= 0 || H <= 0) return 0;
  p.pair_heads = (H / Hkv) % 2 == 0;
  const int rows = p.pair_heads ? kBQ : 2 * kBQ;
  p.n_qb = (Sq + rows - 1) / rows;
  p.nh = p.pair_heads ? H / 2 : H;
  const long long heads = (long long)p.nh * B, items = heads * p.n_qb;
  if (items > INT_MAX - 1024) return -4;
  p.heads = (int)heads;
  p.m_heads = fast_div_of(p.heads);
  p.m_nh = fast_div_of(p.nh);
  p.m_group = fast_div_of(H / Hkv);
  const int grid = items < 148 ? (int)items : 148;
  const size_t smem = 2048 + (size_t)(D / 64) * (2 * 128 + 2 * kFwdSlots * kFK) * 128;
  cudaError_t e;
  if (D == 128) {
    static SmemAsk ask;
    e = ask(flash_fwd_kernel<128>, smem);
    if (e != cudaSuccess) return (int)e;
    flash_fwd_kernel<128><<<grid, kFwdThreads, smem, (cudaStream_t)stream>>>(tq, tk, tv, p);
  } else {
    static SmemAsk ask;
    e = ask(flash_fwd_kernel<64>, smem);
    if (e != cudaSuccess) return (int)e;
    flash_fwd_kernel<64><<<grid, kFwdThreads, smem, (cudaStream_t)stream>>>(tq, tk, tv, p);
  }
  return (int)cudaGetLastError();
}

// dO, O: [B, Sq, H, D] views; dq like q; dk, dv like k. delta: fp32 scratch [B, H, Sq].
extern "C" int e2h_flash_bwd(const void* q, long long q_sb, long long q_ss, long long q_sh,
                             const void* k, const void* v, long long k_sb, long long k_ss,
                             long long k_sh, const void* o, long long o_sb, long long o_ss,
                             long long o_sh, const void* d_o, long long do_sb, long long do_ss,
                             long long do_sh, const float* lse, float* delta, void* dq, void* dk,
                             void* dv, const int* left_pad, int B, int H, int Hkv, int Sq, int Sk,
                             int D, float scale, int* status, void* stream_v) {
  using namespace e2h;
  cudaStream_t stream = (cudaStream_t)stream_v;
  if (D != 128 && D != 64) return -1;
  if (H % Hkv) return -2;
  CUtensorMap tq, tk, tv, tdo;
  int r = make_map4d(&tq, q, D, Sq, H, B, q_sb, q_ss, q_sh, kBQ);
  if (r) return r;
  r = make_map4d(&tk, k, D, Sk, Hkv, B, k_sb, k_ss, k_sh, kBK);
  if (r) return r;
  r = make_map4d(&tv, v, D, Sk, Hkv, B, k_sb, k_ss, k_sh, kBK);
  if (r) return r;
  r = make_map4d(&tdo, d_o, D, Sq, H, B, do_sb, do_ss, do_sh, kBQ);
  if (r) return r;
  {
    const int warps = H * Sq;
    dim3 grid((warps * 32 + 255) / 256, B);
    flash_delta_kernel<<<grid, 256, 0, stream>>>(
        (const __nv_bfloat16*)o, (const __nv_bfloat16*)d_o, delta, o_sb, o_ss, o_sh, do_sb, do_ss,
        do_sh, H, Sq, D);
  }
  FlashBwdParams p;
  p.B = B; p.H = H; p.Hkv = Hkv; p.Sq = Sq; p.Sk = Sk; p.D = D;
  p.scale = scale; p.left_pad = left_pad; p.lse = lse; p.delta = delta;
  p.dq = (__nv_bfloat16*)dq; p.dk = (__nv_bfloat16*)dk; p.dv = (__nv_bfloat16*)dv;
  p.q_sb = q_sb; p.q_ss = q_ss; p.q_sh = q_sh; p.k_sb = k_sb; p.k_ss = k_ss; p.k_sh = k_sh;
  p.status = status;
  const int tile = (D / 64) * 128 * 128;
  const size_t smem_kv = 2048 + 4 * (size_t)tile + 4 * 128 * 128;
  const size_t smem_q = 2048 + 4 * (size_t)tile + 2 * 128 * 128;
  dim3 gkv((Sk + kBK - 1) / kBK, Hkv, B), gq((Sq + kBQ - 1) / kBQ, H, B);
  cudaError_t e;
#define E2H_BWD(D_)                                                                              \
  {                                                                                              \
    static SmemAsk ask_kv, ask_q;                                                                \
    e = ask_kv(flash_bwd_dkdv_kernel<D_>, smem_kv);                                              \
    if (e == cudaSuccess) e = ask_q(flash_bwd_dq_kernel<D_>, smem_q);                            \
    if (e != cudaSuccess) return (int)e;                                                         \
    flash_bwd_dkdv_kernel<D_><<<gkv, kBwdThreads, smem_kv, stream>>>(tq, tk, tv, tdo, p);                \
    flash_bwd_dq_kernel<D_><<<gq, kBwdThreads, smem_q, stream>>>(tq, tk, tv, tdo, p);                    \
  }
  if (D == 128) E2H_BWD(128) else E2H_BWD(64)
#undef E2H_BWD
  return (int)cudaGetLastError();
}
