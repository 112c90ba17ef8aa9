// Mask-free attention (joint text+image self-attention, Wan self- and
// cross-attention) as a tcgen05 flash-attention kernel, head_dim 128, bf16.
//
// A CTA pair (two SMs of a cluster) owns 256 query rows of one (batch, head), 128 per CTA, and streams the keys/values
// in tiles of 128 through cta_group::2 MMAs: each CTA stages half of every K tile (64 keys) and half of every V tile
// (64 of the 128 value columns) and the tensor cores of both read both halves.  The grid is persistent: pair u works
// through items u, u + pairs, ... so the prologue of one item runs under the end of the one before.  Roles per CTA:
//   warp 0      TMA producer of Q (two buffers) and of a 4-stage ring of K half tiles; warp 2: the same ring for V (one
//               thread for all of it takes about 900 cycles per tile, nearly the tile's tensor time)
//   warp 1      MMA issuer (leader CTA only): S_t = Q K_j^T (SS, both operands K-major), O += P_t V_j (TS: P read from
//               TMEM, V MN-major).  The whole warp runs the loop, one elected lane issues.
//   warps 4-7   epilogue: O (TMEM) and the groups' row sums -> output rows, while the next item is already running
//   warps 8-19  three softmax groups of four warps, one thread per query row; group t takes key tiles t, t+3, ...
// TMEM (512 columns): S_0 | S_1 | S_2 | O, 128 fp32 columns each.  A softmax thread turns the 128 scores of its row
// into 64 columns of packed bf16 probabilities written over the first half of the same S (it is always ahead of
// itself: chunk c of 32 scores becomes columns [16c, 16c+16)).  S_t(j+3) is issued right behind O += P_t(j) V_j.
//
// Why three score tiles in flight: one key tile is a serial chain S-MMA (512 tensor cycles) -> wake-up -> 128
// exponentials per row (1024 MUFU cycles) -> hand-over -> P.V (512) of more than 3000 cycles with its hops, of which the
// tensor core and the MUFU are each needed for 1024.  With two query tiles per CTA and S | S | O | O in TMEM only two
// chains can be in flight (2 tiles per ~3450 cycles, tensor pipe 56 %); one query tile per CTA with S | S | S | O has
// three (a tile per ~1490 cycles, 68 %).  What that would cost in shared-memory and L2 traffic (K and V serve 128 rows
// instead of 256) the pair gives back: each SM stages and reads half of every K and V tile.  Short key ranges gain most,
// because an item's Q load, first tile and epilogue now run under its neighbours.  Measured, this form against two query
// tiles per CTA: 24 heads x 4608 229 -> 203 us, 40 heads x 32760 queries x 512 keys 596 -> 348 us, 5 heads x 32768 x
// 32760 2387 -> 2022 us (bursts); under the 1000 W cap 263 -> 232 us, 595 -> 407 us.  Whole-chip runs are bound by that
// cap (1.5 GHz), so instructions count even where issue slots are free: tracking the maximum and cutting the exponents
// score by score was 3 us of the 203; a quarter of the exponentials as a polynomial on the FMA pipe took 4 % of the cycles
// away and gave all of it back in clock.
//
// Exponentials are taken against a reference m_ref per row, shared by the three groups and handed from tile to tile
// (`mslot`).  The first tile sets it to ceil(row maximum); after that the thread of a tile moves it, before it has
// looked at the tile, to the largest exponent that it saw in its own earlier tiles, if that is more than 2^8 above.  So
// the reference trails by up to three tiles, and no maximum sits on the chain above; a tile's entries that exceed it
// simply give p > 1, and row sums and O carry the same reference.  When a reference moves, O is rescaled in place by that
// thread, between O += P(j-1) V (it waits for it) and O += P(j) V (which needs its own P).
//
// Entries that are more than 2^100 above the reference would leave the range of p.  A tile that meets one (its sums tell)
// goes on against a higher reference of its own: what it has of P and of the row sum is scaled down, and O too before P is
// handed over.  The tiles behind it, which may have started with the lower reference, learn of that through a second chain
// (`fin`: one word per warp of rows, written when a tile's P is complete; `fref`: the rows' references, written only when
// one is above what `mslot` gave), and scale their P down before they hand it over.  So O, P and the sums always agree,
// however steeply a row climbs, and nothing is cut.
//
// m_ref is always an INTEGER (in log2 units): rescaling by 2^(integer) is exact in floating point, so the bf16
// rounding of a probability does not depend on which reference it was computed against.  The result therefore equals
// "P = bf16(exp2(s*c - M)), O = P V / sum(exp2(s*c - M))" for ANY integer M, whatever the tile schedule - which is
// what the CPU restatement used by the parity tests evaluates (with M = ceil of the row maximum).
#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "dsb.h"

namespace dsb {

constexpr int kTileQ = 128;   // query rows per CTA
constexpr int kPairQ = 256;   // ... and per CTA pair: the rows of one work item
constexpr int kTileKV = 128;
constexpr int kGroups = 3;    // softmax groups = score tiles in TMEM
constexpr int kQBufs = 2;
constexpr int kRing = 4;      // stages of the K and of the V ring
constexpr int kSumSlots = 8;  // items whose row sums may be published before the epilogue has read them, see below
constexpr int kTmaWarp = 0, kMmaWarp = 1, kTmaVWarp = 2;  // warp 3 only completes the control warps' warpgroup
constexpr int kEpiWarp0 = 4, kSoftmaxWarp0 = 8;
constexpr int kAttnThreads = (kSoftmaxWarp0 + 4 * kGroups) * 32;
// 640 threads are launched with 96 registers each; the control warpgroup gives 48 of its away, 16 for each softmax
// thread (32 scores and 16 packed probabilities at a time): 3 x 112 + 96 + 48 = 5 x 96.
constexpr int kSoftmaxRegs = 112, kControlRegs = 48;
static_assert(kAttnThreads == 640, "the register split assumes five warpgroups");
constexpr int kQBytes = kTileQ * 256;              // two 64-column halves of 128 rows
constexpr int kKBytes = (kTileKV / 2) * 256;       // 64 keys, two 64-column halves
constexpr int kVBytes = kTileKV * 128;             // 128 keys, 64 value columns
constexpr int kBarBytes = 512;
constexpr int kAttnSmem = kQBufs * kQBytes + kRing * (kKBytes + kVBytes) + kBarBytes + kTileQ * 8 +
                          kSumSlots * kGroups * kTileQ * 8 + kTileQ * 4 + 1024;

constexpr int kMaxParts = 8;
constexpr int kWsRow = 132;  // floats per row of a partial result (528 bytes: rows stay 16-byte aligned)
// The query rows (and, independently, the output rows) may be cut into up to kMaxParts equal row ranges that live in
// different buffers - e.g. in the memory of different GPUs of a sequence-parallel group, where rank r holds the
// queries of its own tokens and receives the output rows of its own tokens from every rank.
struct AttnQMaps {
  CUtensorMap m[kMaxParts];
};
struct AttnParams {
  __nv_bfloat16* o;
  __nv_bfloat16* o_part[kMaxParts];
  int out_e4m3;         // 1: the output is written as e4m3 (1 byte per element; strides count elements = bytes)
  // Work items (256 query rows of one head) are numbered query tile fastest, then head, then sample.  Items from n_full
  // on - the ones that would form a partly filled last wave - are each cut into `split` units over contiguous key
  // ranges; those leave unnormalised partial results in `ws` and attn_combine_kernel finishes the rows.
  int n_pairs, n_full, split, n_units, H;
  float* ws;            // [tail item][part][256 rows][kWsRow floats]: 128 output columns, reference exponent, row sum
  int q_rows_per_part;  // 0: one query buffer (map 0); else a multiple of kTileQ
  int o_rows_per_part;  // 0: one output buffer (o); else row s goes to o_part[s / o_rows_per_part]
  int64_t o_stride_b, o_stride_s, o_stride_h;
  int Sq, Sk;
  float scale_log2;  // sm_scale * log2(e)
  // position of the (s, h, b) coordinates inside the tensor-map coordinate list (after d)
  int q_pos[3], k_pos[3], v_pos[3];
  int* status;
};

// The reference of a query row on its way from the thread of one key tile to the thread of the next: a 64-bit slot
// {sequence number, value} written with one store; the reader spins (bounded) until the number it expects is there.
__device__ __forceinline__ void ref_publish(unsigned long long* slot, uint32_t seq, float v) {
  *reinterpret_cast<volatile unsigned long long*>(slot) =
      (static_cast<unsigned long long>(seq) << 32) | static_cast<unsigned long long>(__float_as_uint(v));
}
__device__ __forceinline__ bool ref_read(const unsigned long long* slot, uint32_t seq, float* v, volatile int* abort_flag) {
  unsigned long long w = *reinterpret_cast<const volatile unsigned long long*>(slot);
  if (static_cast<uint32_t>(w >> 32) != seq) {
    const long long t0 = clock64();
    uint32_t spins = 0;
    do {
      if (((++spins) & 0xffu) == 0) {
        if (*abort_flag) return false;
        if (clock64() - t0 > kWaitLimitCycles) {
          *abort_flag = 1;
          return false;
        }
      }
      w = *reinterpret_cast<const volatile unsigned long long*>(slot);
    } while (static_cast<uint32_t>(w >> 32) != seq);
  }
  *v = __uint_as_float(static_cast<uint32_t>(w));
  return true;
}
// The word that says what O's references are once a tile has been added to it: twice {tile number + 1}, plus one if some row
// of the warp has a reference above the one handed on in its slot.  Waits (bounded) for the word of the tile before `t`.
__device__ __forceinline__ bool fin_read(const volatile uint32_t* word, uint32_t t, bool* above, volatile int* abort_flag) {
  uint32_t w = *word;
  if ((w ^ (t << 1)) > 1u) {
    const long long t0 = clock64();
    uint32_t spins = 0;
    do {
      if (((++spins) & 0xffu) == 0) {
        if (*abort_flag) return false;
        if (clock64() - t0 > kWaitLimitCycles) {
          *abort_flag = 1;
          return false;
        }
      }
      w = *word;
    } while ((w ^ (t << 1)) > 1u);
  }
  *above = (w & 1) != 0;
  return true;
}

// Coordinates (s, h, b) in the order of a tensor map, kept in registers: only s changes inside an item.
struct BoxCoords {
  int c0, c1, c2;
  bool s0, s1;  // which of them is s (the third if neither)
  __device__ __forceinline__ BoxCoords(const int (&pos)[3], int h, int b) {
    s0 = pos[0] == 0, s1 = pos[0] == 1;
    c0 = pos[1] == 0 ? h : b;
    c1 = pos[1] == 1 ? h : b;
    c2 = pos[1] == 2 ? h : b;
  }
  __device__ __forceinline__ void load(uint8_t* dst, const CUtensorMap* m, uint32_t bar, int d0, int s) const {
    tma_load_4d_cg2(dst, m, bar, d0, s0 ? s : c0, s1 ? s : c1, (s0 || s1) ? c2 : s);
  }
};

// One unit of work of a pair: 256 query rows from q0 on, of head h of sample b, against key tiles [jb, jb + nkv).
struct AttnUnit {
  int q0, h, b, jb, nkv;
  int tail_part;  // SPLIT: (tail item) * split + part, or -1 for an item that is not cut
};
template <bool SPLIT>
__device__ __forceinline__ AttnUnit attn_unit(const AttnParams& p, int u) {
  AttnUnit w;
  int item = u, part = 0;
  w.tail_part = -1;
  if constexpr (SPLIT) {
    if (u >= p.n_full) {
      w.tail_part = u - p.n_full;
      part = w.tail_part % p.split;
      item = p.n_full + w.tail_part / p.split;
    }
  }
  const int bh = item / p.n_pairs;
  w.q0 = (item - bh * p.n_pairs) * kPairQ;
  w.b = bh / p.H;
  w.h = bh - w.b * p.H;
  const int all = (p.Sk + kTileKV - 1) / kTileKV;
  w.jb = 0, w.nkv = all;
  if (SPLIT && w.tail_part >= 0) {
    w.jb = static_cast<int>(static_cast<int64_t>(part) * all / p.split);
    w.nkv = static_cast<int>(static_cast<int64_t>(part + 1) * all / p.split) - w.jb;
  }
  return w;
}

// 2^(from - to) for integers from <= to (0 when that underflows)
__device__ __forceinline__ float pow2_down(float from, float to) {
  return __int_as_float(max(0, 127 + static_cast<int>(from - to)) << 23);
}

// 16 scores -> 16 probabilities (packed bf16) against the reference, and their sum.  CHECK: columns from `valid` on do not
// exist, and the largest exponent is kept - relative to the reference (1), or by itself (2), which costs a product per score
// and is exact however far the reference is away.
template <int CHECK>
__device__ __forceinline__ void exp_pairs(const uint32_t (&a)[16], uint32_t* pk, float2 cs2, float2 nm2, float2 (&sum)[2],
                                          int valid, float* mx) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 s = make_float2(__uint_as_float(a[2 * i]), __uint_as_float(a[2 * i + 1]));
    const float2 x = __ffma2_rn(s, cs2, nm2);
    float2 pp = make_float2(fast_exp2(x.x), fast_exp2(x.y));
    if constexpr (CHECK != 0) {
      const float2 e = CHECK == 2 ? __fmul2_rn(s, cs2) : x;
      if (2 * i < valid) *mx = fmaxf(*mx, e.x);
      else pp.x = 0.f;
      if (2 * i + 1 < valid) *mx = fmaxf(*mx, e.y);
      else pp.y = 0.f;
    }
    sum[i & 1] = __fadd2_rn(sum[i & 1], pp);
    pk[i] = pack_bf16x2(pp.x, pp.y);
  }
}
// 16 columns of TMEM that hold fp32 values (BF16: pairs of bf16) times a power of two
template <bool BF16>
__device__ __forceinline__ void scale_columns(uint32_t taddr, float f) {
  uint32_t r[16];
  tmem_ld16(taddr, r);
  tc_wait_ld_regs(r);
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    if constexpr (BF16) {
      const float2 v = unpack_bf16x2(r[i]);
      r[i] = pack_bf16x2(v.x * f, v.y * f);
    } else {
      r[i] = __float_as_uint(__uint_as_float(r[i]) * f);
    }
  }
  tmem_st16(taddr, r);
}
__device__ __forceinline__ void max_chunk(const uint32_t (&a)[32], float (&mx)[4], bool neg) {
  if (!neg) {
#pragma unroll
    for (int i = 0; i < 16; ++i) mx[i & 3] = max3f(mx[i & 3], __uint_as_float(a[2 * i]), __uint_as_float(a[2 * i + 1]));
  } else {  // a negative scale turns the largest exponent into the smallest score
#pragma unroll
    for (int i = 0; i < 16; ++i) mx[i & 3] = min3f(mx[i & 3], __uint_as_float(a[2 * i]), __uint_as_float(a[2 * i + 1]));
  }
}

// SPLIT: the launch has items cut along the keys (see AttnParams); the plain instantiation carries none of that code.
template <bool SPLIT>
__global__ void __launch_bounds__(kAttnThreads, 1)
    flash_attn_kernel(const __grid_constant__ AttnQMaps qmaps, const __grid_constant__ CUtensorMap tmap_k,
                      const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + kQBufs * kQBytes;
  uint8_t* sV = sK + kRing * kKBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + kRing * kVBytes);
  // barriers marked (L) count both CTAs' events in the leader CTA; the *_empty, s_full and o_full ones are signalled by the
  // MMA's commits in both CTAs
  uint64_t* q_full = bars;               // kQBufs (L)
  uint64_t* q_empty = q_full + kQBufs;   // kQBufs
  uint64_t* k_full = q_empty + kQBufs;   // kRing (L)
  uint64_t* k_empty = k_full + kRing;    // kRing
  uint64_t* v_full = k_empty + kRing;    // kRing (L)
  uint64_t* v_empty = v_full + kRing;    // kRing: also "O holds P.V of this tile"
  uint64_t* s_full = v_empty + kRing;    // kGroups
  uint64_t* p_full = s_full + kGroups;   // kGroups (L): P of the tile is in TMEM
  uint64_t* o_full = p_full + kGroups;   // 1
  uint64_t* o_empty = o_full + 1;        // 1 (L)
  uint64_t* l_full = o_empty + 1;        // kSumSlots
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(l_full + kSumSlots);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile uint32_t* fin = tmem_slot + 2;  // one word per warp of rows (four)
  unsigned long long* mslot = reinterpret_cast<unsigned long long*>(reinterpret_cast<uint8_t*>(bars) + kBarBytes);
  float2* sums = reinterpret_cast<float2*>(mslot + kTileQ);  // [kSumSlots][kGroups][kTileQ] {row sum, its reference}
  volatile float* fref = reinterpret_cast<volatile float*>(sums + kSumSlots * kGroups * kTileQ);  // per row, see above

  // a warp index that the compiler can see to be uniform: the roles' code then keeps its addresses in uniform registers
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader_cta = rank == 0;
  const int unit0 = blockIdx.x >> 1, n_pairs_grid = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kQBufs; ++i) mbar_init(&q_full[i], 1), mbar_init(&q_empty[i], 1);
    for (int i = 0; i < kRing; ++i) {
      mbar_init(&k_full[i], 1), mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1), mbar_init(&v_empty[i], 1);
    }
    for (int i = 0; i < kGroups; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 8);  // four warps of each CTA
    }
    mbar_init(o_full, 1);
    mbar_init(o_empty, 8);
    for (int i = 0; i < kSumSlots; ++i) mbar_init(&l_full[i], 4 * kGroups);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (threadIdx.x < kTileQ) mslot[threadIdx.x] = 0ull;  // sequence 0 = what the first tile expects
  if (threadIdx.x < 4) fin[threadIdx.x] = 0u;
  if (warp == kTmaWarp && lane == 0) {
    tma_prefetch_desc(&qmaps.m[0]);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
  }
  if (warp == kMmaWarp) {
    tmem_alloc_cg2(tmem_slot, 512);
    tmem_relinquish_cg2();
  }
  tc_fence_before();
  grid_wait();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers are initialised before anyone signals them
  tc_fence_after();
  // All 512 columns are allocated, so the allocation starts at column 0 of lane 0 and TMEM addresses are constants.
  constexpr uint32_t kTmemO = kGroups * 128;
  if (threadIdx.x == 0 && *tmem_slot != 0) *abort_flag = 1;

  if (warp < kEpiWarp0) {
    setmaxnreg_dec<kControlRegs>();
    if (warp == kTmaWarp) {
      // ------------------------------------------------------------ TMA producer of Q and K
      if (lane == 0) {
        const uint32_t b_kf = mapa_u32(smem_u32(k_full), 0), b_qf = mapa_u32(smem_u32(q_full), 0);
        uint32_t n = 0, t = 0;  // items and tiles so far
        for (int u = unit0; u < p.n_units; u += n_pairs_grid, ++n) {
          const AttnUnit w = attn_unit<SPLIT>(p, u);
          const uint32_t qb = n & 1;
          if (!mbar_wait(&q_empty[qb], ((n >> 1) & 1) ^ 1, abort_flag)) goto producer_done;
          {
            int s0 = w.q0 + static_cast<int>(rank) * kTileQ, part = 0;
            if (p.q_rows_per_part > 0) {  // a 128-row tile never straddles two parts
              part = min(s0 / p.q_rows_per_part, kMaxParts - 1);
              s0 -= part * p.q_rows_per_part;
            }
            if (leader_cta) mbar_expect_tx(&q_full[qb], 2 * kQBytes);
            const BoxCoords c(p.q_pos, w.h, w.b);
            c.load(sQ + qb * kQBytes, &qmaps.m[part], b_qf + qb * 8, 0, s0);
            c.load(sQ + qb * kQBytes + kQBytes / 2, &qmaps.m[part], b_qf + qb * 8, 64, s0);
          }
          const BoxCoords c(p.k_pos, w.h, w.b);
          int s0 = w.jb * kTileKV + static_cast<int>(rank) * (kTileKV / 2);
          for (int j = 0; j < w.nkv; ++j, ++t, s0 += kTileKV) {
            const uint32_t st = t & (kRing - 1);
            if (!mbar_wait(&k_empty[st], ((t / kRing) & 1) ^ 1, abort_flag)) goto producer_done;
            if (leader_cta) mbar_expect_tx(&k_full[st], 2 * kKBytes);
            c.load(sK + st * kKBytes, &tmap_k, b_kf + st * 8, 0, s0);
            c.load(sK + st * kKBytes + kKBytes / 2, &tmap_k, b_kf + st * 8, 64, s0);
          }
        }
        grid_release();  // a few key tiles before this CTA is done
      }
    producer_done:;
    } else if (warp == kTmaVWarp) {
      // ------------------------------------------------------------ TMA producer of V
      if (lane == 0) {
        const uint32_t b_vf = mapa_u32(smem_u32(v_full), 0);
        uint32_t t = 0;
        for (int u = unit0; u < p.n_units; u += n_pairs_grid) {
          const AttnUnit w = attn_unit<SPLIT>(p, u);
          const BoxCoords c(p.v_pos, w.h, w.b);
          int s0 = w.jb * kTileKV;
          for (int j = 0; j < w.nkv; ++j, ++t, s0 += kTileKV) {
            const uint32_t st = t & (kRing - 1);
            if (!mbar_wait(&v_empty[st], ((t / kRing) & 1) ^ 1, abort_flag)) goto v_producer_done;
            if (leader_cta) mbar_expect_tx(&v_full[st], 2 * kVBytes);
            c.load(sV + st * kVBytes, &tmap_v, b_vf + st * 8, static_cast<int>(rank) * 64, s0);
          }
        }
      }
    v_producer_done:;
    } else if (warp == kMmaWarp) {
      // -------------------------------------------------------------- MMA issuer
      if (leader_cta) {
        constexpr uint32_t idesc_qk = make_idesc(DFMT_F32, FMT_BF16, FMT_BF16, 0, 0, 256, 128);
        constexpr uint32_t idesc_pv = make_idesc(DFMT_F32, FMT_BF16, FMT_BF16, 0, 1, 256, 128);
        // Every descriptor is the low word of a base (the address field, in 16-byte units, never carries out of it) plus an
        // offset, under one constant high word.
        const uint64_t q_desc0 = make_desc_k_sw128(smem_u32(sQ));
        const uint32_t hi = static_cast<uint32_t>(q_desc0 >> 32), q_lo = static_cast<uint32_t>(q_desc0),
                       k_lo = static_cast<uint32_t>(make_desc_k_sw128(smem_u32(sK))),
                       v_lo = static_cast<uint32_t>(make_desc_mn_sw128(smem_u32(sV), kVBytes, 1024));  // one 64-column chunk
        auto desc = [&](uint32_t l) { return (static_cast<uint64_t>(hi) << 32) | l; };
        const uint32_t b_qf = smem_u32(q_full), b_qe = smem_u32(q_empty), b_kf = smem_u32(k_full), b_ke = smem_u32(k_empty),
                       b_vf = smem_u32(v_full), b_ve = smem_u32(v_empty), b_sf = smem_u32(s_full), b_pf = smem_u32(p_full), b_of = smem_u32(o_full), b_oe = smem_u32(o_empty);
        // The score MMAs run three tiles (across items) ahead of the P.V ones: the first three steps issue scores only.
        // A satisfied wait costs this warp about 100 cycles, most of it the latency of the poll, so the barriers of a step
        // are polled together.
        int qk_u = unit0, qk_left = qk_u < p.n_units ? attn_unit<SPLIT>(p, qk_u).nkv : 0;
        int u = unit0, left = qk_left;
        uint32_t qk_n = 0, n = 0, kt = 0, vt = 0, sb = 0, pph = 1;  // items and tiles so far; score tile; its P phase
        bool q_new = true, o_new = true;
        int lead = kGroups;
        while (u < p.n_units) {
          const bool qk = qk_u < p.n_units;
          const uint32_t kst = kt & (kRing - 1), vst = vt & (kRing - 1), qb = qk_n & 1;
          if (qk && q_new && !mbar_wait_warp<false>(b_qf + qb * 8, (qk_n >> 1) & 1, abort_flag)) goto mma_done;
          const uint32_t k_ok = mbar_peek<false>(b_kf + kst * 8, (kt / kRing) & 1);
          if (lead > 0) {
            --lead;
            if (qk && !mbar_wait_warp<false>(b_kf + kst * 8, (kt / kRing) & 1, abort_flag)) goto mma_done;
          } else {
            const uint32_t v_ok = mbar_peek<false>(b_vf + vst * 8, (vt / kRing) & 1);
            const uint32_t p_ok = mbar_peek<true>(b_pf + sb * 8, pph);
            if (!__all_sync(0xffffffffu, (k_ok & v_ok & p_ok) != 0)) {
              if (qk && !mbar_wait_warp<false>(b_kf + kst * 8, (kt / kRing) & 1, abort_flag)) goto mma_done;
              if (!mbar_wait_warp<false>(b_vf + vst * 8, (vt / kRing) & 1, abort_flag)) goto mma_done;
              if (!mbar_wait_warp<true>(b_pf + sb * 8, pph, abort_flag)) goto mma_done;
            }
            // the epilogue of the item before has read O out
            if (o_new && !mbar_wait_warp<true>(b_oe, (n & 1) ^ 1, abort_flag)) goto mma_done;
            const uint32_t b_lo = v_lo + vst * (kVBytes >> 4), a = sb * 128;
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
              for (int kk = 0; kk < 8; ++kk)  // 16 keys per instruction = 16 rows of 128 bytes of the V tile, 8 columns of P
                mma_f16_pair_ts(kTmemO, a + kk * 8, desc(b_lo + kk * 128u), idesc_pv, (!o_new || kk > 0) ? 1u : 0u);
              tc_commit_pair(b_ve + vst * 8);
              if (left == 1) tc_commit_pair(b_of);
            }
            __syncwarp();
            ++vt;
            o_new = --left == 0;
            if (o_new) {
              ++n;
              u += n_pairs_grid;
              if (u < p.n_units) left = attn_unit<SPLIT>(p, u).nkv;
            }
          }
          // scores of the next tile, into the columns whose probabilities the MMAs above have just consumed
          if (qk) {
            tc_fence_after();
            const uint32_t a_lo = q_lo + qb * (kQBytes >> 4), b_lo = k_lo + kst * (kKBytes >> 4);
            if (elect_one()) {
#pragma unroll
              for (int kk = 0; kk < 8; ++kk)
                mma_f16_pair_ss(sb * 128, desc(a_lo + ((kk >> 2) * (kQBytes / 2 >> 4) + 2 * (kk & 3))),
                                desc(b_lo + ((kk >> 2) * (kKBytes / 2 >> 4) + 2 * (kk & 3))), idesc_qk, kk > 0 ? 1u : 0u);
              tc_commit_pair(b_sf + sb * 8);
              tc_commit_pair(b_ke + kst * 8);
              if (qk_left == 1) tc_commit_pair(b_qe + qb * 8);
            }
            __syncwarp();
            ++kt;
            q_new = --qk_left == 0;
            if (q_new) {
              ++qk_n;
              qk_u += n_pairs_grid;
              if (qk_u < p.n_units) qk_left = attn_unit<SPLIT>(p, qk_u).nkv;
            }
          }
          if (++sb == kGroups) sb = 0, pph ^= 1;
        }
      }
    mma_done:;
    }
  } else if (warp >= kSoftmaxWarp0) {
    // ----------------------------------------------------------------- softmax
    setmaxnreg_inc<kSoftmaxRegs>();
    const int grp = (warp - kSoftmaxWarp0) >> 2, quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t t_s = lane_off + grp * 128;
    const uint32_t t_o = lane_off + kTmemO;
    unsigned long long* slot = mslot + row;
    const float cs = p.scale_log2;
    const bool neg = cs < 0.f;
    const float2 cs2 = make_float2(cs, cs);
    const uint32_t bar_remote = mapa_u32(smem_u32(&p_full[grp]), 0);
    uint32_t sph = 0;
    int g = 0, n = 0, jj = grp;  // tiles of this pair before the item; items before; my next tile inside the item
    // A wait that runs out is noted here and the lane goes on (with whatever it reads) up to the vote below, so that a warp
    // gives up as a whole: a lane that left by itself would let the others' votes and TMEM accesses wait for it.
    bool alive = true;
    for (int u = unit0; u < p.n_units; u += n_pairs_grid, ++n) {
      const AttnUnit w = attn_unit<SPLIT>(p, u);
      float m_ref = 0.f;      // the reference of my last tile
      float run = -INFINITY;  // bounds the largest exponent (score * cs) among my tiles so far
      float2 ls[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      bool first = true;
      int lift_chunk = -1;                    // >= 0: a tile has left the range of p, see behind the loop
      float o_ref = 0.f, lift_grown = 0.f, lift_sum = 0.f;
      for (; jj < w.nkv; jj += kGroups) {
        const uint32_t t = static_cast<uint32_t>(g + jj);
        const int valid = p.Sk - (w.jb + jj) * kTileKV;  // columns of this tile that exist (all of them if >= 128)
        uint32_t a[16], b[16], pk[16];
        // The tile's reference is settled before its scores are there, from what the thread knows of its earlier tiles and
        // from the reference of the tile before (of the item before, for the first tile, which only keeps the order).
        float m_prev = 0.f;
        alive = ref_read(slot, t, &m_prev, abort_flag) && alive;
        const bool move = jj > 0 && run > m_prev + 8.0f;
        float m_new = move ? ceilf(run) : m_prev;
        if (jj > 0) ref_publish(slot, t + 1, m_new);
        const bool any_move = __any_sync(0xffffffffu, move || !alive);
        if (any_move && __any_sync(0xffffffffu, !alive)) goto softmax_done;
        alive = mbar_wait(&s_full[grp], sph, abort_flag);
        sph ^= 1;
        tc_fence_after();
        if (any_move) {
          // O (tiles before this one) is brought to the new reference once P.V of the tile before has been added to it.
          // Only now: S of this tile implies P.V of three tiles before, without which the parity of the V stage's barrier,
          // which comes round every four tiles, could be read one round early.
          alive = mbar_wait(&v_empty[(t - 1) & (kRing - 1)], ((t - 1) / kRing) & 1, abort_flag) && alive;
          tc_fence_after();
          float from = m_prev;
          bool above = false;
          alive = fin_read(fin + quad, t, &above, abort_flag) && alive;
          if (above) {
            __threadfence_block();
            from = fref[row];
          }
          const float alpha = pow2_down(from, fmaxf(m_new, from));
#pragma unroll 1
          for (int c = 0; c < 8; ++c) scale_columns<false>(t_o + c * 16, alpha);
        }
        if (jj == 0) {
          // first tile: the row maximum must be known before anything is exponentiated
          float mx[4];
          mx[0] = mx[1] = mx[2] = mx[3] = neg ? INFINITY : -INFINITY;
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t r[32];
            tmem_ld32(t_s + c * 32, r);
            tc_wait_ld_regs(r);
            if (valid < kTileKV) {
              const uint32_t none = neg ? 0x7f800000u : 0xff800000u;
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (c * 32 + i >= valid) r[i] = none;
            }
            max_chunk(r, mx, neg);
          }
          const float m0 = neg ? fminf(fminf(mx[0], mx[1]), fminf(mx[2], mx[3])) : fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
          m_new = fmaxf(ceilf(m0 * cs), -1e30f);
          ref_publish(slot, t + 1, m_new);
        }
        if (!first && __any_sync(0xffffffffu, m_new != m_ref)) {
          const float alpha = pow2_down(m_ref, m_new);
          ls[0].x *= alpha, ls[0].y *= alpha, ls[1].x *= alpha, ls[1].y *= alpha;
        }
        first = false;
        m_ref = m_new;
        const float2 nm2 = make_float2(-m_new, -m_new);
        float grown_sum = 0.f;
        float grown = -INFINITY;  // the two bound this tile's largest exponent relative to the reference, see below
        // Kept as a short loop: three warps per SM sub-partition run it out of step, and the code of a whole unrolled tile
        // does not stay in the instruction caches.
        tmem_ld16(t_s, a);
        int c = 0;
#pragma unroll 1
        for (; c < 4; ++c) {
          const uint32_t t_c = t_s + c * 32;
          float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
          tc_wait_ld_regs(a);
          tmem_ld16(t_c + 16, b);
          exp_pairs<0>(a, pk, cs2, nm2, sum, 0, nullptr);
          tc_wait_ld_regs(b);
          if (c < 3) tmem_ld16(t_c + 32, a);
          exp_pairs<0>(b, pk + 8, cs2, nm2, sum, 0, nullptr);
          // The sum of the chunk's probabilities bounds their maximum from above and, within a factor of 32, from below:
          // that is all the next reference needs, and takes no instruction per score.
          float total = (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
          if (valid < kTileKV || __any_sync(0xffffffffu, !(total <= 1e30f))) {
            // The last key tile, a score about 2^100 above the reference, or a NaN: once more, with columns masked and the
            // largest exponent known (the chunk's scores are still in TMEM, P has not reached its columns).
            sum[0] = sum[1] = make_float2(0.f, 0.f);
            tmem_ld16(t_c, b);
            tc_wait_ld_regs(b);
            exp_pairs<1>(b, pk, cs2, nm2, sum, valid - c * 32, &grown);
            tmem_ld16(t_c + 16, b);
            tc_wait_ld_regs(b);
            exp_pairs<1>(b, pk + 8, cs2, nm2, sum, valid - c * 32 - 16, &grown);
            if (__any_sync(0xffffffffu, grown > 100.f)) break;  // on from this chunk below
            total = 0.f;
          }
          grown_sum = fmaxf(grown_sum, total);
          ls[0] = __fadd2_rn(ls[0], sum[0]);
          ls[1] = __fadd2_rn(ls[1], sum[1]);
          tmem_st16(t_s + c * 16, pk);
        }
        // In order behind the tile before; on its own path (below) if that one, or this one, has left the range of p.
        const uint32_t fin_seen = fin[quad];
        if (__any_sync(0xffffffffu, c < 4 || fin_seen != t << 1)) {
          bool above = false;
          alive = fin_read(fin + quad, t, &above, abort_flag) && alive;
          if (__any_sync(0xffffffffu, c < 4 || (above && jj > 0))) {
            lift_chunk = c;
            o_ref = m_new;
            lift_grown = fminf(grown, 100.f) + m_ref, lift_sum = grown_sum;
            break;
          }
        }
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          fin[quad] = (t << 1) + 2;
          if (leader_cta) mbar_arrive(&p_full[grp]);
          else mbar_arrive_remote(bar_remote);
        }
        if (grown_sum > 1.f) grown = fmaxf(grown, static_cast<float>((__float_as_int(grown_sum) >> 23) - 126));
        run = fmaxf(run, grown + m_ref);
      }
      if (lift_chunk >= 0) {
        // The group's remaining tiles of the item, the first of them from chunk lift_chunk on: every score is looked at before
        // its P is stored, and the reference of a row is lifted whenever one is more than 2^100 above it.
        // `o_ref`: O's reference before this tile, if the tiles before have not lifted it.
        int c = lift_chunk;
        float grown = lift_grown, grown_sum = lift_sum, m_new = o_ref;
        for (;;) {
          const uint32_t t = static_cast<uint32_t>(g + jj);
          const int valid = p.Sk - (w.jb + jj) * kTileKV;
          uint32_t b[16], pk[16];
          tc_wait_st();
#pragma unroll 1
          for (; c < 4; ++c) {
            const uint32_t t_c = t_s + c * 32;
            for (;;) {
              float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
              const float2 nm2 = make_float2(-m_ref, -m_ref);
              tmem_ld16(t_c, b);
              tc_wait_ld_regs(b);
              exp_pairs<2>(b, pk, cs2, nm2, sum, valid - c * 32, &grown);
              tmem_ld16(t_c + 16, b);
              tc_wait_ld_regs(b);
              exp_pairs<2>(b, pk + 8, cs2, nm2, sum, valid - c * 32 - 16, &grown);
              const float m_to = grown > m_ref + 100.f ? ceilf(grown) : m_ref;
              if (!__any_sync(0xffffffffu, m_to != m_ref)) {
                ls[0] = __fadd2_rn(ls[0], sum[0]);
                ls[1] = __fadd2_rn(ls[1], sum[1]);
                break;
              }
              // the chunk once more, and what there is of the tile and of the row sum scaled down
              const float alpha = pow2_down(m_ref, m_to);
              ls[0].x *= alpha, ls[0].y *= alpha, ls[1].x *= alpha, ls[1].y *= alpha;
#pragma unroll 1
              for (int i = 0; i < c; ++i) scale_columns<true>(t_s + i * 16, alpha);
              if (m_to != m_ref) grown_sum = 0.f;  // `grown` covers it
              m_ref = m_to;
            }
            tmem_st16(t_s + c * 16, pk);
            tc_wait_st();
          }
          if (grown_sum > 1.f) grown = fmaxf(grown, static_cast<float>((__float_as_int(grown_sum) >> 23) - 126) + m_ref);
          // O and P of the warp's rows are brought to the higher of their two references.
          bool above = false;
          alive = fin_read(fin + quad, t, &above, abort_flag) && alive;
          if (jj == 0) {
            o_ref = m_ref;  // the first tile overwrites O
          } else if (above) {
            __threadfence_block();
            o_ref = fmaxf(o_ref, fref[row]);
          }
          const float m_to = fmaxf(m_ref, o_ref);
          if (__any_sync(0xffffffffu, m_to != o_ref)) {
            alive = mbar_wait(&v_empty[(t - 1) & (kRing - 1)], ((t - 1) / kRing) & 1, abort_flag) && alive;
            tc_fence_after();
            const float alpha = pow2_down(o_ref, m_to);
#pragma unroll 1
            for (int i = 0; i < 8; ++i) scale_columns<false>(t_o + i * 16, alpha);
          }
          if (__any_sync(0xffffffffu, m_to != m_ref)) {
            const float alpha = pow2_down(m_ref, m_to);
#pragma unroll 1
            for (int i = 0; i < 4; ++i) scale_columns<true>(t_s + i * 16, alpha);
            ls[0].x *= alpha, ls[0].y *= alpha, ls[1].x *= alpha, ls[1].y *= alpha;
            m_ref = m_to;
          }
          tc_wait_st();
          if (m_to != m_new) grown = fmaxf(grown, m_to + 8.5f);  // the next tile's reference will not be below this one
          run = fmaxf(run, grown);
          const bool lifted = __any_sync(0xffffffffu, m_to != m_new);
          fref[row] = m_to;
          __threadfence_block();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) {
            fin[quad] = (t << 1) + (lifted ? 3 : 2);
            if (leader_cta) mbar_arrive(&p_full[grp]);
            else mbar_arrive_remote(bar_remote);
          }
          jj += kGroups;
          if (jj >= w.nkv) break;
          o_ref = 0.f;
          alive = ref_read(slot, t + kGroups, &o_ref, abort_flag) && alive;
          m_new = run > o_ref + 8.0f ? ceilf(run) : o_ref;
          ref_publish(slot, t + kGroups + 1, m_new);
          if (__any_sync(0xffffffffu, !alive)) goto softmax_done;
          alive = mbar_wait(&s_full[grp], sph, abort_flag);
          sph ^= 1;
          tc_fence_after();
          const float alpha = pow2_down(m_ref, m_new);
          ls[0].x *= alpha, ls[0].y *= alpha, ls[1].x *= alpha, ls[1].y *= alpha;
          m_ref = m_new;
          grown = -INFINITY, grown_sum = 0.f;
          c = 0;
        }
      }
      jj -= w.nkv;
      g += w.nkv;
      // This group's row sums of the item.  Slot n % 8 is free: this group runs at most three tiles ahead of P.V plus the
      // items in which it has no tile, so publishing item n means P.V of an item >= n - 6 has been issued, which waited
      // for the epilogue of item n - 7.
      sums[((n & (kSumSlots - 1)) * kGroups + grp) * kTileQ + row] =
          make_float2((ls[0].x + ls[0].y) + (ls[1].x + ls[1].y), first ? -1e30f : m_ref);
      __syncwarp();
      if (lane == 0) mbar_arrive(&l_full[n & (kSumSlots - 1)]);
    }
  softmax_done:;
  } else {
    // ---------------------------------------------------------------- epilogue
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t t_o = (static_cast<uint32_t>(quad * 32) << 16) + kTmemO;
    const uint32_t bar_empty = mapa_u32(smem_u32(o_empty), 0);
    int n = 0;
    for (int u = unit0; u < p.n_units; u += n_pairs_grid, ++n) {
      const AttnUnit w = attn_unit<SPLIT>(p, u);
      if (!mbar_wait_all(&l_full[n & (kSumSlots - 1)], (n / kSumSlots) & 1, abort_flag)) break;
      const float2* sm = sums + (n & (kSumSlots - 1)) * kGroups * kTileQ + row;
      const float2 l0 = sm[0], l1 = sm[kTileQ], l2 = sm[2 * kTileQ];
      const float m = fmaxf(l0.y, fmaxf(l1.y, l2.y));  // the reference of the last tile, which O is relative to
      const float l = l0.x * pow2_down(l0.y, m) + l1.x * pow2_down(l1.y, m) + l2.x * pow2_down(l2.y, m);
      if (!mbar_wait_all(o_full, n & 1, abort_flag)) break;
      tc_fence_after();
      auto release = [&]() {  // O has been read out: the next item's first P.V may overwrite it
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (leader_cta) mbar_arrive(o_empty);
          else mbar_arrive_remote(bar_empty);
        }
      };
      const int prow = static_cast<int>(rank) * kTileQ + row;  // row inside the item
      const int sq = w.q0 + prow;
      if (SPLIT && w.tail_part >= 0) {
        // one key range of a split item: O (relative to 2^m), m and the row sum go to the workspace
        float* wrow = p.ws + (static_cast<int64_t>(w.tail_part) * kPairQ + prow) * kWsRow;
        wrow[128] = m;
        wrow[129] = l;
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t r[32];
          tmem_ld32(t_o + c * 32, r);
          tc_wait_ld_regs(r);
#pragma unroll
          for (int i = 0; i < 8; ++i)
            *reinterpret_cast<uint4*>(wrow + c * 32 + i * 4) = make_uint4(r[i * 4], r[i * 4 + 1], r[i * 4 + 2], r[i * 4 + 3]);
        }
        release();
        continue;
      }
      const float inv = 1.0f / l;
      __nv_bfloat16* obase = p.o + static_cast<int64_t>(w.b) * p.o_stride_b;
      int so = sq;
      if (p.o_rows_per_part > 0) {
        const int part = min(sq / p.o_rows_per_part, kMaxParts - 1);
        obase = p.o_part[part];
        so = sq - part * p.o_rows_per_part;
      }
      const int64_t ooff = static_cast<int64_t>(so) * p.o_stride_s + static_cast<int64_t>(w.h) * p.o_stride_h;
      __nv_bfloat16* orow = obase + ooff;
      uint8_t* orow8 = reinterpret_cast<uint8_t*>(p.o) + static_cast<int64_t>(w.b) * p.o_stride_b + ooff;
#pragma unroll 1
      for (int c = 0; c < 128; c += 64) {
        uint32_t o[32];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          uint32_t r[16];
          tmem_ld16(t_o + c + k * 16, r);
          tc_wait_ld_regs(r);
#pragma unroll
          for (int i = 0; i < 8; ++i)
            o[k * 8 + i] = pack_bf16x2(__uint_as_float(r[2 * i]) * inv, __uint_as_float(r[2 * i + 1]) * inv);
        }
        if (c) release();
        if (sq < p.Sq) {
          if (p.out_e4m3) {
            // e4m3 output (the operand of a following FP8 Linear with unit activation scale): the value is rounded to
            // bf16 first and then cast with saturation, i.e. exactly what a bf16 output followed by dsb_cast_quant gives
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint32_t e[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const __nv_fp8x2_storage_t e0 = __nv_cvt_float2_to_fp8x2(unpack_bf16x2(o[i * 8 + 2 * k]), __NV_SATFINITE, __NV_E4M3);
                const __nv_fp8x2_storage_t e1 =
                    __nv_cvt_float2_to_fp8x2(unpack_bf16x2(o[i * 8 + 2 * k + 1]), __NV_SATFINITE, __NV_E4M3);
                e[k] = static_cast<uint32_t>(e0) | (static_cast<uint32_t>(e1) << 16);
              }
              *reinterpret_cast<uint4*>(orow8 + c + i * 16) = make_uint4(e[0], e[1], e[2], e[3]);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              *reinterpret_cast<uint4*>(orow + c + i * 8) = make_uint4(o[i * 4], o[i * 4 + 1], o[i * 4 + 2], o[i * 4 + 3]);
          }
        }
        __syncwarp();
      }
    }
  }

  if (*abort_flag) __nanosleep(200000);
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA leaves (or frees TMEM) while its peer may still use it
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc_cg2(*tmem_slot, 512);
  }
  if (threadIdx.x == 0 && *abort_flag && p.status) atomicCAS(p.status, 0, DSB_ERR_TIMEOUT);
}

// Finishes the rows of the split items: with M = max over parts of m_p, O = sum_p 2^(m_p - M) O_p and
// l = sum_p 2^(m_p - M) l_p (the m_p are integers, so the factors are exact), out = O / l.  One warp per row,
// four columns per lane.
__global__ void __launch_bounds__(256) attn_combine_kernel(AttnParams p, int tail_items) {
  grid_wait();
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int rows = kPairQ;
  if (gw >= tail_items * rows) return;
  const int ti = gw / rows, r = gw % rows;
  const int item = p.n_full + ti;
  const int sq = (item % p.n_pairs) * rows + r;
  const int h = item / p.n_pairs;
  if (sq >= p.Sq) return;
  const float* base = p.ws + (static_cast<int64_t>(ti) * p.split * rows + r) * kWsRow;
  float M = -INFINITY;
  for (int s = 0; s < p.split; ++s) M = fmaxf(M, base[static_cast<int64_t>(s) * rows * kWsRow + 128]);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  float l = 0.f;
  for (int s = 0; s < p.split; ++s) {
    const float* pr = base + static_cast<int64_t>(s) * rows * kWsRow;
    const float w = exp2f(pr[128] - M);
    const float4 o = *reinterpret_cast<const float4*>(pr + lane * 4);
    acc.x = fmaf(w, o.x, acc.x), acc.y = fmaf(w, o.y, acc.y), acc.z = fmaf(w, o.z, acc.z), acc.w = fmaf(w, o.w, acc.w);
    l = fmaf(w, pr[129], l);
  }
  const float inv = 1.0f / l;
  __nv_bfloat16* obase = p.o;
  int so = sq;
  if (p.o_rows_per_part > 0) {
    const int part = min(sq / p.o_rows_per_part, kMaxParts - 1);
    obase = p.o_part[part];
    so = sq - part * p.o_rows_per_part;
  }
  __nv_bfloat16* orow = obase + static_cast<int64_t>(so) * p.o_stride_s + static_cast<int64_t>(h) * p.o_stride_h + lane * 4;
  uint2 o2;
  o2.x = pack_bf16x2(acc.x * inv, acc.y * inv);
  o2.y = pack_bf16x2(acc.z * inv, acc.w * inv);
  *reinterpret_cast<uint2*>(orow) = o2;
}

// Rank-4 tensor map over (d, then s/h/b ordered by ascending stride); box = 64 columns x box_rows rows of s.
static int make_tmap_attn(CUtensorMap* out, int (&pos)[3], const void* base, int S, int H, int B, int64_t ss,
                          int64_t sh, int64_t sb, uint32_t box_rows) {
  PFN_encodeTiled enc = get_encode_tiled();
  if (!enc) return DSB_ERR_CUDA;
  struct Dim {
    uint64_t size, stride;
    uint32_t box;
    int id;
  } d[3] = {{static_cast<uint64_t>(S), static_cast<uint64_t>(ss) * 2, box_rows, 0},
            {static_cast<uint64_t>(H), static_cast<uint64_t>(sh) * 2, 1u, 1},
            {static_cast<uint64_t>(B), static_cast<uint64_t>(sb) * 2, 1u, 2}};
  // a dimension of extent 1 never moves: give it a stride that keeps the list ascending
  std::stable_sort(d, d + 3, [](const Dim& a, const Dim& b2) {
    if ((a.size == 1) != (b2.size == 1)) return b2.size == 1;
    return a.stride < b2.stride;
  });
  uint64_t prev = 256;  // bytes of one row of d
  for (int i = 0; i < 3; ++i) {
    if (d[i].size == 1) d[i].stride = prev * (i == 0 ? 1 : d[i - 1].size);
    if (d[i].stride == 0 || (d[i].stride & 15)) return DSB_ERR_ARG;
    prev = d[i].stride;
  }
  for (int i = 0; i < 3; ++i) pos[d[i].id] = i;
  const cuuint64_t dims[4] = {128, d[0].size, d[1].size, d[2].size};
  const cuuint64_t strides[3] = {d[0].stride, d[1].stride, d[2].stride};
  const cuuint32_t box[4] = {64, d[0].box, d[1].box, d[2].box};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? DSB_OK : DSB_ERR_CUDA;
}

}  // namespace dsb

using namespace dsb;

// CTA pairs the current device holds at once (a GPC with an odd SM count leaves one out); 0 on failure.  Also opts both
// kernels into their shared memory.
static int resident_pairs() {
  static std::atomic<int> cached[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int n = cached[dev].load();
  if (n > 0) return n;
  if (cudaFuncSetAttribute(flash_attn_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttnSmem) != cudaSuccess ||
      cudaFuncSetAttribute(flash_attn_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttnSmem) != cudaSuccess)
    return 0;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(sm_count()) & ~1u, 1, 1);
  cfg.blockDim = dim3(kAttnThreads, 1, 1);
  cfg.dynamicSmemBytes = kAttnSmem;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, flash_attn_kernel<false>, &cfg) != cudaSuccess || n <= 0) n = sm_count() / 2;
  cached[dev].store(n);
  return n;
}

// q_parts / o_parts: nullptr for one buffer (q / o), else n equal row ranges in separate buffers
static int launch_attn(const void* q, const void* const* q_parts, int n_q_parts, int q_rows_per_part, const void* k,
                       const void* v, void* o, void* const* o_parts, int n_o_parts, int o_rows_per_part, int B, int H,
                       int Sq, int Sk, int head_dim, int64_t q_stride_b, int64_t q_stride_s, int64_t q_stride_h,
                       int64_t k_stride_b, int64_t k_stride_s, int64_t k_stride_h, int64_t v_stride_b,
                       int64_t v_stride_s, int64_t v_stride_h, int64_t o_stride_b, int64_t o_stride_s,
                       int64_t o_stride_h, float sm_scale, int out_e4m3, void* ws, int64_t ws_bytes, int* status,
                       void* stream) {
  if (!k || !v || B <= 0 || H <= 0 || Sq < 0 || Sk <= 0) return DSB_ERR_ARG;
  if (ws && ((reinterpret_cast<uintptr_t>(ws) & 15u) || ws_bytes < 0)) return DSB_ERR_ARG;
  if (out_e4m3 && (o_parts || ((o_stride_s | o_stride_h | o_stride_b) & 15))) return DSB_ERR_ARG;
  if (head_dim != 128) return DSB_ERR_UNSUPPORTED;
  if (B > 65535) return DSB_ERR_UNSUPPORTED;
  auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  if (!al16(k) || !al16(v)) return DSB_ERR_ARG;
  if (q_parts) {
    if (B != 1 || n_q_parts < 1 || n_q_parts > kMaxParts || q_rows_per_part <= 0 || (q_rows_per_part % kTileQ) ||
        static_cast<int64_t>(n_q_parts) * q_rows_per_part < Sq)
      return DSB_ERR_ARG;
    for (int i = 0; i < n_q_parts; ++i)
      if (!q_parts[i] || !al16(q_parts[i])) return DSB_ERR_ARG;
  } else if (!q || !al16(q)) {
    return DSB_ERR_ARG;
  }
  if (o_parts) {
    if (B != 1 || n_o_parts < 1 || n_o_parts > kMaxParts || o_rows_per_part <= 0 ||
        static_cast<int64_t>(n_o_parts) * o_rows_per_part < Sq)
      return DSB_ERR_ARG;
    for (int i = 0; i < n_o_parts; ++i)
      if (!o_parts[i] || !al16(o_parts[i])) return DSB_ERR_ARG;
  } else if (!o || !al16(o)) {
    return DSB_ERR_ARG;
  }
  const int64_t strides[] = {q_stride_s, q_stride_h, k_stride_s, k_stride_h, v_stride_s, v_stride_h,
                             o_stride_s, o_stride_h, q_stride_b, k_stride_b, v_stride_b, o_stride_b};
  for (int64_t s : strides)
    if (s < 0 || (s & 7)) return DSB_ERR_ARG;
  if (Sq == 0) return DSB_OK;
  AttnParams p = {};
  AttnQMaps qm;
  CUtensorMap tk, tv;
  int rc;
  if (q_parts) {
    // every part is a buffer of q_rows_per_part rows (rows past Sq are read but never used), so all maps share one
    // coordinate order; unused slots repeat the last part
    for (int i = 0; i < kMaxParts; ++i) {
      const void* base = q_parts[i < n_q_parts ? i : n_q_parts - 1];
      if ((rc = make_tmap_attn(&qm.m[i], p.q_pos, base, q_rows_per_part, H, 1, q_stride_s, q_stride_h, q_stride_b,
                               kTileQ)) != DSB_OK)
        return rc;
    }
    p.q_rows_per_part = q_rows_per_part;
  } else {
    if ((rc = make_tmap_attn(&qm.m[0], p.q_pos, q, Sq, H, B, q_stride_s, q_stride_h, q_stride_b, kTileQ)) != DSB_OK)
      return rc;
    for (int i = 1; i < kMaxParts; ++i) qm.m[i] = qm.m[0];
  }
  if ((rc = make_tmap_attn(&tk, p.k_pos, k, Sk, H, B, k_stride_s, k_stride_h, k_stride_b, kTileKV / 2)) != DSB_OK) return rc;
  if ((rc = make_tmap_attn(&tv, p.v_pos, v, Sk, H, B, v_stride_s, v_stride_h, v_stride_b, kTileKV)) != DSB_OK) return rc;
  p.o = reinterpret_cast<__nv_bfloat16*>(o);
  if (o_parts) {
    for (int i = 0; i < kMaxParts; ++i)
      p.o_part[i] = reinterpret_cast<__nv_bfloat16*>(o_parts[i < n_o_parts ? i : n_o_parts - 1]);
    p.o_rows_per_part = o_rows_per_part;
  }
  p.out_e4m3 = out_e4m3 ? 1 : 0;
  p.o_stride_b = o_stride_b;
  p.o_stride_s = o_stride_s;
  p.o_stride_h = o_stride_h;
  p.Sq = Sq;
  p.Sk = Sk;
  p.scale_log2 = sm_scale * 1.4426950408889634f;
  p.status = status;
  const int n_pairs = (Sq + kPairQ - 1) / kPairQ;
  const int64_t items = static_cast<int64_t>(n_pairs) * H * B;
  if (items > 0x3fffffff) return DSB_ERR_UNSUPPORTED;
  const int pairs = resident_pairs();
  if (pairs <= 0) return DSB_ERR_CUDA;
  p.n_pairs = n_pairs;
  p.H = H;
  p.n_full = static_cast<int>(items);
  p.split = 1;
  p.ws = nullptr;
  // The items run in waves of `pairs`.  A partly filled last wave costs a whole item's duration, so when the caller
  // provides a workspace its items are cut along the keys into as many units as fill that wave, plus a combine pass.
  int tail = 0;
  if (ws && B == 1 && !out_e4m3) {
    const int nkv = (Sk + kTileKV - 1) / kTileKV;
    tail = static_cast<int>(items % pairs);
    // cut in `split`: the last wave's items take ceil(tail * split / pairs) rounds of 1/split of an item's duration
    // (plus a few per cent per unit for partial-result stores and the combine pass)
    int split = 1;
    if (tail > 0 && items > pairs) {
      double best = 1.0;
      for (int sp = 2; sp <= 4; ++sp) {
        if (nkv / sp < 8) break;  // every key range keeps at least 8 tiles
        const double cost = static_cast<double>((static_cast<int64_t>(tail) * sp + pairs - 1) / pairs) / sp + 0.05;
        if (cost < best - 1e-9) best = cost, split = sp;
      }
    }
    const int64_t need = static_cast<int64_t>(tail) * split * kPairQ * kWsRow * 4;
    if (split >= 2 && need <= ws_bytes) {
      p.split = split;
      p.n_full = static_cast<int>(items) - tail;
      p.ws = reinterpret_cast<float*>(ws);
    }
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  p.n_units = p.n_full + (p.split > 1 ? tail * p.split : 0);
  const dim3 grid(static_cast<unsigned>(p.n_units < pairs ? p.n_units : pairs) * 2, 1, 1);
  const cudaError_t err = launch_kernel<2>(p.split > 1 ? flash_attn_kernel<true> : flash_attn_kernel<false>, grid, kAttnThreads,
                                           kAttnSmem, st, qm, tk, tv, p);
  if (err != cudaSuccess) return DSB_ERR_CUDA;
  if (p.split > 1) {
    const int warps = tail * kPairQ;
    if (launch_kernel(attn_combine_kernel, (warps + 7) / 8, 256, 0, st, p, tail) != cudaSuccess) return DSB_ERR_CUDA;
  }
  return cudaGetLastError() == cudaSuccess ? DSB_OK : DSB_ERR_CUDA;
}

extern "C" int dsb_flash_attn(const void* q, const void* k, const void* v, void* o, int B, int H, int Sq, int Sk,
                              int head_dim, int64_t q_stride_b, int64_t q_stride_s, int64_t q_stride_h,
                              int64_t k_stride_b, int64_t k_stride_s, int64_t k_stride_h, int64_t v_stride_b,
                              int64_t v_stride_s, int64_t v_stride_h, int64_t o_stride_b, int64_t o_stride_s,
                              int64_t o_stride_h, float sm_scale, int* status, void* stream) {
  return launch_attn(q, nullptr, 0, 0, k, v, o, nullptr, 0, 0, B, H, Sq, Sk, head_dim, q_stride_b, q_stride_s, q_stride_h,
                     k_stride_b, k_stride_s, k_stride_h, v_stride_b, v_stride_s, v_stride_h, o_stride_b, o_stride_s,
                     o_stride_h, sm_scale, 0, nullptr, 0, status, stream);
}

extern "C" int dsb_flash_attn_out8(const void* q, const void* k, const void* v, void* o, int B, int H, int Sq, int Sk,
                                   int head_dim, int64_t q_stride_b, int64_t q_stride_s, int64_t q_stride_h,
                                   int64_t k_stride_b, int64_t k_stride_s, int64_t k_stride_h, int64_t v_stride_b,
                                   int64_t v_stride_s, int64_t v_stride_h, int64_t o_stride_b, int64_t o_stride_s,
                                   int64_t o_stride_h, float sm_scale, int* status, void* stream) {
  return launch_attn(q, nullptr, 0, 0, k, v, o, nullptr, 0, 0, B, H, Sq, Sk, head_dim, q_stride_b, q_stride_s, q_stride_h,
                     k_stride_b, k_stride_s, k_stride_h, v_stride_b, v_stride_s, v_stride_h, o_stride_b, o_stride_s,
                     o_stride_h, sm_scale, 1, nullptr, 0, status, stream);
}

extern "C" int dsb_flash_attn_parts(const void* const* q_parts, int n_q_parts, int q_rows_per_part, const void* k,
                                    const void* v, void* const* o_parts, int n_o_parts, int o_rows_per_part, int H,
                                    int Sq, int Sk, int head_dim, int64_t q_stride_s, int64_t q_stride_h,
                                    int64_t k_stride_s, int64_t k_stride_h, int64_t v_stride_s, int64_t v_stride_h,
                                    int64_t o_stride_s, int64_t o_stride_h, float sm_scale, void* workspace,
                                    int64_t workspace_bytes, int* status, void* stream) {
  if (!q_parts || !o_parts) return DSB_ERR_ARG;
  return launch_attn(nullptr, q_parts, n_q_parts, q_rows_per_part, k, v, nullptr, o_parts, n_o_parts, o_rows_per_part, 1,
                     H, Sq, Sk, head_dim, 0, q_stride_s, q_stride_h, 0, k_stride_s, k_stride_h, 0, v_stride_s,
                     v_stride_h, 0, o_stride_s, o_stride_h, sm_scale, 0, workspace, workspace_bytes, status, stream);
}

extern "C" int64_t dsb_flash_attn_workspace_bytes(void) {
  // a last wave is at least one item short of the pairs that run at once, and its items are cut in at most four
  const int pairs = resident_pairs();
  return pairs > 1 ? static_cast<int64_t>(pairs - 1) * 4 * kPairQ * kWsRow * 4 : 0;
}
