// hb_pair.cu -- Lennard-Jones + erfc-screened real-space Coulomb pair
// kernel over the packed neighbour list.
//
// Physics follows the reference's composed pair kernel
// (src/forces/jit_composed.rs:1490-1831) with the LJ functor
// (src/forces/lj.rs:237-283, optional CHARMM switch) and the SPME real-space
// functor (src/forces/spme.rs:730-759, erfc by the Abramowitz-Stegun 7.1.26
// polynomial in single precision), per-fragment cutoffs, exclusion scales
// applied per fragment, energy and virial split 1/2 per atom.
//
// Structure (own design): persistent warps take (i-tile, run of entries)
// work items; see k_pair below.  Pair forces are summed as integers (int32
// sums folded into int64 fixed point at 2^40), so forces do not depend on
// entry order or on scheduling and repeat runs are byte-identical.
// Exclusions arrive as a 32-bit mask per j-slot built with the list, so an
// ordinary pair costs no exclusion lookup.  Tiles that satisfy the
// single-periodic-copy condition shift i and j positions against the tile
// centre once per entry and skip the per-pair minimum image.
#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

#include "hb_internal.cuh"

// Resident blocks the register budget is cut for.  Force-only: 6 (80
// registers, no spill) runs the 65,536-water list in 245 us against 248 at 5
// (96), 258 at 7 (72, 88 B of spill) and 268 at 8 (64, 240 B); with scaled
// exclusions and a switch the same cap spills 72 B.  With energies or exact
// sums 5, where the kernel needs 96 registers; the multi-system form, which
// carries its member's pointers, spills 72 B there.
#define PAIR_MIN_BLOCKS(EV, EXACT, MULTI) ((EV) || (EXACT) || (MULTI) ? 5 : 6)

namespace {

struct PairParams {
  int n_types;
  int lj_on, coul_on;
  float rc2_max;
  float coul_rc2;
  float alpha;
  float c2a;   // 2 alpha / sqrt(pi)
  float nl2e;  // -log2(e)
  uint32_t n, n_tiles;
  uint32_t slab;
};

// one system of the multi-system pair launch: its lists, positions,
// accumulators and cell, and its first work item in the launch's item space
struct PairMember {
  const float4 *tile_posq;
  const int *tile_type;
  const float4 *center;
  const uint32_t *tile_nent;
  const uint32_t *entry_j;
  const uint32_t *entry_excl;
  const DBox *box;
  unsigned long long *fp;
  uint32_t n, n_tiles, slab, chunks, item0, pad[3];
};

__device__ __forceinline__ void shift_to(float &x, float &y, float &z, const float4 &c,
                                         const DBox &b) {
  float dx = x - c.x, dy = y - c.y, dz = z - c.z;
  x -= b.lx * rintf(dx * b.ilx);
  y -= b.ly * rintf(dy * b.ily);
  z -= b.lz * rintf(dz * b.ilz);
}

__device__ __forceinline__ long long to_fixed(float v) {
  return __float2ll_rn(v * HB_FP_SCALE);
}

__device__ __forceinline__ void red_add(unsigned long long *p, long long v) {
  if (v != 0) atomicAdd(p, (unsigned long long)v);
}

// ---------------------------------------------------------------------
// k_pair: one warp per work item (i-tile, run of entries), one lane per
// i-atom of the tile.  Per entry:
//   stage     the 32 j-atoms go to shared memory, those of a type with a
//             Lennard-Jones term in the highest rows;
//   distance  every lane tests its i-atom against the 32 rows (broadcast
//             loads, two rows per packed FP32x2 step) and keeps the hits as
//             a 32-bit mask, exclusions and padding masked out;
//   drain     while any lane has hits of the older of the two staged
//             entries, each lane takes its own next two hits -- from the
//             older entry, else already from the newer one -- and evaluates
//             them as one packed FP32x2 pair.
// The i-atom and its force sums never leave the lane's registers, and no
// queue is written or read; the two-entry window is what balances the lanes
// (a lane with few hits in one entry works ahead in the next).
//
// Forces are int32 fixed point (scale 2^30, integer sums: order-independent,
// the same run to run and for every split of the work).  The i-side sums of
// at most 32 pairs are folded into int64 at every drain; the j-side sums go
// to shared memory by integer atomics and to int64 global sums once per
// entry.  A pair force component above 0.06 hartree/bohr takes the int64
// path instead, so the int32 sums cannot wrap (32 x 0.06 x 2^30 < 2^31).
// With EV the energy and virial halves of each pair are int32 sums at 2^28
// (guard 0.24 hartree: 32 x 0.24 x 2^28 < 2^31, where 0.25 would wrap), and
// the LJ energy total is summed per lane in int64.
//
// EXACT: every pair force is converted to int64 (2^40) by itself and takes
// the minimum image of the two stored positions, so it is a function of the
// positions alone, not of the tile the pair was packed into.
//
// Bound: instruction issue (about 1,190 warp instructions per entry, of
// which 450 do not depend on the hits) together with shared-memory
// wavefronts; DRAM and MUFU are far from it.  Against one pair queue per
// entry with balanced lane runs (1,776 instructions per entry: the queue's
// scan, writes, reads and the i-side flushes cost more than the idle lanes
// they fill): 286 -> 245 us per force-only evaluation of 65,536 waters,
// 40 -> 19 us for 343 waters (with one entry per item), and the exact form,
// before one warp per tile with six int64 shared atomics per pair,
// 166 -> 51 us for 13,824 ions.  Two copies of the j-side sums (even and odd lanes)
// halve the same-address atomics of a round: 254 -> 248 us.
// ---------------------------------------------------------------------
#define PK_WARPS 4
#define PK_COPY 80
#define PK_SHIFT 10               // 2^40 / 2^30
#define PK_SCALE 1073741824.0f    // 2^30
#define PK_FMAX 0.06f
#define PK_ESHIFT 12              // 2^40 / 2^28
#define PK_ESCALE 268435456.0f    // 2^28
#define PK_EMAX 0.24f
// 32 terms at the guards, each rounded to an integer, fit an int32
static_assert(32.0 * (PK_FMAX * (double)PK_SCALE + 0.5) < 2147483648.0, "force sums may wrap");
static_assert(32.0 * (PK_EMAX * (double)PK_ESCALE + 0.5) < 2147483648.0, "energy sums may wrap");

template <bool EV, bool SCALED, bool EXACT>
struct PairWarp {
  using acc_t = typename std::conditional<EXACT, unsigned long long, int>::type;
  float4 jpos[64];  // two entries of 32 rows
  float4 jxy2[16];  // rows 2k, 2k + 1 of the newer entry, negated: (-x, -x', -y, -y')
  float2 jz2[16];   // (-z, -z')
  int jtype[64];
  uint32_t jslot[64];
  acc_t fj[EV ? 5 : 3][PK_COPY + 64];  // two copies per row, even and odd lanes, 16 banks apart
  uint32_t oj[SCALED ? 64 : 1];
};

// |a|, |b|, |c| maximum that keeps NaN
__device__ __forceinline__ float max_abs3(float a, float b, float c) {
  float r;
  asm("{\n\t.reg .f32 x, y, z;\n\tabs.f32 x, %1;\n\tabs.f32 y, %2;\n\tabs.f32 z, %3;\n\t"
      "max.NaN.f32 x, x, y;\n\tmax.NaN.f32 %0, x, z;\n\t}"
      : "=f"(r)
      : "f"(a), "f"(b), "f"(c));
  return r;
}

// hardware approximations without the scaling steps for subnormal arguments
// and results, which no separation, screening factor or exponent here needs
// (a screening factor below 2^-126 counts as zero)
__device__ __forceinline__ float fast_rsqrt(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <bool EV, bool SCALED, bool SWITCH, bool EXACT, bool MULTI>
__global__ void __launch_bounds__(PK_WARPS * 32, PAIR_MIN_BLOCKS(EV, EXACT, MULTI))
    k_pair(const float4 *__restrict__ a_tile_posq, const int *__restrict__ a_tile_type,
           const float4 *__restrict__ a_center, const uint32_t *__restrict__ a_tile_nent,
           const uint32_t *__restrict__ a_entry_j, const uint32_t *__restrict__ a_entry_excl,
           const DBox *__restrict__ a_box, const float4 *__restrict__ lj_table,
           const float *__restrict__ lj_invd, PairParams a_P, unsigned long long *__restrict__ a_fp,
           const uint32_t *__restrict__ sorted_ids, const uint32_t *__restrict__ eoff,
           const uint32_t *__restrict__ epart, const float2 *__restrict__ escale,
           uint32_t *__restrict__ work, uint32_t a_chunks, uint32_t chunk, uint32_t quota,
           unsigned long long *__restrict__ e_lj_total, const PairMember *__restrict__ members,
           uint32_t n_members, uint32_t n_items_all) {
  static_assert(!(MULTI && (EV || SCALED || EXACT)), "the multi-system form is force-only, unscaled");
  using Warp = PairWarp<EV, SCALED, EXACT>;
  constexpr int NC = EV ? 5 : 3;
  extern __shared__ float4 sm_lj4[];
  __shared__ Warp smw[PK_WARPS];
  __shared__ uint32_t sm_ljtypes[32];  // per i-type: j-types with a Lennard-Jones term
  // multi-system form: the members' first work items, for the per-item
  // member search (members beyond the table search global memory)
  constexpr uint32_t MT = 128u;
  __shared__ uint32_t sm_item0[MULTI ? MT : 1];
  if constexpr (MULTI) {
    for (uint32_t k = threadIdx.x; k < MT && k < n_members; k += blockDim.x) sm_item0[k] = members[k].item0;
  }
  // the fixed-point scale rides on the LJ energy scale and the j-charges
  // (a power of two: every rounding stays where it was)
  constexpr float FSC = EXACT ? 1.0f : PK_SCALE;
  const int nt2 = a_P.n_types * a_P.n_types;
  float *sm_ljd4 = reinterpret_cast<float *>(sm_lj4 + nt2);
  for (int k = threadIdx.x; k < nt2; k += blockDim.x) {
    float4 L = lj_table[k];
    L.y *= FSC;
    sm_lj4[k] = L;
    sm_ljd4[k] = lj_invd[k];
  }
  const bool few_types = a_P.n_types <= 32;
  if (few_types && (int)threadIdx.x < a_P.n_types) {
    uint32_t bits = 0u;
    for (int q = 0; q < a_P.n_types; ++q)
      if (lj_table[threadIdx.x * a_P.n_types + q].y != 0.0f) bits |= 1u << q;
    sm_ljtypes[threadIdx.x] = bits;
  }
  __syncthreads();
  const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t lt = (1u << lane) - 1u, jo = (lane & 1u) * PK_COPY;
  Warp &S = smw[w];
  long long elj_fix = 0;  // LJ energy of this lane's pairs (fixed point)
  const uint32_t n_items = MULTI ? n_items_all : a_P.n_tiles * a_chunks;
  // j-types with a Lennard-Jones term against some type of the table
  uint32_t any_lj = a_P.lj_on ? 0xFFFFFFFFu : 0u;
  if (a_P.lj_on && few_types) {
    any_lj = 0u;
    for (int q = 0; q < a_P.n_types; ++q) any_lj |= sm_ljtypes[q];
  }

  // warps take (tile, run of entries) items from a counter, at most `quota`
  // each (a finite quota retires blocks as they finish); the next item is
  // requested while the current one runs
  uint32_t g_next = 0u;
  if (lane == 0) g_next = atomicAdd(work, 1u);
  for (uint32_t taken = 0; taken < quota; ++taken) {
    uint32_t g = __shfl_sync(0xFFFFFFFFu, g_next, 0);
    if (g >= n_items) break;
    if (lane == 0 && taken + 1u < quota) g_next = atomicAdd(work, 1u);
    // the system this item belongs to: the kernel's own arguments, or (the
    // multi-system form) the member whose item range holds g
    const float4 *__restrict__ tile_posq = a_tile_posq;
    const int *__restrict__ tile_type = a_tile_type;
    const float4 *__restrict__ center = a_center;
    const uint32_t *__restrict__ tile_nent = a_tile_nent;
    const uint32_t *__restrict__ entry_j = a_entry_j;
    const uint32_t *__restrict__ entry_excl = a_entry_excl;
    const DBox *__restrict__ box = a_box;
    unsigned long long *__restrict__ fp = a_fp;
    PairParams P = a_P;
    uint32_t chunks = a_chunks;
    if constexpr (MULTI) {
      uint32_t lo = 0u, hi = n_members;  // largest m with members[m].item0 <= g
      while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if ((mid < MT ? sm_item0[mid] : members[mid].item0) <= g) lo = mid;
        else hi = mid;
      }
      const PairMember &M = members[lo];
      g -= M.item0;
      tile_posq = M.tile_posq;
      tile_type = M.tile_type;
      center = M.center;
      tile_nent = M.tile_nent;
      entry_j = M.entry_j;
      entry_excl = M.entry_excl;
      fp = M.fp;
      P.n = M.n;
      P.n_tiles = M.n_tiles;
      P.slab = M.slab;
      chunks = M.chunks;
      box = M.box;
    }
    const size_t np_all = (size_t)P.n_tiles * 32u;
    const uint32_t I = g / chunks, ch = g - I * chunks;
    const uint32_t tile_e0 = I * P.slab;
    const uint32_t e0 = tile_e0 + ch * chunk;
    // the slab holds entry e0 whether the tile uses it or not: its load does
    // not wait for the tile's entry count
    const uint32_t sj_first = entry_j[(uint64_t)e0 * 32u + lane];
    const uint32_t jm_first = entry_excl[(uint64_t)e0 * 32u + lane];
    const uint32_t tile_e1 = tile_e0 + min(tile_nent[I], P.slab);
    if (e0 >= tile_e1) continue;
    const uint32_t e1 = min(e0 + chunk, tile_e1);
    const DBox b = *box;
    const float4 c = center[I];
    const uint32_t si = I * 32u + lane;
    const bool ivalid = si < P.n;
    const float4 far = make_float4(1.0e18f, 1.0e18f, 1.0e18f, 0.0f);
    // software pipeline: an entry's j-slots and exclusions are requested two
    // entries ahead, its j-atoms one entry ahead
    uint32_t sj_n = sj_first, jm_n = jm_first, sj_nn = HB_SENTINEL, jm_nn = 0u;
    if (e0 + 1u < e1) {
      sj_nn = entry_j[(uint64_t)(e0 + 1u) * 32u + lane];
      jm_nn = entry_excl[(uint64_t)(e0 + 1u) * 32u + lane];
    }
    float4 pi = tile_posq[si];
    const int ti = ivalid ? tile_type[si] : 0;
    const int ti_row = ti * P.n_types;
    const bool i_lj = P.lj_on && (few_types ? sm_ljtypes[ti] != 0u : true);
    const uint32_t oi = SCALED && ivalid ? sorted_ids[si] : HB_SENTINEL;
    const bool has_self = P.n - I * 32u >= 2u;
    long long ax = 0, ay = 0, az = 0, ae = 0, aw = 0;
    float4 pj_n = far;
    int tj_n = 0;
    if (sj_n != HB_SENTINEL) {
      pj_n = tile_posq[sj_n];
      tj_n = tile_type[sj_n];
    }

    auto item = [&](auto form) {
      constexpr int FORM = decltype(form)::value;
      if (!ivalid) pi = make_float4(-1.0e18f, -1.0e18f, -1.0e18f, 0.0f);
      else if (FORM == HB_IMAGE_NONE) shift_to(pi.x, pi.y, pi.z, c, b);
      // the entry whose data the prefetch registers hold goes to rows
      // [base, base + 32); returns the lane's hits, a bound on the mask of its
      // hits without a Lennard-Jones term, and (SCALED) its listed exclusions
      auto stage = [&](uint32_t e, uint32_t base, uint32_t &lj_below, uint32_t &scaled) -> uint32_t {
        const bool self = has_self && (e == tile_e0);
        const uint32_t sj = sj_n, jm = jm_n;
        float4 pj = pj_n;
        const int tj = tj_n;
        const bool jvalid = sj != HB_SENTINEL;
        if (FORM == HB_IMAGE_NONE && jvalid) shift_to(pj.x, pj.y, pj.z, c, b);
        const bool jl = jvalid && (few_types ? ((any_lj >> tj) & 1u) != 0u : any_lj != 0u);
        const uint32_t b_v = __ballot_sync(0xFFFFFFFFu, jvalid), b_l = __ballot_sync(0xFFFFFFFFu, jl);
        const uint32_t n_v = __popc(b_v), n_l = __popc(b_l);
        const uint32_t row = jl ? 31u - __popc(b_l & lt)
                                : (jvalid ? 31u - n_l - __popc(b_v & ~b_l & lt) : __popc(~b_v & lt));
        // a lane's mask above this value holds a Lennard-Jones pair
        lj_below = i_lj && n_l != 0u ? (1u << (32u - n_l)) - 1u : 0xFFFFFFFFu;
        sj_n = sj_nn;
        jm_n = jm_nn;
        sj_nn = HB_SENTINEL;
        if (e + 2u < e1) {
          sj_nn = entry_j[(uint64_t)(e + 2u) * 32u + lane];
          jm_nn = entry_excl[(uint64_t)(e + 2u) * 32u + lane];
        }
        pj_n = far;
        tj_n = 0;
        if (sj_n != HB_SENTINEL) {
          pj_n = tile_posq[sj_n];
          tj_n = tile_type[sj_n];
        }
        __syncwarp();
        {
          float *jn = reinterpret_cast<float *>(&S.jxy2[row >> 1]);
          jn[row & 1u] = -pj.x;
          jn[2u + (row & 1u)] = -pj.y;
          reinterpret_cast<float *>(&S.jz2[row >> 1])[row & 1u] = -pj.z;
        }
        pj.w *= FSC;
        S.jpos[base + row] = pj;
        S.jtype[base + row] = tj;
        S.jslot[base + row] = sj;
        if (SCALED) S.oj[base + row] = jvalid ? sorted_ids[sj] : HB_SENTINEL;
#pragma unroll
        for (int q = 0; q < NC; ++q) S.fj[q][base + lane] = S.fj[q][PK_COPY + base + lane] = 0;
        __syncwarp();
        uint32_t m = 0u;
        const float2 px = make_float2(pi.x, pi.x), py = make_float2(pi.y, pi.y),
                     pz = make_float2(pi.z, pi.z);
        const float2 nrc = make_float2(-P.rc2_max, -P.rc2_max);
        // r2 < rc2 exactly when r2 - rc2 is negative: the sign bits of the
        // packed difference are shifted into the mask, highest row first
#pragma unroll
        for (int k = 15; k >= 0; --k) {
          const float4 a = S.jxy2[k];
          float2 dx = __fadd2_rn(px, make_float2(a.x, a.y));
          float2 dy = __fadd2_rn(py, make_float2(a.z, a.w));
          float2 dz = __fadd2_rn(pz, S.jz2[k]);
          hb_min_image2<FORM>(dx, dy, dz, b);
          float2 r2 = __fmul2_rn(dx, dx);
          r2 = __ffma2_rn(dy, dy, r2);
          r2 = __ffma2_rn(dz, dz, r2);
          const float2 d = __fadd2_rn(r2, nrc);
          m = __funnelshift_l(__float_as_uint(d.y), m, 1);
          m = __funnelshift_l(__float_as_uint(d.x), m, 1);
        }
        // padding takes part in no pair, whatever its placeholder
        // coordinates give under the minimum image
        m &= ivalid && n_v != 0u ? 0xFFFFFFFFu << (32u - n_v) : 0u;
        // exclusions are stored per j-atom (bit i: excluded with i-atom i);
        // few j-atoms of an entry have any.  In the self entry each pair
        // counts once, seen from the lower of its two slots
        uint32_t ex = 0u;
        for (uint32_t todo = __ballot_sync(0xFFFFFFFFu, jm != 0u); todo != 0u; todo &= todo - 1u) {
          const uint32_t src = (uint32_t)__ffs(todo) - 1u;
          const uint32_t jm_s = __shfl_sync(0xFFFFFFFFu, jm, src);
          const uint32_t row_s = __shfl_sync(0xFFFFFFFFu, row, src);
          ex |= ((jm_s >> lane) & 1u) << row_s;
        }
        if (self) {
          for (uint32_t src = 0; src < 32u; ++src) {
            const uint32_t row_s = __shfl_sync(0xFFFFFFFFu, row, src);
            if (src <= lane) m &= ~(1u << row_s);
          }
        }
        if (SCALED) scaled = ex;
        else m &= ~ex;
        return m;
      };

      uint32_t lj_a = 0u, lj_b = 0u, sc_a = 0u, sc_b = 0u, base_a = 0u;
      uint32_t m_a = stage(e0, 0u, lj_a, sc_a);
      for (uint32_t e = e0 + 1u; e <= e1; ++e) {
        const uint32_t base_b = base_a ^ 32u;
        // the newer entry's hits: those without and those with a
        // Lennard-Jones term (the latter wait until the entry is the older)
        uint32_t m_b = 0u, m_bl = 0u;
        if (e < e1) {
          m_b = stage(e, base_b, lj_b, sc_b);
          m_bl = m_b & ~lj_b;
          m_b &= lj_b;
        }
        typename std::conditional<EXACT, long long, int>::type sx = 0, sy = 0, sz = 0, se = 0, sw = 0;
        // one round: the lane's next two hits, the older entry's first,
        // highest row (Lennard-Jones) first
        auto round = [&](auto ljc) {
          constexpr bool LJ = decltype(ljc)::value;
          if ((m_a | m_b) != 0u) {
            const bool a0 = m_a != 0u;
            const uint32_t q0 = 31u - (uint32_t)__clz(a0 ? m_a : m_b);
            if (a0) m_a ^= 1u << q0;
            else m_b ^= 1u << q0;
            const bool a1 = m_a != 0u, two = (m_a | m_b) != 0u;
            const uint32_t q1 = 31u - (uint32_t)__clz(a1 ? m_a : m_b);
            if (a1) m_a ^= 1u << q1;
            else if (two) m_b ^= 1u << q1;
            const uint32_t r0 = q0 + (a0 ? base_a : base_b);
            const uint32_t r1 = two ? q1 + (a1 ? base_a : base_b) : r0;
            const float4 ja = S.jpos[r0], jb = S.jpos[r1];
            float2 dx = make_float2(pi.x - ja.x, pi.x - jb.x);
            float2 dy = make_float2(pi.y - ja.y, pi.y - jb.y);
            float2 dz = make_float2(pi.z - ja.z, pi.z - jb.z);
            hb_min_image2<FORM>(dx, dy, dz, b);
            float2 r2 = __fmul2_rn(dx, dx);
            r2 = __ffma2_rn(dy, dy, r2);
            r2 = __ffma2_rn(dz, dz, r2);
            const float2 inv_r = make_float2(fast_rsqrt(r2.x), fast_rsqrt(r2.y));
            const float2 inv_r2 = __fmul2_rn(inv_r, inv_r);
            float2 s_lj = make_float2(1.0f, 1.0f), s_c = s_lj;
            if (SCALED) {
              const bool xa = ((a0 ? sc_a : sc_b) >> q0) & 1u, xb = two && (((a1 ? sc_a : sc_b) >> q1) & 1u);
              if (xa || xb) {
                auto listed = [&](uint32_t r, float &l, float &q) {
                  l = 0.0f;
                  q = 0.0f;
                  const uint32_t o = S.oj[r];
                  for (uint32_t z = eoff[o]; z < eoff[o + 1]; ++z) {
                    if (epart[z] == oi) {
                      const float2 v = escale[z];
                      l = v.x;
                      q = v.y;
                      break;
                    }
                  }
                };
                if (xa) listed(r0, s_lj.x, s_c.x);
                if (xb) listed(r1, s_lj.y, s_c.y);
              }
            }
            const float2 one2 = make_float2(1.0f, 1.0f);
            float2 fac = make_float2(0.0f, 0.0f), en = fac;
            if constexpr (LJ) {
              const int ta = ti_row + S.jtype[r0], tb = ti_row + S.jtype[r1];
              const float4 La = sm_lj4[ta], Lb = sm_lj4[tb];
              const float2 eps = make_float2(La.y, Lb.y);
              const float2 sr2 = __fmul2_rn(make_float2(La.x, Lb.x), inv_r2);
              const float2 sr6 = __fmul2_rn(__fmul2_rn(sr2, sr2), sr2);
              const float2 sr12 = __fmul2_rn(sr6, sr6);
              const float2 nsr6 = make_float2(-sr6.x, -sr6.y);
              float2 f = __fmul2_rn(__fmul2_rn(eps, inv_r2),
                                    __ffma2_rn(make_float2(2.0f, 2.0f), sr12, nsr6));
              float2 u = one2;
              if (SWITCH || EV)
                u = __fmul2_rn(__fmul2_rn(eps, make_float2(1.0f / 6.0f, 1.0f / 6.0f)),
                               __fadd2_rn(sr12, nsr6));
              if (SWITCH && (r2.x > La.w || r2.y > Lb.w)) {
                const float2 inv_d = make_float2(sm_ljd4[ta], sm_ljd4[tb]);
                const float2 tau = __fmul2_rn(__fadd2_rn(r2, make_float2(-La.w, -Lb.w)), inv_d);
                const float2 omt = __fadd2_rn(one2, make_float2(-tau.x, -tau.y));
                const float2 sw2 = __fmul2_rn(__fmul2_rn(omt, omt),
                                              __ffma2_rn(make_float2(2.0f, 2.0f), tau, one2));
                const float2 chain =
                    __fmul2_rn(__fmul2_rn(__fmul2_rn(make_float2(12.0f, 12.0f), tau), omt), inv_d);
                const float2 fsw = __ffma2_rn(sw2, f, __fmul2_rn(chain, u));
                const float2 usw = __fmul2_rn(sw2, u);
                if (r2.x > La.w) {
                  f.x = fsw.x;
                  u.x = usw.x;
                }
                if (r2.y > Lb.w) {
                  f.y = fsw.y;
                  u.y = usw.y;
                }
              }
              if (SCALED) {
                f = __fmul2_rn(f, s_lj);
                u = __fmul2_rn(u, s_lj);
              }
              // no Lennard-Jones term beyond its cut-off, nor (eps = 0, or a
              // zero exclusion scale, whatever r) where there is none
              const bool on_a = r2.x <= La.z && La.y != 0.0f && (!SCALED || s_lj.x != 0.0f);
              const bool on_b = r2.y <= Lb.z && Lb.y != 0.0f && (!SCALED || s_lj.y != 0.0f);
              if (on_a) fac.x = f.x;
              if (on_b) fac.y = f.y;
              if (EV) {
                if (on_a) {
                  en.x = u.x;
                  elj_fix += to_fixed(u.x * (1.0f / FSC));
                }
                if (on_b && two) {
                  en.y = u.y;
                  elj_fix += to_fixed(u.y * (1.0f / FSC));
                }
              }
            }
            if (P.coul_on) {
              const float2 r = __fmul2_rn(r2, inv_r);
              const float2 ar = __fmul2_rn(make_float2(P.alpha, P.alpha), r);
              const float2 ea = __fmul2_rn(make_float2(P.nl2e, P.nl2e), __fmul2_rn(ar, ar));
              const float2 gg = make_float2(fast_exp2(ea.x), fast_exp2(ea.y));
              const float2 den = __ffma2_rn(make_float2(0.3275911f, 0.3275911f), ar, one2);
              const float2 tt = make_float2(fast_rcp(den.x), fast_rcp(den.y));
              float2 poly = __ffma2_rn(make_float2(1.061405429f, 1.061405429f), tt,
                                       make_float2(-1.453152027f, -1.453152027f));
              poly = __ffma2_rn(poly, tt, make_float2(1.421413741f, 1.421413741f));
              poly = __ffma2_rn(poly, tt, make_float2(-0.284496736f, -0.284496736f));
              poly = __ffma2_rn(poly, tt, make_float2(0.254829592f, 0.254829592f));
              const float2 pt = __fmul2_rn(poly, tt);
              // erfc(ar) / r + c2a exp(-a^2 r^2) = gg (poly tt / r + c2a)
              const float2 wv = __fmul2_rn(gg, __ffma2_rn(pt, inv_r, make_float2(P.c2a, P.c2a)));
              float2 qq = __fmul2_rn(make_float2(pi.w, pi.w), make_float2(ja.w, jb.w));
              if (SCALED) qq = __fmul2_rn(qq, s_c);
              float2 fc = __fmul2_rn(__fmul2_rn(qq, inv_r2), wv);
              const bool on_a = r2.x <= P.coul_rc2 && (!SCALED || s_c.x != 0.0f);
              const bool on_b = r2.y <= P.coul_rc2 && (!SCALED || s_c.y != 0.0f);
              if (!on_a) fc.x = 0.0f;
              if (!on_b) fc.y = 0.0f;
              fac = __fadd2_rn(fac, fc);
              if (EV) {
                const float2 ec = __fmul2_rn(__fmul2_rn(qq, __fmul2_rn(pt, gg)), inv_r);
                if (on_a) en.x += ec.x;
                if (on_b) en.y += ec.y;
              }
            }
            if (!two) fac.y = 0.0f;
            float2 fx = __fmul2_rn(fac, dx), fy = __fmul2_rn(fac, dy), fz = __fmul2_rn(fac, dz);
            if constexpr (EXACT) {
              const long long xa = to_fixed(fx.x), ya = to_fixed(fy.x), za = to_fixed(fz.x);
              atomicAdd(&S.fj[0][jo + r0], (unsigned long long)xa);
              atomicAdd(&S.fj[1][jo + r0], (unsigned long long)ya);
              atomicAdd(&S.fj[2][jo + r0], (unsigned long long)za);
              sx += xa;
              sy += ya;
              sz += za;
              if (two) {
                const long long xb = to_fixed(fx.y), yb = to_fixed(fy.y), zb = to_fixed(fz.y);
                atomicAdd(&S.fj[0][jo + r1], (unsigned long long)xb);
                atomicAdd(&S.fj[1][jo + r1], (unsigned long long)yb);
                atomicAdd(&S.fj[2][jo + r1], (unsigned long long)zb);
                sx += xb;
                sy += yb;
                sz += zb;
              }
              if constexpr (EV) {
                const long long ea = to_fixed(0.5f * en.x), wa = to_fixed(0.5f * fac.x * r2.x);
                atomicAdd(&S.fj[3][jo + r0], (unsigned long long)ea);
                atomicAdd(&S.fj[4][jo + r0], (unsigned long long)wa);
                se += ea;
                sw += wa;
                if (two) {
                  const long long eb = to_fixed(0.5f * en.y), wb = to_fixed(0.5f * fac.y * r2.y);
                  atomicAdd(&S.fj[3][jo + r1], (unsigned long long)eb);
                  atomicAdd(&S.fj[4][jo + r1], (unsigned long long)wb);
                  se += eb;
                  sw += wb;
                }
              }
            } else {
              constexpr float FLIM = PK_FMAX * PK_SCALE;
              const float ma = max_abs3(fx.x, fy.x, fz.x), mb = max_abs3(fx.y, fy.y, fz.y);
              if (!(max_abs3(ma, mb, 0.0f) <= FLIM)) {
                // rare: the exact int64 path for both atoms of the pair
                auto large = [&](uint32_t r, float x, float y, float z) {
                  const uint32_t sj = S.jslot[r];
                  const long long lx = __float2ll_rn(x * (HB_FP_SCALE / PK_SCALE)),
                                  ly = __float2ll_rn(y * (HB_FP_SCALE / PK_SCALE)),
                                  lz = __float2ll_rn(z * (HB_FP_SCALE / PK_SCALE));
                  ax += lx;
                  ay += ly;
                  az += lz;
                  red_add(&fp[0 * np_all + sj], -lx);
                  red_add(&fp[1 * np_all + sj], -ly);
                  red_add(&fp[2 * np_all + sj], -lz);
                };
                if (!(ma <= FLIM)) {
                  large(r0, fx.x, fy.x, fz.x);
                  fx.x = fy.x = fz.x = 0.0f;
                }
                if (!(mb <= FLIM)) {
                  large(r1, fx.y, fy.y, fz.y);
                  fx.y = fy.y = fz.y = 0.0f;
                }
              }
              const int xa = __float2int_rn(fx.x), ya = __float2int_rn(fy.x), za = __float2int_rn(fz.x);
              const int xb = __float2int_rn(fx.y), yb = __float2int_rn(fy.y), zb = __float2int_rn(fz.y);
              atomicAdd(&S.fj[0][jo + r0], xa);
              atomicAdd(&S.fj[1][jo + r0], ya);
              atomicAdd(&S.fj[2][jo + r0], za);
              if (two) {
                atomicAdd(&S.fj[0][jo + r1], xb);
                atomicAdd(&S.fj[1][jo + r1], yb);
                atomicAdd(&S.fj[2][jo + r1], zb);
              }
              sx += xa + xb;
              sy += ya + yb;
              sz += za + zb;
              if constexpr (EV) {
                // half of the pair's energy and virial to each atom
                float2 he = __fmul2_rn(en, make_float2(0.5f / PK_SCALE, 0.5f / PK_SCALE));
                float2 hw = __fmul2_rn(__fmul2_rn(fac, r2), make_float2(0.5f / PK_SCALE, 0.5f / PK_SCALE));
                const float ga = max_abs3(he.x, hw.x, 0.0f), gb = max_abs3(he.y, hw.y, 0.0f);
                if (!(ga <= PK_EMAX) || (two && !(gb <= PK_EMAX))) {
                  auto large = [&](uint32_t r, float x, float y) {
                    const uint32_t sj = S.jslot[r];
                    const long long lx = to_fixed(x), ly = to_fixed(y);
                    ae += lx;
                    aw += ly;
                    red_add(&fp[3 * np_all + sj], lx);
                    red_add(&fp[4 * np_all + sj], ly);
                  };
                  if (!(ga <= PK_EMAX)) {
                    large(r0, he.x, hw.x);
                    he.x = hw.x = 0.0f;
                  }
                  if (two && !(gb <= PK_EMAX)) {
                    large(r1, he.y, hw.y);
                    he.y = hw.y = 0.0f;
                  }
                }
                const int ea = __float2int_rn(he.x * PK_ESCALE), wa = __float2int_rn(hw.x * PK_ESCALE);
                atomicAdd(&S.fj[3][jo + r0], ea);
                atomicAdd(&S.fj[4][jo + r0], wa);
                se += ea;
                sw += wa;
                if (two) {
                  const int eb = __float2int_rn(he.y * PK_ESCALE), wb = __float2int_rn(hw.y * PK_ESCALE);
                  atomicAdd(&S.fj[3][jo + r1], eb);
                  atomicAdd(&S.fj[4][jo + r1], wb);
                  se += eb;
                  sw += wb;
                }
              }
            }
          }
        };
        // rounds with the Lennard-Jones arithmetic while some lane's older
        // entry has such a pair, then rounds without.  A lane takes at most
        // 32 pairs in all (the older entry has 32 rows, two leave per round)
        while (__any_sync(0xFFFFFFFFu, m_a > lj_a)) round(std::true_type{});
        while (__any_sync(0xFFFFFFFFu, m_a != 0u)) round(std::false_type{});
        if constexpr (EXACT) {
          ax += sx;
          ay += sy;
          az += sz;
          ae += se;
          aw += sw;
        } else {
          ax += (long long)sx << PK_SHIFT;
          ay += (long long)sy << PK_SHIFT;
          az += (long long)sz << PK_SHIFT;
          if (EV) {
            ae += (long long)se << PK_ESHIFT;
            aw += (long long)sw << PK_ESHIFT;
          }
        }
        __syncwarp();
        const uint32_t sj = S.jslot[base_a + lane];
        if (sj != HB_SENTINEL) {
          // j-side sums carry the i-atoms' sign
#pragma unroll
          for (int q = 0; q < NC; ++q) {
            const long long t = (long long)S.fj[q][base_a + lane] + (long long)S.fj[q][PK_COPY + base_a + lane];
            const long long v = EXACT ? t : t << (q < 3 ? PK_SHIFT : PK_ESHIFT);
            red_add(&fp[q * np_all + sj], q < 3 ? -v : v);
          }
        }
        base_a = base_b;
        m_a = m_b | m_bl;
        lj_a = lj_b;
        sc_a = sc_b;
      }
    };
    const int flags = (int)c.w;
    if (!EXACT && (flags & 1) != 0) item(std::integral_constant<int, HB_IMAGE_NONE>{});
    else if ((flags & 2) != 0) item(std::integral_constant<int, HB_IMAGE_ORTHO>{});
    else item(std::integral_constant<int, HB_IMAGE_TILTED>{});
    if (ivalid) {
      red_add(&fp[0 * np_all + si], ax);
      red_add(&fp[1 * np_all + si], ay);
      red_add(&fp[2 * np_all + si], az);
      if (EV) {
        red_add(&fp[3 * np_all + si], ae);
        red_add(&fp[4 * np_all + si], aw);
      }
    }
  }
  if (EV) {
    // LJ energy total for the scalar split: one integer reduction per warp
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) elj_fix += __shfl_xor_sync(0xFFFFFFFFu, elj_fix, o);
    if (lane == 0) red_add(e_lj_total, elj_fix);
  }
}

// dynamic shared memory: the type tables
constexpr size_t table_bytes(size_t n_types) { return (sizeof(float4) + sizeof(float)) * n_types * n_types; }

// Tables of more than 28 types may not fit beside the warps' shared memory
// within the default 48 KB.  The limit is a property of the kernel in the
// whole process, so it is only ever set to the largest table's size: another
// thread's launch with a smaller table leaves it where it is.
template <class K>
int allow_smem(K kernel, size_t dynamic) {
  if (dynamic > 16u * 1024u)
    HB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)table_bytes(HB_MAX_TYPES)));
  return HB_OK;
}

// Entries per work item when the caller set none: about half of what each
// resident warp gets, at most 4.  Small systems need every entry as an item
// of its own (343 waters: 19 us at 1, 32 us at 4), large ones gain from
// fewer loads and sums of the i-tile until the last items' length shows
// (65,536 waters: 303, 259, 251, 248, 254 us at 1, 2, 3, 4, 8)
uint32_t pair_chunk_of(const hb_forcefield *ff) {
  if (ff->pair_chunk > 0) return (uint32_t)ff->pair_chunk;
  const uint64_t per_tile = std::max<uint32_t>((ff->slab - std::min(ff->slab, 4u)) * 2u / 3u, 1u);
  const uint64_t warps = (uint64_t)ff->sys->ctx->n_sm * 24u;
  return (uint32_t)std::min<uint64_t>(std::max<uint64_t>(per_tile * ff->n_tiles / (warps * 2u), 1u), 4u);
}

// Resident blocks per SM when the caller set none.  With a reciprocal part
// fewer than fit, so that its chain on the other stream finds SM room beside
// the persistent blocks.  Force-only (6 fit): one fewer where whole planes are
// transformed (graph step of 65,536 waters 414, 392, 453 us at 6, 5, 4; of
// 8,192 103, 97, 106 us), two fewer where five line passes have to find room
// (2,000 waters 69, 64, 60 us; 21,952: 209, 204, 196 us), and the same beside
// the one-cluster transform, where it makes no difference.  With energies or
// exact sums (5 fit) one fewer: beside line passes 1,732, 1,609, 1,596,
// 1,638 us per 20 steps of 1,237 waters with energies at 5, 4, 3, 2 blocks,
// 1,932, 1,770, 1,791, 1,911 us per relaxation of 2,000 waters, 961, 856, 832,
// 848 us per 10 exact steps of 13,824 ions.  The multi-system form takes the
// same four (12 replicas 2,809, 2,844, 2,941 us per 10 steps at 5, 4, 3)
uint32_t pair_blocks_of(const hb_forcefield *ff, bool wide) {
  if (ff->pair_blocks_per_sm > 0) return (uint32_t)ff->pair_blocks_per_sm;
  const uint32_t fit = wide ? PAIR_MIN_BLOCKS(true, false, false) : PAIR_MIN_BLOCKS(false, false, false);
  if (!ff->spme.on) return fit;
  return ff->spme.use_plane || wide ? fit - 1u : fit - 2u;
}

template <bool EV, bool SCALED, bool SWITCH, bool EXACT>
int launch_t(hb_forcefield *ff, cudaStream_t s, const PairParams &P) {
  const size_t smem = table_bytes((size_t)P.n_types);
  const uint32_t chunk = pair_chunk_of(ff);  // entries per work item
  const uint32_t chunks = hb_div_up(P.slab, chunk);
  const uint32_t items = P.n_tiles * chunks;
  // persistent (quota 0): that many blocks of 4 warps per SM, or fewer for
  // small systems; with a quota of q items per
  // warp, enough blocks that every item is taken
  uint32_t grid, quota = 0xFFFFFFFFu;
  if (ff->pair_quota > 0) {
    quota = (uint32_t)ff->pair_quota;
    grid = hb_div_up(items, PK_WARPS * quota);
  } else {
    grid = std::min<uint32_t>((uint32_t)ff->sys->ctx->n_sm * pair_blocks_of(ff, EV || EXACT),
                              hb_div_up(items, PK_WARPS));
  }
  HB_TRY(allow_smem(k_pair<EV, SCALED, SWITCH, EXACT, false>, smem));
  k_pair<EV, SCALED, SWITCH, EXACT, false><<<std::max(grid, 1u), PK_WARPS * 32, smem, s>>>(
      ff->d_tile_posq, ff->d_tile_type, ff->d_tile_center, ff->d_tile_nent, ff->d_entry_j,
      ff->d_entry_excl, ff->sys->d_box, ff->d_lj, ff->d_lj_invd, P, ff->d_fp, ff->d_sorted_ids,
      ff->d_excl_off, ff->d_excl_partner, ff->d_excl_scale, ff->d_work, chunks, chunk, quota,
      ff->d_acc, nullptr, 0u, 0u);
  HB_CUDA(cudaGetLastError());
  return HB_OK;
}

}  // namespace

int pair_launch(hb_forcefield *ff, bool ev, cudaStream_t s) {
  if (ff->sys->n < 2 || ff->n_tiles == 0) return HB_OK;
  if (!ff->lj_on && !ff->coul_on) return HB_OK;
  PairParams P;
  P.n_types = (int)ff->n_types;
  P.lj_on = ff->lj_on;
  P.coul_on = ff->coul_on;
  P.rc2_max = ff->rc_max * ff->rc_max;
  P.coul_rc2 = ff->coul_rc2;
  P.alpha = ff->alpha;
  P.c2a = 2.0f * ff->alpha / 1.7724538509055160273f;
  P.nl2e = -1.44269504088896340736f;
  P.n = ff->sys->n;
  P.n_tiles = ff->n_tiles;
  P.slab = ff->slab;
  const bool sc = ff->excl_scaled != 0, sw = ff->any_switch != 0;
  auto with = [&](auto e, auto c, auto w) {
    constexpr bool EV = decltype(e)::value, SC = decltype(c)::value, SW = decltype(w)::value;
    return ff->exact_pairs ? launch_t<EV, SC, SW, true>(ff, s, P) : launch_t<EV, SC, SW, false>(ff, s, P);
  };
  using T = std::true_type;
  using F = std::false_type;
  if (ev) {
    if (sc) return sw ? with(T{}, T{}, T{}) : with(T{}, T{}, F{});
    return sw ? with(T{}, F{}, T{}) : with(T{}, F{}, F{});
  }
  if (sc) return sw ? with(F{}, T{}, T{}) : with(F{}, T{}, F{});
  return sw ? with(F{}, F{}, T{}) : with(F{}, F{}, F{});
}

// ---------------------------------------------------------------------
// Multi-system pair launch (replica batches): one persistent k_pair over
// the work items of every member, each item finding its member by a binary
// search of the members' first items.  Members must share the pair physics
// (types, tables, cut-offs, Ewald alpha, switch) and take the force-only,
// unscaled, tile-shifted form; their own lists, positions, cells and
// accumulators stay where they are.
// ---------------------------------------------------------------------
size_t pair_member_bytes() { return sizeof(PairMember); }

bool pair_batchable(hb_forcefield *const *ffs, uint32_t n) {
  if (n == 0) return false;
  const hb_forcefield *a = ffs[0];
  for (uint32_t k = 0; k < n; ++k) {
    const hb_forcefield *f = ffs[k];
    if (f->exact_pairs || f->excl_scaled || f->n_tiles == 0 || f->sys->n < 2) return false;
    if (f->lj_on != a->lj_on || f->coul_on != a->coul_on || f->any_switch != a->any_switch ||
        f->n_types != a->n_types || f->rc_max != a->rc_max || f->coul_rc2 != a->coul_rc2 ||
        f->alpha != a->alpha)
      return false;
    // the switch factors (lj_invd) follow from these tables
    if (f->h_lj.size() != a->h_lj.size()) return false;
    if (std::memcmp(f->h_lj.data(), a->h_lj.data(), sizeof(float4) * a->h_lj.size()) != 0) return false;
  }
  return a->lj_on || a->coul_on;
}

// the member table (host-built, copied synchronously: call outside capture).
// One work-item length for all members, the first one's: with items of all
// members to take from, the length does not show (12 replicas 2,846, 2,830,
// 2,838, 2,824 us per 10 steps at 1, 2, 3, 4 entries; with a kernel per member
// 2,460, 2,416, 2,504, 2,479)
int pair_batch_table(hb_forcefield *const *ffs, uint32_t n, void *d_table, uint32_t *items_total) {
  std::vector<PairMember> t(n);
  uint32_t item0 = 0;
  const uint32_t chunk = pair_chunk_of(ffs[0]);
  for (uint32_t k = 0; k < n; ++k) {
    hb_forcefield *f = ffs[k];
    PairMember &m = t[k];
    std::memset(&m, 0, sizeof(m));
    m.tile_posq = f->d_tile_posq;
    m.tile_type = f->d_tile_type;
    m.center = f->d_tile_center;
    m.tile_nent = f->d_tile_nent;
    m.entry_j = f->d_entry_j;
    m.entry_excl = f->d_entry_excl;
    m.box = f->sys->d_box;
    m.fp = f->d_fp;
    m.n = f->sys->n;
    m.n_tiles = f->n_tiles;
    m.slab = f->slab;
    m.chunks = hb_div_up(f->slab, chunk);
    m.item0 = item0;
    item0 += m.n_tiles * m.chunks;
  }
  HB_CUDA(cudaMemcpy(d_table, t.data(), sizeof(PairMember) * n, cudaMemcpyHostToDevice));
  *items_total = item0;
  return HB_OK;
}

int pair_launch_batch(hb_forcefield *const *ffs, uint32_t n, const void *d_table,
                      uint32_t items_total, uint32_t *d_work, cudaStream_t s) {
  const hb_forcefield *a = ffs[0];
  PairParams P;
  std::memset(&P, 0, sizeof(P));
  P.n_types = (int)a->n_types;
  P.lj_on = a->lj_on;
  P.coul_on = a->coul_on;
  P.rc2_max = a->rc_max * a->rc_max;
  P.coul_rc2 = a->coul_rc2;
  P.alpha = a->alpha;
  P.c2a = 2.0f * a->alpha / 1.7724538509055160273f;
  P.nl2e = -1.44269504088896340736f;
  const size_t smem = table_bytes((size_t)P.n_types);
  const uint32_t grid = std::min<uint32_t>(
      (uint32_t)a->sys->ctx->n_sm * pair_blocks_of(a, true), hb_div_up(items_total, PK_WARPS));
  HB_CUDA(cudaMemsetAsync(d_work, 0, sizeof(uint32_t), s));
  const PairMember *tab = static_cast<const PairMember *>(d_table);
  auto launch = [&](auto kernel) {
    HB_TRY(allow_smem(kernel, smem));
    kernel<<<std::max(grid, 1u), PK_WARPS * 32, smem, s>>>(
        nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, a->sys->d_box, a->d_lj, a->d_lj_invd, P,
        nullptr, nullptr, nullptr, nullptr, nullptr, d_work, 1u, pair_chunk_of(a), 0xFFFFFFFFu,
        nullptr, tab, n, items_total);
    HB_CUDA(cudaGetLastError());
    return (int)HB_OK;
  };
  return a->any_switch ? launch(k_pair<false, false, true, false, true>)
                       : launch(k_pair<false, false, false, false, true>);
}
