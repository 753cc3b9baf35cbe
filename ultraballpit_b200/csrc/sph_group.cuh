// sph_group.cuh - the neighbour kernels with G lanes per particle.
//
// One thread per particle walks its candidates, its 80 or so neighbours and
// its boundary candidates in series: below some 50,000 particles the GPU then
// holds too few warps to hide that chain, and a step costs the chain's latency
// whatever its size. Here a group of G consecutive lanes shares a particle:
// each lane evaluates one pair of a round, and the terms go to shared memory
// in visit order, from where the lanes add them up, one component of the sums
// per lane, one term after the other: the additions, and their order, are the
// reference's. A term then costs its store and its turn in the additions on
// top, so that above those sizes a thread per particle is the faster form.
// Dam break, us per kernel, thread form | 8 | 16 | 32 lanes:
//   particles   density                forces               XSPH + drift
//     2,000     92 | 27 | 21 | 18      39 | 16 | 14 | 14    24 | 17 | 14 | 16
//     5,292     98 | 27 | 23 | 29      37 | 18 | 16 | 21    23 | 16 | 16 | 20
//    11,664     96 | 31 | 39 | 53      37 | 21 | 23 | 29    22 | 18 | 20 | 26
//    31,250    103 | 66 | 82 | 127     41 | 37 | 43 | 59    24 | 30 | 34 | 50
//    72,963    119 | 131               49 | 68              31 | 53
// (the warp-cooperative density scan, 32 particles a warp: 113 at 72,963).
// Hence 16 lanes up to 56 particles per SM, 8 above, for density and forces up
// to 240 and 256 per SM, for XSPH up to 128; density then takes two lanes per
// particle (k_density_pair) up to 1300 per SM.
#pragma once
#include "sph_kernels.cuh"

namespace sph {

constexpr int kGroupThreads = 128;  // threads per block of the group forms
constexpr int kGroupBlocks = 5;     // per SM: 96 registers, no spills (7 blocks at 72: 10 % slower below 10k particles)
constexpr int kRepCap = 32;         // noted repulsion candidates per particle

// Shared memory of one group: NC components of CH ordered terms (the terms
// between two rounds of additions), rows 16 bytes apart in the banks.
template <int NC, int CH>
struct __align__(16) GroupTerms {
  float t[NC][CH + 4];
};
constexpr int kRounds = 2;  // rounds whose gathers are in flight together
template <int G>
constexpr int kChunkOf = G * kRounds;  // the terms they make

template <int G>
struct Group {
  static constexpr int kPer = kGroupThreads / G;  // particles per block
  int sub;         // lane within the group
  unsigned mask;   // the group's lanes within the warp
  int shift;       // first lane of the group
  __device__ __forceinline__ Group()
      : sub((int)(threadIdx.x & (G - 1))), shift((int)(threadIdx.x & 31u & ~(unsigned)(G - 1))) {
    mask = ((1u << G) - 1u) << shift;
  }
  // the group's bits of a warp ballot, at bit 0
  __device__ __forceinline__ uint32_t bits(uint32_t ballot) const { return (ballot & mask) >> shift; }
  __device__ __forceinline__ uint32_t below() const { return (1u << sub) - 1u; }
  __device__ __forceinline__ float get(float v, int lane) const {
    return __shfl_sync(0xffffffffu, v, shift + lane);
  }
};

// A lane's entries of its particle's stored list: sub, sub + G, ... in turn.
template <int G>
struct GroupList {
  const uint32_t* p;
  size_t step;  // words from one round's entry to the next
  __device__ __forceinline__ GroupList(const uint32_t* nbr, int n, int i, int sub)
      : p(nbr + nbr_index((uint32_t)sub, n, i)), step((size_t)n * G) {}
  __device__ __forceinline__ uint32_t next() {
    const uint32_t v = __ldg(p);
    p += step;
    return v;
  }
};

// Adds the first `m` terms (m <= CH, group-uniform; terms past it up to a
// multiple of four are zeros) of the lane's component, in order. Adding a
// zero leaves a sum that is not -0 as it is.
template <int NC, int CH>
__device__ __forceinline__ float add_terms(const GroupTerms<NC, CH>& T, int c, uint32_t m, float acc) {
  const float* t = T.t[c];
  for (uint32_t e = 0; e < m; e += 4) {
    const float4 v = *reinterpret_cast<const float4*>(t + e);
    acc += v.x;
    acc += v.y;
    acc += v.z;
    acc += v.w;
  }
  return acc;
}

// Boundary particles entry(q0 .. q1), G at a time, each loaded a round ahead:
// f(valid, index, position) with every lane of the warp taking part
// (groups of a warp may differ in their ranges).
template <int G, class L, class F>
__device__ __forceinline__ void group_candidates(const Group<G>& g, uint32_t q0, uint32_t q1, L&& entry,
                                                 const float4* __restrict__ bpos, F&& f) {
  uint32_t q = q0 + g.sub, ahead = q + G;
  uint32_t bi = q < q1 ? entry(q) : 0u;
  uint32_t bn = ahead < q1 ? entry(ahead) : 0u;
  float4 bp = q < q1 ? __ldg(&bpos[bi]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (uint32_t r = q0; __any_sync(0xffffffffu, r < q1); r += G) {
    const bool valid = q < q1;
    const uint32_t b = bi;
    const float4 p = bp;
    q = ahead;
    ahead += G;
    bi = bn;
    if (ahead < q1) bn = entry(ahead);
    if (q < q1) bp = __ldg(&bpos[bi]);
    f(valid, b, p);
  }
}

// ---------------------------------------------------------------------------
// XSPH + drift (k_xsph_drift's work)
// ---------------------------------------------------------------------------
// The neighbours' half-kicked velocities (k_xsph_prep's records in the thread
// form) are computed here from velocity and acceleration: a launch less, where
// launches count. With `red` the kernel also computes the step's dt from the
// last step's maxima, for every instance's own particles; the first block
// stores it, for all `ninst` instances, those without particles among them.
template <class KP, int G>
__global__ void __launch_bounds__(kGroupThreads, kGroupBlocks)
k_xsph_group(KP kp, int n, int ninst, float* __restrict__ dtp, const float* __restrict__ red,
             const float4* __restrict__ pos,
             const float4* __restrict__ velout, const float4* __restrict__ acc,
             const uint32_t* __restrict__ id, const uint2* __restrict__ ctab,
             const uint32_t* __restrict__ rank_of_lin, float4* __restrict__ posU, float4* __restrict__ velU,
             uint32_t* __restrict__ idU, uint32_t* __restrict__ keyU, uint32_t* __restrict__ hist,
             const uint32_t* __restrict__ err, const uint32_t* __restrict__ nbr,
             const uint32_t* __restrict__ ncount) {
  constexpr int U = kRounds, CH = kChunkOf<G>;
  __shared__ GroupTerms<3, CH> s_terms[kGroupThreads / G];
  const Group<G> g;
  GroupTerms<3, CH>& T = s_terms[threadIdx.x / G];
  const int slot = (int)((blockIdx.x * kGroupThreads + threadIdx.x) / G);
  const bool live = slot < n && !*err;
  const int i = live ? slot : 0;
  const SimConst& k = kp.at(i);
  float dt;
  if (red) {
    dt = cfl_dt(k.h, k.c, k.cfl, red[2 * k.inst], red[2 * k.inst + 1]);
    if (blockIdx.x == 0)
      for (int q = threadIdx.x; q < ninst; q += kGroupThreads)
        dtp[q] = cfl_dt(kp.tab[q].h, kp.tab[q].c, kp.tab[q].cfl, red[2 * q], red[2 * q + 1]);
  } else {
    dt = dtp[k.inst];
  }
  const float4 pi = pos[i];
  const float4 vi = velout[i];
  const float4 ai = acc[i];
  const float hdt = 0.5f * dt;
  const float vx = vi.x + ai.x * hdt;
  const float vy = vi.y + ai.y * hdt;
  const float vz = vi.z + ai.z * hdt;
  float sum = 0.0f;  // lanes 0..2: the components of the XSPH sum
  const bool xsph = live && (k.flags & kFlagXsph);
  const uint32_t counts = xsph ? (k.fast ? __ldg(&ncount[i]) : kRescanBit) : 0u;
  const bool listed = counts_listed(counts);
  const uint32_t mine = listed ? counts_neighbours(counts) : 0u;
  const uint32_t most = __reduce_max_sync(0xffffffffu, mine);
  // the quotient's operands are watched here: the largest density, and whether
  // a mass lies outside the range
  float rho_max = vi.w;
  bool odd = false;
  GroupList<G> list(nbr, n, i, g.sub);
  for (uint32_t c0 = 0; c0 < most; c0 += CH) {
    // the entries past the list's end are in bounds and not used: their lanes
    // gather the particle itself and put zeros
    float4 pj[U], vj[U], aj[U];
    uint32_t s[U];
#pragma unroll
    for (int u = 0; u < U; ++u) s[u] = list.next();
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!(c0 + u * G + g.sub < mine)) s[u] = (uint32_t)i;
      pj[u] = __ldg(&pos[s[u]]);
      vj[u] = __ldg(&velout[s[u]]);
      aj[u] = __ldg(&acc[s[u]]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float dx = pi.x - pj[u].x, dy = pi.y - pj[u].y, dz = pi.z - pj[u].z;
      const float factor = xsph_factor(dx * dx + dy * dy + dz * dz, 2.0f * pj[u].w, vi.w + vj[u].w, k);
      const float m = fabsf(pj[u].w);
      rho_max = fmaxf(rho_max, vj[u].w);
      odd = odd || !(m == 0.0f || (m >= kMassMin && m <= kMassMax));
      const bool in = c0 + u * G + g.sub < mine;
      T.t[0][u * G + g.sub] = in ? factor * ((vj[u].x + aj[u].x * hdt) - vx) : 0.0f;
      T.t[1][u * G + g.sub] = in ? factor * ((vj[u].y + aj[u].y * hdt) - vy) : 0.0f;
      T.t[2][u * G + g.sub] = in ? factor * ((vj[u].z + aj[u].z * hdt) - vz) : 0.0f;
    }
    __syncwarp();
    if (g.sub < 3 && c0 < mine) sum = add_terms(T, g.sub, min(mine - c0, (uint32_t)CH), sum);
    __syncwarp();
  }
  odd = g.bits(__ballot_sync(0xffffffffu, odd || rho_max > kRhoMax)) != 0u;
  float sx = g.get(sum, 0), sy = g.get(sum, 1), sz = g.get(sum, 2);
  if (xsph && (!listed || odd || !finite3(sx, sy, sz))) {
    const Sum3 e = xsph_exact(kp.ref(i), i, pi, make_float4(vx, vy, vz, vi.w), hdt, pos, velout, acc, ctab);
    sx = e.x;
    sy = e.y;
    sz = e.z;
  }
  if (!live || g.sub != 0) return;
  drift_and_bin(k, i, dt, pi, vi.w, vx, vy, vz, sx, sy, sz, id, rank_of_lin, posU, velU, idU, keyU, hist);
}

// ---------------------------------------------------------------------------
// density + density diffusion + equation of state (k_density's work)
// ---------------------------------------------------------------------------
// A warp holds P = 32 / G consecutive slots, G lanes each. The scan is
// scan_warp's with the P slots' segments (scan_segment: the lanes are 32
// candidates, four particles a step), so a warp of fewer particles is a
// shorter chain; then the lanes of a group turn its masks into its list, each
// a run of the words, and share its terms and boundary candidates.
template <int G, int NC>
struct __align__(16) CoopWarp {
  static constexpr int P = 32 / G, kPad = (P + 3) & ~3, kCols = 4 * P;
  float px[kPad], py[kPad], pz[kPad];  // a segment's particles
  union {
    uint32_t mask[kScanWords * kCols];  // per segment [word][particle]
    GroupTerms<NC, kChunkOf<G>> terms[P];  // once the masks are lists
  };
  uint32_t list[P][kNbrCap];
  uint32_t vstart[P][kScanRanges + 1], sstart[P][kScanRanges];  // as ScanWarp's, per segment
  uint32_t mbase[kPad], mquad[kPad];
};

// The closure's feature probes (feature_probe) of a particle held by L lanes,
// `sub` this one's number and get(v, l) lane l's v: each lane reads its share
// and every lane ends up with all twelve. Every lane of the warp takes part,
// `near` if its particle is near the wall. Bound by latency: one lane alone
// read them in turn, some 100 gathers and 36 divisions, and they took 22 of
// the 107 us of a 24k-particle tank's density pass; shared by 8 lanes they
// take 6, by the pair form's 2 some 6 of 133 us at 42k particles.
template <int L, class Get>
__device__ __forceinline__ void share_probes(const SimConst& k, const float* __restrict__ sdf, const float4& pi,
                                             int sub, bool near, float centre, Get get, float out[12]) {
  if (!__any_sync(0xffffffffu, near)) return;
  const bool grad = near && wall_is_sdf(k, pi, centre);
  constexpr int R = (12 + L - 1) / L;
  float own[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int a = r * L + sub;
    own[r] = a < 12 && (a < 6 ? grad : near) ? feature_probe(k, sdf, pi, a) : 0.0f;
  }
#pragma unroll
  for (int a = 0; a < 12; ++a) out[a] = get(own[a / L], a % L);
}

// The closure network's tile of a block in the group form: a row per
// particle, taken by the block's last warp to arrive, which nobody waits for.
// A tile a warp was 4 rows of 16 with 8 lanes a particle: the network took 27
// us of the same pass, and takes 14 with one tile a block. The two together:
// 45 -> 37 / 63 -> 55 / 107 -> 86 us at 5k / 13k / 24k particles.
struct BlockTile {
  uint32_t xy[kClTileWords];  // network_epilogue's tile
  int owner[16];              // the row's particle, -1 for none
  float rho_pre[16];
  uint32_t arrived;           // warps, and (from bit 16 up) their particles near the wall
};

template <class KP, int CL, int G>
__global__ void __launch_bounds__(kGroupThreads, kGroupBlocks)
k_density_group(KP kp, int n, const float* __restrict__ dtp, const float4* __restrict__ pos, Planes pl,
                const float2* __restrict__ rv, const uint32_t* __restrict__ id, const uint2* __restrict__ ctab,
                const uint32_t* __restrict__ bc_start, const uint32_t* __restrict__ bc_list,
                const float4* __restrict__ bpos, float2* __restrict__ rf, float* __restrict__ pr,
                const uint32_t* __restrict__ err, uint32_t* __restrict__ nbr, uint32_t* __restrict__ ncount,
                const float* __restrict__ sdf, const float2* __restrict__ wall_tab, ClosureBufs cb,
                uint32_t* __restrict__ slow, WallLists wl) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int NC = CL ? 3 : 2, P = 32 / G;
  extern __shared__ __align__(16) unsigned char s_dyn[];
  using SW = CoopWarp<G, NC>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  SW& S = reinterpret_cast<SW*>(s_dyn)[warp];
  BlockTile& B = *reinterpret_cast<BlockTile*>(s_dyn + (kGroupThreads / 32) * sizeof(SW));  // CL == 2
  const Group<G> g;
  const int base = (int)((blockIdx.x * kGroupThreads + threadIdx.x) >> 5) * P;
  if (CL == 2) {
    B.xy[threadIdx.x] = 0u;  // the x tile: 128 words
    if (threadIdx.x < 16) B.owner[threadIdx.x] = -1;
    if (threadIdx.x == 0) B.arrived = 0u;
    __syncthreads();
  }
  if (base >= n || *err) return;  // whole warps
  const int mine_p = lane / G;    // the group's particle within the warp
  const bool live = base + mine_p < n;
  const int i = live ? base + mine_p : base;
  const SimConst& k = kp.at(i);
  const float4 pi = pos[i];
  const int cx = axis_cell(pi.x, k.gmin[0], k.cell, k.dims[0]);
  const int cy = axis_cell(pi.y, k.gmin[1], k.cell, k.dims[1]);
  const int cz = axis_cell(pi.z, k.gmin[2], k.cell, k.dims[2]);
  const int lin = cell_hash(cx, cy, cz, k);
  // Phase 1: the segments' masks. Lane p < P stands for particle p here.
  const int src = (lane < P ? lane : 0) * G;
  const bool slot_live = __shfl_sync(kAll, live ? 1 : 0, src) && lane < P;
  const float qx = __shfl_sync(kAll, pi.x, src), qy = __shfl_sync(kAll, pi.y, src), qz = __shfl_sync(kAll, pi.z, src);
  const int ix = __shfl_sync(kAll, cx, src), iy = __shfl_sync(kAll, cy, src), iz = __shfl_sync(kAll, cz, src);
  const int islot = __shfl_sync(kAll, i, src);
  const uint32_t gkey = __shfl_sync(kAll, (uint32_t)(k.coff + lin), src);
  const uint32_t gprev = __shfl_up_sync(kAll, gkey, 1);
  const uint32_t heads = __ballot_sync(kAll, slot_live && (lane == 0 || gprev != gkey));
  const int nlive = __popc(__ballot_sync(kAll, slot_live));
  {
    int seg = 0;
    uint32_t mbase = 0;
    for (uint32_t hh = heads; hh; hh &= hh - 1u, ++seg) {
      const int hl = __ffs(hh) - 1;
      const uint32_t after = heads & ~((2u << hl) - 1u);  // hl < P <= 16
      const int he = after ? __ffs(after) - 1 : nlive;
      const int sx = __shfl_sync(kAll, ix, hl), sy = __shfl_sync(kAll, iy, hl), sz = __shfl_sync(kAll, iz, hl);
      const SimConst& ks = kp.at(__shfl_sync(kAll, islot, hl));
      const int nw = scan_segment(S, seg, hl, he, mbase, ks, sx, sy, sz, qx, qy, qz, pl, ctab);
      if (nw <= kScanWords) mbase += (uint32_t)(nw * ((he - hl + 3) & ~3));
      __syncwarp();
    }
  }
  // Phase 2: each lane of a group expands a run of its particle's mask words
  // into the list, from the count of the lanes before it.
  uint32_t listed = 0;
  {
    const uint32_t upto = heads & ((2u << mine_p) - 1u);  // mine_p < P <= 16
    const int s = __popc(upto) - 1;
    const int head = 31 - __clz(upto);
    const int R = k.rows ? 9 : 27;
    const uint32_t total = S.vstart[s][R];
    const int nw = (int)((total + 31u) / 32u);
    if (nw > kScanWords) {  // too dense for the masks: the per-thread scan
      if (live && g.sub == 0) listed = record_neighbors(pi.x, pi.y, pi.z, i, pl, ctab, ScanGeo(k), nbr, n);
      listed = __shfl_sync(g.mask, listed, g.shift);
      __syncwarp(g.mask);
      if (live)
        for (uint32_t e = g.sub; e < min(listed, kNbrCap); e += G) S.list[mine_p][e] = nbr[nbr_index(e, n, i)];
    } else {
      const uint32_t q4 = S.mquad[s];
      const uint32_t* words = S.mask + S.mbase[s] + (mine_p - head);
      const uint32_t vself = S.vstart[s][R / 2] + ((uint32_t)i - S.sstart[s][R / 2]);
      const int wself = (int)(vself >> 5);
      const uint32_t bself = ~(1u << (vself & 31u));
      const int w0 = g.sub * nw / G, w1 = (g.sub + 1) * nw / G;
      uint32_t count = 0;
      for (int w = w0; live && w < w1; ++w) count += __popc(w == wself ? words[w * q4] & bself : words[w * q4]);
      uint32_t incl = count;
#pragma unroll
      for (int o = 1; o < G; o <<= 1) {
        const uint32_t v = __shfl_up_sync(g.mask, incl, o, G);
        if (g.sub >= o) incl += v;
      }
      listed = __shfl_sync(g.mask, incl, G - 1, G);
      uint32_t e = incl - count;
      int r = 0;
      uint32_t vnext = S.vstart[s][1];
      uint32_t delta = S.sstart[s][0] - S.vstart[s][0];
      uint32_t* const out = S.list[mine_p];
      int w = w0 - 1;
      uint32_t M = 0;
      for (; count; --count) {
        while (M == 0u) {
          ++w;
          M = words[w * q4];
          if (w == wself) M &= bself;
        }
        const uint32_t v = (uint32_t)(w * 32 + __ffs(M) - 1);
        M &= M - 1u;
        while (v >= vnext) {
          ++r;
          vnext = S.vstart[s][r + 1];
          delta = S.sstart[s][r] - S.vstart[s][r];
        }
        if (e < kNbrCap) out[e] = v + delta;
        ++e;
      }
    }
  }
  __syncwarp();
  // Phase 3: the terms over the list. Lane 0 sums the density, lane 1 the
  // diffusion, lane 2 the closure's kernel sum.
  constexpr int U = kRounds, CH = kChunkOf<G>;
  GroupTerms<NC, CH>& T = S.terms[mine_p];
  uint32_t* const list = S.list[mine_p];
  const float rho_old_i = rv[i].x;
  const bool delta = (k.flags & kFlagDelta) != 0;
  uint32_t key = 0xffffffffu;
  float dmin = INFINITY;
  float sum = g.sub == 0 ? pi.w * k.norm_h3 : 0.0f;
  const uint32_t mine = live && listed <= kNbrCap ? listed : 0u;
  const uint32_t most = __reduce_max_sync(kAll, mine);
  for (uint32_t c0 = 0; c0 < most; c0 += CH) {
    float4 pj[U];
    float2 rvj[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {  // a lane past the list's end gathers the particle itself and puts zeros
      const uint32_t e = c0 + u * G + g.sub;
      const uint32_t s = e < mine ? list[e] : (uint32_t)i;
      pj[u] = __ldg(&pos[s]);
      rvj[u] = __ldg(&rv[s]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = c0 + u * G + g.sub < mine;
      const float dx = pi.x - pj[u].x, dy = pi.y - pj[u].y, dz = pi.z - pj[u].z;
      const float d2 = in ? dx * dx + dy * dy + dz * dz : 1.0f;
      float w, half_diff;
      if (delta) density_fast<true>(k, pj[u].w, rvj[u], rho_old_i, dx, dy, dz, d2, key, dmin, w, half_diff);
      else density_fast<false>(k, pj[u].w, rvj[u], rho_old_i, dx, dy, dz, d2, key, dmin, w, half_diff);
      T.t[0][u * G + g.sub] = in ? pj[u].w * w : 0.0f;
      T.t[1][u * G + g.sub] = in ? 2.0f * half_diff : 0.0f;
      if (CL) T.t[2][u * G + g.sub] = in ? rvj[u].y * w : 0.0f;
    }
    __syncwarp();
    if (g.sub < NC && c0 < mine) sum = add_terms(T, g.sub, min(mine - c0, (uint32_t)CH), sum);
    __syncwarp();
  }
  float rho = g.get(sum, 0), diff_sum = g.get(sum, 1), ssum = CL ? g.get(sum, 2) : 0.0f;
  const bool close = g.bits(__ballot_sync(kAll, dmin < kTinyD2)) != 0u;
  const bool small = g.bits(__ballot_sync(kAll, key < k.diff_key)) != 0u;
  if (live && (listed > kNbrCap || !k.fast || close || small || !finite3(rho, diff_sum, 0.0f))) {
    const DensitySum e = density_exact(kp.ref(i), i, pi, rho_old_i, pos, rv, ctab);
    rho = e.rho;
    diff_sum = e.diff;
    if (CL) ssum = e.ssum;
  }
  __syncwarp();
  // Phase 4: boundary terms m_b w in ascending boundary index, added to the
  // density by lane 0 and to the closure's wall density by lane 1; the
  // boundary particles in support follow the neighbours in the list.
  const uint32_t b0 = live ? __ldg(&bc_start[k.coff + lin]) : 0u, b1 = live ? __ldg(&bc_start[k.coff + lin + 1]) : 0u;
  float wsum = g.sub == 0 ? rho : 0.0f;
  uint32_t nwall = 0, held = 0;  // held: terms waiting in shared memory
  auto flush = [&] {
    __syncwarp();
    if (g.sub < 4 && (held & 3u) && ((held + g.sub) & ~3u) == (held & ~3u)) T.t[0][held + g.sub] = 0.0f;
    __syncwarp();
    if (g.sub < (CL ? 2 : 1)) wsum = add_terms(T, 0, held, wsum);
    __syncwarp();
    held = 0;
  };
  group_candidates(g, b0, b1, [&](uint32_t q) { return __ldg(&bc_list[q]); }, bpos,
                   [&](bool valid, uint32_t bi, const float4& bp) {
    const float dx = pi.x - bp.x, dy = pi.y - bp.y, dz = pi.z - bp.z;
    const float d2 = dx * dx + dy * dy + dz * dz;
    const bool in = valid && d2 <= k.sup_d2;
    const uint32_t ballot = __ballot_sync(kAll, in);
    if (ballot == 0u) return;
    const uint32_t m = g.bits(ballot);
    if (__any_sync(kAll, held + __popc(m) > (uint32_t)CH)) flush();
    if (in) {
      const uint32_t rank = __popc(m & g.below());
      T.t[0][held + rank] = bp.w * w_c2(sqrt_any(d2), k);
      const uint32_t e = listed + nwall + rank;
      if (e < kNbrCap) list[e] = bi;
    }
    held += __popc(m);
    nwall += __popc(m);
  });
  flush();
  // the list leaves in quads: lane l stores those of particle l % P
  {
    const int p = lane % P;
    const uint32_t entries = __shfl_sync(kAll, min(listed + nwall, kNbrCap), p * G);
    const int ip = base + p;
    if (ip < n)
      for (uint32_t q = lane / P; q * 4 < entries; q += G)
        reinterpret_cast<uint4*>(nbr)[(size_t)q * (size_t)n + (size_t)ip] =
            *reinterpret_cast<const uint4*>(&S.list[p][q * 4]);
  }
  const uint32_t counts = live ? pack_counts(listed, nwall, close) : 0u;
  if (CL == 0 && wl.list) {
    const uint32_t theirs = __shfl_sync(kAll, counts, (lane % P) * G);
    scatter_walls(kp, base, lane < P ? theirs : 0u, pos, bc_start, bc_list, bpos, wl,
                  [&](int src, uint32_t e) { return S.list[src][e]; });
  }
  rho = g.get(wsum, 0);
  const DensityState st{rho, diff_sum, ssum, CL ? g.get(wsum, 1) : 0.0f, nwall, listed};
  const float centre = live ? centre_sdf<CL>(k, sdf, pi) : 0.0f;
  float probes[CL ? 12 : 1];
  if (CL)
    share_probes<G>(k, sdf, pi, g.sub, live && k.feat_sdf && centre_feature(k, pi, centre) < k.support, centre,
                    [&](float v, int l) { return g.get(v, l); }, probes);
  float f[16];
  float rho_pre = 0.0f;
  bool near_wall = false;
  if (live && g.sub == 0) {
    ncount[i] = counts;
    near_wall = density_finish<CL>(k, i, dtp[k.inst], pi, st, rv, id, rf, pr, centre,
                                   [&](int a) { return probes[CL ? a : 0]; }, wall_tab, cb, slow, f, rho_pre);
  }
  if (CL == 2) {
    constexpr int W = kGroupThreads / 32;
    static_assert(W * P <= 16 && kGroupThreads == 16 * 16 / 2, "a block's particles are one tile");
    __nv_bfloat16* xt = reinterpret_cast<__nv_bfloat16*>(B.xy);
    float* yt = reinterpret_cast<float*>(B.xy + 16 * 16 / 2);
    const int row = warp * P + mine_p;
    if (near_wall) {
#pragma unroll
      for (int a = 0; a < 16; ++a) xt[row * 16 + a] = __float2bfloat16_rn(f[a]);
      B.owner[row] = i;
      B.rho_pre[row] = rho_pre;
    }
    const uint32_t rows = (uint32_t)__popc(__ballot_sync(kAll, near_wall));
    // the rows, and density_finish's results, are there for the last to arrive
    __threadfence_block();
    __syncwarp();
    const uint32_t before = __shfl_sync(kAll, lane == 0 ? atomicAdd(&B.arrived, 1u + (rows << 16)) : 0u, 0);
    const int warps = min(W, (n - (base - warp * P) + P - 1) / P);
    if ((int)(before & 0xffffu) != warps - 1 || (before >> 16) + rows == 0u) return;
    __threadfence_block();
    sphmlp::forward_tile_regs(xt, cb.wq, cb.wf, yt, lane);
    __syncwarp();
    const int o = lane < 16 ? B.owner[lane] : -1;
    if (o >= 0)
      closure_apply_one(kp.at(o), o, (id[o] & kAirBit) != 0, B.rho_pre[lane], yt + lane * 4, rf, pr, cb.corr, slow);
  }
}

// Between the group form's sizes and those whose warps of 32 particles fill
// the GPU: 16 particles a warp, two lanes each. The scan is scan_warp's with
// 16 particles; in a round the pair's lanes take two neighbours each (entries
// 4r, 4r + 1 and 4r + 2, 4r + 3 of the list), and the first adds its own terms,
// then the other's. It executes 38 % more instructions than 32 particles a warp
// and halves the chain. Density, us, 8 lanes | pair | 32 particles a warp:
//   31k 66 | 66 | 103   50k 96 | 79 | 104   73k 131 | 95 | 111
//   146k - | 166 | 178   250k - | 251 | 241
// A tank with SDF walls:   24k  49 | 53 | 88     35k  66 | 55 | 88     73k 125 | 82 | 104
//                         115k 186 | 119 | 115  163k 260 | 160 | 154  191k 301 | 174 | 162
// and with the closure:    24k  80 | 94 | 135    35k 111 | 109 | 131   73k 195 | 152 | 164
//                         115k 291 | 223 | 213  163k 379 | 270 | 254  191k 436 | 307 | 300
// There two lanes and one cross at some 100k, not at the 192k that the rule has
// for all: up to 7 % of those passes (SDF walls with the closure 14 %).
// Eight blocks per SM at 64 registers; with six or five, 73k takes 113 or 117.
constexpr int kPairParticles = 16;
constexpr int kPairBlocks = 8;
template <class KP, int CL>
__global__ void __launch_bounds__(kGroupThreads, kPairBlocks)
k_density_pair(KP kp, int n, const float* __restrict__ dtp, const float4* __restrict__ pos, Planes pl,
               const float2* __restrict__ rv, const uint32_t* __restrict__ id, const uint2* __restrict__ ctab,
               const uint32_t* __restrict__ bc_start, const uint32_t* __restrict__ bc_list,
               const float4* __restrict__ bpos, float2* __restrict__ rf, float* __restrict__ pr,
               const uint32_t* __restrict__ err, uint32_t* __restrict__ nbr, uint32_t* __restrict__ ncount,
               const float* __restrict__ sdf, const float2* __restrict__ wall_tab, ClosureBufs cb,
               uint32_t* __restrict__ slow, WallLists wl) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int P = kPairParticles;
  extern __shared__ __align__(16) unsigned char s_dyn[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  ScanWarp& S = reinterpret_cast<ScanWarp*>(s_dyn)[warp];
  const int base = (int)((blockIdx.x * kGroupThreads + threadIdx.x) >> 5) * P;
  if (base >= n || *err) return;  // whole warps
  const int p = lane & (P - 1);
  const bool second = lane >= P;
  const bool live = base + p < n;
  const int i = live ? base + p : base;
  const SimConst& k = kp.at(i);
  const float4 pi = pos[i];
  const float rho_old_i = rv[i].x;
  const bool delta = (k.flags & kFlagDelta) != 0;
  const int cx = axis_cell(pi.x, k.gmin[0], k.cell, k.dims[0]);
  const int cy = axis_cell(pi.y, k.gmin[1], k.cell, k.dims[1]);
  const int cz = axis_cell(pi.z, k.gmin[2], k.cell, k.dims[2]);
  const int lin = cell_hash(cx, cy, cz, k);
  const uint32_t gkey = (uint32_t)(k.coff + lin);
  const uint32_t gprev = __shfl_up_sync(kAll, gkey, 1);
  const uint32_t heads = __ballot_sync(kAll, live && !second && (lane == 0 || gprev != gkey));
  const int nlive = min(P, n - base);
  const int myhead = 31 - __clz(heads & ((2u << p) - 1u));
  const uint32_t hmask = 1u << myhead;
  float rho = pi.w * k.norm_h3, diff_sum = 0.0f, ssum = 0.0f;  // the first lane's
  uint32_t key = 0xffffffffu, mine = 0;  // mine: the neighbours this lane takes
  float dmin = INFINITY;
  bool fed = true;
  uint32_t dense = 0;  // neighbours of a particle whose neighbourhood passes the masks
  uint32_t rem = heads;
  while (rem) {
    uint32_t batch = 0, t = rem;  // the next kScanSegs segments
    for (int q = 0; q < kScanSegs && t; ++q) {
      batch |= t & (0u - t);
      t &= t - 1u;
    }
    rem = t;
    __syncwarp();
    int seg = 0;
    uint32_t mbase = 0;
    for (uint32_t bb = batch; bb; bb &= bb - 1u, ++seg) {
      const int hl = __ffs(bb) - 1;
      const uint32_t after = heads & ~((2u << hl) - 1u);
      const int he = after ? __ffs(after) - 1 : nlive;
      const int sx = __shfl_sync(kAll, cx, hl), sy = __shfl_sync(kAll, cy, hl), sz = __shfl_sync(kAll, cz, hl);
      const SimConst& ks = kp.at(__shfl_sync(kAll, i, hl));
      const int nw = scan_segment(S, seg, hl, he, mbase, ks, sx, sy, sz, pi.x, pi.y, pi.z, pl, ctab);
      if (nw <= kScanWords) mbase += (uint32_t)(nw * ((he - hl + 3) & ~3));
      __syncwarp();
    }
    const bool in_batch = live && (batch & hmask);
    const int s = __popc(batch & (hmask - 1u));
    const int R = k.rows ? 9 : 27;
    const uint32_t total = in_batch ? S.vstart[s][R] : 0u;
    const int nw = (int)((total + 31u) / 32u);
    const bool act = in_batch && nw <= kScanWords;
    if (in_batch && !act) {
      fed = false;
      if (!second) {
        dense = record_neighbors(pi.x, pi.y, pi.z, i, pl, ctab, ScanGeo(k), nbr, n);
        for (uint32_t e = 0; e < min(dense, kNbrCap); ++e) {  // no terms here: the closest is looked for by itself
          const float4 pj = __ldg(&pos[nbr[nbr_index(e, n, i)]]);
          const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
          dmin = fminf(dmin, dx * dx + dy * dy + dz * dz);
        }
      }
    }
    __syncwarp();
    const uint32_t q4 = act ? S.mquad[s] : 0u;
    const uint32_t* words = S.mask + (act ? S.mbase[s] + (uint32_t)(p - myhead) : 0u);
    const uint32_t vself = act ? S.vstart[s][R / 2] + ((uint32_t)i - S.sstart[s][R / 2]) : 0u;
    const int wself = act ? (int)(vself >> 5) : -1;
    const uint32_t bself = ~(1u << (vself & 31u));
    int w = 0, r = 0;
    uint32_t M = act ? words[0] : 0u;
    if (wself == 0) M &= bself;
    uint32_t vnext = act ? S.vstart[s][1] : 0u;
    uint32_t off = act ? S.sstart[s][0] - S.vstart[s][0] : 0u;
    auto more = [&] {  // the next set bit's word, if any is left
      while (M == 0u && w + 1 < nw) {
        M = words[++w * q4];
        if (w == wself) M &= bself;
      }
      return M != 0u;
    };
    auto next = [&](uint32_t& slot) {
      if (!act || !more()) return false;
      const uint32_t v = (uint32_t)(w * 32 + __ffs(M) - 1);
      M &= M - 1u;
      while (v >= vnext) {
        ++r;
        vnext = S.vstart[s][r + 1];
        off = S.sstart[s][r] - S.vstart[s][r];
      }
      slot = v + off;
      ++mine;
      return true;
    };
    auto skip2 = [&] {
      if (act && more()) {
        M &= M - 1u;
        if (more()) M &= M - 1u;
      }
    };
    if (second) skip2();
    uint2* at = reinterpret_cast<uint2*>(reinterpret_cast<uint4*>(nbr) + i) + (second ? 1 : 0);
    for (uint32_t q = 0;; ++q, at += 2 * (size_t)n) {
      uint32_t sa = (uint32_t)i, sb = (uint32_t)i;
      const bool g0 = next(sa), g1 = g0 && next(sb);
      if (!__any_sync(kAll, g0)) break;
      const float4 p0 = __ldg(&pos[sa]), p1 = __ldg(&pos[sb]);
      const float2 r0 = __ldg(&rv[sa]), r1 = __ldg(&rv[sb]);
      auto term = [&](bool in, const float4& pj, const float2& rvj, float& a, float& d, float& v) {
        const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
        const float d2 = in ? dx * dx + dy * dy + dz * dz : 1.0f;
        float wt, half_diff;
        if (delta) density_fast<true>(k, pj.w, rvj, rho_old_i, dx, dy, dz, d2, key, dmin, wt, half_diff);
        else density_fast<false>(k, pj.w, rvj, rho_old_i, dx, dy, dz, d2, key, dmin, wt, half_diff);
        a = in ? pj.w * wt : 0.0f;
        d = in ? 2.0f * half_diff : 0.0f;
        v = CL && in ? rvj.y * wt : 0.0f;
      };
      float a0, a1, d0, d1, v0, v1;
      term(g0, p0, r0, a0, d0, v0);
      term(g1, p1, r1, a1, d1, v1);
      if (g0 && q < kNbrCap / 4) *at = make_uint2(sa, sb);
      const float b0 = __shfl_down_sync(kAll, a0, P), b1 = __shfl_down_sync(kAll, a1, P);
      const float e0 = __shfl_down_sync(kAll, d0, P), e1 = __shfl_down_sync(kAll, d1, P);
      rho += a0;
      rho += a1;
      rho += b0;
      rho += b1;
      diff_sum += d0;
      diff_sum += d1;
      diff_sum += e0;
      diff_sum += e1;
      if (CL) {
        const float f0 = __shfl_down_sync(kAll, v0, P), f1 = __shfl_down_sync(kAll, v1, P);
        ssum += v0;
        ssum += v1;
        ssum += f0;
        ssum += f1;
      }
      skip2();
    }
    __syncwarp();
  }
  const uint32_t listed = __shfl_sync(kAll, dense, p) + mine + __shfl_xor_sync(kAll, mine, P);
  key = min(key, __shfl_xor_sync(kAll, key, P));
  dmin = fminf(dmin, __shfl_xor_sync(kAll, dmin, P));
  const bool close = dmin < kTinyD2;
  if (live && !second && (!fed || !k.fast || close || key < k.diff_key || !finite3(rho, diff_sum, 0.0f))) {
    const DensitySum e = density_exact(kp.ref(i), i, pi, rho_old_i, pos, rv, ctab);
    rho = e.rho;
    diff_sum = e.diff;
    if (CL) ssum = e.ssum;
  }
  __syncwarp();
  // boundary terms, four candidates a round, two a lane; those in support
  // follow the neighbours in the list
  float rho_wall = 0.0f;
  uint32_t nwall = 0;
  const uint32_t q0 = live ? __ldg(&bc_start[k.coff + lin]) : 0u, q1 = live ? __ldg(&bc_start[k.coff + lin + 1]) : 0u;
  const uint32_t mine0 = min(q0 + (second ? 2u : 0u), q1);
  BoundaryWalk<2> walk(q0 < q1 ? mine0 : 0u, q0 < q1 ? q1 : 0u, bc_list, bpos, 4u);
  for (uint32_t q = q0; __any_sync(kAll, q < q1); q += 4) {
    const uint32_t qa = q + (second ? 2u : 0u);
    const bool va = qa < q1, vb = qa + 1 < q1;
    uint32_t bi[2] = {0u, 0u};
    float4 bp[2] = {make_float4(0.0f, 0.0f, 0.0f, 0.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f)};
    if (va) walk.round(qa, bi, bp);
    const uint32_t ia = bi[0], ib = bi[1];
    const float4 ba = bp[0], bb = bp[1];
    auto d2_of = [&](const float4& b) {
      const float dx = pi.x - b.x, dy = pi.y - b.y, dz = pi.z - b.z;
      return dx * dx + dy * dy + dz * dz;
    };
    const float da = d2_of(ba), db = d2_of(bb);
    const bool ina = va && da <= k.sup_d2, inb = vb && db <= k.sup_d2;
    const uint32_t ma = __ballot_sync(kAll, ina), mb = __ballot_sync(kAll, inb);
    if ((ma | mb) == 0u) continue;
    const float wa = ina ? ba.w * w_c2(sqrt_any(da), k) : 0.0f, wb = inb ? bb.w * w_c2(sqrt_any(db), k) : 0.0f;
    const float xa = __shfl_down_sync(kAll, wa, P), xb = __shfl_down_sync(kAll, wb, P);
    rho += wa;
    rho += wb;
    rho += xa;
    rho += xb;
    if (CL) {
      rho_wall += wa;
      rho_wall += wb;
      rho_wall += xa;
      rho_wall += xb;
    }
    const uint32_t first = ((ma >> p) & 1u) + ((mb >> p) & 1u);  // the first lane's
    uint32_t e = listed + nwall + (second ? first : 0u);
    if (ina && e < kNbrCap) nbr[nbr_index(e, n, i)] = ia;
    e += ina ? 1u : 0u;
    if (inb && e < kNbrCap) nbr[nbr_index(e, n, i)] = ib;
    nwall += first + ((ma >> (p + P)) & 1u) + ((mb >> (p + P)) & 1u);
  }
  const uint32_t counts = live && !second ? pack_counts(listed, nwall, close) : 0u;
  if (CL == 0 && wl.list) {
    __syncwarp();
    scatter_walls(kp, base, counts, pos, bc_start, bc_list, bpos, wl,
                  [&](int src, uint32_t e) { return nbr[nbr_index(e, n, base + src)]; });
  }
  const float centre = live ? centre_sdf<CL>(k, sdf, pi) : 0.0f;
  float probes[CL ? 12 : 1];
  if (CL)
    share_probes<2>(k, sdf, pi, second ? 1 : 0, live && k.feat_sdf && centre_feature(k, pi, centre) < k.support, centre,
                    [&](float v, int l) { return __shfl_sync(kAll, v, p + l * P); }, probes);
  float f[16];
  float rho_pre = 0.0f;
  bool near_wall = false;
  if (live && !second) {
    ncount[i] = counts;
    near_wall = density_finish<CL>(k, i, dtp[k.inst], pi, DensityState{rho, diff_sum, ssum, rho_wall, nwall, listed},
                                   rv, id, rf, pr, centre, [&](int a) { return probes[CL ? a : 0]; }, wall_tab, cb,
                                   slow, f, rho_pre);
  }
  if (CL == 2) {
    uint32_t* tile = reinterpret_cast<uint32_t*>(s_dyn + (kGroupThreads / 32) * sizeof(ScanWarp)) + warp * kClTileWords;
    network_epilogue(kp, i, near_wall, f, rho_pre, tile, id, rf, pr, cb, slow);
  }
}

// ---------------------------------------------------------------------------
// forces + kick 2 (k_forces' work)
// ---------------------------------------------------------------------------
template <int G>
struct __align__(16) ForceGroup {
  GroupTerms<6, kChunkOf<G>> terms;
  uint32_t rep[kRepCap];  // boundary candidates within the repulsion radius, in order
};

template <class KP, int CL, int G, bool MIXED>
__global__ void __launch_bounds__(kGroupThreads, kGroupBlocks)
k_forces_group(KP kp, int n, const float* __restrict__ dtp, float hdt_scale, const float4* __restrict__ pos,
               const float4* __restrict__ vel, const float2* __restrict__ rf, const float* __restrict__ pr,
               const uint32_t* __restrict__ id, const uint2* __restrict__ ctab,
               const uint32_t* __restrict__ bc_start, const uint32_t* __restrict__ bc_list,
               const float4* __restrict__ bpos, const float* __restrict__ bpress, float4* __restrict__ acc,
               float4* __restrict__ velout, float* __restrict__ red, const uint32_t* __restrict__ err,
               const uint32_t* __restrict__ nbr, const uint32_t* __restrict__ ncount,
               const float* __restrict__ sdf, const float2* __restrict__ wall_tab,
               const float4* __restrict__ corr, const uint32_t* __restrict__ slow) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int U = kRounds, CH = kChunkOf<G>;
  __shared__ ForceGroup<G> s_group[kGroupThreads / G];
  const Group<G> g;
  ForceGroup<G>& S = s_group[threadIdx.x / G];
  const int slot = (int)((blockIdx.x * kGroupThreads + threadIdx.x) / G);
  if (__all_sync(kAll, slot >= n)) return;
  const bool live = slot < n && !*err;
  const int i = live ? slot : 0;
  const SimConst& k = kp.at(i);
  const float4 pi = pos[i];
  const float4 vi = vel[i];
  const float2 rfi = rf[i];
  const float rho_i = rfi.x;
  const float neg_mi = -pi.w;
  uint32_t key = 0xffffffffu;
  float sum = 0.0f;  // lanes 0..2: the pressure force, 3..5: the viscous acceleration
  const uint32_t counts = live ? __ldg(&ncount[i]) : 0u;
  const bool listed = counts_listed(counts) && !slow[k.inst];
  const uint32_t mine = listed ? counts_neighbours(counts) : 0u;
  const uint32_t most = __reduce_max_sync(kAll, mine);
  GroupList<G> list(nbr, n, i, g.sub);
  for (uint32_t c0 = 0; c0 < most; c0 += CH) {
    float4 pj[U], vj[U];
    float2 rfj[U];
    uint32_t s[U];
#pragma unroll
    for (int u = 0; u < U; ++u) s[u] = list.next();  // in bounds; not used past the list's end
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!(c0 + u * G + g.sub < mine)) s[u] = (uint32_t)i;
      pj[u] = __ldg(&pos[s[u]]);
      vj[u] = __ldg(&vel[s[u]]);
      rfj[u] = __ldg(&rf[s[u]]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = c0 + u * G + g.sub < mine;
      const float dx = pi.x - pj[u].x, dy = pi.y - pj[u].y, dz = pi.z - pj[u].z;
      uint32_t kk = 0xffffffffu;
      float factor, fv, gx, gy, gz;
      forces_fast<MIXED>(k, neg_mi, vi, rfi, pj[u], vj[u], rfj[u], dx, dy, dz, dx * dx + dy * dy + dz * dz, kk, factor,
                         fv, gx, gy, gz);
      if (in) key = min(key, kk);
      S.terms.t[0][u * G + g.sub] = in ? factor * gx : 0.0f;
      S.terms.t[1][u * G + g.sub] = in ? factor * gy : 0.0f;
      S.terms.t[2][u * G + g.sub] = in ? factor * gz : 0.0f;
      S.terms.t[3][u * G + g.sub] = in ? fv * gx : 0.0f;
      S.terms.t[4][u * G + g.sub] = in ? fv * gy : 0.0f;
      S.terms.t[5][u * G + g.sub] = in ? fv * gz : 0.0f;
    }
    __syncwarp();
    if (c0 < mine) {
      const uint32_t m = min(mine - c0, (uint32_t)CH);
      if (g.sub < 6) sum = add_terms(S.terms, g.sub, m, sum);
    }
    __syncwarp();
  }
  const bool odd = g.bits(__ballot_sync(kAll, key < k.visc_key || !finite3(sum, 0.0f, 0.0f))) != 0u;
  if (live && (!listed || odd)) {
    const PairForce e = forces_exact(kp.ref(i), i, pi, vi, rfi, pos, vel, rf, ctab);
    sum = g.sub == 0 ? e.fp.x : g.sub == 1 ? e.fp.y : g.sub == 2 ? e.fp.z
          : g.sub == 3 ? e.fv.x : g.sub == 4 ? e.fv.y : e.fv.z;
  }
  __syncwarp();
  // wall pressure, added to the pressure force in ascending boundary index,
  // over the boundary particles in support, which the density pass listed (or,
  // past the list's capacity, over the cell's candidates); those within the
  // repulsion radius are noted on the way
  const bool walls_listed = counts_walls_listed(counts);
  uint32_t b0 = 0, b1 = 0;
  if (walls_listed) {
    b0 = counts_first_wall(counts);
    b1 = b0 + counts_walls(counts);
  } else {
    const int lin = cell_hash(axis_cell(pi.x, k.gmin[0], k.cell, k.dims[0]),
                              axis_cell(pi.y, k.gmin[1], k.cell, k.dims[1]),
                              axis_cell(pi.z, k.gmin[2], k.cell, k.dims[2]), k);
    b0 = __ldg(&bc_start[k.coff + lin]);
    b1 = __ldg(&bc_start[k.coff + lin + 1]);
  }
  auto wall = [&](uint32_t e) { return __ldg(walls_listed ? &nbr[nbr_index(e, n, i)] : &bc_list[e]); };
  const bool air = (id[i] & kAirBit) != 0;
  uint32_t nrep = 0;
  {
    const float pic = fmaxf(pr[i], 0.0f);
    const float pic_over = pic / (rho_i * rho_i);
    const float brho = air ? kAirRho0 : kWaterRho0;
    const float brho2 = brho * brho;
    uint32_t held = 0;
    auto flush = [&] {
      __syncwarp();
      if (g.sub < 4 && ((held + g.sub) & ~3u) == (held & ~3u) && (held & 3u))
        for (int c = 0; c < 3; ++c) S.terms.t[c][held + g.sub] = 0.0f;
      __syncwarp();
      if (g.sub < 3) sum = add_terms(S.terms, g.sub, held, sum);
      __syncwarp();
      held = 0;
    };
    const bool repulsion = (k.flags & kFlagRepulsion) != 0;
    group_candidates(g, b0, b1, wall, bpos, [&](bool valid, uint32_t bi, const float4& bp) {
      const float dx = pi.x - bp.x, dy = pi.y - bp.y, dz = pi.z - bp.z;
      const float d2 = dx * dx + dy * dy + dz * dz;
      const bool in = valid && d2 <= k.sup_d2;
      const uint32_t ballot = __ballot_sync(kAll, in);
      const bool near = repulsion && valid && d2 <= k.r0_d2 && d2 > k.tiny_d2;
      const uint32_t nm = g.bits(__ballot_sync(kAll, near));
      if (near) {
        const uint32_t e = nrep + __popc(nm & g.below());
        if (e < (uint32_t)kRepCap) S.rep[e] = bi;
      }
      nrep += __popc(nm);
      if (ballot == 0u) return;
      const uint32_t m = g.bits(ballot);
      if (__any_sync(kAll, held + __popc(m) > (uint32_t)CH)) flush();
      if (in) {
        const uint32_t e = held + __popc(m & g.below());
        float gx, gy, gz;
        grad_wall(dx, dy, dz, d2, k, gx, gy, gz);
        const float pb_over = __ldg(&bpress[bi]) / brho2;
        const float factor = neg_mi * bp.w * (pic_over + pb_over);
        S.terms.t[0][e] = factor * gx;
        S.terms.t[1][e] = factor * gy;
        S.terms.t[2][e] = factor * gz;
      }
      held += __popc(m);
    });
    flush();
  }
  // the lanes of the group hold the acceleration whole from here on
  float ax = 0.0f + g.get(sum, 0) / pi.w, ay = 0.0f + g.get(sum, 1) / pi.w, az = 0.0f + g.get(sum, 2) / pi.w;
  ax += g.get(sum, 3);
  ay += g.get(sum, 4);
  az += g.get(sum, 5);
  ax += k.grav[0];
  ay += k.grav[1];
  az += k.grav[2];
  if (k.sdf_mode && g.sub == 0) sdf_wall_force(k, sdf, wall_tab, pi, pr[i], rho_i, air, ax, ay, az);
  // repulsion (boundary.rs:143-181), in ascending boundary index
  {
    const uint32_t few = nrep <= (uint32_t)kRepCap ? nrep : 0u;
    const uint32_t rounds = __reduce_max_sync(kAll, few);
    for (uint32_t e0 = 0; e0 < rounds; e0 += G) {
      const uint32_t e = e0 + g.sub;
      float fx = 0.0f, fy = 0.0f, fz = 0.0f;
      if (e < few) repulsion_term(k, pi, __ldg(&bpos[S.rep[e]]), fx, fy, fz);
      S.terms.t[0][g.sub] = fx;
      S.terms.t[1][g.sub] = fy;
      S.terms.t[2][g.sub] = fz;
      __syncwarp();
      if (e0 < few) {
        ax = add_terms(S.terms, 0, G, ax);
        ay = add_terms(S.terms, 1, G, ay);
        az = add_terms(S.terms, 2, G, az);
      }
      __syncwarp();
    }
    if (nrep > (uint32_t)kRepCap)  // more than the list holds: one after the other
      for (uint32_t q = b0; q < b1; ++q) {
        const float4 bp = __ldg(&bpos[wall(q)]);
        const float dx = pi.x - bp.x, dy = pi.y - bp.y, dz = pi.z - bp.z;
        const float d2 = dx * dx + dy * dy + dz * dz;
        if (d2 <= k.r0_d2 && d2 > k.tiny_d2) {
          float fx, fy, fz;
          repulsion_term(k, pi, bp, fx, fy, fz);
          ax += fx;
          ay += fy;
          az += fz;
        }
      }
  }
  float sig = 0.0f, amag = 0.0f;
  int inst = -1;
  if (live && g.sub == 0) {
    inst = k.inst;
    forces_finish<CL>(k, i, (0.5f * dtp[k.inst]) * hdt_scale, vi, rho_i, ax, ay, az, corr, acc, velout, sig, amag);
  }
  reduce_maxima(inst, sig, amag, red);
}

}  // namespace sph
