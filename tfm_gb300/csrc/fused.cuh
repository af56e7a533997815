// Heun stages of small batches in one kernel each.
//
// A batch that does not fill the GPU is bound by the launches of a step and
// by the latency of each kernel, not by its arithmetic: scan (3), scatter,
// pair and update, twice per step, are twelve kernels of 3-12 us each (12 to
// 16 of 152 SMs busy at 2048 beads). Here a stage is one kernel, so a step is
// two: positions live in fixed-capacity cell buckets, so no counting sort is
// needed; every bead sums its own pair force over the full 27-cell stencil,
// so no force is exchanged between beads; and the same CTA integrates its
// beads and inserts their new positions into the next stage's buckets. The
// full stencil costs two to three times the pair tests of the sorted half
// stencil, which is what ends the range of this path.
//
// Measured on a GB300, us per Heun step, sorted path / this one (single
// systems at packing fraction 0.08, ccp, and 0.2, baseline):
//   beads          1024         2048         8192         24000        40000
//   ccp        35.3 /  8.9  38.7 / 10.8  41.6 / 17.9  48.2 / 28.6  52.8 / 42.1
//   baseline   43.0 / 12.9  42.0 / 13.5  45.9 / 31.4  58.4 / 59.9  62.1 / 75.4
//
// Buckets. Every system has a grid of cells of side the largest pair cutoff.
// A cell holds up to FUSED_CAP (x, y, z, index << 3 | flags) slots; beads
// beyond that go to an overflow list that every bead scans (empty unless the
// density is several times that of a relaxed system). There are two sets of
// slots (positions and predictor) and three of counts: the kernel that reads
// set k fills set k + 1 and clears set k + 2.
//
// CTA: 8 warps of pair lanes (L = S G lanes a bead, 256 / L beads), which also
// take the lamina sites, and two threads a bead that meanwhile compute its
// bonded and wall forces and its noise (one thread a bead for all of these,
// sites included, took 12.9 instead of 9.5 us a step at 1024 ccp beads then: its
// serial chain was longer than the pair loop).
#pragma once

#include "kernels.cuh"

namespace ccpgpu {

constexpr int FUSED_SLOTS = 32;         // a cell's slots in memory
// ... of which it fills 31: a cell of the sort, which is no wider than a bucket,
// meets at most eight buckets, so one that holds more than the 255 beads the sort
// can count leaves some in the overflow list, where the bead's CTA looks for that.
constexpr int FUSED_CAP = 31;
static_assert(8 * FUSED_CAP <= 255, "an over-full cell of the sort shows as overflow");
constexpr int FUSED_PAIR_THREADS = 256;
// pair lanes, then a thread per bead for the other forces and one for the noise
// (whole warps)
__host__ __device__ constexpr int fused_own(int lanes) { return lanes > 8 ? 32 : FUSED_PAIR_THREADS / lanes; }
__host__ __device__ constexpr int fused_threads(int lanes) { return FUSED_PAIR_THREADS + 2 * fused_own(lanes); }

struct FusedGrid {  // one system's bucket grid, with a border of empty cells
  int32_t cell_off, cps;  // cps: cells per side, border included
  float inv_csl;
  int32_t pad;
};

struct FusedArgs {
  const Tile *tiles;  // 256 / L beads each
  const SysDesc *sys;
  const FusedGrid *grid;
  float4 *pos, *er, *fbuf, *rnb;
  float *force;  // STAGE 0
  const float4 *slots_in;
  float4 *slots_out;
  const uint32_t *cnt_in;  // per cell; [n_cells]: length of the overflow list
  uint32_t *cnt_out, *cnt_zero;
  const float4 *ovf_in;
  float4 *ovf_out;
  const float4 *lbs;
  const uint32_t *lbs_start;
  unsigned long long *step;
  int *err;
  int n_cells;
};

__device__ __forceinline__ int fused_cell(float4 p, const FusedGrid &g, bool &esc) {
  const int n = g.cps - 2;
  const int x = cell_coord(p.x, g.inv_csl, n, esc), y = cell_coord(p.y, g.inv_csl, n, esc),
            z = cell_coord(p.z, g.inv_csl, n, esc);
  return g.cell_off + ((z + 1) * g.cps + y + 1) * g.cps + x + 1;
}

// Inserts bead i at p (flags in w) into its cell's bucket. A bead has escaped
// where the sort would clamp it: outside the system's sort grid.
__device__ __forceinline__ void fused_insert(float4 p, int i, const SysDesc &s, const FusedGrid &g,
                                             uint32_t *cnt, float4 *slots, float4 *ovf, int n_cells,
                                             int *err) {
  bool esc = false, clamped = false;
  const int c = fused_cell(p, g, clamped);
  cell_of(p, s, esc);
  if (esc) set_err(err, ERR_ESCAPE);
  const float4 q = make_float4(p.x, p.y, p.z,
                               __uint_as_float(((uint32_t)i << BF_BITS) | (wbits(p) & 7u)));
  const uint32_t r = atomicAdd(&cnt[c], 1u);
  if (r < (uint32_t)FUSED_CAP)
    slots[(size_t)c * FUSED_SLOTS + r] = q;
  else
    ovf[atomicAdd(&cnt[n_cells], 1u)] = q;
}

// Buckets of the current positions (counts cleared by the host).
__global__ void k_fused_build(const Tile *__restrict__ tiles, const SysDesc *__restrict__ sys,
                              const FusedGrid *__restrict__ grid, int tile,
                              const float4 *__restrict__ pos, uint32_t *cnt, float4 *slots,
                              float4 *ovf, int n_cells, int *err) {
  const Tile t = tiles[blockIdx.x];
  const SysDesc &s = sys[t.sys];
  const int i = t.begin + threadIdx.x;
  if ((int)threadIdx.x >= tile || i >= s.bead_off + s.n) return;
  fused_insert(pos[i], i, s, grid[t.sys], cnt, slots, ovf, n_cells, err);
}

// Slots of a cell that the lanes of a bead read together; the beads beyond them
// take a loop of their own. Cells hold 2-3 beads in ccp's field (side 2), 6 in
// the baseline (2.5).
__host__ __device__ constexpr int fused_read(int pot) { return pot == POT_WF ? 4 : 8; }

// Number of beads in cells that hold more than `most`, added to *sum.
__global__ void __launch_bounds__(256)
    k_fused_crowd(const uint32_t *__restrict__ cnt, int n_cells, uint32_t most,
                  unsigned int *__restrict__ sum) {
  unsigned int s = 0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n_cells; c += gridDim.x * blockDim.x)
    s += cnt[c] > most ? cnt[c] : 0u;
  s = __reduce_add_sync(0xffffffffu, s);
  if ((threadIdx.x & 31u) == 0u && s) atomicAdd(sum, s);
}

// Whether the pair of the bead at p (word wi, `near` = (index - 1) << 3) and
// the candidate q is within its class's cutoff and not |i - j| <= 1.
__device__ __forceinline__ bool fused_hit(float4 p, uint32_t wi, uint32_t near, float4 q,
                                          float rc2_att, float rc2_rep) {
  const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
  const float d2 = pair_d2(dx, dy, dz);
  const uint32_t wj = wbits(q);
  return d2 <= ((wi & wj & BF_HET) ? rc2_att : rc2_rep) && wj - near >= (3u << BF_BITS);
}

// A bead's force terms, summed so that the order of the slots, which differs
// from run to run, hardly shows: each term is split at 2^-10 (adding and
// subtracting 1.5 * 2^13), the upper parts add up without rounding while the
// sum is below 2^12, and the rounding of the lower ones is 2^-20 of what
// plain sums leave. Two runs of one system of 2048 ccp beads give the same
// positions over 3000 steps (20 pairs of runs); with plain sums they were up to
// 1.1e-2 apart. 1024 beads 9.65 -> 9.79 us a step, 30386 beads 27.3 -> 27.6.
struct ForceSum {
  float3 hi = make_float3(0.0f, 0.0f, 0.0f), lo = make_float3(0.0f, 0.0f, 0.0f);
  static __device__ __forceinline__ void split_add(float t, float &h, float &l) {
    const float u = __fsub_rn(__fadd_rn(t, 12288.0f), 12288.0f);
    h = __fadd_rn(h, u);
    l = __fadd_rn(l, __fsub_rn(t, u));
  }
  __device__ __forceinline__ void add(float x, float y, float z) {
    split_add(x, hi.x, lo.x);
    split_add(y, hi.y, lo.y);
    split_add(z, hi.z, lo.z);
  }
};

// Adds the pair's force on the bead at p; HH: both are A beads.
template <int POT, bool HH>
__device__ __forceinline__ void fused_add(float4 p, float4 q, const ForceField &ff, ForceSum &acc) {
  const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
  const float d2 = pair_d2(dx, dy, dz);
  const float cf = POT == POT_WF ? wf_coef(ff.e_att, d2)
                                 : lj_coef<!HH>(HH ? ff.e_att : ff.e_rep, dx, dy, dz, d2);
  acc.add(cf * dx, cf * dy, cf * dz);
}

template <int POT>
__device__ __forceinline__ void fused_test_add(float4 p, uint32_t wi, uint32_t near, float4 q,
                                               float rc2_att, float rc2_rep, const ForceField &ff,
                                               ForceSum &acc) {
  if (!fused_hit(p, wi, near, q, rc2_att, rc2_rep)) return;
  if (POT == POT_LJ && !(wi & wbits(q) & BF_HET))
    fused_add<POT, false>(p, q, ff, acc);
  else
    fused_add<POT, true>(p, q, ff, acc);
}

// Warp mask of the L lanes that share the calling lane's bead.
template <int L>
__device__ __forceinline__ uint32_t fused_lanes() {
  const uint32_t lane = threadIdx.x & 31u;
  return (uint32_t)(((1ull << L) - 1ull) << (lane & ~(uint32_t)(L - 1)));
}

// Offset of cell `it` (0 .. 26) of the stencil from its centre.
__device__ __forceinline__ int fused_offset(int it, int cps) {
  const int dz = it / 9, r = it - 9 * dz, dy = r / 3, dx = r - 3 * dy;
  return ((dz - 1) * cps + dy - 1) * cps + dx - 1;
}

// Lamina-binding force on a LAD bead (lbs_force) from the (z, y) rows of cells
// first, first + stride, ...: the bead's pair lanes take a row each.
__device__ __forceinline__ float3 fused_lbs(float4 x, const SysDesc &s, const ForceField &ff,
                                            const float4 *__restrict__ lbs,
                                            const uint32_t *__restrict__ lbs_start, int first,
                                            int stride) {
  float3 f = make_float3(0.0f, 0.0f, 0.0f);
  float d2 = x.x * x.x + x.y * x.y + x.z * x.z;
  float m = ff.lco * 1.001f + 1e-4f;
  float lo = fmaxf(s.lbs_rmin - m, 0.0f), hi = s.lbs_rmax + m;
  if (d2 < lo * lo || d2 > hi * hi) return f;  // no site within reach
  bool esc = false;
  int xl = cell_coord(x.x - m, s.inv_csl, s.cps, esc), xh = cell_coord(x.x + m, s.inv_csl, s.cps, esc);
  int yl = cell_coord(x.y - m, s.inv_csl, s.cps, esc), yh = cell_coord(x.y + m, s.inv_csl, s.cps, esc);
  int zl = cell_coord(x.z - m, s.inv_csl, s.cps, esc), zh = cell_coord(x.z + m, s.inv_csl, s.cps, esc);
  const float cl = ff.e_l * (8.0f / (3.0f * ff.lco * ff.lco));
  const float l2h = __fmul_rn(ff.lco, ff.lco), l2l = __fmaf_rn(ff.lco, ff.lco, -l2h);
  const int ny = yh - yl + 1, rows = ny * (zh - zl + 1);
  for (int r = first; r < rows; r += stride) {
    const int z = zl + r / ny, y = yl + r % ny;
    int row = s.cell_off + (z * s.cps + y) * s.cps;
    uint32_t b = lbs_start[row + xl], e = lbs_start[row + xh + 1];
    for (uint32_t k = b; k < e; ++k) {
      float4 q = lbs[k];
      float vx = x.x - q.x, vy = x.y - q.y, vz = x.z - q.z;
      // (d/lco)^6 - 1 = (n2 - 1)(n2^2 + n2 + 1) with n2 - 1 = (d^2 - lco^2) / lco^2:
      // no cancellation as d -> lco, where the force goes to zero
      float dd = sq3_minus(vx, vy, vz, l2h, l2l);
      if (dd > 0.0f) continue;  // beyond the cutoff
      float m1 = dd / l2h;
      float n2 = 1.0f + m1;
      float cf = cl * m1 * (n2 * n2 + n2 + 1.0f);
      f.x += cf * vx;
      f.y += cf * vy;
      f.z += cf * vz;
    }
  }
  return f;
}

// One Heun stage (see k_update): STAGE 1 reads pos and writes er, STAGE 2
// reads er and writes pos. STAGE 0 writes the total force at pos (k_total_force)
// as packed xyz triples: forces of 2048 ccp beads take this kernel and the
// filling of the buckets, 12 us on the device, instead of the sort's four kernels,
// the pair pass, the total and the packing, 33 us. S lanes read the first S slots of a cell together
// and G cells are read at once by the S G lanes of a bead. Every lane notes
// its hits in a bit mask (one bit per cell visited) and evaluates them
// afterwards: few candidates are within the cutoff, and evaluated in place
// nearly every visit would run the coefficient for one or two lanes of 32.
template <int STAGE, int POT, int S, int G, int MINB>
__global__ void __launch_bounds__(fused_threads(S * G), MINB)
    k_fused(const __grid_constant__ FusedArgs a, const __grid_constant__ ForceField ff) {
  constexpr int L = S * G, B = FUSED_PAIR_THREADS / L;
  constexpr int NV = (27 + G - 1) / G;
  constexpr int OWN = fused_own(L), THREADS = fused_threads(L);
  __shared__ float4 fpair[B], fnoise[B];
  __shared__ int off[32];
  const Tile t = a.tiles[blockIdx.x];
  const SysDesc &s = a.sys[t.sys];
  const FusedGrid g = a.grid[t.sys];
  const int end = s.bead_off + s.n;
  if (threadIdx.x < 32) off[threadIdx.x] = fused_offset(threadIdx.x, g.cps);
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  const float4 *X = (STAGE == 2) ? a.er : a.pos;
  if (STAGE != 0)
    for (int c = blockIdx.x * THREADS + threadIdx.x; c <= a.n_cells; c += gridDim.x * THREADS)
      a.cnt_zero[c] = 0u;

  float4 xi, r0, f1;
  float3 F;
  const int bo = (int)threadIdx.x - FUSED_PAIR_THREADS;  // bead of the own-force threads
  const int io = t.begin + bo;
  const bool mine = bo >= 0 && bo < B && io < end;
  if (bo < 0) {
    const int sub = threadIdx.x % L, b = threadIdx.x / L;
    const int ss = sub % S, gs = sub / S;
    const int i = t.begin + b;
    const bool valid = i < end;
    ForceSum acc;
    const uint32_t n_ovf = a.cnt_in[a.n_cells];
    const float4 p = X[valid ? i : t.begin];
    const uint32_t wi = wbits(p), near = (uint32_t)(i - 1) << BF_BITS;
    bool esc = false;
    const int c0 = fused_cell(p, g, esc);
    const float rc2_att = ff.rc_att * ff.rc_att, rc2_rep = ff.rc_rep * ff.rc_rep;
    const uint32_t *cnt = a.cnt_in + c0;
    const float4 *slots = a.slots_in + (size_t)c0 * FUSED_SLOTS + ss;
    // one bit per cell visited: hits of A-A pairs, of other pairs, cells with
    // more than S beads
    uint32_t hit_a = 0, hit_x = 0, over = 0;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int it = v * G + gs;
      const int o = G == 1 ? fused_offset(v, g.cps) : off[it];
      if (G == 1 || 27 % G == 0 || it < 27) {
        // the slot is read without waiting for the count (a slot beyond it
        // holds an old position and is not a hit)
        const uint32_t n = cnt[o];
        const float4 q = slots[(ptrdiff_t)o * FUSED_SLOTS];
        if ((uint32_t)ss < n && fused_hit(p, wi, near, q, rc2_att, rc2_rep)) {
          if (POT == POT_LJ && !(wi & wbits(q) & BF_HET))
            hit_x |= 1u << v;
          else
            hit_a |= 1u << v;
        }
        if (n > (uint32_t)S) over |= 1u << v;
      }
    }
    if (!valid) hit_a = hit_x = over = 0;
    while (__any_sync(0xffffffffu, hit_a != 0u)) {
      if (hit_a) {
        const int o = off[(__ffs(hit_a) - 1) * G + gs];
        hit_a &= hit_a - 1u;
        fused_add<POT, true>(p, slots[(ptrdiff_t)o * FUSED_SLOTS], ff, acc);
      }
    }
    if (POT == POT_LJ) {
      while (__any_sync(0xffffffffu, hit_x != 0u)) {
        if (hit_x) {
          const int o = off[(__ffs(hit_x) - 1) * G + gs];
          hit_x &= hit_x - 1u;
          fused_add<POT, false>(p, slots[(ptrdiff_t)o * FUSED_SLOTS], ff, acc);
        }
      }
    }
    while (over) {  // cells with more than S beads
      const int o = off[(__ffs(over) - 1) * G + gs];
      over &= over - 1u;
      const uint32_t n = min(cnt[o], (uint32_t)FUSED_CAP);
      for (uint32_t k = S + ss; k < n; k += S)
        fused_test_add<POT>(p, wi, near, slots[(ptrdiff_t)o * FUSED_SLOTS + (k - ss)], rc2_att, rc2_rep,
                            ff, acc);
    }
    if (n_ovf && valid) {
      uint32_t mates = 0;
      for (uint32_t k = sub; k < n_ovf; k += L) {
        const float4 q = a.ovf_in[k];
        const int gj = (int)(wbits(q) >> BF_BITS);
        if (gj >= s.bead_off && gj < end) {
          fused_test_add<POT>(p, wi, near, q, rc2_att, rc2_rep, ff, acc);
          mates += bead_cell(q, s, esc) == bead_cell(p, s, esc);
        }
      }
      // more beads in the bead's cell of the sort than its byte counts hold
      // (cell_add): the state is refused here too
      for (int it = 0; it < 27; ++it) {
        const uint32_t n = min(cnt[off[it]], (uint32_t)FUSED_CAP);
        for (uint32_t k = sub; k < n; k += L)
          mates += bead_cell(slots[(ptrdiff_t)off[it] * FUSED_SLOTS + k - ss], s, esc) == bead_cell(p, s, esc);
      }
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1)
        mates += __shfl_xor_sync(fused_lanes<L>(), mates, o);
      if (mates > 255u) set_err(a.err, ERR_SLOT);
    }
    if ((wi & BF_LAD) && valid && s.n_lbs > 0) {
      const float3 fl3 = fused_lbs(p, s, ff, a.lbs, a.lbs_start, sub, L);
      acc.add(fl3.x, fl3.y, fl3.z);
    }
    __syncwarp();
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
      acc.hi.x += __shfl_xor_sync(0xffffffffu, acc.hi.x, o);
      acc.hi.y += __shfl_xor_sync(0xffffffffu, acc.hi.y, o);
      acc.hi.z += __shfl_xor_sync(0xffffffffu, acc.hi.z, o);
      acc.lo.x += __shfl_xor_sync(0xffffffffu, acc.lo.x, o);
      acc.lo.y += __shfl_xor_sync(0xffffffffu, acc.lo.y, o);
      acc.lo.z += __shfl_xor_sync(0xffffffffu, acc.lo.z, o);
    }
    if (sub == 0)
      fpair[b] = make_float4(acc.hi.x + acc.lo.x, acc.hi.y + acc.lo.y, acc.hi.z + acc.lo.z, 0.0f);
  } else if (bo >= OWN) {
    // the noise warp: stage 1 draws, stage 2 takes what stage 1 drew
    const int in = io - OWN;
    if (STAGE != 0 && bo - OWN < B && in < end) {
      float3 z = make_float3(0.0f, 0.0f, 0.0f);
      if (ff.sd > 0.0f) {
        if (STAGE == 1) {
          // the counter holds the last step taken; the second stage advances it
          z = bead_noise((uint32_t)(in - s.bead_off), *a.step + 1ull, s.seed_lo, s.seed_hi, a.err);
          z = make_float3(ff.sd * z.x, ff.sd * z.y, ff.sd * z.z);
          a.rnb[in] = make_float4(z.x, z.y, z.z, 0.0f);
        } else {
          const float4 r4 = a.rnb[in];
          z = make_float3(r4.x, r4.y, r4.z);
        }
      }
      fnoise[bo - OWN] = make_float4(z.x, z.y, z.z, 0.0f);
    }
  } else if (mine) {
    // the neighbours are read at once: their flags decide what is used
    xi = X[io];
    float4 nb[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      nb[k] = X[min(max(io + (k < 2 ? k - 2 : k - 1), s.bead_off), end - 1)];
    if (STAGE == 2) {
      r0 = a.pos[io];
      f1 = a.fbuf[io];
    }
    F = bonded_force_at([&](int j) { return j < io ? nb[j - io + 2] : nb[j - io + 1]; }, io, xi, end,
                        ff);
    add_wall<MODE_DST>(xi, s, ff, F);
  }
  __syncthreads();
  if (!mine) return;
  const float4 fp = fpair[bo];
  F.x += fp.x;
  F.y += fp.y;
  F.z += fp.z;
  if (STAGE == 0) {
    float *f = a.force + 3 * (size_t)io;
    f[0] = F.x;
    f[1] = F.y;
    f[2] = F.z;
    return;
  }
  const float4 rn = fnoise[bo];
  float4 out;
  if (STAGE == 1) {
    float3 D = make_float3(F.x * ff.dt, F.y * ff.dt, F.z * ff.dt);
    cap_step(D, ff.max_step);
    out = make_float4(xi.x + D.x + rn.x, xi.y + D.y + rn.y, xi.z + D.z + rn.z, xi.w);
    a.er[io] = out;
    a.fbuf[io] = make_float4(F.x, F.y, F.z, 0.0f);
  } else {
    const float h = 0.5f * ff.dt;
    float3 D = make_float3((f1.x + F.x) * h, (f1.y + F.y) * h, (f1.z + F.z) * h);
    cap_step(D, ff.max_step);
    out = make_float4(r0.x + D.x + rn.x, r0.y + D.y + rn.y, r0.z + D.z + rn.z, r0.w);
    a.pos[io] = out;
    if (blockIdx.x == 0 && bo == 0) *a.step += 1ull;
  }
  if (!(isfinite(out.x) && isfinite(out.y) && isfinite(out.z))) {
    // within no bead's cutoff, so left out: a state that is lost as a whole
    // would otherwise fill the overflow list
    set_err(a.err, ERR_NAN);
    set_err(a.err, ERR_ESCAPE);
    return;
  }
  fused_insert(out, io, s, g, a.cnt_out, a.slots_out, a.ovf_out, a.n_cells, a.err);
}

}  // namespace ccpgpu
