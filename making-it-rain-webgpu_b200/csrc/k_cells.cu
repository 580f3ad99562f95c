// k_cells.cu -- folding positions into the cell, the deterministic spatial
// sort, and the cluster-pair tile list with its interaction masks.
//
// Replaces the reference's wrap + counting-sort cell list + sort_cells
// (src/gpu/kernels/cell-list.wgsl:140-331) and its three-pass Verlet list
// (nonbonded-pairs.wgsl:412-497) with a B200-shaped design:
//   * atoms are sorted along a Hilbert curve of ~0.25 nm fractional cells, so 32
//     consecutive slots form a compact cluster (a "block");
//   * the list holds block pairs (tiles) whose bounding boxes come within
//     cutoff + skin, plus one 32-bit interaction mask per tile row that removes
//     exclusions, padding and the lower triangle of diagonal tiles;
//   * the order inside a cell is ascending atom index, written by rank rather
//     than by atomics, so two runs hold the same tiles (their rows in any
//     order, which the pair kernel's sums do not depend on).
// A rebuild happens only when the integrator saw an atom move more than skin/2
// (verlet.wgsl:57), decided on the device; every phase kernel returns at once
// when no system asked for one.
#include <algorithm>

#include "device_state.h"

namespace mdb {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ int grid_stride_start() { return blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ int grid_stride() { return gridDim.x * blockDim.x; }

// Fractional coordinates of a 2^32 fixed-point position, exactly, and the
// position folded into the cell (fixed64.wgsl:335 does the same with f32
// estimates and a bounded loop; here the lattice count is exact).
struct Folded {
  long long x, y, z;           // folded position, 2^32 fixed
  unsigned int fa, fb, fc;     // fractional parts, 2^-32 units
  long long na, nb, nc;        // lattice translation taken off
};

__device__ __forceinline__ Folded fold(const SysDev& S, long long x, long long y, long long z) {
  const long long fa = fixed_mul(x, S.inv_fx[0]) + fixed_mul(y, S.inv_fx[3]) + fixed_mul(z, S.inv_fx[6]);
  const long long fb = fixed_mul(y, S.inv_fx[4]) + fixed_mul(z, S.inv_fx[7]);
  const long long fc = fixed_mul(z, S.inv_fx[8]);
  const long long na = fa >> 32, nb = fb >> 32, nc = fc >> 32;
  Folded f;
  f.x = x - na * S.box_fx[0] - nb * S.box_fx[3] - nc * S.box_fx[6];
  f.y = y - nb * S.box_fx[4] - nc * S.box_fx[7];
  f.z = z - nc * S.box_fx[8];
  f.fa = static_cast<unsigned int>(fa & 0xffffffffll);
  f.fb = static_cast<unsigned int>(fb & 0xffffffffll);
  f.fc = static_cast<unsigned int>(fc & 0xffffffffll);
  f.na = na;
  f.nb = nb;
  f.nc = nc;
  return f;
}

__device__ __forceinline__ int cell_index(unsigned int frac, int dim) {
  const int c = static_cast<int>((static_cast<unsigned long long>(frac) * static_cast<unsigned>(dim)) >> 32);
  return c < dim ? c : dim - 1;
}

// ---------------------------------------------------------------- phases --

// A rebuild is a chain of phases with a grid barrier (or a launch) between
// them, so their number counts as much as their work: counters are cleared by
// the phase that last reads them, an atom's place in its cell comes with the
// count, everything written by slot is written where the slot is decided, and
// a row is searched, pruned and written by one pass:
//   cells assigned | scan | scatter | slots placed | boxes | rows | exclusions
//
// Every system about to be pruned only (no rebuild) gets its references here
// too: its atoms' positions, its clusters' boxes at the pair coordinates the
// integrator wrote, and an empty inner list.
__device__ void phase_prune_references(const Dev& d) {
  if (blockIdx.x == 0)
    for (int s = threadIdx.x; s < d.S; s += blockDim.x)
      if (d.prune_now[s] && !d.rebuild_now[s]) d.in_count[s] = 0;
  // Lanes of a warp hold 32 consecutive slots (n_slots is a multiple of 32),
  // one system's, so the branch below is warp-uniform.
  for (int gs = grid_stride_start(); gs < d.n_slots; gs += grid_stride()) {
    const int s = d.slot_sys[gs];
    if (!d.prune_now[s] || d.rebuild_now[s]) continue;
    const int a = d.order[gs];
    const float inv = d.sys[s].pc_inv;
    float lo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, hi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
    if (a >= 0) {
      d.prx[a] = d.px[a];
      d.pry[a] = d.py[a];
      d.prz[a] = d.pz[a];
      const int4 p = d.pc[gs];
      lo[0] = hi[0] = p.x * inv;
      lo[1] = hi[1] = p.y * inv;
      lo[2] = hi[2] = p.z * inv;
    }
    const int C = d.cluster;
    for (int o = C / 2; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o, C));
        hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o, C));
      }
    if ((gs & (C - 1)) == 0) {
      d.cb_lo[gs / C] = make_float4(lo[0], lo[1], lo[2], 0.f);
      d.cb_hi[gs / C] = make_float4(hi[0], hi[1], hi[2], 0.f);
    }
  }
}

// Each atom's cell and its arrival number there; the cells' counts and the
// counts of each chunk of kCellChunk consecutive cells.
__device__ void phase_cells_assign(const Dev& d) {
  const int lane = threadIdx.x & 31;
  for (int a0 = grid_stride_start() - lane; a0 < d.n_atoms; a0 += grid_stride()) {
    const int a = a0 + lane, s = a < d.n_atoms ? d.atom_sys[a] : 0;
    int chunk = -1;
    if (a < d.n_atoms && d.rebuild_now[s]) {
      const SysDev& S = d.sys[s];
      const Folded f = fold(S, d.px[a], d.py[a], d.pz[a]);
      const int cx = cell_index(f.fa, S.cdim[0]), cy = cell_index(f.fb, S.cdim[1]),
                cz = cell_index(f.fc, S.cdim[2]);
      const int local = d.cell_map[S.cell_off + (cx * S.cdim[1] + cy) * S.cdim[2] + cz];
      const int gc = S.cell_off + local;
      d.cell_of[a] = gc;
      d.cell_arrival[a] = atomicAdd(&d.cell_cnt[gc], 1);
      chunk = S.chunk_off + local / kCellChunk;
    }
    // neighbours in index are neighbours in space: one atomic for the lanes of
    // a chunk (one each took 96 us over the ensemble's 627k atoms, on 1,300 words)
    const unsigned int same = __match_any_sync(0xffffffffu, chunk);
    if (chunk >= 0 && lane == __ffs(same) - 1) atomicAdd(&d.chunk_cnt[chunk], __popc(same));
  }
}

// The cells' starts: a block to a chunk, from the sum of the chunks before it
// (a block to a system took 106 us over the 64,000 cells of a 100k-atom box).
__device__ void phase_cells_scan(const Dev& d) {
  static_assert(kCellChunk == 2 * kThreads, "two cells a thread");
  __shared__ int part[kThreads / 32], before[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int ch = blockIdx.x; ch < d.n_chunks; ch += gridDim.x) {
    const int s = d.chunk_sys[ch];
    if (!d.rebuild_now[s]) continue;
    const SysDev& S = d.sys[s];
    const int c = ch - S.chunk_off, first = c * kCellChunk + 2 * threadIdx.x;
    int sum = 0;
    for (int i = threadIdx.x; i < c; i += kThreads) sum += d.chunk_cnt[S.chunk_off + i];
    const int v0 = first < S.n_cells ? d.cell_cnt[S.cell_off + first] : 0;
    const int v1 = first + 1 < S.n_cells ? d.cell_cnt[S.cell_off + first + 1] : 0;
    int x = v0 + v1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 31) part[warp] = x;
    if (lane == 0) before[warp] = sum;
    __syncthreads();
    int start = x - v0 - v1;
    for (int w = 0; w < kThreads / 32; ++w) start += before[w] + (w < warp ? part[w] : 0);
    if (first < S.n_cells) d.cell_start[S.cell_off + first] = start;
    if (first + 1 < S.n_cells) d.cell_start[S.cell_off + first + 1] = start + v0;
    __syncthreads();  // the shared words are free for the next chunk
  }
}

__device__ void phase_cells_scatter(const Dev& d) {
  for (int a = grid_stride_start(); a < d.n_atoms; a += grid_stride()) {
    const int s = d.atom_sys[a];
    if (!d.rebuild_now[s]) continue;
    d.tmp_order[d.sys[s].slot_off + d.cell_start[d.cell_of[a]] + d.cell_arrival[a]] = a;
  }
}

// Ascending atom index inside each cell, by rank: the order is a function of
// the positions alone, whatever order the counts' atomics landed in
// (cell-list.wgsl:319 sort_cells).  With its slot an atom gets everything kept
// by slot: pair coordinates as int32 at 2^pc_shift per nm under the lattice
// translation that folds it into the cell now (cell-list.wgsl:140 `wrap`;
// three signed 10-bit counts, applied until the next rebuild, so the
// coordinates move continuously and the tiles' lattice shifts stay valid),
// parameters, and the positions the displacement tests measure against.
__device__ void phase_place(const Dev& d) {
  for (int gs = grid_stride_start(); gs < d.n_slots; gs += grid_stride()) {
    const int s = d.slot_sys[gs];
    if (!d.rebuild_now[s]) continue;
    const SysDev& S = d.sys[s];
    if (gs - S.slot_off >= S.n_atoms) {
      d.order[gs] = -1;
      d.pc[gs] = make_int4(0, 0, 0, 0);
      d.prm[gs] = make_float4(0.f, 0.f, 0.f, 0.f);
      continue;
    }
    const int a = d.tmp_order[gs];
    const int gc = d.cell_of[a];
    const long long x = d.px[a], y = d.py[a], z = d.pz[a];
    const float4 prm = d.prm_atom[a];
    const int st = d.cell_start[gc], cnt = d.cell_cnt[gc];
    int r = st;
    for (int k = 0; k < cnt; ++k) r += d.tmp_order[S.slot_off + st + k] < a;
    const int to = S.slot_off + r;
    const Folded f = fold(S, x, y, z);
    d.order[to] = a;
    d.rank[a] = r;
    d.islot[d.entry[a]] = to;
    d.fold[to] = int((f.na & 1023) | ((f.nb & 1023) << 10) | ((f.nc & 1023) << 20));
    d.pc[to] = pair_coordinate(S, x, y, z, f.na, f.nb, f.nc);
    d.prm[to] = prm;
    d.refx[a] = x;
    d.refy[a] = y;
    d.refz[a] = z;
    if (d.inner) {
      d.prx[a] = x;
      d.pry[a] = y;
      d.prz[a] = z;
    }
  }
}

// A group of C lanes per cluster (32/C clusters per warp): the cluster's
// bounding box and its super-cluster's.  Every lane takes part in every
// shuffle; only the writes depend on whether the cluster's system rebuilds.
// The sort's counters are cleared for the next rebuild, the lists emptied.
template <int C>
__device__ void phase_boxes(const Dev& d) {
  constexpr int G = 32 / C;
  const int lane = threadIdx.x & 31, g = lane / C, l = lane & (C - 1);
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int c = grid_stride_start(); c < d.n_cells; c += grid_stride())
    if (d.rebuild_now[d.cell_sys[c]]) d.cell_cnt[c] = 0;
  for (int c = grid_stride_start(); c < d.n_chunks; c += grid_stride())
    if (d.rebuild_now[d.chunk_sys[c]]) d.chunk_cnt[c] = 0;
  if (blockIdx.x == 0)
    for (int s = threadIdx.x; s < d.S; s += blockDim.x)
      if (d.rebuild_now[s]) {
        d.tile_need[s] = 0;
        if (d.inner) d.in_count[s] = 0;
      }
  for (int wb = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; wb * G < d.n_blocks; wb += warps) {
    const int b = wb * G + g;
    const bool valid = b < d.n_blocks;
    const int s = valid ? d.block_sys[b] : 0;
    const bool work = valid && d.rebuild_now[s];
    const float inv = d.sys[s].pc_inv;
    const int gs = b * C + l;
    float lo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, hi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
    if (work && d.order[gs] >= 0) {
      const int4 p = d.pc[gs];
      lo[0] = hi[0] = p.x * inv;
      lo[1] = hi[1] = p.y * inv;
      lo[2] = hi[2] = p.z * inv;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int o = C / 2; o > 0; o >>= 1) {
        lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o, C));
        hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o, C));
      }
    if (work && l == 0) {
      const float4 low = make_float4(lo[0], lo[1], lo[2], 0.f), high = make_float4(hi[0], hi[1], hi[2], 0.f);
      d.bb_lo[b] = low;
      d.bb_hi[b] = high;
      if (d.inner) {
        d.cb_lo[b] = low;
        d.cb_hi[b] = high;
      }
    }
    if (C < 32) {
      // the warp's 32/C clusters form one super-cluster (a system's clusters
      // start at a multiple of 32 slots, so it never straddles two systems)
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int o = C; o < 32; o <<= 1) {
          lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
          hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
      if (work && lane == 0) {
        d.sb_lo[wb] = make_float4(lo[0], lo[1], lo[2], 0.f);
        d.sb_hi[wb] = make_float4(hi[0], hi[1], hi[2], 0.f);
      }
    }
  }
}

// What the box tests of a row need of its system, in registers.
struct Cell {
  float b0, b3, b4, b6, b7, b8;  // the lattice, reduced form
  float i0, i4, i8;              // reciprocals of its diagonal
  float list2;
  float one_image2;  // see S.one_image2
};
__device__ __forceinline__ Cell cell_of_system(const SysDev& S) {
  return Cell{S.box_f[0], S.box_f[3], S.box_f[4], S.box_f[6], S.box_f[7], S.box_f[8],
              S.inv_f[0], S.inv_f[4], S.inv_f[8], S.list2, S.one_image2};
}

// Centre separation and half-extents of two boxes, the separation reduced
// sequentially against c, b, a (src/reference/forces/nonbonded.ts:241); the
// counts taken off come back in n.
struct BoxPair {
  float dx, dy, dz, hx, hy, hz;
};
__device__ __forceinline__ BoxPair box_pair(const Cell& B, float4 li, float4 hi_, float4 lj, float4 hj, float* n) {
  BoxPair p;
  p.hx = 0.5f * (hi_.x - li.x) + 0.5f * (hj.x - lj.x);
  p.hy = 0.5f * (hi_.y - li.y) + 0.5f * (hj.y - lj.y);
  p.hz = 0.5f * (hi_.z - li.z) + 0.5f * (hj.z - lj.z);
  p.dx = 0.5f * (lj.x + hj.x) - 0.5f * (li.x + hi_.x);
  p.dy = 0.5f * (lj.y + hj.y) - 0.5f * (li.y + hi_.y);
  p.dz = 0.5f * (lj.z + hj.z) - 0.5f * (li.z + hi_.z);
  n[2] = rintf(p.dz * B.i8);
  p.dx -= n[2] * B.b6; p.dy -= n[2] * B.b7; p.dz -= n[2] * B.b8;
  n[1] = rintf(p.dy * B.i4);
  p.dx -= n[1] * B.b3; p.dy -= n[1] * B.b4;
  n[0] = rintf(p.dx * B.i0);
  p.dx -= n[0] * B.b0;
  return p;
}

__device__ __forceinline__ float gap2(float d, float h) {
  const float g = fmaxf(fabsf(d) - h, 0.f);
  return g * g;
}

// When every centre distance that could pass (list + both half-diagonals) is
// below half the cell's narrowest width, the sequential reduction already
// gives the minimum image, as it does for the reference's cutoff: in
// one_image2, (half the width - list)^2, the bound on the half-diagonals'
// square (without bound in a rectangular cell, where it always does).
__device__ __forceinline__ bool one_image(const Cell& B, const BoxPair& p) {
  return p.hx * p.hx + p.hy * p.hy + p.hz * p.hz < B.one_image2;
}

// Do two boxes of one system come within cutoff + skin under some periodic
// image?  Box-to-box gap distance, minimised over images.  An empty
// cluster's box is inverted (lo = +3e38, hi = -3e38): its gap is infinite.
// Images out of reach along one axis are not tried along the others (small
// triclinic cells: 27 images a test otherwise).
__device__ __forceinline__ bool boxes_near(const Cell& B, float4 li, float4 hi_, float4 lj, float4 hj) {
  float n[3];
  const BoxPair p = box_pair(B, li, hi_, lj, hj, n);
  if (one_image(B, p)) return gap2(p.dx, p.hx) + gap2(p.dy, p.hy) + gap2(p.dz, p.hz) < B.list2;
  for (int k = -1; k <= 1; ++k) {
    const float z2 = gap2(p.dz + k * B.b8, p.hz);
    if (!(z2 < B.list2)) continue;
    for (int j = -1; j <= 1; ++j) {
      const float y2 = z2 + gap2(p.dy + j * B.b4 + k * B.b7, p.hy);
      if (!(y2 < B.list2)) continue;
      for (int i = -1; i <= 1; ++i)
        if (y2 + gap2(p.dx + i * B.b0 + j * B.b3 + k * B.b6, p.hx) < B.list2) return true;
    }
  }
  return false;
}

// The lattice shift (in pair-coordinate units, applied to J) of the image
// that brings box J nearest box I, as boxes_near finds it; w carries that
// image's lattice counts (so a box change can recompute the shift without a
// rebuild) and the per-pair flag, set when that
// one image might not hold every pair of the tile within the cutoff: when
// 2 (|h_I| + |h_J|) + list + cutoff reaches the cell's narrowest width (h the
// half-diagonals), another image of some pair could come inside the cutoff,
// and the pair kernel takes the minimum image per pair instead.
__device__ __forceinline__ int4 tile_image(const SysDev& S, const Cell& B, float4 li, float4 hi_, float4 lj, float4 hj) {
  float n[3];
  const BoxPair p = box_pair(B, li, hi_, lj, hj, n);
  int na = -int(n[0]), nb = -int(n[1]), nc = -int(n[2]);
  if (!one_image(B, p)) {
    float best = 3.0e38f;
    int bi = 0, bj = 0, bk = 0;
    for (int k = -1; k <= 1; ++k) {
      const float z2 = gap2(p.dz + k * B.b8, p.hz);
      if (!(z2 < best)) continue;
      for (int j = -1; j <= 1; ++j) {
        const float y2 = z2 + gap2(p.dy + j * B.b4 + k * B.b7, p.hy);
        if (!(y2 < best)) continue;
        for (int i = -1; i <= 1; ++i) {
          const float g = y2 + gap2(p.dx + i * B.b0 + j * B.b3 + k * B.b6, p.hx);
          if (g < best) {
            best = g;
            bi = i;
            bj = j;
            bk = k;
          }
        }
      }
    }
    na += bi;
    nb += bj;
    nc += bk;
  }
  const float ei = 0.5f * sqrtf((hi_.x - li.x) * (hi_.x - li.x) + (hi_.y - li.y) * (hi_.y - li.y) +
                                (hi_.z - li.z) * (hi_.z - li.z));
  const float ej = 0.5f * sqrtf((hj.x - lj.x) * (hj.x - lj.x) + (hj.y - lj.y) * (hj.y - lj.y) +
                                (hj.z - lj.z) * (hj.z - lj.z));
  const bool per_pair = 2.f * (ei + ej) + sqrtf(S.list2) + sqrtf(S.cut2) >= S.min_width;
  // wrapping 32-bit arithmetic: the pair kernel adds the shift to a coordinate
  // and subtracts another; the result, a separation inside the cutoff, fits
  return tile_shift_for(S, tile_flags(per_pair, na, nb, nc));
}

// Position of the k-th (from 0) set bit of m, or -1.
__device__ __forceinline__ int nth_set_bit(unsigned int m, int k) {
  for (int i = 0; i < k && m; ++i) m &= m - 1;
  return m ? __ffs(m) - 1 : -1;
}

// Row `r` of the mask of tile (I, J) (indices within their system): every pair
// of atoms, without padding and, on the diagonal, one half.
template <int C>
__device__ __forceinline__ unsigned int valid_row(const SysDev& S, int I, int J, int r) {
  constexpr unsigned kAll = C == 32 ? 0xffffffffu : ((1u << C) - 1u);
  const int nj = max(0, min(C, S.n_atoms - J * C));
  unsigned int row = nj >= C ? kAll : ((1u << nj) - 1u);
  if (J == I) row &= r == C - 1 ? 0u : ((kAll << (r + 1)) & kAll);
  return I * C + r < S.n_atoms ? row : 0u;
}

// The candidates of row I among super-clusters [sI, sEnd), in ascending J: the
// 32-slot super-cluster of J (kSub = 32 / C clusters) must come near I's
// cluster before the clusters inside it are tested, 32 / kSub super-clusters to
// a pass of the warp.
// `batch(J)` is called by the whole warp, J < 0 in lanes without a candidate.
template <int C, class Batch>
__device__ __forceinline__ void walk_row(const Dev& d, const Cell& B, int I, float4 li, float4 hi_, int sI, int sEnd,
                                         Batch batch) {
  constexpr int kSub = 32 / C, kBatch = 32 / kSub;
  const int lane = threadIdx.x & 31;
  for (int J0 = sI; J0 < sEnd; J0 += 32) {
    const int SJ = J0 + lane;
    const bool near = SJ < sEnd && boxes_near(B, li, hi_, d.sb_lo[SJ], d.sb_hi[SJ]);
    if (C == 32) {
      batch(near ? SJ : -1);  // no super level: the boxes tested are the clusters themselves
      continue;
    }
    unsigned int rest = __ballot_sync(0xffffffffu, near);
    while (rest) {
      // lanes k * kSub .. k * kSub + kSub - 1 take the k-th remaining near super-cluster
      const int nth = nth_set_bit(rest, lane / kSub);
      const int J = nth >= 0 ? (J0 + nth) * kSub + lane % kSub : -1;
      batch(J >= I && boxes_near(B, li, hi_, d.bb_lo[J], d.bb_hi[J]) ? J : -1);
      for (int b = 0; b < kBatch && rest; ++b) rest &= rest - 1;  // the super-clusters this pass took
    }
  }
}

// Which of a warp's candidate tiles of row I (lane's J and shift; `here`: the
// lanes that have one) hold a pair closer than reach: 32/C tiles at a time, C
// lanes to a tile, the pair kernel's rotation on distances only.  `pi` is the
// row's atom lane mod C.
template <int C>
__device__ __forceinline__ unsigned int tiles_with_pair(const Dev& d, const SysDev& S, int I, int4 pi, int J, int4 sh,
                                                        unsigned int here, float reach2) {
  constexpr int G = 32 / C;
  constexpr unsigned kGroup = C == 32 ? 0xffffffffu : ((1u << C) - 1u);
  const int lane = threadIdx.x & 31, g = lane / C, l = lane & (C - 1), src = (l + 1) & (C - 1);
  const float inv = S.pc_inv;
  unsigned int keep = 0u;
  // the next group's atoms are on their way while one group is tested
  struct Group {
    int J, w;
    int4 pj;
  };
  auto fetch = [&](int t0) {
    Group r;
    const int from = (t0 + g) & 31;
    r.J = t0 < 32 ? __shfl_sync(0xffffffffu, J, from) : -1;
    const int sx = __shfl_sync(0xffffffffu, sh.x, from), sy = __shfl_sync(0xffffffffu, sh.y, from),
              sz = __shfl_sync(0xffffffffu, sh.z, from);
    r.w = __shfl_sync(0xffffffffu, sh.w, from);
    r.pj = make_int4(0, 0, 0, 0);
    if (r.J >= 0) {
      r.pj = d.pc[r.J * C + l];
      if (!tile_per_pair(r.w)) {
        r.pj.x = int(unsigned(r.pj.x) + unsigned(sx));
        r.pj.y = int(unsigned(r.pj.y) + unsigned(sy));
        r.pj.z = int(unsigned(r.pj.z) + unsigned(sz));
      }
    }
    return r;
  };
  Group next = fetch(0);
  const int end = 32 - __clz(here);  // no candidate from here on
  for (int t0 = 0; t0 < end; t0 += G) {
    const Group now = next;
    next = fetch(t0 + G);
    if (!__any_sync(0xffffffffu, now.J >= 0)) continue;
    const bool per_pair = now.J >= 0 && tile_per_pair(now.w);
    unsigned int mask = now.J >= 0 ? valid_row<C>(S, I - S.block_off, now.J - S.block_off, l) : 0u;
    int4 pj = now.pj;
    // bit k <-> j = l + k (mod C)
    mask = C == 32 ? __funnelshift_r(mask, mask, l) : (mask >> l) | (mask << ((C - l) & (C - 1)));
    const bool images = __any_sync(0xffffffffu, per_pair);
    bool hit = false;
#pragma unroll 8
    for (int k = 0; k < C; ++k) {
      int dx = int(unsigned(pj.x) - unsigned(pi.x)), dy = int(unsigned(pj.y) - unsigned(pi.y)),
          dz = int(unsigned(pj.z) - unsigned(pi.z));
      if (images) {
        // (a tile that needs none is left as it is: see the pair kernel)
        if (S.triclinic) min_image<true>(S, dx, dy, dz);
        else min_image<false>(S, dx, dy, dz);
      }
      const float rx = dx * inv, ry = dy * inv, rz = dz * inv;
      hit |= ((mask >> k) & 1u) && rx * rx + ry * ry + rz * rz < reach2;
      pj.x = __shfl_sync(0xffffffffu, pj.x, src, C);
      pj.y = __shfl_sync(0xffffffffu, pj.y, src, C);
      pj.z = __shfl_sync(0xffffffffu, pj.z, src, C);
    }
    const unsigned int hits = __ballot_sync(0xffffffffu, hit);
#pragma unroll
    for (int q = 0; q < G; ++q)
      if ((hits >> (q * C)) & kGroup) keep |= 1u << (t0 + q);
  }
  return keep;
}

// A warp to a segment of a row (row_supers super-clusters of J: whole rows in
// large engines, fewer where rows alone would leave warps idle; row_segments
// to a row): its candidates are found once, into shared memory; with pruning, those whose atoms are all farther apart than cutoff + skin are
// dropped (the box test is conservative: about a fifth of 8x8 tiles have no
// pair inside); one atomic reserves its place in its system's list, and
// the tiles are written there, in ascending J.  Rows land in any order: the
// pair kernel's sums do not depend on it (per-tile f32 partials become int64
// fixed point).  A row longer than the buffer (a cluster that straddles a jump
// of the space-filling curve has a large box and may reach half the system)
// is walked again instead.  Measured alone against a count pass, a scan, a fill
// pass that tested every box again, and prune, scan and copy passes: 2,652
// atoms 83 -> 23 us, 12k 115 -> 77, 27k (no pruning) 164 -> 70, 100k 316 -> 206,
// the 64-system ensemble 1.52 -> 0.71 ms.  Reserving by block (one atomic for its
// eight warps, between two barriers) was slower: 12k 119 us, the warps wait for
// the longest of the eight.
constexpr int kRowBuffer = 512;

template <int C>
__device__ void phase_rows(const Dev& d, int (*buffers)[kRowBuffer]) {
  constexpr int kWords = C * C / 32;
  const int lane = threadIdx.x & 31;
  int* buf = buffers[threadIdx.x >> 5];
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const unsigned below = (1u << lane) - 1u;
  constexpr int kSub = 32 / C;
  const int tasks = d.n_blocks * d.row_segments;
  for (int task = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; task < tasks; task += warps) {
    const int I = task / d.row_segments, seg = task - I * d.row_segments;
    const int s = d.block_sys[I];
    if (!d.rebuild_now[s]) continue;
    const SysDev& S = d.sys[s];
    const int super0 = S.block_off / kSub, supers = S.n_blocks / kSub;
    const int sI = max(I / kSub, super0 + seg * d.row_supers), sEnd = super0 + min(supers, (seg + 1) * d.row_supers);
    if (sI >= sEnd) continue;  // no J from I up: the exclusions never look here
    const Cell B = cell_of_system(S);
    const float4 li = d.bb_lo[I], hi_ = d.bb_hi[I];
    const float reach2 = S.list2 * (1.0f + 1e-5f);
    const int4 pi = d.prune ? d.pc[I * C + (lane & (C - 1))] : make_int4(0, 0, 0, 0);
    // which of a batch's candidates (a lane's J, or none: J < 0) stay, as a
    // warp mask: with pruning, those with a pair within cutoff + skin
    auto keepers = [&](int J) {
      const unsigned int here = __ballot_sync(0xffffffffu, J >= 0);
      if (!d.prune) return here;
      int4 sh = make_int4(0, 0, 0, 0);
      if (J >= 0) sh = tile_image(S, B, li, hi_, d.bb_lo[J], d.bb_hi[J]);
      return tiles_with_pair<C>(d, S, I, pi, J, sh, here, reach2);
    };
    int found = 0;
    walk_row<C>(d, B, I, li, hi_, sI, sEnd, [&](int J) {
      const unsigned int here = __ballot_sync(0xffffffffu, J >= 0);
      const int at = found + __popc(here & below);
      if (J >= 0 && at < kRowBuffer) buf[at] = J;
      found += __popc(here);
    });
    __syncwarp();
    const bool fits = found <= kRowBuffer;
    int count = found;
    if (d.prune && fits) {
      count = 0;
      for (int k0 = 0; k0 < found; k0 += 32) {
        const int J = k0 + lane < found ? buf[k0 + lane] : -1;
        const unsigned int keep = keepers(J);
        if ((keep >> lane) & 1u) buf[count + __popc(keep & below)] = J;  // never past what was read
        count += __popc(keep);
        __syncwarp();
      }
    } else if (d.prune) {
      count = 0;
      walk_row<C>(d, B, I, li, hi_, sI, sEnd, [&](int J) { count += __popc(keepers(J)); });
    }
    int start = 0;
    if (lane == 0) {
      if (count) start = atomicAdd(&d.tile_need[s], count);
      d.tile_start[task] = start;
      d.tile_cnt[task] = count;
    }
    start = __shfl_sync(0xffffffffu, start, 0);
    const long long base = static_cast<long long>(S.tile_off) + start;
    const int cap = S.tile_cap - start;
    // tiles past the system's capacity are dropped; the finish phase sees the
    // count and stops the step
    auto write = [&](int at, int J) {
      if (C == 8) {
        if (J < 0 || at >= cap) return;
        d.tiles[base + at] = make_int2(I, J);
        d.tile_shift[base + at] = tile_image(S, B, li, hi_, d.bb_lo[J], d.bb_hi[J]);
        unsigned int words[2] = {0u, 0u};
#pragma unroll
        for (int r = 0; r < 8; ++r) words[r >> 2] |= valid_row<8>(S, I - S.block_off, J - S.block_off, r) << ((r & 3) * 8);
        *reinterpret_cast<uint2*>(d.masks + (base + at) * kWords) = make_uint2(words[0], words[1]);
      }
    };
    auto write_batch = [&](int at0, int J, unsigned int keep) {
      if (C == 8) {
        write(at0 + __popc(keep & below), (keep >> lane) & 1u ? J : -1);
        return;
      }
      // a 32x32 tile's mask is one word per row: every lane writes its row
      for (int n = 0; keep; ++n) {
        const int src = __ffs(keep) - 1;
        keep &= keep - 1;
        const int Jt = __shfl_sync(0xffffffffu, J, src), at = at0 + n;
        if (at >= cap) continue;
        if (lane == 0) {
          d.tiles[base + at] = make_int2(I, Jt);
          d.tile_shift[base + at] = tile_image(S, B, li, hi_, d.bb_lo[Jt], d.bb_hi[Jt]);
        }
        d.masks[(base + at) * kWords + lane] = valid_row<C>(S, I - S.block_off, Jt - S.block_off, lane);
      }
    };
    if (fits) {
      for (int k0 = 0; k0 < count; k0 += 32) {
        const int J = k0 + lane < count ? buf[k0 + lane] : -1;
        write_batch(k0, J, __ballot_sync(0xffffffffu, J >= 0));
      }
      __syncwarp();  // the buffer is free for the warp's next row
    } else {
      int written = 0;
      walk_row<C>(d, B, I, li, hi_, sI, sEnd, [&](int J) {
        const unsigned int keep = keepers(J);
        write_batch(written, J, keep);
        written += __popc(keep);
      });
    }
  }
}

// Clear the mask bit of every excluded pair in the tile that holds it.
template <int C>
__device__ void phase_tiles_exclusions(const Dev& d) {
  for (int e = grid_stride_start(); e < d.n_excl; e += grid_stride()) {
    const int s = d.excl_sys[e];
    if (!d.rebuild_now[s]) continue;
    const SysDev& S = d.sys[s];
    const int2 pr = d.excl[e];
    int sa = d.rank[pr.x], sb = d.rank[pr.y];
    if (sa > sb) { const int t = sa; sa = sb; sb = t; }
    const int I = S.block_off + sa / C, J = S.block_off + sb / C;
    const int row = sa % C, bit = sb % C;
    // the row's segment that would hold the tile, in ascending J
    const int task = I * d.row_segments + (J - S.block_off) / (32 / C) / d.row_supers;
    int lo = d.tile_start[task];
    const int end = lo + d.tile_cnt[task];
    int hi = end;
    if (hi > S.tile_cap) hi = S.tile_cap;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      const int Jm = d.tiles[S.tile_off + mid].y;
      if (Jm < J) lo = mid + 1;
      else hi = mid;
    }
    if (lo < end && lo < S.tile_cap && d.tiles[S.tile_off + lo].y == J) {
      const long long t = static_cast<long long>(S.tile_off) + lo;
      if (C == 32) atomicAnd(&d.masks[t * 32 + row], ~(1u << bit));
      else atomicAnd(&d.masks[t * (C * C / 32) + (row >> 2)], ~(1u << ((row & 3) * 8 + bit)));
    }
  }
}

// The inner list of every system that rebuilt or is due a prune: the outer
// tiles with an unexcluded pair closer than cutoff + inner skin (GROMACS's
// dynamic pruning, Pall et al., J. Chem. Phys. 153, 134110 (2020), made
// exact: a prune is due as soon as any atom has moved half the inner skin, so
// a dropped tile has no pair inside the cutoff until the next one and the
// pair kernel's results are bit-identical to running the whole outer list).
// A warp takes 32 consecutive outer tiles and one atomicAdd reserves room for
// the survivors, which keep their order.  Chunks land in any order; the pair
// kernel's sums do not depend on it (per-tile f32 partials become int64 fixed
// point), and a chunk spans at most two rows.
//
// 8x8 tiles: one lane per tile; a tile whose clusters' current boxes are out
// of reach is dropped at once, the others test their pairs until the first one
// within reach, on f32 offsets from the tile's first atom (exact integer
// differences, then one rounding), with the J cluster in registers --
// independent loads and no shuffles.  Tiles flagged for per-pair images (the
// cell is too small for one shift per tile) take each pair's minimum image, as
// the pair kernel does, in cells narrower than cutoff + list radius + 1 nm,
// where nearly every tile is flagged; in wider cells the few flagged tiles
// are kept without a test.  32x32 tiles (too many registers for that) keep a tile if some
// atom of I is within reach of J's current bounding box and some atom of J of
// I's, which any pair within reach implies: conservative, one lane per atom.
template <int C>
__device__ bool tile_within_reach(const Dev& d, const SysDev& S, long long ti, float reach2, int lane);

// Some pair of an 8x8 tile's mask closer than reach (a lane's own tile; every
// pair's minimum image if the tile is flagged for it).
__device__ __forceinline__ bool tile_has_pair(const Dev& d, const SysDev& S, int2 tile, int4 sh,
                                              const unsigned int* mask, float reach2) {
  const float inv = S.pc_inv;
  if (tile_per_pair(sh.w)) {
    int4 qj[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) qj[j] = d.pc[tile.y * 8 + j];
    for (int i = 0; i < 8; ++i) {
      const unsigned int row = ((i < 4 ? mask[0] : mask[1]) >> ((i & 3) * 8)) & 0xFFu;
      if (!row) continue;
      const int4 qi = d.pc[tile.x * 8 + i];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (!((row >> j) & 1u)) continue;
        int dx = int(unsigned(qj[j].x) - unsigned(qi.x)), dy = int(unsigned(qj[j].y) - unsigned(qi.y)),
            dz = int(unsigned(qj[j].z) - unsigned(qi.z));
        if (S.triclinic) min_image<true>(S, dx, dy, dz);
        else min_image<false>(S, dx, dy, dz);
        const float rx = dx * inv, ry = dy * inv, rz = dz * inv;
        if (rx * rx + ry * ry + rz * rz < reach2) return true;
      }
    }
    return false;
  }
  // both clusters' sixteen atoms in one round of loads, then the 64 tests
  // (loading each i atom inside the loop made a chain of eight round trips)
  int4 qi[8], qj[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    qi[k] = d.pc[tile.x * 8 + k];
    qj[k] = d.pc[tile.y * 8 + k];
  }
  const int4 r0 = qi[0];
  const unsigned ox = unsigned(r0.x) - unsigned(sh.x), oy = unsigned(r0.y) - unsigned(sh.y),
                 oz = unsigned(r0.z) - unsigned(sh.z);
  float jx[8], jy[8], jz[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    jx[j] = int(unsigned(qj[j].x) - ox) * inv;
    jy[j] = int(unsigned(qj[j].y) - oy) * inv;
    jz[j] = int(unsigned(qj[j].z) - oz) * inv;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const unsigned int row = ((i < 4 ? mask[0] : mask[1]) >> ((i & 3) * 8)) & 0xFFu;
    const float ix = int(unsigned(qi[i].x) - unsigned(r0.x)) * inv,
                iy = int(unsigned(qi[i].y) - unsigned(r0.y)) * inv,
                iz = int(unsigned(qi[i].z) - unsigned(r0.z)) * inv;
    bool hit = false;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float dx = jx[j] - ix, dy = jy[j] - iy, dz = jz[j] - iz;
      hit |= ((row >> j) & 1u) && dx * dx + dy * dy + dz * dz < reach2;
    }
    if (hit) return true;  // most kept tiles stop at their first rows
  }
  return false;
}

template <>
__device__ bool tile_within_reach<8>(const Dev& d, const SysDev& S, long long ti, float reach2, int) {
  const int2 tile = __ldcg(&d.tiles[ti]);
  const int4 sh = __ldcg(&d.tile_shift[ti]);
  const bool per_pair = tile_per_pair(sh.w);
  if (per_pair && !S.prune_per_pair) return true;
  if (!per_pair) {
    // the clusters' current boxes first: most outer tiles of a long skin are
    // out of reach box to box and need no pair loop (the margin covers the
    // boxes' f32 rounding)
    const float inv = S.pc_inv;
    const float4 ilo = d.cb_lo[tile.x], ihi = d.cb_hi[tile.x], jlo = d.cb_lo[tile.y], jhi = d.cb_hi[tile.y];
    const float sx = sh.x * inv, sy = sh.y * inv, sz = sh.z * inv;
    const float gx = fmaxf(fmaxf(jlo.x + sx - ihi.x, ilo.x - (jhi.x + sx)), 0.f);
    const float gy = fmaxf(fmaxf(jlo.y + sy - ihi.y, ilo.y - (jhi.y + sy)), 0.f);
    const float gz = fmaxf(fmaxf(jlo.z + sz - ihi.z, ilo.z - (jhi.z + sz)), 0.f);
    if (gx * gx + gy * gy + gz * gz >= reach2 * (1.0f + 4e-5f)) return false;
  }
  const unsigned int mask[2] = {__ldcg(&d.masks[ti * 2]), __ldcg(&d.masks[ti * 2 + 1])};
  return tile_has_pair(d, S, tile, sh, mask, reach2);
}

template <>
__device__ bool tile_within_reach<32>(const Dev& d, const SysDev& S, long long ti, float reach2, int l) {
  const int2 tile = __ldcg(&d.tiles[ti]);
  const int4 sh = __ldcg(&d.tile_shift[ti]);
  const unsigned int row = __ldcg(&d.masks[ti * 32 + l]);
  const unsigned int cols = __reduce_or_sync(0xffffffffu, row);
  if (tile_per_pair(sh.w)) return true;  // warp-uniform: one tile per warp
  const float inv = S.pc_inv;
  const float4 ilo = d.cb_lo[tile.x], ihi = d.cb_hi[tile.x];
  const float4 jlo = d.cb_lo[tile.y], jhi = d.cb_hi[tile.y];
  const float sx = sh.x * inv, sy = sh.y * inv, sz = sh.z * inv;
  const int4 qi = d.pc[tile.x * 32 + l], qj = d.pc[tile.y * 32 + l];
  const float ix = qi.x * inv, iy = qi.y * inv, iz = qi.z * inv;
  const float jx = qj.x * inv + sx, jy = qj.y * inv + sy, jz = qj.z * inv + sz;
  const float ax = fmaxf(fmaxf(jlo.x + sx - ix, ix - (jhi.x + sx)), 0.f);
  const float ay = fmaxf(fmaxf(jlo.y + sy - iy, iy - (jhi.y + sy)), 0.f);
  const float az = fmaxf(fmaxf(jlo.z + sz - iz, iz - (jhi.z + sz)), 0.f);
  const float bx = fmaxf(fmaxf(ilo.x - jx, jx - ihi.x), 0.f);
  const float by = fmaxf(fmaxf(ilo.y - jy, jy - ihi.y), 0.f);
  const float bz = fmaxf(fmaxf(ilo.z - jz, jz - ihi.z), 0.f);
  const bool hit_i = row != 0u && ax * ax + ay * ay + az * az < reach2;
  const bool hit_j = ((cols >> l) & 1u) && bx * bx + by * by + bz * bz < reach2;
  return __any_sync(0xffffffffu, hit_i) && __any_sync(0xffffffffu, hit_j);
}

template <int C>
__device__ void phase_inner(const Dev& d) {
  constexpr int kWords = C * C / 32;
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  for (int s = 0; s < d.S; ++s) {
    if (!d.rebuild_now[s] && !d.prune_now[s]) continue;
    const SysDev& S = d.sys[s];
    const int n = min(d.tile_count[s], S.tile_cap);
    const float reach2 = S.inner2 * (1.0f + 1e-5f);
    // each system's first chunk goes to the warp after the previous system's
    // last (the outer list's offsets, which this kernel only reads), so a
    // batch of small systems spreads over every warp instead of the first few
    const int first = (d.tile_prefix[s] >> 5) % warps;
    for (int c0 = ((warp - first + warps) % warps) * 32; c0 < n; c0 += warps * 32) {
      unsigned int keep = 0u;  // bit k: outer tile c0 + k survives (the same in every lane)
      if (C == 8) {
        const bool alive = c0 + lane < n && tile_within_reach<C>(d, S, S.tile_off + c0 + lane, reach2, lane);
        keep = __ballot_sync(0xffffffffu, alive);
      } else {
        for (int k = 0; k < 32 && c0 + k < n; ++k)
          if (tile_within_reach<C>(d, S, S.tile_off + c0 + k, reach2, lane)) keep |= 1u << k;
      }
      const int count = __popc(keep);
      int base = 0;
      if (lane == 0 && count) base = atomicAdd(&d.in_count[s], count);
      base = __shfl_sync(0xffffffffu, base, 0);
      if ((keep >> lane) & 1u) {
        const long long from = static_cast<long long>(S.tile_off) + c0 + lane;
        const long long to = static_cast<long long>(S.tile_off) + base + __popc(keep & ((1u << lane) - 1u));
        d.in_tiles[to] = __ldcg(&d.tiles[from]);
        d.in_shift[to] = __ldcg(&d.tile_shift[from]);
        if (C < 32) {
#pragma unroll
          for (int w = 0; w < kWords; ++w) d.in_masks[to * kWords + w] = __ldcg(&d.masks[from * kWords + w]);
        }
      }
      if (C == 32) {
        // a 32x32 tile's mask is 32 words: the warp copies each kept tile's
        unsigned int f = keep;
        while (f) {
          const int k = __ffs(f) - 1;
          f &= f - 1;
          const long long from = static_cast<long long>(S.tile_off) + c0 + k;
          const long long to = static_cast<long long>(S.tile_off) + base + __popc(keep & ((1u << k) - 1u));
          d.in_masks[to * kWords + lane] = __ldcg(&d.masks[from * kWords + lane]);
        }
      }
    }
  }
}

// Exclusive offsets of per-system counts (one warp): prefix[s] and, at
// prefix[S], the total; `count(s)` is called once per system.
template <class Count>
__device__ __forceinline__ void system_offsets(const Dev& d, int* prefix, Count count) {
  const int lane = threadIdx.x & 31;
  int carry = 0;
  for (int s0 = 0; s0 < d.S; s0 += 32) {
    const int s = s0 + lane, n = s < d.S ? count(s) : 0;
    int x = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (s < d.S) prefix[s] = carry + x - n;
    carry += __shfl_sync(0xffffffffu, x, 31);
  }
  if (lane == 0) prefix[d.S] = carry;
}

// After the outer list (one warp): per-system counts, offsets and rebuild
// counts.  Without an inner list the rebuild requests are cleared here; with
// one, the inner-list kernel that follows still needs them and clears them
// itself.
__device__ void list_finish(const Dev& d) {
  system_offsets(d, d.tile_prefix, [&](int s) {
    int n = d.tile_count[s];
    if (d.rebuild_now[s]) {
      // a list that needs more tiles than the system's capacity is cut there,
      // and the engine's halt word stops the integrator, so no step runs on
      // the cut list: the host grows the capacity to `tile_need` and rebuilds
      // before it runs the remaining steps
      const int need = __ldcg(&d.tile_need[s]), cap = d.sys[s].tile_cap;
      if (need > cap) {
        atomicOr(&d.err[s], kErrTileCapacity);
        atomicExch(d.halt, 1);
      }
      d.tile_count[s] = n = min(need, cap);
      d.rebuild_count[s] += 1;
      if (!d.inner) d.rebuild_now[s] = 0;
    }
    return n;
  });
  if (!d.inner && (threadIdx.x & 31) == 0) *d.any_rebuild = 0;
}

// After the inner list (one warp): its offsets, the prune count, and every
// list request cleared for the next step.
__device__ void inner_finish(const Dev& d) {
  system_offsets(d, d.in_prefix, [&](int s) {
    if (d.prune_now[s] && !d.rebuild_now[s]) d.prune_count[s] += 1;
    d.prune_now[s] = 0;
    d.rebuild_now[s] = 0;
    return __ldcg(&d.in_count[s]);
  });
  if ((threadIdx.x & 31) == 0) {
    *d.any_rebuild = 0;
    *d.any_prune = 0;
  }
}

// True in every thread of the block that finishes last, whose view of global
// memory then holds every block's writes.
__device__ __forceinline__ bool last_block(int* ticket) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1) == int(gridDim.x) - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  if (threadIdx.x == 0) *ticket = 0;
  return true;
}

// Grid-wide barrier for the cooperative list kernel: arrive on a counter,
// the last arrival bumps the generation, the others wait on it with a bounded
// spin.  A wait that gives up records kErrTimeout and returns, so a scheduling
// fault becomes an error status and never a hung GPU.
__device__ bool grid_barrier(unsigned int* bar, int* err) {
  __syncthreads();
  __shared__ int ok;
  if (threadIdx.x == 0) {
    ok = 1;
    volatile unsigned int* gen = bar + 1;
    const unsigned int mine = *gen;
    __threadfence();
    if (atomicAdd(bar, 1u) + 1u == gridDim.x) {
      bar[0] = 0u;
      __threadfence();
      atomicAdd(bar + 1, 1u);
    } else {
      long long spins = 0;
      while (*gen == mine) {
        if (++spins > (1ll << 22)) {
          atomicOr(err, kErrTimeout);
          ok = 0;
          break;
        }
        __nanosleep(32);
      }
    }
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

// The exclusions, and the list's finish by the last block to end: every block
// has read the rebuild requests by then.
template <int C>
__device__ void phase_exclusions_finish(const Dev& d) {
  phase_tiles_exclusions<C>(d);
  if (last_block(d.list_ticket) && threadIdx.x < 32) list_finish(d);
}

// One launch per step.  With no rebuild requested it returns at once, or takes
// the references of a prune that is due; otherwise it runs the sort and
// tile-list phases with a grid barrier between them.
template <int C>
__global__ void __launch_bounds__(kThreads, 4) k_list(Dev d) {
  __shared__ int buffers[kThreads / 32][kRowBuffer];
  const bool rebuild = *d.any_rebuild != 0, prune = d.inner && *d.any_prune != 0;
  int* err = d.err;  // system 0's word carries a barrier timeout
  if (prune) phase_prune_references(d);
  if (!rebuild) return;
  phase_cells_assign(d);
  if (!grid_barrier(d.list_barrier, err)) return;
  phase_cells_scan(d);
  if (!grid_barrier(d.list_barrier, err)) return;
  phase_cells_scatter(d);
  if (!grid_barrier(d.list_barrier, err)) return;
  phase_place(d);
  if (!grid_barrier(d.list_barrier, err)) return;
  phase_boxes<C>(d);
  if (!grid_barrier(d.list_barrier, err)) return;
  phase_rows<C>(d, buffers);
  if (!grid_barrier(d.list_barrier, err)) return;
  phase_exclusions_finish<C>(d);
}

// The same phases as separate launches (the path the graph-free debug mode,
// large batches and devices without cooperative launch take).
__global__ void __launch_bounds__(kThreads) k_prune_references(Dev d) {
  if (d.inner && *d.any_prune) phase_prune_references(d);
}
__global__ void __launch_bounds__(kThreads) k_cells_assign(Dev d) {
  if (*d.any_rebuild) phase_cells_assign(d);
}
__global__ void __launch_bounds__(kThreads) k_cells_scan(Dev d) {
  if (*d.any_rebuild) phase_cells_scan(d);
}
__global__ void __launch_bounds__(kThreads) k_cells_scatter(Dev d) {
  if (*d.any_rebuild) phase_cells_scatter(d);
}
__global__ void __launch_bounds__(kThreads) k_place(Dev d) {
  if (*d.any_rebuild) phase_place(d);
}
template <int C>
__global__ void __launch_bounds__(kThreads) k_boxes(Dev d) {
  if (*d.any_rebuild) phase_boxes<C>(d);
}
template <int C>
__global__ void __launch_bounds__(kThreads, 3) k_rows(Dev d) {
  __shared__ int buffers[kThreads / 32][kRowBuffer];
  if (*d.any_rebuild) phase_rows<C>(d, buffers);
}
template <int C>
__global__ void __launch_bounds__(kThreads) k_exclusions(Dev d) {
  if (*d.any_rebuild) phase_exclusions_finish<C>(d);
}
// The inner list, its own launch after the list kernels (a full grid, where
// the cooperative list kernel has one or two blocks per SM): nothing to do unless a
// system rebuilt or is due a prune.  The last block to finish writes the
// offsets and clears the requests; every block has read them by then, since
// each reads them before taking its ticket.
template <int C>
__global__ void __launch_bounds__(kThreads) k_inner_prune(Dev d) {
  wait_for_predecessor();
  release_successor();
  if (!*d.any_rebuild && !*d.any_prune) return;
  phase_inner<C>(d);
  if (last_block(d.inner_ticket) && threadIdx.x < 32) inner_finish(d);
}

int blocks_for(int n, int threads, int cap = 148 * 8) {
  const int b = (n + threads - 1) / threads;
  return b < 1 ? 1 : (b > cap ? cap : b);
}

int g_list_grid = 0;

}  // namespace

// Size the cooperative grid once: every block resident at the same time.
int prepare_list_kernel(int device) {
  int per_sm = 0, sms = 0;
  int per_sm8 = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_list<32>, kThreads, 0) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm8, k_list<8>, kThreads, 0) != cudaSuccess) return 0;
  per_sm = std::min(per_sm, per_sm8);
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
  int coop = 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device);
  g_list_grid = coop ? std::max(1, std::min(per_sm, 2)) * sms : 0;
  return g_list_grid;
}

bool launch_list(const Dev& d, cudaStream_t st) {
  if (g_list_grid <= 0) return false;
  cudaLaunchConfig_t cfg = {};
  // Two blocks per SM, or one where an inner list makes rebuilds rare and the
  // system is small: most launches then find nothing to do, and the fewer
  // blocks cost the spread beside them less.  A step with one and with two, us
  // (skin 0.5, inner skin 0.1, TIP3P cubes): 2.7k atoms 45.6, 45.7; 9.8k 59.2,
  // 58.7; 27k 103.1, 109.6; 55k 196.5, 201.4; 64k 233, 237; from 2^16 slots the
  // rebuild outweighs it (100k 400, 392).  An evaluation at new positions
  // always rebuilds and would take two: 340, 317; 600, 559; 993, 901; 1161,
  // 1042 for 9.8k, 27k, 55k and 64k (rebuild alone 108, 90; 186, 144; 325, 238;
  // 410, 291).  Rebuilds before the phases
  // were joined and the rows searched once: 2,652 atoms (defaults) 111 -> 72
  // us, 12k 163 -> 146, 27k 305 -> 267, 100k 694 -> 414, the 64-system ensemble
  // (all systems, separate launches) 2.58 -> 1.73 ms.
  const bool few = d.inner && d.n_slots < (1 << 16) && g_list_grid > 1;
  cfg.gridDim = dim3(few ? (g_list_grid + 1) / 2 : g_list_grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (d.cluster == 8) return cudaLaunchKernelEx(&cfg, k_list<8>, d) == cudaSuccess;
  return cudaLaunchKernelEx(&cfg, k_list<32>, d) == cudaSuccess;
}

void launch_rebuild_sort(const Dev& d, cudaStream_t st) {
  k_cells_assign<<<blocks_for(d.n_atoms, kThreads), kThreads, 0, st>>>(d);
  k_cells_scan<<<blocks_for(d.n_chunks, 1), kThreads, 0, st>>>(d);
  k_cells_scatter<<<blocks_for(d.n_atoms, kThreads), kThreads, 0, st>>>(d);
  k_place<<<blocks_for(d.n_slots, kThreads), kThreads, 0, st>>>(d);
}

void launch_prune_references(const Dev& d, cudaStream_t st) {
  if (d.inner) k_prune_references<<<blocks_for(d.n_slots, kThreads), kThreads, 0, st>>>(d);
}

template <int C>
void rebuild_tiles(const Dev& d, cudaStream_t st) {
  const int warp_blocks = blocks_for(d.n_blocks * d.row_segments * 32, kThreads);
  k_boxes<C><<<blocks_for(d.n_slots, kThreads), kThreads, 0, st>>>(d);
  k_rows<C><<<warp_blocks, kThreads, 0, st>>>(d);
  k_exclusions<C><<<blocks_for(d.n_excl, kThreads), kThreads, 0, st>>>(d);
}

void launch_inner_prune(const Dev& d, cudaStream_t st) {
  if (!d.inner) return;
  if (d.cluster == 8) launch_chained(k_inner_prune<8>, 148 * 4, kThreads, 0, st, d);
  else launch_chained(k_inner_prune<32>, 148 * 4, kThreads, 0, st, d);
}

void launch_rebuild_tiles(const Dev& d, cudaStream_t st) {
  if (d.cluster == 8) rebuild_tiles<8>(d, st);
  else rebuild_tiles<32>(d, st);
}

}  // namespace mdb
