// The cluster-pair neighbor build on sm_100a.
//
// Replaces MDIR's emitted groups build (lib/Conversion/MDExecKernels/
// GroupsBuild.cpp: emitKeys 520, sortByKey 429, emitChunks 741, emitBoxes
// 912, emitLists 1098) behind the same contract (docs/neighbor-groups.md,
// Sections 1.1-1.3 and 4-5.2): every image of every non-excluded pair whose
// f32 distance is within the widened reach R' = R + 3e-6 (Lx+Ly+Lz) has
// exactly one bit, in the list of the group of the earlier place.
//
// The B200 design differs from the reference's: the cell sort is a counting
// sort into columns of about 16 atoms per column-width of height (so a
// group of 16 consecutive places of a column is close to a cube, with no
// sorting network); the search takes a run of places from each column around
// a group by the z bins of the sort (no candidate's box is read), tests the
// places against the group's box, 32 or 128 at a time, and those that pass
// against its 16 members; the exclusion partners of the 16 members are
// sorted in shared memory and
// looked up by binary search; and the list of a group is a fixed slab of C
// entries (grown by the host when a build reports a longer list), so that
// the units of work come out in group order and every result is
// deterministic.
//
// Kernels (in launch order): nb_keys, scan, nb_scatter, nb_columns,
// nb_places, nb_search_t, nb_unit_blocks, nb_unit_write.
#include <cmath>
#include <cstdio>

#include "nb_context.h"
#include "nb_prune.cuh"
#include "nb_scan.cuh"

#define NB_EXCL_MAX 256

// The atom of a place in xw.w, and above it whether its type has LJ terms.
#define NB_ATOM_BITS 0x3fffffff
#define NB_ATOM_LJ 0x40000000

namespace {

// The brick of a cell: x + S H in [0, ax) x [0, by) x [0, cz), S found
// along c, then b, then a (with no tilts, per axis), each product and sum
// of f64 rounded as written.
__global__ void nb_keys(int64_t n, const double *__restrict__ x, double Lx, double Ly, double Lz,
                        double bx, double cx, double cy,
                        int Nx, int Ny, int Nz, float inv_wx, float inv_wy, float inv_hz,
                        int32_t *__restrict__ key, int32_t *__restrict__ rank, int32_t *__restrict__ bin_count,
                        float4 *__restrict__ atom_xw, char4 *__restrict__ atom_shift, double *__restrict__ x_build) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double v0 = x[3 * i], v1 = x[3 * i + 1], v2 = x[3 * i + 2];
  if (x_build) {  // the positions of the build, for the displacement test
    x_build[3 * i] = v0;
    x_build[3 * i + 1] = v1;
    x_build[3 * i + 2] = v2;
  }
  bool ok = isfinite(v0) && isfinite(v1) && isfinite(v2);
  double S0 = 0, S1 = 0, S2 = 0;
  double p0 = 0, p1 = 0, p2 = 0;
  if (ok) {
    S2 = -floor(v2 / Lz);
    p2 = __dadd_rn(v2, __dmul_rn(S2, Lz));
    p1 = __dadd_rn(v1, __dmul_rn(S2, cy));
    S1 = -floor(p1 / Ly);
    p1 = __dadd_rn(p1, __dmul_rn(S1, Ly));
    p0 = __dadd_rn(__dadd_rn(v0, __dmul_rn(S2, cx)), __dmul_rn(S1, bx));
    S0 = -floor(p0 / Lx);
    p0 = __dadd_rn(p0, __dmul_rn(S0, Lx));
    ok = fabs(S0) <= 100.0 && fabs(S1) <= 100.0 && fabs(S2) <= 100.0;
  }
  if (!ok) {
    key[i] = Nx * Ny * Nz;  // the bin of the positions that have no key
    rank[i] = atomicAdd(&bin_count[Nx * Ny * Nz], 1);
    atom_xw[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    atom_shift[i] = make_char4(0, 0, 0, 0);
    return;
  }
  float w0 = (float)p0, w1 = (float)p1, w2 = (float)p2;
  int kx = min(max((int)(w0 * inv_wx), 0), Nx - 1);
  int ky = min(max((int)(w1 * inv_wy), 0), Ny - 1);
  int kz = min(max((int)(w2 * inv_hz), 0), Nz - 1);
  int k = (ky * Nx + kx) * Nz + kz;
  key[i] = k;
  rank[i] = atomicAdd(&bin_count[k], 1);
  atom_xw[i] = make_float4(w0, w1, w2, 1.f);
  atom_shift[i] = make_char4((signed char)S0, (signed char)S1, (signed char)S2, 0);
}

// The atoms of each bin, in the order they came (nb_places orders them).
__global__ void nb_scatter(int64_t n, const int32_t *__restrict__ key, const int32_t *__restrict__ rank,
                           const int32_t *__restrict__ bin_start, int32_t *__restrict__ sorted) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  sorted[bin_start[key[i]] + rank[i]] = (int32_t)i;
}

// The groups of 16 places of column c.  With `frames` (a batch), the column
// is of frame col_frame[c].
template <bool BATCH>
__device__ __forceinline__ int nb_column_groups(int c, int Nz, const int32_t *__restrict__ bin_start,
                                                const NbFrameDev *__restrict__ frames,
                                                const int32_t *__restrict__ col_frame) {
  int b0 = c * Nz, nz = Nz;
  if (BATCH) {
    const NbFrameDev &F = frames[col_frame[c]];
    nz = F.Nz;
    b0 = F.bin0 + (c - F.col0) * nz;
  }
  return (bin_start[b0 + nz] - bin_start[b0] + NB_GROUP - 1) / NB_GROUP;
}

// The columns' first groups, in one block: a thread a column counts its
// groups and a scan places them, a block's threads of columns at a time.
template <bool BATCH>
__global__ void __launch_bounds__(1024) nb_columns(int ncol, int Nz, const int32_t *__restrict__ bin_start,
                                                   const NbFrameDev *__restrict__ frames,
                                                   const int32_t *__restrict__ col_frame,
                                                   int32_t *__restrict__ group_start) {
  __shared__ int sw[32];
  int before = 0;
  for (int c0 = 0; c0 < ncol; c0 += blockDim.x) {
    const int c = c0 + threadIdx.x;
    const int groups = c < ncol ? nb_column_groups<BATCH>(c, Nz, bin_start, frames, col_frame) : 0;
    int total;
    const int first = before + nb_block_exclusive_scan(groups, sw, total);
    before += total;
    if (c < ncol) group_start[c] = first;
  }
  if (threadIdx.x == 0) group_start[ncol] = before;
}

// The columns' groups, a thread a column over the whole GPU (nb_scan places
// them).
template <bool BATCH>
__global__ void nb_column_counts(int ncol, int Nz, const int32_t *__restrict__ bin_start,
                                 const NbFrameDev *__restrict__ frames, const int32_t *__restrict__ col_frame,
                                 int32_t *__restrict__ groups) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < ncol) groups[c] = nb_column_groups<BATCH>(c, Nz, bin_start, frames, col_frame);
}

// The places, a thread an atom of the bin order: within its bin (half an
// atom on average) an atom comes after those of a smaller number, so that the
// order does not depend on the threads.  Also clears the build's sizes and
// writes those that the columns give, with the positions that have no key (the
// bin past the grid).  With `frames`, the columns of a batch.
template <bool BATCH>
__global__ void nb_places(int nsorted_max, int ncol, const int32_t *__restrict__ bin_start, int nvalid_bins,
                          const int32_t *__restrict__ sorted, const int32_t *__restrict__ key, int Nz,
                          const NbFrameDev *__restrict__ frames, const int32_t *__restrict__ atom_frame,
                          const int32_t *__restrict__ group_start, int64_t places_cap,
                          const float4 *__restrict__ atom_xw, const char4 *__restrict__ atom_shift,
                          const int32_t *__restrict__ type, const int32_t *__restrict__ lj_on,
                          int32_t *__restrict__ order, int32_t *__restrict__ place_of,
                          char4 *__restrict__ shift, float4 *__restrict__ xw, int32_t *__restrict__ sizes) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s == 0) {
    const int groups = group_start[ncol];
    for (int k = 0; k < NB_SIZE_COUNT; ++k) sizes[k] = 0;
    sizes[NB_SIZE_GROUPS] = groups;
    sizes[NB_SIZE_PLACES] = groups * NB_GROUP;
    sizes[NB_SIZE_NAN] = bin_start[nvalid_bins + 1] - bin_start[nvalid_bins];
    sizes[NB_SIZE_OVERFLOW] = (int64_t)groups * NB_GROUP > places_cap ? 1 : 0;
  }
  if (s >= nsorted_max) return;
  const int a = sorted[s], k = key[a];
  if (k >= nvalid_bins) {  // positions with no key are in no group
    place_of[a] = -1;
    return;
  }
  int c = k / Nz, b0 = c * Nz;
  if (BATCH) {
    const NbFrameDev &F = frames[atom_frame[a]];
    const int col = (k - F.bin0) / F.Nz;
    c = F.col0 + col;
    b0 = F.bin0 + col * F.Nz;
  }
  const int lo = bin_start[k], hi = bin_start[k + 1];
  int col_rank = lo - bin_start[b0];
  for (int j = lo; j < hi; ++j) col_rank += sorted[j] < a ? 1 : 0;
  int64_t p = (int64_t)group_start[c] * NB_GROUP + col_rank;
  if (p >= places_cap) {
    place_of[a] = -1;
    return;
  }
  order[p] = a;
  place_of[a] = (int32_t)p;
  shift[p] = atom_shift[a];
  float4 v = atom_xw[a];
  // the search reads place, atom and whether its type has LJ terms together
  v.w = __int_as_float(a | (lj_on && lj_on[type[a]] != 0 ? NB_ATOM_LJ : 0));
  xw[p] = v;
}

// The f32 distance of the pair test, the same for both orders of the pair:
// d = (x_B + s L) - x_A with A the atom of the smaller number and s the
// image of B relative to A; products and sums rounded one at a time.
__device__ __forceinline__ float nb_pair_r2(float4 xa, float4 xb, float sx, float sy, float sz) {
  float dx = __fsub_rn(__fadd_rn(xb.x, sx), xa.x);
  float dy = __fsub_rn(__fadd_rn(xb.y, sy), xa.y);
  float dz = __fsub_rn(__fadd_rn(xb.z, sz), xa.z);
  return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

struct SearchParams {
  float Lx, Ly, Lz;
  float bx, cx, cy;  // the tilts of a triclinic cell (TRI), else 0
  float wx, wy, inv_hz;
  int Nx, Ny, Nz;
  float R2f;     // (float)(R'^2)
  float Rbox;    // R' plus a margin, for the conservative box and window tests
  int64_t groups_cap;
  int64_t list_cap;
  int lj;  // 1: the entries of a partner with LJ terms first; 0: as found, every partner with them; -1: none with them
};

// A coordinate no position comes near: an empty member place lies beyond
// any reach of every candidate (its square stays finite in f32).
#define NB_NOWHERE 1e18f

// W warps build the list of one group (W = 1: a warp a group, four groups
// a block; W = 4: a block a group).
//
// The window.  A lane takes one (column, image) of the window around the
// group's box and finds the run of places of that column that can lie within
// the reach: the columns are sorted by z bin, so the height the reach leaves
// at the column's distance in x and y gives the run from two bin starts, with
// no look at the places.  The runs of 32 such lanes are laid end to end (a
// warp scan) and cut into chunks of 32 candidates, so no lane waits for the
// longest run and a column's far places are never read.
//
// The tests.  A lane takes one candidate place against the group's box;
// those that pass wait in a queue in window order, and whole warps of them
// run the 16 member tests.  With P.lj == 1 (no pruned reach) the entries of a
// partner with Lennard-Jones terms go to the front of the row and the others
// to its back, last one lowest, moved down when the list is done: the order
// the adjoint's rounds ask for, without a pass of its own over the lists
// (320 µs for the 1.07 M-atom box, 18 µs for 900 atoms).  With W = 4 a chunk is 128 candidates, the
// queue is the block's, and counts of the four warps keep the order, so a
// list is the same for every W.
//
// What bounds it: the member tests' arithmetic (16 tests of 8 operations, each
// rounded once, packed in pairs, for about two thirds of the candidates); a
// chunk's place loads are issued two chunks at a time.  Reading whole columns of groups, their
// boxes, then their places one pair of groups at a time took 3,350 µs for the
// 1.07 M-atom box at 1.0 nm and 27 ms at 1.6 nm; this takes 631 and 1,570.
template <int W, bool BATCH, bool TRI = false>
__global__ void __launch_bounds__(128) nb_search_t(SearchParams P0, const NbFrameDev *__restrict__ frames,
                                                   const int32_t *__restrict__ group_frame,
                                                   const int32_t *sizes_in,
                                                   const int32_t *__restrict__ order,
                                                   const float4 *__restrict__ xw,
                                                   const int32_t *__restrict__ group_start,
                                                   const int32_t *__restrict__ bin_start,
                                                   const int32_t *__restrict__ excl_off,
                                                   const int32_t *__restrict__ excl,
                                                   int2 *__restrict__ slab, int32_t *__restrict__ counts,
                                                   int32_t *__restrict__ counts_lj, int32_t *sizes) {
  constexpr int GPB = 4 / W;       // groups per block
  constexpr int CHUNK = 32 * W;    // candidates a step
  constexpr int QCAP = 2 * CHUNK;  // the queue (a step adds at most CHUNK to fewer than CHUNK)
  __shared__ float4 s_qx[GPB][QCAP];  // the queue: the place's position, its atom in w
  __shared__ int2 s_qi[GPB][QCAP];    // and the place and the image code
  __shared__ float4 s_run[4][32];     // a warp's runs: the image's shift, its code in w
  __shared__ int2 s_runp[4][32];      // and its first place less its offset, and the offset
  __shared__ float4 s_mem[GPB][NB_GROUP];  // the members, the atom in w
  // members m and m + 8 side by side for the packed tests: (x, x', y, y'), (z, z')
  __shared__ float4 s_mxy[GPB][NB_GROUP / 2];
  __shared__ float2 s_mz[GPB][NB_GROUP / 2];
  __shared__ int s_raw[GPB][NB_EXCL_MAX], s_key[GPB][NB_EXCL_MAX];  // exclusions: partner * 16 + member
  __shared__ int s_meta[GPB][4];  // nkeys, wide, kmin, kmax
  __shared__ int s_kept[W], s_has[W];
  const unsigned FULL = 0xffffffffu;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int u = lane & 15, half = lane >> 4;
  const int gi = warp / W, part = warp % W;
  const unsigned below = (1u << lane) - 1u;
  const int64_t g = (int64_t)blockIdx.x * GPB + gi;
  // W = 4: the same for the whole block; W = 1: for the warp
  if (g >= sizes_in[NB_SIZE_GROUPS] || g >= P0.groups_cap) return;
  auto sync = [&]() {
    if (W > 1)
      __syncthreads();
    else
      __syncwarp();
  };
  // a frame of a batch: its cell, grid, reach, first column and first bin
  SearchParams P = P0;
  int col0 = 0, bin0 = 0;
  if (BATCH) {
    const NbFrameDev &F = frames[group_frame[g]];
    P.Lx = F.Lf0;
    P.Ly = F.Lf1;
    P.Lz = F.Lf2;
    P.wx = F.wx;
    P.wy = F.wy;
    P.inv_hz = F.inv_hz;
    P.Nx = F.Nx;
    P.Ny = F.Ny;
    P.Nz = F.Nz;
    P.R2f = F.R2f;
    P.Rbox = F.Rbox;
    col0 = F.col0;
    bin0 = F.bin0;
  }

  // the members and their box, in every warp of the group
  const int ai = order[g * NB_GROUP + u];
  float4 xi = ai >= 0 ? xw[g * NB_GROUP + u] : make_float4(NB_NOWHERE, NB_NOWHERE, NB_NOWHERE, 0.f);
  xi.w = __int_as_float(ai);
  float3 lo, hi;
  nb_live_box(xi, ai >= 0, lo, hi);
  // the exclusion partners of the members: keys (partner atom, member),
  // sorted; by the first warp of the group
  if (part == 0) {
    if (half == 0) s_mem[gi][u] = xi;
    const float ox = __shfl_sync(FULL, xi.x, lane + 8), oy = __shfl_sync(FULL, xi.y, lane + 8);
    const float oz = __shfl_sync(FULL, xi.z, lane + 8);
    if (lane < NB_GROUP / 2) {
      s_mxy[gi][lane] = make_float4(xi.x, ox, xi.y, oy);
      s_mz[gi][lane] = make_float2(xi.z, oz);
    }
    int rs = 0, re = 0;
    if (excl_off && half == 0 && ai >= 0) {
      rs = excl_off[ai];
      re = excl_off[ai + 1];
    }
    int cnt = re - rs;
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y;
    }
    int nkeys = __shfl_sync(FULL, incl, 31);
    bool wide = nkeys > NB_EXCL_MAX;
    if (!wide) {
      int at = incl - cnt;
      for (int k = 0; k < cnt; ++k) s_raw[gi][at + k] = excl[rs + k] * NB_GROUP + u;
    } else if (lane == 0) {
      atomicAdd(&sizes[NB_SIZE_EXCL_WIDE], 1);
    }
    __syncwarp();
    int kmin = INT_MAX, kmax = INT_MIN;
    if (!wide) {
      // rank sort of the keys (atom numbers stay below 2^26: they fit)
      for (int k = lane; k < nkeys; k += 32) {
        const int kv = s_raw[gi][k];
        int r = 0;
        for (int t = 0; t < nkeys; ++t) {
          const int tv = s_raw[gi][t];
          r += (tv < kv) || (tv == kv && t < k);
        }
        s_key[gi][r] = kv;
        kmin = min(kmin, kv / NB_GROUP);
        kmax = max(kmax, kv / NB_GROUP);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        kmin = min(kmin, __shfl_xor_sync(FULL, kmin, o));
        kmax = max(kmax, __shfl_xor_sync(FULL, kmax, o));
      }
    }
    if (lane == 0) {
      s_meta[gi][0] = nkeys;
      s_meta[gi][1] = wide;
      s_meta[gi][2] = kmin;
      s_meta[gi][3] = kmax;
    }
  }
  sync();
  const int nkeys = s_meta[gi][0];
  const bool wide = s_meta[gi][1] != 0;
  const int kmin = s_meta[gi][2], kmax = s_meta[gi][3];
  NbCell H;
  H.ax = P.Lx;
  H.by = P.Ly;
  H.cz = P.Lz;
  H.bx = P.bx;
  H.cx = P.cx;
  H.cy = P.cy;
  const float Rb2 = P.Rbox * P.Rbox;
  int2 *const row = slab + g * P.list_cap;
  float4 *const qx = s_qx[gi];
  int2 *const qi = s_qi[gi];
  int qh = 0, qn = 0;  // the queue's first entry and size (the same in every warp of the group)
  int front = 0, back = 0;  // entries written from the row's start, and from its end

  // The member tests of the first `take` places of the queue, a lane each
  // (warp `part` takes the part-th 32 of them), in queue order.
  auto drain = [&](int take) {
    unsigned mask = 0;
    int pj = 0, code = 0;
    const int k = 32 * part + lane;
    const bool on = k < take;
    float4 xj = make_float4(0.f, 0.f, 0.f, 0.f);
    if (on) {
      int2 e = qi[(qh + k) & (QCAP - 1)];
      xj = qx[(qh + k) & (QCAP - 1)];
      pj = e.x;
      code = e.y;
    }
    const int home = nb_image_code(0, 0, 0);
    int sx, sy, sz;
    nb_decode_image(on ? code : home, sx, sy, sz);
    const float3 t = nb_lattice_shift(sx, sy, sz, H);
    // x_j + s L - x_m, two members at a time in packed f32x2 arithmetic (each
    // difference, product and sum rounded once, as nb_pair_r2's).  In the
    // home cell the two orientations of the canonical distance differ in sign
    // alone, so this is it.  Through an image it is within `slack` of it: what
    // lies that near the reach is tested again in the canonical orientation.
    const float ix = __fadd_rn(xj.x, t.x), iy = __fadd_rn(xj.y, t.y), iz = __fadd_rn(xj.z, t.z);
    const float2 nx = make_float2(-ix, -ix), ny = make_float2(-iy, -iy), nz = make_float2(-iz, -iz);
    auto tests = [&](float limit) {
      unsigned in = 0;
#pragma unroll
      for (int m = 0; m < NB_GROUP / 2; ++m) {
        const float4 a = s_mxy[gi][m];
        const float2 dx = __fadd2_rn(make_float2(a.x, a.y), nx), dy = __fadd2_rn(make_float2(a.z, a.w), ny);
        const float2 dz = __fadd2_rn(s_mz[gi][m], nz);
        const float2 r2 = __fadd2_rn(__fadd2_rn(__fmul2_rn(dx, dx), __fmul2_rn(dy, dy)), __fmul2_rn(dz, dz));
        in |= r2.x <= limit ? (1u << m) : 0u;
        in |= r2.y <= limit ? (1u << (m + 8)) : 0u;
      }
      return in;
    };
    mask = tests(P.R2f);
    if (__ballot_sync(FULL, on && code != home) != 0u) {
      const float slack = 4e-6f * P.Rbox * (H.ax + H.by + H.cz + fabsf(H.bx) + fabsf(H.cx) + fabsf(H.cy));
      unsigned doubt = tests(P.R2f + slack) & ~tests(P.R2f - slack);
      if (!on || code == home) doubt = 0;
      const int aj = __float_as_int(xj.w) & NB_ATOM_BITS;
      while (doubt) {
        const int m = __ffs(doubt) - 1;
        doubt &= doubt - 1;
        const float4 xm = s_mem[gi][m];
        // canonical orientation: A the smaller atom number, d = (x_B + s L) - x_A
        const bool jfirst = aj < __float_as_int(xm.w);
        const float sgn = jfirst ? -1.f : 1.f;
        const float r2 = nb_pair_r2(jfirst ? xj : xm, jfirst ? xm : xj, sgn * t.x, sgn * t.y, sgn * t.z);
        mask = r2 <= P.R2f ? mask | (1u << m) : mask & ~(1u << m);
      }
    }
    if (!on) mask = 0;
    if ((pj >> 4) == (int)g) mask &= (1u << (pj & 15)) - 1u;  // inside the group, each pair once
    if (mask) {
      const int aj = __float_as_int(xj.w) & NB_ATOM_BITS;
      if (!wide) {
        if (nkeys > 0 && aj >= kmin && aj <= kmax) {
          int lo_i = 0, hi_i = nkeys;
          while (lo_i < hi_i) {
            int mid = (lo_i + hi_i) >> 1;
            if (s_key[gi][mid] < aj * NB_GROUP) lo_i = mid + 1; else hi_i = mid;
          }
          for (int e = lo_i; e < nkeys && s_key[gi][e] / NB_GROUP == aj; ++e)
            mask &= ~(1u << (s_key[gi][e] & (NB_GROUP - 1)));
        }
      } else {
        unsigned mm = mask;
        while (mm) {
          int m = __ffs(mm) - 1;
          mm &= mm - 1;
          int am = __float_as_int(s_mem[gi][m].w);
          for (int e = excl_off[am]; e < excl_off[am + 1]; ++e)
            if (excl[e] == aj) mask &= ~(1u << m);
        }
      }
    }
    const bool first = P.lj != 1 || (__float_as_int(xj.w) & NB_ATOM_LJ) != 0;
    const unsigned has = __ballot_sync(FULL, mask != 0), hf = __ballot_sync(FULL, mask != 0 && first);
    const unsigned hb = has & ~hf;
    int at = first ? front + __popc(hf & below) : back + __popc(hb & below);
    if (W > 1) {
      if (lane == 0) s_has[part] = __popc(hf) | (__popc(hb) << 16);
      sync();
#pragma unroll
      for (int w = 0; w < W; ++w) {
        const int f = s_has[w] & 0xffff, r = s_has[w] >> 16;
        if (w < part) at += first ? f : r;
        front += f;
        back += r;
      }
    } else {
      front += __popc(hf);
      back += __popc(hb);
      __syncwarp();
    }
    if (!first) at = (int)P.list_cap - 1 - at;
    if (mask && at >= 0 && at < P.list_cap) row[at] = make_int2(pj, (int)(mask | ((unsigned)code << 16)));
    qh = (qh + take) & (QCAP - 1);
    qn -= take;
  };

  // The places that pass the test against the group's box into the queue, in
  // candidate order; a full chunk of the queue is drained.
  auto push = [&](bool valid, int p, float4 xj, float4 run) {
    bool keep = false;
    if (valid) {
      const float xs = xj.x + run.x, ys = xj.y + run.y, zs = xj.z + run.z;
      const float gx = fmaxf(fmaxf(lo.x - xs, xs - hi.x), 0.f);
      const float gy = fmaxf(fmaxf(lo.y - ys, ys - hi.y), 0.f);
      const float gz = fmaxf(fmaxf(lo.z - zs, zs - hi.z), 0.f);
      keep = gx * gx + gy * gy + gz * gz <= Rb2;
    }
    const unsigned kb = __ballot_sync(FULL, keep);
    int at = qh + qn + __popc(kb & below);
    if (W > 1) {
      if (lane == 0) s_kept[part] = __popc(kb);
      sync();
#pragma unroll
      for (int w = 0; w < W; ++w) {
        if (w < part) at += s_kept[w];
        qn += s_kept[w];
      }
    } else {
      qn += __popc(kb);
    }
    if (keep) {
      qx[at & (QCAP - 1)] = xj;
      qi[at & (QCAP - 1)] = make_int2(p, __float_as_int(run.w));
    }
    sync();  // the queue is written (and s_kept read) before the drain and the next push
    if (qn >= CHUNK) drain(CHUNK);
  };

  // 32 columns of the window (one a lane; `on` marks those in it) seen
  // through the image t: their runs of places, laid end to end.
  auto columns = [&](bool on, int cx, int cy, float3 t, int code) {
    int p0 = 0, len = 0;
    if (on) {
      const int c = col0 + cy * P.Nx + cx;
      const int gs = group_start[c];
      if (group_start[c + 1] > (int)g) {
        // the column's distance from the group's box in x and y leaves the
        // height the reach can take in z (the margin of Rbox covers the
        // rounding of the columns' edges)
        const float x0 = cx * P.wx + t.x, y0 = cy * P.wy + t.y;
        const float dx = fmaxf(fmaxf(x0 - hi.x, lo.x - (x0 + P.wx)), 0.f);
        const float dy = fmaxf(fmaxf(y0 - hi.y, lo.y - (y0 + P.wy)), 0.f);
        const float z2 = Rb2 - dx * dx - dy * dy;
        if (z2 >= 0.f) {
          const float zr = sqrtf(z2);
          const float z0 = lo.z - zr - t.z, z1 = hi.z + zr - t.z;
          if (z1 >= 0.f && z0 <= P.Lz) {
            // the bins as nb_keys takes them: (int)(z inv_hz) does not decrease with z
            const int k0 = min(max((int)(z0 * P.inv_hz), 0), P.Nz - 1);
            const int k1 = min(max((int)(z1 * P.inv_hz), 0), P.Nz - 1);
            const int b = bin0 + (c - col0) * P.Nz;
            const int s0 = bin_start[b];
            p0 = max(gs * NB_GROUP + bin_start[b + k0] - s0, (int)g * NB_GROUP);
            const int p1 = min(gs * NB_GROUP + bin_start[b + k1 + 1] - s0, (int)P.groups_cap * NB_GROUP);
            len = max(p1 - p0, 0);
          }
        }
      }
    }
    const unsigned full = __ballot_sync(FULL, len > 0);
    if (full == 0u) return;
    int incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y;
    }
    const int total = __shfl_sync(FULL, incl, 31), runs = __popc(full);
    __syncwarp();
    if (len > 0) {
      const int r = __popc(full & below);
      s_run[warp][r] = make_float4(t.x, t.y, t.z, __int_as_float(code));
      s_runp[warp][r] = make_int2(p0 - (incl - len), incl - len);
    }
    __syncwarp();
    const int off = lane < runs ? s_runp[warp][lane].y : INT_MAX;  // the lane-th run's offset
    // candidate t0 + lane: its run is the last that starts at or before it
    auto find = [&](int t0, bool &valid, int &p, float4 &run) {
      const bool in = off > t0 && off < t0 + 32;
      const unsigned starts = __reduce_or_sync(FULL, in ? 1u << (off - t0) : 0u);
      const int first = __popc(__ballot_sync(FULL, off <= t0)) - 1;
      const int k = (first < 0 ? 0 : first) + __popc(starts & ((2u << lane) - 1u));
      valid = t0 + lane < total;
      p = 0;
      run = s_run[warp][k & 31];
      if (valid) p = s_runp[warp][k].x + t0 + lane;
    };
    for (int t0 = 32 * part; t0 - 32 * part < total; t0 += 2 * CHUNK) {
      bool va, vb;
      int pa, pb;
      float4 ra, rb;
      find(t0, va, pa, ra);
      find(t0 + CHUNK, vb, pb, rb);
      const float4 xa = va ? xw[pa] : make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 xb = vb ? xw[pb] : make_float4(0.f, 0.f, 0.f, 0.f);
      push(va, pa, xa, ra);
      if (t0 - 32 * part + CHUNK < total) push(vb, pb, xb, rb);
    }
  };

  if (!TRI) {
    // orthorhombic: the window of columns around the box, wrapped per axis,
    // each with the images in z that its height cuts
    const int kx0 = (int)floorf((lo.x - P.Rbox) / P.wx), kx1 = (int)floorf((hi.x + P.Rbox) / P.wx);
    const int ky0 = (int)floorf((lo.y - P.Rbox) / P.wy), ky1 = (int)floorf((hi.y + P.Rbox) / P.wy);
    const int sz0 = (lo.z - P.Rbox < 0.f) ? -1 : 0;
    const int sz1 = (hi.z + P.Rbox >= P.Lz) ? 1 : 0;
    const int nz = sz1 - sz0 + 1, nx = kx1 - kx0 + 1, nwin = (ky1 - ky0 + 1) * nx * nz;
    for (int base = 0; base < nwin; base += 32) {
      const int s = base + lane, wi = s / nz;
      const int ky = ky0 + wi / nx, kx = kx0 + wi % nx;
      const int cy = ((ky % P.Ny) + P.Ny) % P.Ny, cx = ((kx % P.Nx) + P.Nx) % P.Nx;
      const int sx = (kx - cx) / P.Nx, sy = (ky - cy) / P.Ny, sz = sz0 + s % nz;
      columns(s < nwin, cx, cy, nb_lattice_shift(sx, sy, sz, H), nb_image_code(sx, sy, sz));
    }
  } else {
    // triclinic: every lattice vector n that can bring a brick position
    // within the reach of the box (along c, then b, then a), each with the
    // brick's columns its window cuts
    const float R = P.Rbox;
    const int nc0 = (int)floorf((lo.z - R) / H.cz), nc1 = (int)floorf((hi.z + R) / H.cz);
    for (int nc = nc0; nc <= nc1; ++nc) {
      const float yc = (float)nc * H.cy, xc = (float)nc * H.cx;
      const int nb0 = (int)floorf((lo.y - R - yc) / H.by), nb1 = (int)floorf((hi.y + R - yc) / H.by);
      for (int nb = nb0; nb <= nb1; ++nb) {
        const float xb = xc + (float)nb * H.bx;
        const int na0 = (int)floorf((lo.x - R - xb) / H.ax), na1 = (int)floorf((hi.x + R - xb) / H.ax);
        for (int na = na0; na <= na1; ++na) {
          const float3 t = nb_lattice_shift(na, nb, nc, H);
          if (hi.z + R - t.z < 0.f || lo.z - R - t.z >= H.cz) continue;
          const int ax0 = max(0, (int)floorf((lo.x - R - t.x) / P.wx));
          const int ax1 = min(P.Nx - 1, (int)floorf((hi.x + R - t.x) / P.wx));
          const int ay0 = max(0, (int)floorf((lo.y - R - t.y) / P.wy));
          const int ay1 = min(P.Ny - 1, (int)floorf((hi.y + R - t.y) / P.wy));
          if (ax0 > ax1 || ay0 > ay1) continue;
          const int nx = ax1 - ax0 + 1, nwin = nx * (ay1 - ay0 + 1);
          for (int base = 0; base < nwin; base += 32) {
            const int s = base + lane;
            columns(s < nwin, ax0 + s % nx, ay0 + s / nx, t, nb_image_code(na, nb, nc));
          }
        }
      }
    }
  }
  sync();  // every warp is past the last drain's counts
  if (qn > 0) drain(qn);
  const int count = front + back, cap = (int)P.list_cap;
  if (back > 0 && count <= cap) {
    // the back entries down behind the front ones, the first of them (at the
    // row's end) first
    const int t = 32 * part + lane, low = cap - back;
    sync();
    if (count <= low) {
      for (int k = t; k < back; k += CHUNK) row[front + k] = row[cap - 1 - k];
    } else {
      // the two stretches overlap: turned round in place, then moved chunk by chunk
      for (int k = t; k < back / 2; k += CHUNK) {
        const int2 a = row[cap - 1 - k], b = row[low + k];
        row[cap - 1 - k] = b;
        row[low + k] = a;
      }
      sync();
      for (int k0 = 0; k0 < back; k0 += CHUNK) {
        const int k = k0 + t;
        const int2 v = k < back ? row[low + k] : make_int2(0, 0);
        sync();
        if (k < back) row[front + k] = v;
        sync();
      }
    }
  }
  if (part == 0 && lane == 0) {
    counts[g] = count;
    if (counts_lj) counts_lj[g] = P.lj < 0 ? 0 : front;
    atomicMax(&sizes[NB_SIZE_LONGEST], count);
    if (count > P.list_cap) atomicOr(&sizes[NB_SIZE_OVERFLOW], 2);
  }
}

// The units of the lists (64 entries each), in group order: the units of
// blocks of NB_SCAN_TILE groups, then a pass in which each block adds the
// units before its own, scans its groups and writes their units.  One block
// takes the second pass alone.  With a gate (a pruning of the MD step),
// nothing unless it is set.  `entries` counts the lists' entries.
__device__ __forceinline__ int nb_group_units(int64_t g, int groups, const int32_t *__restrict__ counts,
                                              int64_t list_cap) {
  return g < groups ? ((int)min((int64_t)counts[g], list_cap) + NB_UNIT - 1) / NB_UNIT : 0;
}

__global__ void __launch_bounds__(NB_SCAN_THREADS) nb_unit_blocks(int64_t groups_cap,
                                                                  const int32_t *__restrict__ sizes,
                                                                  const int32_t *__restrict__ counts,
                                                                  int64_t list_cap, int32_t *__restrict__ block_units,
                                                                  const int *gate) {
  __shared__ int sw[32];
  if (gate && *gate == 0) return;
  const int groups = (int)min((int64_t)sizes[NB_SIZE_GROUPS], groups_cap);
  int n = 0;
#pragma unroll
  for (int k = 0; k < NB_SCAN_PER_THREAD; ++k)
    n += nb_group_units((int64_t)blockIdx.x * NB_SCAN_TILE + k * NB_SCAN_THREADS + threadIdx.x, groups, counts,
                        list_cap);
  int total;
  nb_block_exclusive_scan(n, sw, total);
  if (threadIdx.x == 0) block_units[blockIdx.x] = total;
}

__global__ void __launch_bounds__(NB_SCAN_THREADS) nb_unit_write(
    int64_t groups_cap, const int32_t *__restrict__ sizes, const int32_t *__restrict__ counts, int64_t list_cap,
    const int32_t *__restrict__ block_units, int64_t units_cap, int32_t *__restrict__ unit_start,
    int2 *__restrict__ units, int32_t *sizes_out, int entries, const int *gate, double *prunes) {
  __shared__ int sw[32];
  if (gate && *gate == 0) return;
  const int groups = (int)min((int64_t)sizes[NB_SIZE_GROUPS], groups_cap);
  int at = nb_sum_before(block_units, blockIdx.x, sw);
  int listed = 0;
  for (int k = 0; k < NB_SCAN_PER_THREAD; ++k) {
    const int64_t g0 = (int64_t)blockIdx.x * NB_SCAN_TILE + k * NB_SCAN_THREADS, g = g0 + threadIdx.x;
    if (g0 >= groups) break;  // the same for the block: a small system scans once
    const int n = nb_group_units(g, groups, counts, list_cap);
    int total;
    const int first = at + nb_block_exclusive_scan(n, sw, total);
    at += total;
    if (g < groups) {
      unit_start[g] = first;
      for (int o = 0; o < n; ++o)
        if (first + o < units_cap) units[first + o] = make_int2((int)g, o);
      listed += counts[g];
    }
  }
  if (entries) {
    int total;
    nb_block_exclusive_scan(listed, sw, total);
    if (threadIdx.x == 0 && total > 0) atomicAdd(&sizes_out[NB_SIZE_ENTRIES], total);
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    sizes_out[NB_SIZE_UNITS] = at;
    if (at > units_cap) atomicOr(&sizes_out[NB_SIZE_OVERFLOW], 4);
    unit_start[groups] = at;
    if (prunes) *prunes += 1.0;
  }
}

// The pruning of the dual list (MDIR: emitGroupsPrune,
// lib/Conversion/MDExecToGPU/MDExecToGPU.cpp:9588; docs/neighbor-groups.md,
// Section 6.2): inner mask = outer mask and [r^2 <= R_in'^2] at the current
// frames, entries whose inner mask is empty dropped, the rest written in
// their order (a warp per group, ballot compaction), so that the inner list
// of a group is a deterministic function of the outer one and the frames.
__global__ void __launch_bounds__(128) nb_prune(int64_t groups_cap, const int32_t *__restrict__ sizes,
                                                NbCell H, float rin2, int64_t list_cap,
                                                const int2 *__restrict__ slab, const int32_t *__restrict__ counts,
                                                const int32_t *__restrict__ order, const float4 *__restrict__ xq,
                                                int2 *__restrict__ slab_in, int32_t *__restrict__ counts_in,
                                                const int *gate, const double *__restrict__ x,
                                                double *__restrict__ x_prune) {
  __shared__ float4 s_m[4][NB_GROUP];
  const unsigned FULL = 0xffffffffu;
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int64_t g = (int64_t)blockIdx.x * 4 + warp;
  if (gate && *gate == 0) return;
  if (g >= groups_cap || g >= sizes[NB_SIZE_GROUPS]) return;
  if (x_prune) {
    for (int k = lane; k < 3 * NB_GROUP; k += 32) {
      int a = order[g * NB_GROUP + k / 3];
      if (a >= 0) x_prune[3 * a + k % 3] = x[3 * a + k % 3];
    }
  }
  float4 xme = xq[g * NB_GROUP + (lane & 15)];
  if (lane < NB_GROUP) s_m[warp][lane] = xme;
  bool on = lane < NB_GROUP && order[g * NB_GROUP + (lane & 15)] >= 0;
  unsigned live = __ballot_sync(FULL, on) & 0xffffu;
  float3 box_lo, box_hi;
  nb_live_box(xme, on, box_lo, box_hi);
  const float far2 = rin2 * 1.0001f;
  __syncwarp();
  int cnt = (int)min((int64_t)counts[g], list_cap);
  int out = 0;
  for (int base = 0; base < cnt; base += 32) {
    int e = base + lane;
    unsigned inner = 0;
    int2 en = make_int2(0, 0);
    if (e < cnt) {
      en = slab[g * list_cap + e];
      unsigned mm = (unsigned)en.y & live & 0xffffu;
      int sx, sy, sz;
      nb_decode_image(((unsigned)en.y >> 16) & NB_IMAGE_BITS, sx, sy, sz);
      float4 xj = xq[en.x];
      float3 t = nb_lattice_shift(sx, sy, sz, H);
      float jx = __fadd_rn(xj.x, t.x), jy = __fadd_rn(xj.y, t.y), jz = __fadd_rn(xj.z, t.z);
      if (nb_beyond_box(box_lo, box_hi, jx, jy, jz, far2)) mm = 0;
      while (mm) {
        int m = __ffs(mm) - 1;
        mm &= mm - 1;
        float r2 = nb_prune_r2(s_m[warp][m], jx, jy, jz);
        if (r2 <= rin2) inner |= 1u << m;
      }
    }
    unsigned has = __ballot_sync(FULL, inner != 0);
    if (inner) {
      int at = out + __popc(has & ((1u << lane) - 1));
      slab_in[g * list_cap + at] = make_int2(en.x, (int)(inner | ((unsigned)en.y & 0xffff0000u)));
    }
    out += __popc(has);
  }
  if (lane == 0) counts_in[g] = out;
}

// 8 blocks an SM (64 registers, 8 bytes spilled) rather than the 7 that 66
// registers allowed: the 1,526 groups of the 23,550-atom box take 1.29 waves
// of blocks instead of 1.47 (the MD step 54.45 against 54.70 µs, side by side)
__global__ void __launch_bounds__(NB_PRUNE_WARPS * 32, 8)
    nb_prune_block(int64_t groups_cap, const int32_t *__restrict__ sizes, NbCell H, float rin2,
                   int64_t list_cap, const int2 *__restrict__ slab, const int32_t *__restrict__ counts,
                   const int32_t *__restrict__ order, const float4 *__restrict__ xq, int2 *__restrict__ slab_in,
                   int32_t *__restrict__ counts_in, const int *gate, const double *__restrict__ x,
                   double *__restrict__ x_prune, int32_t *unit_counter, int2 *__restrict__ units,
                   int64_t units_cap, double *prunes) {
  int64_t g = blockIdx.x;
  nb_grid_wait();  // the gate and the frames of the kernels before (a chained launch)
  if (gate && *gate == 0) return;  // no pruning due (decided on the device)
  if (g >= groups_cap || g >= sizes[NB_SIZE_GROUPS]) return;
  nb_prune_group(g, H, rin2, list_cap, slab, counts, order, xq, slab_in, counts_in, x, x_prune, unit_counter, units,
                 units_cap, prunes);
}

inline int blocks_for(int64_t n, int t) { return (int)((n + t - 1) / t > 0 ? (n + t - 1) / t : 1); }

}  // namespace

// Grid of the counting sort: columns of about 16 atoms per column-width of
// height, z bins of about half an atom.
static NbGrid nb_plan_grid(int64_t n, const double box[3]) {
  NbGrid G;
  double V = box[0] * box[1] * box[2];
  double rho = (n > 0 ? (double)n : 1.0) / V;
  double dcol = cbrt((double)NB_GROUP / rho);
  G.Nx = (int)std::min(256.0, std::max(1.0, std::floor(box[0] / dcol)));
  G.Ny = (int)std::min(256.0, std::max(1.0, std::floor(box[1] / dcol)));
  int64_t nz = 2 * n / (G.Nx * G.Ny);
  G.Nz = (int)std::max<int64_t>(1, std::min<int64_t>(nz, 1 << 20));
  G.wx = (float)(box[0] / G.Nx);
  G.wy = (float)(box[1] / G.Ny);
  G.hz = (float)(box[2] / G.Nz);
  return G;
}

#define NB_CHECK(x)                                                  \
  do {                                                               \
    cudaError_t e_ = (x);                                            \
    if (e_ != cudaSuccess) {                                         \
      fprintf(stderr, "mdrt_nb: %s: %s\n", #x, cudaGetErrorString(e_)); \
      return -1;                                                     \
    }                                                                \
  } while (0)

template <typename T>
static int nb_realloc(T *&p, int64_t count) {
  if (p) cudaFree(p);
  p = nullptr;
  if (count <= 0) count = 1;
  cudaError_t e = cudaMalloc((void **)&p, sizeof(T) * (size_t)count);
  return e == cudaSuccess ? 0 : -1;
}

// Sizes the buffers for n atoms, the planned columns and bins
// (c.plan_cols, c.plan_bins) and the list capacity C.  Fresh accumulators
// are cleared on s, the stream of the launches that use them (the null
// stream's memset would not come before those of a non-blocking stream).
static int nb_reserve(NbCtx &c, int64_t list_cap, cudaStream_t s) {
  int64_t n = c.n;
  int64_t cols = c.plan_cols;
  int64_t groups = (n + NB_GROUP - 1) / NB_GROUP + cols;  // at most one partial group a column
  int64_t bins = c.plan_bins + 1;
  if (bins > c.bins_cap) {
    int64_t cap = bins + bins / 4;
    if (nb_realloc(c.bin_count, cap) || nb_realloc(c.bin_start, cap + 1))
      return -1;
    int64_t scr = cap / NB_SCAN_TILE + 8;
    int64_t scr2 = (groups + groups / 4) / NB_SCAN_TILE + 8;
    if (nb_realloc(c.scan_scratch, std::max(scr, std::max<int64_t>(scr2, 64)) + 4096)) return -1;
    c.bins_cap = cap;
  }
  if (cols + 1 > c.cols_cap) {
    int64_t cap = cols + cols / 4 + 1;
    if (nb_realloc(c.group_start, cap + 1)) return -1;
    c.cols_cap = cap;
  }
  bool regroup = groups > c.groups_cap;
  if (regroup) {
    int64_t cap = groups + groups / 4 + 16;
    if (nb_realloc(c.order, cap * NB_GROUP) || nb_realloc(c.shift, cap * NB_GROUP) ||
        nb_realloc(c.xw, cap * NB_GROUP) ||
        nb_realloc(c.counts, cap) || nb_realloc(c.counts_lj, cap) ||
        nb_realloc(c.unit_start, cap + 1) || nb_realloc(c.xq, cap * NB_GROUP) ||
        nb_realloc(c.xq_lo, cap * NB_GROUP) ||
        nb_realloc(c.typ_p, cap * NB_GROUP) || nb_realloc(c.acc, cap * NB_GROUP) ||
        nb_realloc(c.acc_fixed, cap * NB_GROUP * 3))
      return -1;
    if (c.pme.on) {
      if (nb_realloc(c.pme.pme_force, cap * NB_GROUP * 4) || nb_realloc(c.pme.potential, cap * NB_GROUP) ||
          nb_realloc(c.pme.tile_bin, cap * NB_GROUP) || nb_realloc(c.pme.tile_rank, cap * NB_GROUP) ||
          nb_realloc(c.pme.tile_sorted, cap * NB_GROUP))
        return -1;
    }
    NB_CHECK(cudaMemsetAsync(c.acc, 0, sizeof(float4) * cap * NB_GROUP, s));
    NB_CHECK(cudaMemsetAsync(c.acc_fixed, 0, sizeof(unsigned long long) * cap * NB_GROUP * 3, s));
    c.groups_cap = cap;
    c.places_cap = cap * NB_GROUP;
  }
  if (regroup || list_cap != c.list_cap) {
    if (nb_realloc(c.slab, c.groups_cap * list_cap)) return -1;
    c.list_cap = list_cap;
    int64_t units = c.groups_cap * ((list_cap + NB_UNIT - 1) / NB_UNIT);
    if (units > c.units_cap) {
      if (nb_realloc(c.units, units) || nb_realloc(c.unit_partials, units * 8)) return -1;
      c.units_cap = units;
    }
  }
  return 0;
}

static int64_t nb_initial_list_cap(int64_t n, const double box[3], double reach, const NbGrid &G) {
  double V = box[0] * box[1] * box[2];
  double rho = n / V;
  double R = reach + 3e-6 * (box[0] + box[1] + box[2]);
  double hz = NB_GROUP / (rho * G.wx * G.wy);
  double w0 = 0.5 * G.wx, w1 = 0.5 * G.wy, w2 = 0.5 * hz;
  double VR = 8 * w0 * w1 * w2 + 8 * (w0 * w1 + w1 * w2 + w2 * w0) * R +
              2 * M_PI * (w0 + w1 + w2) * R * R + 4.0 / 3.0 * M_PI * R * R * R;
  double est = 0.5 * rho * VR * 1.6 + 64;
  est = std::min(est, (double)n * 27.0 + 64);
  return ((int64_t)est + NB_UNIT - 1) / NB_UNIT * NB_UNIT;
}

// Lets `kernel` take `bytes` of dynamic shared memory on the current device
// beside its static shared memory (the default cap is 48 KB for both
// together); once per device and size.
#define NB_MAX_DEVICES 64
template <typename K>
static void nb_allow_smem(K kernel, size_t bytes, size_t (&configured)[NB_MAX_DEVICES]) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (bytes > 16 * 1024 && dev >= 0 && dev < NB_MAX_DEVICES && configured[dev] < bytes) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    configured[dev] = bytes;
  }
}

// The order of a build's lists by their partners' LJ terms (SearchParams::lj):
// without a pruned reach, and where only some types have any.
static int nb_lj_order(const NbCtx &c) {
  if (c.inner_reach > 0.0) return 0;
  const uint32_t all = c.ntypes >= 32 ? 0xffffffffu : (1u << c.ntypes) - 1u;
  return c.lj_mask == 0 ? -1 : c.lj_mask == all ? 0 : 1;
}

// Four warps a group (else one) for a system of this many groups: with one
// warp each, fewer groups leave the GPU's warp slots empty and a group's
// chunks come one after the other (23,550 atoms at 1.0 nm: 31 µs with four,
// 45 with one; at 1.7 nm 74 and 134); with more, the block's waits cost more
// than they bring (192,000 atoms: 179 and 128; at 1.6 nm 396 and 315;
// 1.07 M: 965 and 631).  72,000 atoms are even (72 and 65).
#define NB_SEARCH_FOUR_GROUPS 4000
static bool nb_search_four(int64_t groups) { return groups < NB_SEARCH_FOUR_GROUPS; }

// The units of the lists `counts` into `units` (nb_unit_write).
static void nb_units_run(NbCtx &c, const int32_t *counts, int32_t *unit_start, int2 *units, int32_t *sizes_out,
                         int entries, const int *gate, double *prunes, cudaStream_t s) {
  const int blocks = blocks_for(c.groups_cap, NB_SCAN_TILE);
  if (blocks > 1)
    nb_unit_blocks<<<blocks, NB_SCAN_THREADS, 0, s>>>(c.groups_cap, c.sizes, counts, c.list_cap, c.scan_scratch, gate);
  nb_unit_write<<<blocks, NB_SCAN_THREADS, 0, s>>>(c.groups_cap, c.sizes, counts, c.list_cap, c.scan_scratch,
                                                   c.units_cap, unit_start, units, sizes_out, entries, gate, prunes);
}

// The columns' first groups: one block up to this many columns, above it a
// count by all of the GPU and a scan, two launches more.  The block's passes of
// 1,024 columns come one after the other (three dependent loads a column):
// 6.3 µs for 4,096 columns and 20.3 for 16,384, in a batch 10.1 for 5,500 and
// 18.7 for 11,000, where the three kernels take 5.3, 8.0, 8.3 and 8.5 beside
// their launches.
#define NB_COLUMNS_ONE_BLOCK 8192
template <bool BATCH>
static void nb_columns_run(NbCtx &c, int ncol, int Nz, const NbFrameDev *frames, const int32_t *col_frame,
                           cudaStream_t s) {
  if (ncol <= NB_COLUMNS_ONE_BLOCK) {
    nb_columns<BATCH><<<1, 1024, 0, s>>>(ncol, Nz, c.bin_start, frames, col_frame, c.group_start);
    return;
  }
  // the counts of the bins are scanned: their buffer takes the columns' (no
  // more columns than bins)
  nb_column_counts<BATCH><<<blocks_for(ncol, 256), 256, 0, s>>>(ncol, Nz, c.bin_start, frames, col_frame, c.bin_count);
  nb_scan(c.bin_count, c.group_start, ncol, nullptr, c.scan_scratch, s);
}

// Launches one build on `s`; the sizes are left in c.sizes (device).  The
// chain is nine launches and two memsets (keys, scan, scatter, columns, places,
// search, units), two fewer where a block takes a scan alone: the small
// kernels of a build are each a launch's latency, and 24 of them took as
// long as the search for 900 atoms.
static void nb_build_launch(NbCtx &c, const double *x, const double box[3], bool keep_x, cudaStream_t s) {
  const NbGrid &G = c.grid;
  int64_t n = c.n;
  int nbins = G.nbins();
  cudaMemsetAsync(c.bin_count, 0, sizeof(int32_t) * (nbins + 1), s);
  cudaMemsetAsync(c.order, 0xff, sizeof(int32_t) * c.places_cap, s);
  nb_keys<<<blocks_for(n, 256), 256, 0, s>>>(n, x, box[0], box[1], box[2], c.tilt[0], c.tilt[1], c.tilt[2],
                                            G.Nx, G.Ny, G.Nz,
                                            1.0f / G.wx, 1.0f / G.wy, 1.0f / G.hz, c.key, c.rank,
                                            c.bin_count, c.atom_xw, c.atom_shift, keep_x ? c.x_build : nullptr);
  nb_scan(c.bin_count, c.bin_start, nbins + 1, nullptr, c.scan_scratch, s);
  nb_scatter<<<blocks_for(n, 256), 256, 0, s>>>(n, c.key, c.rank, c.bin_start, c.sorted);
  nb_columns_run<false>(c, G.ncol(), G.Nz, nullptr, nullptr, s);
  nb_places<false><<<blocks_for(n, 256), 256, 0, s>>>((int)n, G.ncol(), c.bin_start, nbins, c.sorted, c.key, G.Nz, nullptr,
                                                     nullptr, c.group_start, c.places_cap, c.atom_xw, c.atom_shift,
                                                     c.type, nb_lj_order(c) == 1 ? c.lj_on : nullptr, c.order,
                                                     c.place_of, c.shift, c.xw, c.sizes);
  SearchParams P;
  P.Lx = (float)box[0];
  P.Ly = (float)box[1];
  P.Lz = (float)box[2];
  P.bx = (float)c.tilt[0];
  P.cx = (float)c.tilt[1];
  P.cy = (float)c.tilt[2];
  P.wx = G.wx;
  P.wy = G.wy;
  P.inv_hz = 1.0f / G.hz;
  P.Nx = G.Nx;
  P.Ny = G.Ny;
  P.Nz = G.Nz;
  // the widening: 3e-6 of the sum of the diagonal and the tilts' magnitudes
  double span = box[0] + box[1] + box[2] + fabs(c.tilt[0]) + fabs(c.tilt[1]) + fabs(c.tilt[2]);
  double Rw = c.reach + 3e-6 * span;
  P.R2f = (float)(Rw * Rw);
  P.Rbox = (float)(Rw + 2e-5 * span + 1e-6);
  P.groups_cap = c.groups_cap;
  P.list_cap = c.list_cap;
  P.lj = nb_lj_order(c);
  const bool four = nb_search_four((n + NB_GROUP - 1) / NB_GROUP);
  const int blocks = four ? (int)c.groups_cap : blocks_for(c.groups_cap, 4);
  auto kernel = nb_triclinic(c) ? (four ? nb_search_t<4, false, true> : nb_search_t<1, false, true>)
                                : (four ? nb_search_t<4, false> : nb_search_t<1, false>);
  kernel<<<blocks, 128, 0, s>>>(P, nullptr, nullptr, c.sizes, c.order, c.xw, c.group_start, c.bin_start, c.excl_off,
                                c.excl, c.slab, c.counts, c.counts_lj, c.sizes);
  nb_units_run(c, c.counts, c.unit_start, c.units, c.sizes, 1, nullptr, nullptr, s);
}

void nb_build_launch_public(NbCtx &c, const double *x, const double box[3], cudaStream_t s) {
  nb_build_launch(c, x, box, false, s);  // the build of record is the host's last
}

int nb_reserve_inner(NbCtx &c, cudaStream_t s) {
  // the inner buffers follow the outer capacities
  int64_t G = c.groups_cap, C = c.list_cap, U = c.units_cap;
  c.slab_in_entries = 0;
  if (nb_realloc(c.slab_in, G * C) || nb_realloc(c.counts_in, G) ||
      nb_realloc(c.unit_start_in, G + 1) || nb_realloc(c.units_in, U))
    return -1;
  c.slab_in_entries = G * C;
  if (!c.sizes_in) {
    if (cudaMalloc(&c.sizes_in, sizeof(int32_t) * NB_SIZE_COUNT) != cudaSuccess) return -1;
  }
  if (cudaMemsetAsync(c.sizes_in, 0, sizeof(int32_t) * NB_SIZE_COUNT, s) != cudaSuccess) return -1;
  c.inner_valid = false;
  return 0;
}

void nb_prune_run(NbCtx &c, const double box[3], cudaStream_t s) {
  double Rw = c.inner_reach + 3e-6 * (box[0] + box[1] + box[2] + fabs(c.tilt[0]) + fabs(c.tilt[1]) + fabs(c.tilt[2]));
  size_t stage = sizeof(int2) * (size_t)c.list_cap;
  if (stage <= 200 * 1024) {
    static size_t configured[NB_MAX_DEVICES] = {};
    nb_allow_smem(nb_prune_block, stage, configured);
    nb_prune_block<<<(int)c.groups_cap, NB_PRUNE_WARPS * 32, stage, s>>>(
        c.groups_cap, c.sizes, nb_cell(c, box), (float)(Rw * Rw), c.list_cap, c.slab,
        c.counts, c.order, c.xq, c.slab_in, c.counts_in, nullptr, nullptr, nullptr, nullptr, nullptr, 0, nullptr);
  } else {
    nb_prune<<<blocks_for(c.groups_cap, 4), 128, 0, s>>>(c.groups_cap, c.sizes, nb_cell(c, box),
                                                        (float)(Rw * Rw), c.list_cap, c.slab,
                                                        c.counts, c.order, c.xq, c.slab_in, c.counts_in, nullptr,
                                                        nullptr, nullptr);
  }
  nb_units_run(c, c.counts_in, c.unit_start_in, c.units_in, c.sizes_in, 0, nullptr, nullptr, s);
}

void nb_prune_gated(NbCtx &c, const double box[3], const int *gate, const double *x, double *x_prune,
                    double *prunes, int32_t *unit_counter, cudaStream_t s) {
  double Rw = c.inner_reach + 3e-6 * (box[0] + box[1] + box[2] + fabs(c.tilt[0]) + fabs(c.tilt[1]) + fabs(c.tilt[2]));
  size_t stage = sizeof(int2) * (size_t)c.list_cap;
  if (stage <= 200 * 1024) {
    static size_t configured[NB_MAX_DEVICES] = {};
    nb_allow_smem(nb_prune_block, stage, configured);
    // outside the deterministic mode the blocks claim their units themselves
    // (the counter is zeroed by the update that asked for the pruning)
    bool claim = !c.deterministic && unit_counter;
    nb_launch_chained(nb_prune_block, dim3((int)c.groups_cap), dim3(NB_PRUNE_WARPS * 32), stage, s, c.groups_cap,
                      c.sizes, nb_cell(c, box), (float)(Rw * Rw), c.list_cap, c.slab,
                      c.counts, c.order, c.xq, c.slab_in, c.counts_in, gate, x, x_prune,
                      claim ? unit_counter : nullptr, claim ? c.units_in : nullptr, c.units_cap,
                      claim ? prunes : nullptr);
    if (claim) return;
  } else {
    nb_prune<<<blocks_for(c.groups_cap, 4), 128, 0, s>>>(c.groups_cap, c.sizes, nb_cell(c, box),
                                                        (float)(Rw * Rw), c.list_cap, c.slab,
                                                        c.counts, c.order, c.xq, c.slab_in, c.counts_in, gate, x,
                                                        x_prune);
  }
  nb_units_run(c, c.counts_in, c.unit_start_in, c.units_in, c.sizes_in, 0, gate, prunes, s);
}

// One complete build with count-then-grow: the list capacity C grows to a
// quarter more than the longest list and the build runs again until every
// list fits (MDIR: mdrtGroupsGrow, runtime/mdrt_cuda.c:3185, and the build
// loop of lib/Conversion/MDExecToGPU/MDExecToGPU.cpp:10107-10175).
int nb_build_run(NbCtx &c, const double *x, const double box[3], cudaStream_t s) {
  NbGrid G = nb_plan_grid(c.n, box);
  int64_t cap = c.list_cap;
  if (cap == 0) cap = nb_initial_list_cap(c.n, box, c.reach, G);
  c.grid = G;
  c.plan_cols = G.ncol();
  c.plan_bins = G.nbins();
  if (!c.key) {
    if (nb_realloc(c.key, c.n) || nb_realloc(c.sorted, c.n) || nb_realloc(c.atom_xw, c.n) ||
        nb_realloc(c.atom_shift, c.n) || nb_realloc(c.place_of, c.n) || nb_realloc(c.rank, c.n) ||
        nb_realloc(c.x_build, 3 * c.n))
      return -1;
  }
  for (int attempt = 0; attempt < 8; ++attempt) {
    if (nb_reserve(c, cap, s)) return -1;
    nb_build_launch(c, x, box, true, s);
    NB_CHECK(cudaMemcpyAsync(c.h_sizes, c.sizes, sizeof(int32_t) * NB_SIZE_COUNT,
                             cudaMemcpyDeviceToHost, s));
    NB_CHECK(cudaStreamSynchronize(s));
    NB_CHECK(cudaGetLastError());
    if (c.h_sizes[NB_SIZE_OVERFLOW] == 0) {
      c.built = true;
      c.builds++;
      c.lj_part_build = c.inner_reach > 0.0 ? -1 : c.builds;
      c.lj_part_mask = c.lj_mask;
      for (int k = 0; k < 3; ++k) c.box_built[k] = box[k];
      c.inner_valid = false;
      if (c.inner_reach > 0.0) {
        int64_t key = c.groups_cap * 1000003 + c.list_cap * 7 + c.units_cap;
        if (key != c.inner_key || !c.slab_in) {
          if (nb_reserve_inner(c, s)) return -1;
          c.inner_key = key;
        }
      }
      return 0;
    }
    int64_t longest = c.h_sizes[NB_SIZE_LONGEST];
    int64_t want = (longest + longest / 4 + NB_UNIT - 1) / NB_UNIT * NB_UNIT;
    cap = std::max(cap, want);
    c.grows++;
  }
  return -1;
}

namespace {

// Copies the entries of each list from a slab of old_cap entries a group to
// one of new_cap (a thread per entry of the old slab).
__global__ void nb_copy_lists(int64_t groups, const int32_t *__restrict__ sizes, int64_t old_cap, int64_t new_cap,
                              const int32_t *__restrict__ counts, const int2 *__restrict__ src,
                              int2 *__restrict__ dst) {
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t g = t / old_cap, e = t - g * old_cap;
  if (g >= groups || g >= sizes[NB_SIZE_GROUPS]) return;
  if (e >= min((int64_t)counts[g], old_cap)) return;
  dst[g * new_cap + e] = src[g * old_cap + e];
}

}  // namespace

int nb_grow_lists_keep(NbCtx &c, int64_t longest, cudaStream_t s) {
  int64_t want = (longest + longest / 4 + NB_UNIT - 1) / NB_UNIT * NB_UNIT;
  if (want <= c.list_cap || !c.built) return 0;
  int64_t G = c.groups_cap, C0 = c.list_cap;
  int64_t units = G * ((want + NB_UNIT - 1) / NB_UNIT);
  bool inner = c.slab_in != nullptr;
  int2 *slab = nullptr, *slab_in = nullptr, *units_new = nullptr, *units_in = nullptr;
  double *partials = nullptr;
  auto fail = [&]() {
    for (void *p : {(void *)slab, (void *)slab_in, (void *)units_new, (void *)units_in, (void *)partials})
      if (p) cudaFree(p);
    return -1;
  };
  if (cudaMalloc(&slab, sizeof(int2) * G * want) != cudaSuccess) return fail();
  if (inner && cudaMalloc(&slab_in, sizeof(int2) * G * want) != cudaSuccess) return fail();
  if (units > c.units_cap) {
    if (cudaMalloc(&units_new, sizeof(int2) * units) != cudaSuccess ||
        cudaMalloc(&partials, sizeof(double) * 8 * units) != cudaSuccess)
      return fail();
    if (inner && cudaMalloc(&units_in, sizeof(int2) * units) != cudaSuccess) return fail();
  }
  int blocks = blocks_for(G * C0, 256);
  nb_copy_lists<<<blocks, 256, 0, s>>>(G, c.sizes, C0, want, c.counts, c.slab, slab);
  if (inner) nb_copy_lists<<<blocks, 256, 0, s>>>(G, c.sizes, C0, want, c.counts_in, c.slab_in, slab_in);
  if (units_new) {
    cudaMemcpyAsync(units_new, c.units, sizeof(int2) * c.units_cap, cudaMemcpyDeviceToDevice, s);
    if (inner) cudaMemcpyAsync(units_in, c.units_in, sizeof(int2) * c.units_cap, cudaMemcpyDeviceToDevice, s);
  }
  NB_CHECK(cudaStreamSynchronize(s));
  NB_CHECK(cudaGetLastError());
  cudaFree(c.slab);
  c.slab = slab;
  if (inner) {
    cudaFree(c.slab_in);
    c.slab_in = slab_in;
    c.slab_in_entries = G * want;
  }
  if (units_new) {
    cudaFree(c.units);
    cudaFree(c.unit_partials);
    c.units = units_new;
    c.unit_partials = partials;
    if (inner) {
      cudaFree(c.units_in);
      c.units_in = units_in;
    }
    c.units_cap = units;
  }
  c.list_cap = want;
  c.inner_key = c.groups_cap * 1000003 + c.list_cap * 7 + c.units_cap;
  c.grows++;
  return 0;
}

int nb_grow_lists(NbCtx &c, int64_t longest) {
  int64_t want = (longest + longest / 4 + NB_UNIT - 1) / NB_UNIT * NB_UNIT;
  if (want <= c.list_cap) return 0;
  c.grows++;
  return nb_reserve(c, want, nullptr);  // the groups stay: nothing is cleared
}

// ---------------------------------------------------------------------------
// The build of a batch of frames (mdrtNbBatch).  The same stages as one
// system's, each one launch over all frames: the bins and columns of frame
// f start at F.bin0 and F.col0, so that the counting sort, the scans and
// the groups are those of one grid laid end to end, and the search of a
// group reads its frame's cell, grid and reach.

namespace {

__global__ void nb_batch_keys(int64_t n, const double *__restrict__ x, const int32_t *__restrict__ atom_frame,
                              const NbFrameDev *__restrict__ frames, int nbins, int32_t *__restrict__ key,
                              int32_t *__restrict__ rank, int32_t *__restrict__ bin_count,
                              float4 *__restrict__ atom_xw, char4 *__restrict__ atom_shift) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const NbFrameDev &F = frames[atom_frame[i]];
  double v0 = x[3 * i], v1 = x[3 * i + 1], v2 = x[3 * i + 2];
  bool ok = isfinite(v0) && isfinite(v1) && isfinite(v2);
  double S0 = 0, S1 = 0, S2 = 0;
  if (ok) {
    S0 = -floor(v0 / F.L0);
    S1 = -floor(v1 / F.L1);
    S2 = -floor(v2 / F.L2);
    ok = fabs(S0) <= 100.0 && fabs(S1) <= 100.0 && fabs(S2) <= 100.0;
  }
  if (!ok) {
    key[i] = nbins;
    rank[i] = atomicAdd(&bin_count[nbins], 1);
    atom_xw[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    atom_shift[i] = make_char4(0, 0, 0, 0);
    return;
  }
  float w0 = (float)(v0 + S0 * F.L0), w1 = (float)(v1 + S1 * F.L1), w2 = (float)(v2 + S2 * F.L2);
  int kx = min(max((int)(w0 * F.inv_wx), 0), F.Nx - 1);
  int ky = min(max((int)(w1 * F.inv_wy), 0), F.Ny - 1);
  int kz = min(max((int)(w2 * F.inv_hz), 0), F.Nz - 1);
  int col = ky * F.Nx + kx;
  int k = F.bin0 + col * F.Nz + kz;
  key[i] = k;
  rank[i] = atomicAdd(&bin_count[k], 1);
  atom_xw[i] = make_float4(w0, w1, w2, 1.f);
  atom_shift[i] = make_char4((signed char)S0, (signed char)S1, (signed char)S2, 0);
}

// Each group's frame and its frame's cell, a thread a column.
__global__ void nb_batch_group_frames(int ncol, const int32_t *__restrict__ group_start, int64_t groups_cap,
                                      const int32_t *__restrict__ col_frame, const NbFrameDev *__restrict__ frames,
                                      int32_t *__restrict__ group_frame, float4 *__restrict__ group_L) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncol) return;
  const int f = col_frame[c];
  const float4 L = make_float4(frames[f].Lf0, frames[f].Lf1, frames[f].Lf2, 0.f);
  for (int g = group_start[c]; g < group_start[c + 1] && g < groups_cap; ++g) {
    group_frame[g] = f;
    group_L[g] = L;
  }
}

// The units of frame f: [frame_units[2f], frame_units[2f + 1]).
__global__ void nb_batch_frame_units(int nframes, const NbFrameDev *__restrict__ frames,
                                     const int32_t *__restrict__ group_start, const int32_t *__restrict__ unit_start,
                                     int32_t *__restrict__ frame_units) {
  int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nframes) return;
  const NbFrameDev &F = frames[f];
  int g0 = group_start[F.col0], g1 = group_start[F.col0 + F.ncol];
  frame_units[2 * f] = unit_start[g0];
  frame_units[2 * f + 1] = unit_start[g1];
}

}  // namespace

// The grids of the frames (host): columns and bins end to end, the widened
// reach of each cell; uploads the frames and the column -> frame map.
static int nb_batch_plan(mdrtNbBatch &b, int64_t *list_cap_hint) {
  NbCtx &c = b.nb->c;
  int64_t bins = 0, cols = 0, cap = 0;
  std::vector<int32_t> col_frame;
  for (int f = 0; f < b.frames; ++f) {
    NbFrameDev &F = b.h_frames[f];
    const double *L = &b.h_boxes[3 * f];
    int64_t nf = b.atom0[f + 1] - b.atom0[f];
    NbGrid G = nb_plan_grid(std::max<int64_t>(nf, 1), L);
    F.L0 = L[0];
    F.L1 = L[1];
    F.L2 = L[2];
    F.Lf0 = (float)L[0];
    F.Lf1 = (float)L[1];
    F.Lf2 = (float)L[2];
    F.Nx = G.Nx;
    F.Ny = G.Ny;
    F.Nz = G.Nz;
    F.wx = G.wx;
    F.wy = G.wy;
    F.inv_wx = 1.0f / G.wx;
    F.inv_wy = 1.0f / G.wy;
    F.inv_hz = 1.0f / G.hz;
    F.bin0 = (int)bins;
    F.col0 = (int)cols;
    F.ncol = G.ncol();
    F.atom0 = (int)b.atom0[f];
    F.natoms = (int)nf;
    double Rw = c.reach + 3e-6 * (L[0] + L[1] + L[2]);
    F.R2f = (float)(Rw * Rw);
    F.Rbox = (float)(Rw + 2e-5 * (L[0] + L[1] + L[2]) + 1e-6);
    F.pref = c.coulomb / (M_PI * L[0] * L[1] * L[2]);
    F.pi2_beta2 = c.beta > 0 ? M_PI * M_PI / (c.beta * c.beta) : 0.0;
    bins += G.nbins();
    cols += G.ncol();
    col_frame.insert(col_frame.end(), G.ncol(), f);
    cap = std::max(cap, nb_initial_list_cap(std::max<int64_t>(nf, 1), L, c.reach, G));
  }
  if (bins >= (1ll << 31) - 2 || cols >= (1ll << 31) - 2) return -1;
  c.plan_cols = cols;
  c.plan_bins = bins;
  if (list_cap_hint) *list_cap_hint = cap;
  if (!b.frames_dev && nb_realloc(b.frames_dev, b.frames)) return -1;
  NB_CHECK(cudaMemcpy(b.frames_dev, b.h_frames.data(), sizeof(NbFrameDev) * b.frames, cudaMemcpyHostToDevice));
  if (cols > b.cols_alloc) {
    if (nb_realloc(b.col_frame, cols)) return -1;
    b.cols_alloc = cols;
  }
  NB_CHECK(cudaMemcpy(b.col_frame, col_frame.data(), sizeof(int32_t) * cols, cudaMemcpyHostToDevice));
  return 0;
}

static void nb_batch_build_launch(mdrtNbBatch &b, const double *x, cudaStream_t s) {
  NbCtx &c = b.nb->c;
  int64_t n = c.n;
  int nbins = (int)c.plan_bins;
  int ncol = (int)c.plan_cols;
  cudaMemsetAsync(c.bin_count, 0, sizeof(int32_t) * (nbins + 1), s);
  cudaMemsetAsync(c.order, 0xff, sizeof(int32_t) * c.places_cap, s);
  nb_batch_keys<<<blocks_for(n, 256), 256, 0, s>>>(n, x, b.atom_frame, b.frames_dev, nbins, c.key, c.rank,
                                                  c.bin_count, c.atom_xw, c.atom_shift);
  nb_scan(c.bin_count, c.bin_start, nbins + 1, nullptr, c.scan_scratch, s);
  nb_scatter<<<blocks_for(n, 256), 256, 0, s>>>(n, c.key, c.rank, c.bin_start, c.sorted);
  nb_columns_run<true>(c, ncol, 1, b.frames_dev, b.col_frame, s);
  nb_batch_group_frames<<<blocks_for(ncol, 128), 128, 0, s>>>(ncol, c.group_start, c.groups_cap, b.col_frame,
                                                             b.frames_dev, b.group_frame, b.group_L);
  nb_places<true><<<blocks_for(n, 256), 256, 0, s>>>((int)n, ncol, c.bin_start, nbins, c.sorted, c.key, 1, b.frames_dev,
                                                    b.atom_frame, c.group_start, c.places_cap, c.atom_xw,
                                                    c.atom_shift, c.type, nb_lj_order(c) == 1 ? c.lj_on : nullptr,
                                                    c.order, c.place_of, c.shift, c.xw, c.sizes);
  SearchParams P = {};
  P.groups_cap = c.groups_cap;
  P.list_cap = c.list_cap;
  P.lj = nb_lj_order(c);  // as a single system's lists, so that the f32 sums are the same
  const bool four = b.search_warps ? b.search_warps == 4 : nb_search_four((n + NB_GROUP - 1) / NB_GROUP);
  const int blocks = four ? (int)c.groups_cap : blocks_for(c.groups_cap, 4);
  auto kernel = four ? nb_search_t<4, true> : nb_search_t<1, true>;
  kernel<<<blocks, 128, 0, s>>>(P, b.frames_dev, b.group_frame, c.sizes, c.order, c.xw, c.group_start, c.bin_start,
                                c.excl_off, c.excl, c.slab, c.counts, c.counts_lj, c.sizes);
  nb_units_run(c, c.counts, c.unit_start, c.units, c.sizes, 1, nullptr, nullptr, s);
  nb_batch_frame_units<<<blocks_for(b.frames, 128), 128, 0, s>>>(b.frames, b.frames_dev, c.group_start,
                                                                c.unit_start, b.frame_units);
}

int nb_batch_build_run(mdrtNbBatch &b, const double *x, cudaStream_t s) {
  NbCtx &c = b.nb->c;
  int64_t hint = 0;
  if (nb_batch_plan(b, &hint)) return -1;
  int64_t cap = std::max<int64_t>(c.list_cap, hint);
  if (!c.key) {
    if (nb_realloc(c.key, c.n) || nb_realloc(c.sorted, c.n) || nb_realloc(c.atom_xw, c.n) ||
        nb_realloc(c.atom_shift, c.n) || nb_realloc(c.place_of, c.n) || nb_realloc(c.rank, c.n))
      return -1;
  }
  if (!b.frame_units && nb_realloc(b.frame_units, 2 * (int64_t)b.frames)) return -1;
  for (int attempt = 0; attempt < 8; ++attempt) {
    if (nb_reserve(c, cap, s)) return -1;
    if (c.groups_cap > b.groups_alloc) {
      if (nb_realloc(b.group_frame, c.groups_cap) || nb_realloc(b.group_L, c.groups_cap)) return -1;
      b.groups_alloc = c.groups_cap;
    }
    nb_batch_build_launch(b, x, s);
    NB_CHECK(cudaMemcpyAsync(c.h_sizes, c.sizes, sizeof(int32_t) * NB_SIZE_COUNT, cudaMemcpyDeviceToHost, s));
    NB_CHECK(cudaStreamSynchronize(s));
    NB_CHECK(cudaGetLastError());
    if (c.h_sizes[NB_SIZE_OVERFLOW] == 0) {
      c.built = true;
      c.builds++;
      c.inner_valid = false;
      return 0;
    }
    int64_t longest = c.h_sizes[NB_SIZE_LONGEST];
    int64_t want = (longest + longest / 4 + NB_UNIT - 1) / NB_UNIT * NB_UNIT;
    cap = std::max(cap, want);
    c.grows++;
  }
  return -1;
}
