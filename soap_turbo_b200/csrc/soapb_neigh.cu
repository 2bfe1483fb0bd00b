// soapb_neigh.cu -- neighbour lists of periodic structures on the device, in
// the CSR layout get_soap takes (src/soap_turbo.f90:139-169): one row per
// central site, the site itself first (r = 0, theta = phi = 0), then every
// periodic image of every atom within rcut, with theta = acos(dz / r) and
// phi = atan2(dy, dx) of the displacement, and the species mask of
// assign_species_multiplicity (src/soap_turbo.f90:2188-2214).
//
// Atoms are binned into a cell list over the (possibly triclinic) cell: cells
// are at least rcut wide along each axis, and a site visits the cells within
// R = ceil(rcut * n_cells / plane_spacing) of its own along each axis, with the
// lattice translation each wrap implies (so small cells, where R cells reach
// around the box, visit several images of the same atoms).  The atoms are
// copied in cell order, so the cells of one (x, y) column of a site's stencil are
// one run of them, and a warp takes a site's runs end to end, a candidate per lane.
// Two passes: count (whose last CTA scans the counts into CSR offsets where the
// sites are few), then fill.  One to four warps per site; the fill gathers the site's
// row in shared memory and sorts it by (neighbour atom, distance) so the order
// depends on nothing but the inputs.
// What bounds it, at some thousand atoms: the launches and each pass's chain of
// dependent loads.  A cell at a time (27 of some 12 atoms, read through their
// indices) count and fill took 32 and 57 us for 1679 sites of 4096 atoms; see
// soapb_build_neighbors for the whole.
#include "soapb_scan.cuh"

namespace soapb {

namespace {

constexpr int kNbWarps = 4;      // warps per CTA of the count kernel
constexpr int kNbFillWarps = 2;  // warps per CTA of the fill kernel where each has a site (its rows sit in shared memory)
constexpr int kNbShift = 512;    // image components are stored as n + kNbShift in 10 bits
constexpr int kNbOneThreads = 1024;
static_assert(kNbMaxReach + 1 + 2 * kNbMaxWrap < kNbShift, "image translations must fit 10 bits");

__device__ __forceinline__ int floor_div(int a, int b) { return a >= 0 ? a / b : -((-a + b - 1) / b); }

// Displacement of atom j's image n (integer lattice vector) from atom i:
// (r_j + n . lattice) - r_i.  Both passes call this, so they agree bit for bit.
__device__ __forceinline__ void image_disp(const NbGeom &g, double xj, double yj, double zj, double xi, double yi,
                                           double zi, int nx, int ny, int nz, double &dx, double &dy, double &dz) {
  const double tx = nx * g.lat[0] + ny * g.lat[3] + nz * g.lat[6];
  const double ty = nx * g.lat[1] + ny * g.lat[4] + nz * g.lat[7];
  const double tz = nx * g.lat[2] + ny * g.lat[5] + nz * g.lat[8];
  dx = (xj + tx) - xi;
  dy = (yj + ty) - yi;
  dz = (zj + tz) - zi;
}

// ---- an atom's cell and the lattice translation that wraps it into the cell
// (image translations then stay within +-(kNbMaxReach + 1 + 2 kNbMaxWrap) <
// kNbShift, the packing range of the fill pass; farther atoms, and non-finite
// positions, are reported and put in cell 0)
__device__ __forceinline__ int4 bin_atom(const NbGeom &g, const double *pos, int a, unsigned long long *err) {
  const double x = pos[3 * a], y = pos[3 * a + 1], z = pos[3 * a + 2];
  int c[3], w[3];
  bool bad = false;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double s = x * g.inv[d] + y * g.inv[3 + d] + z * g.inv[6 + d];
    const double f = floor(s);
    if (!(fabs(f) <= (double)kNbMaxWrap)) {
      bad = true;
      w[d] = 0;
      c[d] = 0;
    } else {
      w[d] = (int)f;
      c[d] = min(g.nc[d] - 1, max(0, (int)((s - f) * g.nc[d])));
    }
  }
  if (bad) atomicMax(err, kErrTop - kErrWrap);
  return make_int4((c[0] * g.nc[1] + c[1]) * g.nc[2] + c[2], w[0], w[1], w[2]);
}
__device__ __forceinline__ int pack3(int x, int y, int z) {
  return ((x + kNbShift) << 20) | ((y + kNbShift) << 10) | (z + kNbShift);
}
__device__ __forceinline__ NbAtom cell_atom(const double *pos, int a, int4 c) {
  return NbAtom{pos[3 * a], pos[3 * a + 1], pos[3 * a + 2], a, pack3(c.y, c.z, c.w)};
}

// The cell list of few atoms by one CTA: counts in shared memory, scanned, and the
// atoms copied to their slots (the order inside a cell is arbitrary).
__global__ void __launch_bounds__(kNbOneThreads) k_nb_cells(NbGeom g, int n_cells, const double *pos, int4 *atom_cell,
                                                            int *cell_start, NbAtom *cells, unsigned long long *err) {
  __shared__ int cnt[kNbOneCells];
  __shared__ int wsum[kNbOneThreads / 32];
  constexpr int PER = kNbOneAtoms / kNbOneThreads, CPT = kNbOneCells / kNbOneThreads;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < n_cells; i += kNbOneThreads) cnt[i] = 0;
  __syncthreads();
  int4 c[PER];
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int a = tid + j * kNbOneThreads;
    if (a < g.n_atoms) {
      c[j] = bin_atom(g, pos, a, err);
      atom_cell[a] = c[j];
      atomicAdd(&cnt[c[j].x], 1);
    }
  }
  __syncthreads();
  int own[CPT], sum = 0;
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    const int q = tid * CPT + i;
    own[i] = q < n_cells ? cnt[q] : 0;
    sum += own[i];
  }
  int x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  int run = x - sum;
  for (int w = 0; w < warp; ++w) run += wsum[w];
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    const int q = tid * CPT + i;
    if (q < n_cells) {
      cell_start[q] = run;
      cnt[q] = run;
    }
    run += own[i];
  }
  if (tid == 0) cell_start[n_cells] = g.n_atoms;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int a = tid + j * kNbOneThreads;
    if (a < g.n_atoms) cells[atomicAdd(&cnt[c[j].x], 1)] = cell_atom(pos, a, c[j]);
  }
}

// ... and of many, in three launches: bin, the scan, place
__global__ void k_nb_bin(NbGeom g, const double *pos, int4 *atom_cell, int *cell_count,
                         unsigned long long *err) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= g.n_atoms) return;
  const int4 c = bin_atom(g, pos, a, err);
  atom_cell[a] = c;
  atomicAdd(&cell_count[c.x], 1);
}
__global__ void k_nb_place(NbGeom g, const double *pos, const int4 *atom_cell, const int *cell_start, int *cell_fill,
                           NbAtom *cells) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= g.n_atoms) return;
  const int4 c = atom_cell[a];
  cells[cell_start[c.x] + atomicAdd(&cell_fill[c.x], 1)] = cell_atom(pos, a, c);
}

// Visits every candidate image of a site's stencil: visit(j, nx, ny, nz, r2, ok)
// is called by all lanes of the warp together (ok false on padding lanes), so
// it may use warp collectives.  A run is the stencil's cells of one x, y and wrap
// in z, contiguous in the cell order; 32 runs are laid end to end at a time.  Of
// `parts` warps that share the site, warp `part` takes every parts-th 64 candidates.
template <typename Visit>
__device__ __forceinline__ void for_each_neighbour(const NbGeom &g, const double *pos, const int4 *atom_cell,
                                                   const int *cell_start, const NbAtom *cells, int a, int part,
                                                   int parts, Visit visit) {
  const int lane = threadIdx.x & 31;
  const int4 ca = atom_cell[a];
  const double xi = pos[3 * a], yi = pos[3 * a + 1], zi = pos[3 * a + 2];
  const int cz = ca.x % g.nc[2], cy = (ca.x / g.nc[2]) % g.nc[1], cx = ca.x / (g.nc[2] * g.nc[1]);
  const int wz0 = floor_div(cz - g.R[2], g.nc[2]), nz = floor_div(cz + g.R[2], g.nc[2]) - wz0 + 1;
  const int ny = 2 * g.R[1] + 1, n_run = (2 * g.R[0] + 1) * ny * nz;
  for (int r0 = 0; r0 < n_run; r0 += 32) {
    int start = 0, len = 0, tr = 0;  // the lane's run, and the translation of its cells
    if (r0 + lane < n_run) {
      const int rr = r0 + lane, iz = rr % nz, t = rr / nz, iy = t % ny, ix = t / ny;
      const int X = cx + ix - g.R[0], wx = floor_div(X, g.nc[0]), qx = X - wx * g.nc[0];
      const int Y = cy + iy - g.R[1], wy = floor_div(Y, g.nc[1]), qy = Y - wy * g.nc[1];
      const int wz = wz0 + iz, lo = max(cz - g.R[2] - wz * g.nc[2], 0),
                hi = min(cz + g.R[2] - wz * g.nc[2], g.nc[2] - 1);
      const int q = (qx * g.nc[1] + qy) * g.nc[2];
      start = cell_start[q + lo];
      len = cell_start[q + hi + 1] - start;
      tr = pack3(wx + ca.y, wy + ca.z, wz + ca.w);
    }
    int incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    // two candidates a lane at a time, so that their loads overlap
    for (int c0 = 64 * part; c0 < total; c0 += 64 * parts) {
      NbAtom b[2];
      int w[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = c0 + 32 * h + lane;
        int r = 0;  // the run of candidate c: how many end at or before it
#pragma unroll
        for (int step = 16; step > 0; step >>= 1)
          if (__shfl_sync(0xffffffffu, incl, r + step - 1) <= c) r += step;
        const int at = c - __shfl_sync(0xffffffffu, incl, r) + __shfl_sync(0xffffffffu, len, r) +
                       __shfl_sync(0xffffffffu, start, r);
        w[h] = __shfl_sync(0xffffffffu, tr, r);
        if (c < total) b[h] = cells[at];
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (c0 + 32 * h >= total) break;
        int j = 0, nx = 0, ny_ = 0, nz_ = 0;
        double r2 = 0.0;
        bool ok = false;
        if (c0 + 32 * h + lane < total) {
          j = b[h].atom;
          // the image of j in the run's cells: translation (w - w_j + w_a) lattice vectors
          nx = (w[h] >> 20) - (b[h].wrap >> 20);
          ny_ = ((w[h] >> 10) & 1023) - ((b[h].wrap >> 10) & 1023);
          nz_ = (w[h] & 1023) - (b[h].wrap & 1023);
          double dx, dy, dz;
          image_disp(g, b[h].x, b[h].y, b[h].z, xi, yi, zi, nx, ny_, nz_, dx, dy, dz);
          r2 = dx * dx + dy * dy + dz * dz;
          ok = r2 < g.rcut2 && !(j == a && nx == 0 && ny_ == 0 && nz_ == 0);
        }
        visit(j, nx, ny_, nz_, r2, ok);
      }
    }
  }
}

// ---- pass 1: neighbours of each site (the row length is one more: the site itself),
// by W warps.
// done (may be null): the CTAs finished; the last one then scans the counts of up to
// kNbOneSites sites into the CSR offsets.
template <int W>
__global__ void __launch_bounds__(32 * kNbWarps) k_nb_count(NbGeom g, const double *pos, const int *sites,
                                                            const int4 *atom_cell, const int *cell_start,
                                                            const NbAtom *cells, int *counts, int *off, int *done,
                                                            unsigned long long *err) {
  constexpr int NT = 32 * kNbWarps;
  const int warp = threadIdx.x >> 5, w = blockIdx.x * (kNbWarps / W) + warp / W, lane = threadIdx.x & 31;
  __shared__ int s_cnt[kNbWarps];
  int cnt = 0;
  const int a = w < g.n_sites ? sites[w] : -1;
  if (a >= 0 && a < g.n_atoms)
    for_each_neighbour(g, pos, atom_cell, cell_start, cells, a, warp % W, W,
                       [&](int, int, int, int, double, bool ok) { cnt += __popc(__ballot_sync(0xffffffffu, ok)); });
  if (W > 1) {
    if (lane == 0) s_cnt[warp] = cnt;
    __syncthreads();
    if (warp % W == 0)
#pragma unroll
      for (int v = 1; v < W; ++v) cnt += s_cnt[warp + v];
  }
  if (lane == 0 && warp % W == 0 && w < g.n_sites) {
    unsigned long long bad = 0ull;
    if (a < 0 || a >= g.n_atoms) bad = kErrTop - (unsigned long long)w;  // site index out of range
    else if (cnt > kNbCap) bad = kErrTop - ((1ull << 32) + (unsigned long long)w);  // row too long
    counts[w] = 1 + cnt;
    if (bad) atomicMax(err, bad);
  }
  if (!done) return;
  __shared__ int s_last;
  __shared__ int wsum[kNbWarps];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(done, 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int per = (g.n_sites + NT - 1) / NT, i0 = threadIdx.x * per, i1 = min(g.n_sites, i0 + per);
  int sum = 0;
#pragma unroll 8
  for (int i = i0; i < i1; ++i) sum += __ldcg(counts + i);
  int x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[threadIdx.x >> 5] = x;
  __syncthreads();
  int run = x - sum;
  for (int v = 0; v < (int)(threadIdx.x >> 5); ++v) run += wsum[v];
#pragma unroll 8
  for (int i = i0; i < i1; ++i) {
    off[i] = run;
    run += __ldcg(counts + i);
  }
  if (threadIdx.x == NT - 1) off[g.n_sites] = run;
}

// The species bits of neighbour j in the row of central atom a, as
// assign_species_multiplicity sets mask(k2, :) (src/soap_turbo.f90:2203-2211):
// the loop runs over the central atom's multiplicity, reading j's species.
__device__ __forceinline__ unsigned mask_bits(const NbGeom &g, const int *atom_species, const int *atom_mult,
                                              int a, int j) {
  unsigned bits = 0;
  const int mc = min(atom_mult[a], g.max_mult), mj = atom_mult[j];
  for (int i2 = 0; i2 < mc; ++i2) {
    const int sp = i2 < mj ? atom_species[(size_t)j * g.max_mult + i2] : 0;
    if (sp > 0 && sp <= g.n_species) bits |= 1u << (sp - 1);
  }
  return bits;
}

// ---- pass 2: each site's row, sorted by (neighbour atom, distance), by W warps.
// Bound by latency: the candidates' loads and the FP64 chain of a pair's distance and
// angles, with few warps on an SM (40 us at 1679 sites of one warp each; the step
// from positions 234 us so, 223 with two).  The pair count
// comes from the offsets; nothing is written where it is above the buffers'
// capacity, o.n_pairs (the host then makes room and launches again).  status, in
// page-locked host memory, receives the pair count and the three error words.
template <int W>
__global__ void __launch_bounds__(W > kNbFillWarps ? 32 * W : 32 * kNbFillWarps)
    k_nb_fill(NbGeom g, const double *pos, const int *sites,
                                                           const int *atom_species, const int *atom_mult,
                                                           const int4 *atom_cell, const int *cell_start,
                                                           const NbAtom *cells, const int *off, NbOut o,
                                                           const unsigned long long *err, int w_cells,
                                                           volatile unsigned long long *status) {
  constexpr int S = W > 1 ? 1 : kNbFillWarps, NT = 32 * W;  // sites of the CTA, threads of a site
  __shared__ unsigned long long s_key[S][kNbCap];
  __shared__ unsigned s_img[S][kNbCap];
  __shared__ int s_filled;
  const int wl = W > 1 ? 0 : threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x % NT;
  const int w = blockIdx.x * S + wl;
  auto sync = [] {
    if (W > 1) __syncthreads();
    else __syncwarp();
  };
  const int n_pairs = g.n_sites > 0 ? off[g.n_sites] : 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    status[0] = (unsigned long long)(long long)n_pairs;
    status[1] = err[0];
    status[2] = err[1];
    status[3] = err[1 + w_cells];
  }
  if (w >= g.n_sites || n_pairs < 0 || n_pairs > o.n_pairs) return;
  const int a = sites[w];
  const int base = off[w], cnt = off[w + 1] - base - 1;
  if (a < 0 || a >= g.n_atoms || cnt > kNbCap) return;  // reported by the count pass
  unsigned long long *key = s_key[wl];
  unsigned *img = s_img[wl];
  int filled = 0;
  if (W > 1) {
    if (tid == 0) s_filled = 0;
    __syncthreads();
  }
  const unsigned lt = (1u << lane) - 1u;
  for_each_neighbour(g, pos, atom_cell, cell_start, cells, a, tid >> 5, W,
                     [&](int j, int nx, int ny, int nz, double r2, bool ok) {
    const unsigned bal = __ballot_sync(0xffffffffu, ok);
    if (W > 1) {
      if (lane == 0 && bal) filled = atomicAdd(&s_filled, __popc(bal));
      filled = __shfl_sync(0xffffffffu, filled, 0);
    }
    if (ok) {
      const int slot = filled + __popc(bal & lt);
      if (slot < kNbCap) {
        const float r = (float)sqrt(r2);
        key[slot] = ((unsigned long long)(unsigned)j << 32) | __float_as_uint(r);
        img[slot] = (unsigned)pack3(nx, ny, nz);
      }
    }
    if (W == 1) filled += __popc(bal);
  });
  sync();
  // the row sorted by (atom, FP32 distance, image translation in x, y, z order):
  // every candidate differs in that triple, so the row's order does not depend on
  // the order the cell list happened to hold the atoms in or the warps found them
  if (cnt <= 64) {  // each thread ranks its entries among all: no steps between which the site waits
    constexpr int PER = NT < 64 ? 64 / NT : 1;
    unsigned long long k[PER];
    unsigned im[PER];
    int n[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      k[i] = tid + i * NT < cnt ? key[tid + i * NT] : ~0ull;
      im[i] = tid + i * NT < cnt ? img[tid + i * NT] : ~0u;
      n[i] = 0;
    }
    if (NT <= 64 || tid < 64)
#pragma unroll 4
      for (int t = 0; t < cnt; ++t) {
        const unsigned long long kt = key[t];
        const unsigned it = img[t];
#pragma unroll
        for (int i = 0; i < PER; ++i) n[i] += kt < k[i] || (kt == k[i] && it < im[i]);
      }
    sync();
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (tid + i * NT < cnt) {
        key[n[i]] = k[i];
        img[n[i]] = im[i];
      }
    sync();
  } else {  // a bitonic sort, padded with the largest key
    int npow = 1;
    while (npow < cnt) npow <<= 1;
    for (int t = cnt + tid; t < npow; t += NT) {
      key[t] = ~0ull;
      img[t] = ~0u;
    }
    sync();
    for (int k = 2; k <= npow; k <<= 1)
      for (int jj = k >> 1; jj > 0; jj >>= 1) {
        for (int t = tid; t < npow; t += NT) {
          const int p = t ^ jj;
          if (p > t) {
            const bool up = (t & k) == 0;
            const unsigned long long kt = key[t], kp = key[p];
            const bool gt = kt > kp || (kt == kp && img[t] > img[p]);
            if (gt == up) {
              key[t] = kp;
              key[p] = kt;
              const unsigned it = img[t];
              img[t] = img[p];
              img[p] = it;
            }
          }
        }
        sync();
      }
  }
  // the site itself first, then its sorted neighbours
  for (int e = tid - 1; e < cnt; e += NT) {
    const int k = base + 1 + e;
    int j;
    double r = 0.0, th = 0.0, ph = 0.0;
    if (e < 0) {
      j = a;
    } else {
      j = (int)(key[e] >> 32);
      const unsigned im = img[e];
      const int nx = (int)(im >> 20) - kNbShift, ny = (int)((im >> 10) & 1023u) - kNbShift,
                nz = (int)(im & 1023u) - kNbShift;
      double dx, dy, dz;
      image_disp(g, pos[3 * j], pos[3 * j + 1], pos[3 * j + 2], pos[3 * a], pos[3 * a + 1], pos[3 * a + 2], nx, ny, nz,
                 dx, dy, dz);
      r = sqrt(dx * dx + dy * dy + dz * dz);
      th = acos(fmin(1.0, fmax(-1.0, dz / r)));
      ph = atan2(dy, dx);
    }
    o.rjs[k] = r;
    o.thetas[k] = th;
    o.phis[k] = ph;
    o.neigh_atom[k] = j;
    const unsigned bits = mask_bits(g, atom_species, atom_mult, a, j);
    for (int s = 0; s < g.n_species; ++s) o.mask[(size_t)s * n_pairs + k] = (uint8_t)((bits >> s) & 1u);
  }
  if (tid == 0) {
    o.n_neigh[w] = cnt + 1;
    o.species_mult[w] = atom_mult[a];
  }
  for (int m = tid; m < g.max_mult; m += NT) o.species[(size_t)w * g.max_mult + m] = atom_species[(size_t)a * g.max_mult + m];
}

__global__ void __launch_bounds__(256) k_nb_scan(DevBatch B, int tiles, int max_spins) {
  __shared__ int sv[kScanTile];
  prep_scan_tile<256>(B, tiles, sv, max_spins);
}

}  // namespace

// Warps that share a site in the count and the fill: the number with the cheapest
// waves of the fill (18, 14 and 7 sites fit an SM at 1, 2 and 4 warps), a site at 2
// and 4 warps taking 0.8 and 0.7 of its time at one.  Builds at 1, 2 and 4 warps, us:
// 64 sites 124, 106, 99; 600 96, 89, 85; 1200 98, 90, 101; 1700 101, 97, 105; 2400 107,
// 114, 120; 8000 177, 168, 199; 32768 382, 380, 515.
static int nb_warps(int n_sites) {
  const int sms = sm_count(), slots[3] = {18 * sms, 14 * sms, 7 * sms};
  const double cost[3] = {1.0, 0.8, 0.7};
  int best = 0;
  double least = 0.0;
  for (int i = 0; i < 3; ++i) {
    const double t = ((n_sites - 1) / slots[i] + 1) * cost[i];
    if (i == 0 || t < least) {
      least = t;
      best = i;
    }
  }
  return 1 << best;
}

cudaError_t launch_nb_cells(const NbGeom &g, int n_cells, const double *pos, int4 *atom_cell, int *cell_count,
                            int *cell_start, int *cell_fill, NbAtom *cells, unsigned long long *err,
                            unsigned long long *scan_state, int *launches, cudaStream_t s) {
  if (g.n_atoms <= kNbOneAtoms && n_cells <= kNbOneCells) {
    k_nb_cells<<<1, kNbOneThreads, 0, s>>>(g, n_cells, pos, atom_cell, cell_start, cells, err);
    *launches += 1;
    return cudaGetLastError();
  }
  k_nb_bin<<<(g.n_atoms + 255) / 256, 256, 0, s>>>(g, pos, atom_cell, cell_count, err);
  cudaError_t e = launch_scan(cell_count, n_cells, cell_start, scan_state, s);
  if (e != cudaSuccess) return e;
  k_nb_place<<<(g.n_atoms + 255) / 256, 256, 0, s>>>(g, pos, atom_cell, cell_start, cell_fill, cells);
  *launches += 3;
  return cudaGetLastError();
}

cudaError_t launch_nb_count(const NbGeom &g, const double *pos, const int *sites, const int4 *atom_cell,
                            const int *cell_start, const NbAtom *cells, int *counts, int *off, int *done,
                            unsigned long long *err, unsigned long long *scan_state, int *launches, cudaStream_t s) {
  if (g.n_sites <= 0) return cudaSuccess;
  const bool one = g.n_sites <= kNbOneSites;
  const int W = nb_warps(g.n_sites), per = kNbWarps / W;
  auto kern = W == 4 ? k_nb_count<4> : W == 2 ? k_nb_count<2> : k_nb_count<1>;
  kern<<<(g.n_sites + per - 1) / per, 32 * kNbWarps, 0, s>>>(g, pos, sites, atom_cell, cell_start, cells, counts, off,
                                                             one ? done : nullptr, err);
  *launches += 1;
  if (one) return cudaGetLastError();
  *launches += 1;
  return launch_scan(counts, g.n_sites, off, scan_state, s);
}

cudaError_t launch_nb_fill(const NbGeom &g, const double *pos, const int *sites, const int *atom_species,
                           const int *atom_mult, const int4 *atom_cell, const int *cell_start, const NbAtom *cells,
                           const int *off, const NbOut &o, const unsigned long long *err, int w_cells,
                           unsigned long long *status, cudaStream_t s) {
  const int W = nb_warps(g.n_sites), per = W > 1 ? 1 : kNbFillWarps;
  const int blocks = g.n_sites > 0 ? (g.n_sites + per - 1) / per : 1;
  auto kern = W == 4 ? k_nb_fill<4> : W == 2 ? k_nb_fill<2> : k_nb_fill<1>;
  kern<<<blocks, W > 1 ? 32 * W : 32 * kNbFillWarps, 0, s>>>(g, pos, sites, atom_species, atom_mult, atom_cell,
                                                             cell_start, cells, off, o, err, w_cells, status);
  return cudaGetLastError();
}

cudaError_t launch_scan(const int *counts, int n, int *off, unsigned long long *state, cudaStream_t s,
                        int blocks, int max_spins) {
  DevBatch B{};
  B.n_sites = n;
  B.n_pairs = -1;
  B.n_neigh = counts;
  B.off = off;
  B.err = state;
  const int tiles = prep_scan_tiles(n);
  if (blocks < 0 || blocks > tiles) blocks = tiles;
  if (blocks > 0) k_nb_scan<<<blocks, 256, 0, s>>>(B, tiles, max_spins);
  return cudaGetLastError();
}

}  // namespace soapb
