// soapb_mixed.cu -- the mixed-precision descriptor and force-VJP kernels.
//
// k_pair, one thread per pair, does the FP64 work of the path and leaves rows in
// FP32; the site kernels, one CTA per central site ("environment"), read them.  A
// site's CSR row of neighbour pairs is walked in chunks; each chunk is turned into
// "entries", one per (pair, species) the radial expansion applies to (mask set,
// inside that species' rcut_hard, the self pair only when its central weight is
// used), sorted by species with ballot ranks so every species' entries are a
// contiguous run.
//
// k_descriptor (get_soap, src/soap_turbo.f90:491-909): c_nlm with a thread per k
//   and NH radial indices, each summing its species' entries in CSR order (a
//   fixed-order segmented reduction, no atomics); the power spectrum of the kept
//   components (a dot product per component), compression, norm, normalise.
// k_contract (soap_contract, src/soap_turbo.f90:1723-1884): G -> Gp -> Gu -> H(n,k)
//   in shared memory, then a half-warp per entry contracts the four angular
//   factors and R_n, dR_n/dr of its row against H; per-pair forces are rotated to
//   Cartesian and the self pair gets minus their sum, all in fixed order.
// k_descriptor_tc, k_contract_tc: the same with the contractions on the tensor
//   cores, where the caller turns them on.
//
// Everything is deterministic: no atomics touch results, and every reduction
// runs in an order fixed by the launch shape.
#include <atomic>
#include <cstdio>
#include <mutex>
#include <type_traits>
#include <vector>

#include "soapb_device.cuh"
#include "soapb_scan.cuh"
#include "soapb_tc.cuh"

namespace soapb {

constexpr double kFourPi = 12.566370614359172954;



// ------------------------------------------------------------------ prep
// The species bits of pair k from the reference's mask(n_pairs, n_species),
// written to B.bits, with the pair's inputs checked.
__device__ __forceinline__ unsigned prep_pair(const DevBatch &B, int k, int n_species) {
  unsigned bits = 0;
  for (int s = 0; s < n_species; ++s)
    if (B.mask[(size_t)s * B.n_pairs + k]) bits |= 1u << s;
  B.bits[k] = (uint8_t)bits;
  const double r = B.rjs[k], t = B.thetas[k], f = B.phis[k];
  if (!(r >= 0.0) || !isfinite(r) || !isfinite(t) || !isfinite(f)) prep_error(B, (unsigned long long)k);
  return bits;
}

// The prep kernel of the plain FP64 path: scan tiles first, then one thread per pair.
constexpr int kPrepThreads = 256;
__global__ void __launch_bounds__(kPrepThreads) k_prep(DevBatch B, int n_species, int scan_tiles) {
  if ((int)blockIdx.x < scan_tiles) {
    __shared__ int sv[kScanTile];
    prep_scan_tile<kPrepThreads>(B, scan_tiles, sv);
    return;
  }
  const int k = ((int)blockIdx.x - scan_tiles) * kPrepThreads + threadIdx.x;
  if (k < B.n_pairs) prep_pair(B, k, n_species);
}

// ------------------------------------------------------------- utilities
template <int NT>
__device__ __forceinline__ double block_sum(double v, double *red) {
  // fixed-order tree: xor shuffles within warps, then warp 0 over partials
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    double t = (lane < NT / 32) ? red[lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}

// Three sums at once, same fixed order as block_sum.
template <int NT>
__device__ __forceinline__ void block_sum3(double &a, double &b, double &c, double *red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) {
    red[warp] = a;
    red[8 + warp] = b;
    red[16 + warp] = c;
  }
  __syncthreads();
  if (warp == 0) {
    double x = (lane < NT / 32) ? red[lane] : 0.0;
    double y = (lane < NT / 32) ? red[8 + lane] : 0.0;
    double z = (lane < NT / 32) ? red[16 + lane] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      x += __shfl_xor_sync(0xffffffffu, x, o);
      y += __shfl_xor_sync(0xffffffffu, y, o);
      z += __shfl_xor_sync(0xffffffffu, z, o);
    }
    if (lane == 0) {
      red[32] = x;
      red[33] = y;
      red[34] = z;
    }
  }
  __syncthreads();
  a = red[32];
  b = red[33];
  c = red[34];
}

// Builds the entry list of one chunk of NT pairs.  Returns, per thread, the
// radial-valid species bits of its own pair, its distance (my_r) and (in
// slot[]) the entry slot of each of them.  Shared: ent[] = chunk-local pair |
// species << 24, and sbase/scnt per species.
template <int NT>
__device__ __forceinline__ int build_entries(const DevParams &P, const DevBatch &B, int p_begin,
                                             int chunk, int p_end, bool vjp, int *ent, int *wcnt,
                                             int *sbase, int *scnt, int *n_ent_out,
                                             int (&slot)[SOAPB_MAX_SPECIES], unsigned &my_bits,
                                             double &my_r) {
  constexpr int NW = NT / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int k = chunk + tid;
  unsigned rb = 0;
  my_r = 1.0;
  if (k < p_end) {
    const double r = B.rjs[k];
    my_r = r;
    const unsigned bits = B.bits[k];
    const int j = k - p_begin;
#pragma unroll
    // a pair at or beyond rcut_max has no angular row (the reference zeroes
    // its angular coefficients, src/soap_turbo_angular.f90:549-574); it only
    // matters for poly3operator, whose radial part has no rcut_hard cut
    for (int s = 0; s < SOAPB_MAX_SPECIES; ++s) {
      if (s >= P.n_species) break;
      const bool ok = ((bits >> s) & 1u) && r < P.rad[s].rcut_hard && r < P.rcut_max &&
                      (vjp ? (j > 0) : (j > 0 || P.rad[s].do_central));
      if (ok) rb |= 1u << s;
    }
  }
  my_bits = rb;
  const unsigned lt = (1u << lane) - 1u;
  int rank[SOAPB_MAX_SPECIES];
#pragma unroll
  for (int s = 0; s < SOAPB_MAX_SPECIES; ++s) {
    rank[s] = 0;
    if (s >= P.n_species) break;
    const unsigned bal = __ballot_sync(0xffffffffu, (rb >> s) & 1u);
    rank[s] = __popc(bal & lt);
    if (lane == 0) wcnt[s * NW + warp] = __popc(bal);
  }
  __syncthreads();
  if (tid < P.n_species) {
    int acc = 0;
    for (int w = 0; w < NW; ++w) {
      const int t = wcnt[tid * NW + w];
      wcnt[tid * NW + w] = acc;
      acc += t;
    }
    scnt[tid] = acc;
  }
  __syncthreads();
  if (tid == 0) {
    int b = 0;
    for (int s = 0; s < P.n_species; ++s) {
      sbase[s] = b;
      b += scnt[s];
    }
    *n_ent_out = b;
  }
  __syncthreads();
#pragma unroll
  for (int s = 0; s < SOAPB_MAX_SPECIES; ++s) slot[s] = -1;
#pragma unroll
  for (int s = 0; s < SOAPB_MAX_SPECIES; ++s) {
    if (s >= P.n_species) break;
    if ((rb >> s) & 1u) {
      const int e = sbase[s] + wcnt[s * NW + warp] + rank[s];
      ent[e] = tid | (s << 24);
      slot[s] = e;
    }
  }
  __syncthreads();
  return *n_ent_out;
}

__device__ __forceinline__ int first_species(unsigned bits) { return __ffs(bits) - 1; }

// ------------------------------------------------------------ pair rows
// The angular row of a pair (floats), written by k_pair and read by the site
// kernels; the descriptor reads its first part alone:
//   amp i_l for l <= LC (amp = rcut_max^2 / sigma_t^2), a pad, and
//   (cos(m phi), -sin(m phi)) for m <= LC;
//   preflm_k P_l^m for l <= l_max (+1 with derivatives), k = l(l+1)/2 + m;
//   amp di_l/dr, 2 sigma_t_scaling / sigma_t, cos(theta), sqrt(1 - cos^2(theta)).
// So u_k = amp preflm_k P_k i_l of src/soap_turbo_angular.f90:590-594 is one
// product of two row values.  LC is a multiple of 4: every part is one of 16 bytes.
__host__ __device__ constexpr int row_il(int) { return 0; }
__host__ __device__ constexpr int row_e(int LC) { return LC + 2; }
__host__ __device__ constexpr int row_p(int LC) { return 3 * LC + 4; }
__host__ __device__ constexpr int row_tail(int LC) { return (row_p(LC) + (LC + 2) * (LC + 3) / 2 + 3) / 4 * 4; }
__host__ __device__ constexpr int row_ild(int LC) { return row_tail(LC); }
__host__ __device__ constexpr int row_sf(int LC) { return row_tail(LC) + LC + 1; }
__host__ __device__ constexpr int row_x(int LC) { return row_tail(LC) + LC + 2; }
__host__ __device__ constexpr int row_sq(int LC) { return row_tail(LC) + LC + 3; }
__host__ __device__ constexpr int row_len(int LC) { return row_tail(LC) + LC + 4; }

int ang_row_floats(const DevParams &P) { return row_len(P.amax_t == 8 ? 8 : 12); }
// The pair kernel stages a warp's rows in two parts, head and tail and then the
// P_l^m values, as four-float pieces; the stride in pieces (odd, so that the lanes'
// rows start in distinct banks) holds the larger of the two.
__host__ __device__ constexpr int pair_stage_stride(int LC) {
  const int np = (row_tail(LC) - row_p(LC)) / 4, rest = row_len(LC) / 4 - np;
  return (np > rest ? np : rest) | 1;
}

// ------------------------------------------------------------ pair kernel
// One thread per pair, all FP64 work of the path:
//  * the radial expansion of every (pair, species) entry
//    (src/soap_turbo_radial.f90:281-1004), rounded to FP32 with 4 pi and
//    global_scaling folded in, into the radial buffer;
//  * the angular row (src/soap_turbo_angular.f90:267-463, 549-607), staged by the
//    warp in shared memory, four values at a time, and copied out with coalesced
//    stores.
// Bound by instructions (44 % of the issue slots at 1679 sites, 55 % at 16384; 30 % of
// them index arithmetic) and the warps' waits on tables and FP64 chains; without tables by
// the FP64 chain of a pair alone (12 and 20 % of the slots, 179 and 122 registers: sigma
// scaling at l_max 12, poly3operator).  So a warp shares nothing but the
// constants with its CTA and takes no barrier after theirs, the table reads of
// one warp run under the FP64 of others, and the copies' loops are of compile-time
// length.  Whole-step times with rows staged by value, CTA-wide copies behind
// barriers and the tables between the two: 128.5 us at 1679 sites, 717 at 16384
// and 75 at 777 without tables; in this form, beside the same site kernels, 124.5, 707
// and 72.6.  Eight CTAs an SM (64 registers, spills) or CTA-wide copies in this form: 125
// and 128.4 us at 1679.
// The site kernels only read these rows; soap_contract reads the rows of the
// descriptor call that kept its state, as the reference keeps the radial and
// angular expansions between get_soap and soap_contract.
// TAB: R_n and dR_n/dr come from the context's piecewise-polynomial tables
// (FP32 evaluation of the FP64 expansion fitted per species; see RadTab)
// instead of the FP64 expansion itself.
constexpr int kPairThreads = 128;
constexpr int kTabUnroll = 4;
// CTAs of the pair kernel before its pair CTAs: the scan tiles, and one that
// orders the sites when the batch is one tile and has an order to fill
__host__ __device__ inline int pair_cta_offset(const DevBatch &B, int scan_tiles) {
  return scan_tiles + ((B.order != nullptr && scan_tiles == 1) ? 1 : 0);
}
template <int AMAX, int LC, bool OP, bool TAB>
__global__ void __launch_bounds__(kPairThreads)
    k_pair(const DevParams P, const DevBatch B, int do_der, int scan_tiles, int pair_lo, int pair_hi) {
  constexpr int NT = kPairThreads;
  extern __shared__ __align__(16) unsigned char smem[];
  // the first CTAs scan n_neigh; with a site order to build, one more orders
  // the sites (pair_cta_offset gives the host the same count)
  const int lead = pair_cta_offset(B, scan_tiles);
  if ((int)blockIdx.x < scan_tiles) {
    prep_scan_tile<NT>(B, scan_tiles, (int *)smem);
    return;
  }
  if ((int)blockIdx.x < lead) {
    order_sites<NT>(B, (int *)smem, (int *)smem + kScanTile);
    return;
  }
  constexpr int S4 = pair_stage_stride(LC), AW4 = row_len(LC) / 4, H4 = row_p(LC) / 4, T4 = row_tail(LC) / 4;
  // what the descriptor alone reads ends here, rounded up to 64 bytes: a row that
  // stops within a sector is merged with memory's (a descriptor of 32768 atoms
  // 395 us, with whole rows 375, so 366)
  constexpr int ND4 = (H4 + ((LC + 1) * (LC + 2) / 2 + 3) / 4 + 3) / 4 * 4;
  static_assert(ND4 <= T4 && ND4 - H4 <= S4 && H4 + AW4 - T4 <= S4, "the staged pieces");
  const int head = (P.off_rad + P.n_species * SOAPB_RADSP_BYTES) / 16;
  for (int t = threadIdx.x; t < head; t += NT) ((uint4 *)smem)[t] = ((const uint4 *)P.blob)[t];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float4 *rows = (float4 *)(smem + (size_t)head * 16) + warp * 32 * S4, *row = rows + lane * S4;
  __syncthreads();
  const int k0 = pair_lo + ((int)blockIdx.x - lead) * NT + 32 * warp;  // the warp's pairs
  const int k = k0 + lane, nrow = min(32, pair_hi - k0);
  bool active = false;
  double x = 0.0, sq = 0.0;
  unsigned todo = 0u;  // the species whose radial expansion applies
  double r = 0.0;
  if (k < pair_hi) {
    const unsigned bits = prep_pair(B, k, P.n_species);
    r = B.rjs[k];
    if (bits != 0u && r < P.rcut_max) {
      active = true;
      const int isp = __ffs(bits) - 1;
      if (do_der)
        angular_stage<LC, true>(P, isp, r, B.thetas[k], B.phis[k], row, row + H4, x, sq);
      else
        angular_stage<LC, false>(P, isp, r, B.thetas[k], B.phis[k], row, row + H4, x, sq);
      for (int s = 0; s < P.n_species; ++s) {
        const RadSp &RS = *(const RadSp *)(smem + P.off_rad + (size_t)s * SOAPB_RADSP_BYTES);
        if (((bits >> s) & 1u) && r < RS.rcut_hard) todo |= 1u << s;
      }
      // the radial expansion of each species in range, as for a neighbour: the
      // central pair's expansion (:342-355) differs only by the factor
      // central_weight (:638-646), which the descriptor applies to that entry.  It
      // stands inside the branch for its bits: after it, the compiler fuses other
      // products into multiply-adds in k_pair<8, 8, false, false>, and up to 2e-4 of the
      // values (which W's cancellation amplifies) come out one or more FP32 ulps apart
      // from the other instantiation's
      if constexpr (!TAB) {
        const double *sW = (const double *)(smem + P.off_W);
        // species are data, not control flow: lanes of different species share
        // one expansion call
        while (todo) {
          const int s = __ffs(todo) - 1;
          todo &= todo - 1u;
          const RadSp &RS = *(const RadSp *)(smem + P.off_rad + (size_t)s * SOAPB_RADSP_BYTES);
          float4 *o = (float4 *)(B.rad + ((size_t)k * P.n_species + s) * 2 * AMAX);
          double val[AMAX], der[AMAX];
          radial_entry<AMAX, OP>(P, RS, sW + s * AMAX * AMAX, r, false, do_der != 0, val, der);
          const double g4 = kFourPi * RS.gscale;
#pragma unroll
          for (int n4 = 0; n4 < AMAX / 4; ++n4)
            o[n4] = make_float4((float)(g4 * val[4 * n4]), (float)(g4 * val[4 * n4 + 1]),
                                (float)(g4 * val[4 * n4 + 2]), (float)(g4 * val[4 * n4 + 3]));
          if (do_der)
#pragma unroll
            for (int n4 = 0; n4 < AMAX / 4; ++n4)
              o[AMAX / 4 + n4] = make_float4((float)(g4 * der[4 * n4]), (float)(g4 * der[4 * n4 + 1]),
                                             (float)(g4 * der[4 * n4 + 2]), (float)(g4 * der[4 * n4 + 3]));
        }
      }
    }
  }
  if constexpr (TAB) {
    // R_n and dR_n/dr from the tables, a warp's entries of one species at a
    // time: 2 AMAX lanes per entry, lane f evaluating function f, so that the
    // segment's coefficients (stored [degree][function]) are read and the
    // entry's radial row is written as contiguous 64-byte runs.  kTabUnroll groups
    // of entries at a time, all their loads before the first product: an entry's
    // eight coefficients are a round trip to L1 or L2 (one group at a time: steps
    // of 64 and 16384 sites 37.0 and 725 us, four: 35.6 and 717)
    constexpr int G = 2 * AMAX, EPW = 32 / G;
    static_assert(32 % G == 0, "lanes per entry");
    const int f = lane % G, sub = lane / G;
    const bool want = f < (do_der ? G : AMAX);
    __shared__ int s_who[kPairThreads];
    int *who = s_who + 32 * warp;
    for (int s = 0; s < P.n_species; ++s) {
      const bool mine = (todo >> s) & 1u;
      const unsigned m = __ballot_sync(0xffffffffu, mine);
      if (!m) continue;
      const int cnt = __popc(m);
      float t = 0.f;
      int cb = -1;
      if (mine) {
        const RadSp &RS = *(const RadSp *)(smem + P.off_rad + (size_t)s * SOAPB_RADSP_BYTES);
        cb = radial_table_locate<AMAX>(P, RS, P.rtab_sp[s], r, t);
        who[__popc(m & ((1u << lane) - 1u))] = lane;
      }
      __syncwarp();
      const float *coef = P.rtab_coef + f;
      float *out = B.rad + ((size_t)k0 * P.n_species + s) * G + f;
      for (int e0 = sub; e0 - sub < cnt; e0 += kTabUnroll * EPW) {
        int src[kTabUnroll];
        float te[kTabUnroll], a[kTabUnroll][kRadTabDeg + 1];
        bool on[kTabUnroll];
#pragma unroll
        for (int q = 0; q < kTabUnroll; ++q) {
          const int e = e0 + q * EPW;
          src[q] = who[min(e, cnt - 1)];
          on[q] = e < cnt && want;
          const int cbe = __shfl_sync(0xffffffffu, cb, src[q]);
          te[q] = __shfl_sync(0xffffffffu, t, src[q]);
          const float *c = coef + cbe;
#pragma unroll
          for (int d = 0; d <= kRadTabDeg; ++d) a[q][d] = on[q] && cbe >= 0 ? __ldg(c + d * G) : 0.f;
        }
#pragma unroll
        for (int q = 0; q < kTabUnroll; ++q) {
          float v = a[q][kRadTabDeg];
#pragma unroll
          for (int d = kRadTabDeg - 1; d >= 0; --d) v = fmaf(v, te[q], a[q][d]);
          if (on[q]) out[src[q] * P.n_species * G] = v;
        }
      }
      __syncwarp();  // the lanes' list is read
    }
  }
  // pieces 0 .. n - 1 of each of the warp's staged rows to their places in global
  // memory, from `at` on, those from `from` on `gap` pieces farther
  auto copy_out = [&](auto pieces, int at, int from, int gap) {
    constexpr int n = decltype(pieces)::value;
    float4 *dst = (float4 *)B.ang + (size_t)k0 * AW4 + at;
#pragma unroll 4
    for (int t = lane; t < nrow * n; t += 32) {
      const int i = t / n, j = t - i * n;
      dst[i * AW4 + j + (j >= from ? gap : 0)] = rows[i * S4 + j];
    }
  };
  __syncwarp();
  if (do_der)
    copy_out(std::integral_constant<int, H4 + AW4 - T4>(), 0, H4, T4 - H4);
  else
    copy_out(std::integral_constant<int, H4>(), 0, H4, 0);
  __syncwarp();
  const int l_top = P.l_max + (do_der ? 1 : 0), n_p = (l_top + 1) * (l_top + 2) / 2;
  if (active) {
    const float *kpx = (const float *)(smem + P.off_kpx);
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    plm_rows<LC + 1>(l_top, (float)x, (float)sq, [&](int kk, float p) {
      v[kk & 3] = p * kpx[kk];
      if ((kk & 3) == 3) row[kk / 4] = make_float4(v[0], v[1], v[2], v[3]);
    });
    if (n_p & 3) row[n_p / 4] = make_float4(v[0], v[1], v[2], v[3]);
  }
  __syncwarp();
  if (do_der)
    copy_out(std::integral_constant<int, T4 - H4>(), H4, AW4, 0);
  else
    copy_out(std::integral_constant<int, ND4 - H4>(), H4, AW4, 0);
}

// ------------------------------------------------------------ layouts
__host__ __device__ inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }
// Staged rows are 16 bytes longer than the global ones: consecutive rows start in
// distinct bank groups and stay 16-byte aligned for the asynchronous copies.
__host__ __device__ inline int stage_stride(int LC) { return row_len(LC) + 4; }
// row stride of H: the species blocks padded to AMAX, plus 4 so that 128-bit
// loads of consecutive k rows fall in distinct banks
__host__ __device__ inline int h_stride(int n_species, int AMAX) { return n_species * AMAX + 4; }
// floats per site of the kept c_nlm, (n, k_max | 1) of (re, im), padded to a multiple of 4 so that every
// site's block starts 16-byte aligned
__host__ __device__ inline size_t keep_stride(const DevParams &P) {
  return ((size_t)2 * P.n_max * (size_t)(P.k_max | 1) + 3) / 4 * 4;
}
// bytes of constants a site kernel keeps in shared memory (mode 0 descriptor, 1 contract)
__host__ __device__ inline size_t site_blob_bytes(const DevParams &P, int mode) {
  return mode ? (size_t)P.blob_c_bytes : (size_t)(P.blob_bytes - P.off_rad);
}

template <int NT>
__device__ __forceinline__ void copy_site_blob(const DevParams &P, unsigned char *smem, int mode) {
  const uint4 *src = (const uint4 *)(mode ? P.blob_c : P.blob + P.off_rad);
  uint4 *dst = (uint4 *)smem;
  for (int t = threadIdx.x; t < (int)(site_blob_bytes(P, mode) / 16); t += NT) dst[t] = src[t];
}

// Offset of a blob section inside the site kernels' shared copy.
#define SBLOB(off) (smem + (P.off) - P.off_rad)
#define SBLOBC(off) (smem + (P.off))

__device__ __forceinline__ const RadSp &rad_of(const unsigned char *smem, const DevParams &P, int s) {
  return *(const RadSp *)(smem + (size_t)s * SOAPB_RADSP_BYTES);
}

// Persistent scheduling of the tensor-core kernels: every CTA takes sites from a
// counter until none are left; which CTA computes a site does not change its result.  The next site
// is fetched ahead, so that neither the ticket nor the CSR bounds are a round
// trip between two sites: thread 0 takes the next ticket when a site starts,
// loads that site's bounds part-way through (ahead_bounds) and hands the three
// values to the CTA in cur[] when the site ends (ahead_publish, which also
// synchronises).  The first site is fetched by first_site.
// A launch processes the sites [site_lo, site_hi) of the batch.  Each CTA takes
// tickets until one is past the last site, so a launch hands out exactly
// (site_hi - site_lo) + gridDim.x of them; the CTA holding the last one puts
// the counter back to 0 for the next launch.  Returns the site (>= site_hi: none left).
__device__ __forceinline__ int take_ticket(const DevBatch &B, int *ticket) {
  const int n = B.site_hi - B.site_lo;
  const int t = atomicAdd(ticket, 1);
  if (t == n + (int)gridDim.x - 1) atomicExch(ticket, 0);
  return (B.order != nullptr && t < n) ? B.order[t] : B.site_lo + min(t, n);
}
__device__ __forceinline__ void first_site(const DevBatch &B, int *ticket, int *cur) {
  if (threadIdx.x == 0) {
    const int s0 = take_ticket(B, ticket);
    cur[0] = s0;
    cur[1] = s0 < B.site_hi ? B.off[s0] : 0;
    cur[2] = s0 < B.site_hi ? B.off[s0 + 1] : 0;
  }
  __syncthreads();
}
__device__ __forceinline__ void ahead_bounds(const DevBatch &B, int nx, int &nx0, int &nx1) {
  if (threadIdx.x == 0 && nx < B.site_hi) {
    nx0 = B.off[nx];
    nx1 = B.off[nx + 1];
  }
}
// Callers guarantee a __syncthreads between their reads of cur[] at the top of
// the site and this call.
__device__ __forceinline__ void ahead_publish(int *cur, int nx, int nx0, int nx1) {
  if (threadIdx.x == 0) {
    cur[0] = nx;
    cur[1] = nx0;
    cur[2] = nx1;
  }
  __syncthreads();
}

// 16-byte asynchronous global -> shared copy (no register staging).
__device__ __forceinline__ void cp_async16(void *dst_smem, const void *src_gmem) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src_gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// Copies the rows of entries [ebase, ebase + n_round) of a chunk into the
// staging area (the angular rows and the radial rows), every 16-byte piece an
// independent asynchronous copy.  The caller synchronises afterwards.
template <int NT, int AMAX, int LC>
__device__ __forceinline__ void stage_entries(const DevParams &P, const DevBatch &B, const int *sEnt,
                                              int chunk, int ebase, int n_round, float *sA, float *sR) {
  constexpr int AW4 = row_len(LC) / 4;
  const int AS = stage_stride(LC);
  for (int t = threadIdx.x; t < n_round * AW4; t += NT) {
    const int el = t / AW4, j4 = t - el * AW4;
    const int k = chunk + (sEnt[ebase + el] & 0xffffff);
    cp_async16(sA + (size_t)el * AS + 4 * j4, B.ang + (size_t)k * (4 * AW4) + 4 * j4);
  }
  constexpr int R4 = AMAX / 4;
  for (int t = threadIdx.x; t < n_round * R4; t += NT) {
    const int el = t / R4, j4 = t - el * R4;
    const int code = sEnt[ebase + el];
    const int k = chunk + (code & 0xffffff), s = code >> 24;
    cp_async16(sR + (size_t)el * AMAX + 4 * j4, B.rad + ((size_t)k * P.n_species + s) * 2 * AMAX + 4 * j4);
  }
  cp_async_wait_all();
}

// ------------------------------------------------------------ tensor cores
// 3xTF32 on mma.sync m16n8k8: each FP32 operand is split into a TF32 head and
// a TF32 tail, x = hi + lo to ~22 bits, and a*b is taken as
// lo_a*hi_b + hi_a*lo_b + hi_a*hi_b (small terms first) with FP32 accumulation.
__device__ __forceinline__ unsigned to_tf32(float x) {
  unsigned r;
  asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void split_tf32(float x, unsigned &hi, unsigned &lo) {
  hi = to_tf32(x);
  lo = to_tf32(x - __uint_as_float(hi));
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma_3xtf32(float (&d)[4], const float (&a)[4], const float (&b)[2]) {
  unsigned ah[4], al[4], bh[2], bl[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) split_tf32(a[i], ah[i], al[i]);
#pragma unroll
  for (int i = 0; i < 2; ++i) split_tf32(b[i], bh[i], bl[i]);
  mma_tf32(d, al, bh);
  mma_tf32(d, ah, bl);
  mma_tf32(d, ah, bh);
}

// Power spectrum tiles P_l[n][j] = sum_c X_l[n][c] X_l[J_j][c] with
// X_l[n] = (Re c_nl0, r2 Re c_nl1 .. r2 Re c_nll, Im c_nl0, r2 Im c_nl1 ..), r2 = sqrt 2,
// i.e. P_l[n][j] = sum_m w_m Re(c_nlm conj c_{J_j}lm), w_0 = 1, w_m = 2
// (src/soap_turbo.f90:750-795).  A warp per (l, 16-row tile, 8-column tile);
// fragment layouts of m16n8k8: lane = 4 g + t, A rows g / g+8 and columns
// t / t+4, B row t / t+4 and column g, D rows g / g+8 and columns 2t, 2t+1.
template <int NT>
__device__ __forceinline__ void ps_tensor(const DevParams &P, const float *sC, float *sPl, const int *J) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int MT = P.ps_mt, NTJ = P.ps_nt, MR = 16 * MT, JP = 8 * NTJ;
  const int n_max = P.n_max, KS = P.k_max | 1;
  const int per_l = MT * NTJ, n_units = (P.l_max + 1) * per_l;
  for (int u = warp; u < n_units; u += NT / 32) {
    const int l = u / per_l, r = u - l * per_l, mt = r / NTJ, nt = r - mt * NTJ;
    const int kb = l * (l + 1) / 2, KL = 2 * (l + 1);
    const int n0 = 16 * mt + g, n1 = n0 + 8, jn = J[8 * nt + g];
    float d[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c0 = 0; c0 < KL; c0 += 8) {
      float a[4], b[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int col = c0 + t + 4 * h;
        float x0 = 0.f, x1 = 0.f, xj = 0.f;
        if (col < KL) {
          const int im = col > l, m = im ? col - l - 1 : col;
          const float w = m ? 1.41421356237309504880f : 1.f;
          const int off = (im ? n_max * KS : 0) + kb + m;
          if (n0 < n_max) x0 = w * sC[n0 * KS + off];
          if (n1 < n_max) x1 = w * sC[n1 * KS + off];
          if (jn >= 0) xj = w * sC[jn * KS + off];
        }
        a[2 * h] = x0;
        a[2 * h + 1] = x1;
        b[h] = xj;
      }
      mma_3xtf32(d, a, b);
    }
    float *o = sPl + (size_t)(l * MR + n0) * JP + 8 * nt + 2 * t;
    o[0] = d[0];
    o[1] = d[1];
    o[8 * JP] = d[2];
    o[8 * JP + 1] = d[3];
  }
}

// ---- C. of a site, from its c_nlm in sC (FP32, (re/im, n, KS)): the power
// spectrum of the kept components (src/soap_turbo.f90:750-795), the
// compression, the norm and the normalised FP64 output (:798-809, 904-909),
// and with keep the c_nlm and norm the contract reads.  keep: bit 0 keeps, bit
// 1 accumulates into soap_out.  tiles: the power spectrum from tensor-core
// tiles in sPl (the tcgen05 kernel: formed there when ps_ready, else here with
// mma.sync 3xTF32 tiles); else one dot product per kept component on the CUDA
// cores (k_descriptor: measured faster than the mma.sync tiles).
template <int NT>
__device__ __forceinline__ void site_output(const DevParams &P, unsigned char *smem, const float *sC, float *sP,
                                            float *sS, float *sPl, const int *kept, double *sRed, int site,
                                            double *__restrict__ soap_out, float *__restrict__ keep_c,
                                            double *__restrict__ keep_norm, int keep, bool tiles,
                                            bool ps_ready = false) {
  const int tid = threadIdx.x;
  const int KS = P.k_max | 1;
  const int n_max = P.n_max;
    // ---- C. power spectrum of the kept components (src/soap_turbo.f90:750-795)
    float *pout = P.cmap_identity ? sS : sP;
    double nrm2 = 0.0;
    if (tiles) {
      // on the tensor cores, then gathered into the kept components with the
      // sqrt 2 of n != n'
      if (!ps_ready) {
        ps_tensor<NT>(P, sC, sPl, (const int *)SBLOB(off_psj));
        __syncthreads();
      }
      const int *kpos = (const int *)SBLOB(off_kpos);
      for (int q = tid; q < P.n_kept; q += NT) {
        const int code = kpos[q];
        const float v = (code < 0 ? 1.41421356237309504880f : 1.f) * sPl[code & 0x7fffffff];
        pout[q] = v;
        nrm2 += (double)v * (double)v;
      }
    } else
    for (int q = tid; q < P.n_kept; q += NT) {
      const int code = kept[q];
      const int n = code & 0xff, np = (code >> 8) & 0xff, l = code >> 16;
      const int kb = l * (l + 1) / 2;
      const float *cn_r = sC + (size_t)n * KS + kb, *cn_i = sC + (size_t)(n_max + n) * KS + kb;
      const float *cp_r = sC + (size_t)np * KS + kb, *cp_i = sC + (size_t)(n_max + np) * KS + kb;
      const float acc0 = cn_r[0] * cp_r[0] + cn_i[0] * cp_i[0];
      float acc = 0.f;
      for (int m = 1; m <= l; ++m) acc += cn_r[m] * cp_r[m] + cn_i[m] * cp_i[m];
      const float base = (n == np) ? 1.f : 1.41421356237309504880f;
      const float v = base * (acc0 + 2.f * acc);
      pout[q] = v;
      nrm2 += (double)v * (double)v;
    }
    if (!P.cmap_identity) {
      // compression through the map (:798-802)
      __syncthreads();
      nrm2 = 0.0;
      for (int o = tid; o < P.n_soap; o += NT) {
        float v = 0.f;
        for (int t = P.pi_off[o]; t < P.pi_off[o + 1]; ++t) v += P.pi_el[t] * sP[P.pi_q[t]];
        sS[o] = v;
        nrm2 += (double)v * (double)v;
      }
    }
    double *out = soap_out + (size_t)site * P.n_soap;
    // accumulate: the caller's soap row is added before the norm is taken, as
    // the reference adds the compressed descriptor into soap (:798-802).  Each
    // thread reads and writes the same components of the row.
    const bool acc = (keep & 2) != 0;
    if (acc) {
      nrm2 = 0.0;
      for (int o = tid; o < P.n_soap; o += NT) {
        const double v = (double)sS[o] + out[o];
        nrm2 += v * v;
      }
    }
    nrm2 = block_sum<NT>(nrm2, sRed);  // (:805-809)
    double norm = sqrt(nrm2);
    if (norm < 1.0e-5) norm = 1.0;
    const double inv = 1.0 / norm;
    if (acc)
      for (int o = tid; o < P.n_soap; o += NT) out[o] = ((double)sS[o] + out[o]) * inv;
    else
      for (int o = tid; o < P.n_soap; o += NT) out[o] = (double)sS[o] * inv;
    if (keep & 1) {
      float2 *kc = (float2 *)(keep_c + (size_t)site * keep_stride(P));
      for (int t = tid; t < n_max * KS; t += NT) kc[t] = make_float2(sC[t], sC[n_max * KS + t]);
      if (tid == 0) keep_norm[site] = norm;
    }
}

// ------------------------------------------------------------ entries of a warp
// The species the radial expansion of each pair of [c0, c1) applies to, for the
// calling warp: byte c of the result is pair c0 + 32 c + lane, bit s species s
// (mask set, inside the species' rcut_hard and rcut_max, the self pair only when
// its expansion is used, and not for the force contraction, vjp).
__device__ __forceinline__ unsigned long long valid_species(const DevParams &P, const DevBatch &B, int p_begin,
                                                            int c0, int c1, bool vjp) {
  const int lane = threadIdx.x & 31;
  unsigned long long v = 0ull;
  // four pairs a lane at a time under one look at each species' constants: a site of
  // several chunks comes here once per chunk and species, and pair by pair its rows of
  // 340 pairs and eight species took the descriptor 163 us at 100 sites, so 103
  for (int cb = 0; c0 + 32 * cb < c1; cb += 4) {
    double r[4];
    unsigned bits[4], ok[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int k = c0 + 32 * (cb + c) + lane;
      r[c] = k < c1 ? B.rjs[k] : 0.0;
      bits[c] = k < c1 ? B.bits[k] : 0u;
      ok[c] = 0u;
    }
    // a pair at or beyond rcut_max has no angular row (the reference zeroes its
    // angular coefficients, src/soap_turbo_angular.f90:549-574); it only matters
    // for poly3operator, whose radial part has no rcut_hard cut
    for (int s = 0; s < P.n_species; ++s) {
      const double cut = fmin(P.rad[s].rcut_hard, P.rcut_max);
      const bool central = !vjp && P.rad[s].do_central;
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (r[c] < cut && (c0 + 32 * (cb + c) + lane > p_begin || central)) ok[c] |= bits[c] & (1u << s);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) v |= (unsigned long long)ok[c] << (8 * (cb + c));
  }
  return v;
}

// Appends species s's entries of a chunk of n_chunk pairs, in order, as chunk-local
// pair | s << 8 from list[e] on; returns the end.  Every warp of a CTA may write
// the same list: it writes the same values.
__device__ __forceinline__ int list_species(unsigned long long valid, int s, int n_chunk, int e, unsigned short *list) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  for (int c = 0; 32 * c < n_chunk; ++c) {
    const bool on = (valid >> (8 * c + s)) & 1ull;
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (on) list[e + __popc(m & lt)] = (unsigned short)((32 * c + lane) | (s << 8));
    e += __popc(m);
  }
  return e;
}

// Two FP32 values in a 64-bit register pair, and two fused multiply-adds in one
// instruction, each rounded as fmaf's.  Kept as 64-bit values from the load to
// the last use: a float2 would be taken apart and put together around each one.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float x, float y) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
  return d;
}
__device__ __forceinline__ f32x2 ffma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

__device__ __forceinline__ f32x2 fmul2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// The site kernels' FP64 sums (the norm, q . G, the central pair) run over slots: slot
// v of `slots` (64, 128 or 256) adds its terms v, v + slots, .. in order, 32 slots are
// added by warp_sum and the warps' sums by slot_tree, as block_sum of so many threads
// adds them.  So a result does not depend on the CTA size that a site was given.
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <int STRIDE = 1>
__device__ __forceinline__ double slot_tree(const double *r, int slots) {
  constexpr int S = STRIDE;
  if (slots == 128) return (r[0] + r[2 * S]) + (r[S] + r[3 * S]);
  if (slots == 64) return r[0] + r[S];
  return ((r[0] + r[4 * S]) + (r[2 * S] + r[6 * S])) + ((r[S] + r[5 * S]) + (r[3 * S] + r[7 * S]));
}

// slot_tree over the warp_sums of the four slots (lane, lane + 32, ..) that a lane
// holds, in eight shuffles: each half of the lanes keeps half of the sums.
__device__ __forceinline__ double slots_by_warp(const double (&v)[4]) {
  const bool up = threadIdx.x & 16, odd = threadIdx.x & 8;
  const double a = (up ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], 16);
  const double b = (up ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], 16);
  double t = (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  t += __shfl_xor_sync(0xffffffffu, t, 16);
  return t + __shfl_xor_sync(0xffffffffu, t, 8);
}

// The norm of a site's components (:805-809), squared: over 128 slots by every warp for
// itself, or over `slots` of them by the CTA through red (slots / 32 doubles).
__device__ __forceinline__ double norm2_by_warp(const float *s, int n) {
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  for (int o = threadIdx.x & 31; o < n; o += 128)
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const double y = o + 32 * w < n ? (double)s[o + 32 * w] : 0.0;
      v[w] = fma(y, y, v[w]);
    }
  return slots_by_warp(v);
}
template <typename Value>
__device__ __forceinline__ double norm2_by_slots(int n, int slots, double *red, Value value) {
  const int lane = threadIdx.x & 31;
  for (int w = threadIdx.x >> 5; 32 * w < slots; w += blockDim.x >> 5) {
    double v = 0.0;
    for (int o = 32 * w + lane; o < n; o += slots) {
      const double y = value(o);
      v = fma(y, y, v);
    }
    v = warp_sum(v);
    if (lane == 0) red[w] = v;
  }
  __syncthreads();
  return slot_tree(red, slots);
}

// A site's components s added to the caller's row before the norm is taken, as the
// reference adds the compressed descriptor into soap (:798-802); returns the norm.  The row
// may lie in host memory, a round trip over the link away: with room for the sums (sum)
// it is read once, by loads that overlap (page-locked soap of 5000 and 1679 sites, both
// calls: 5163 -> 4743 and 1605 -> 1560 us).  An instantiation of its own: beside the other
// outcome in one kernel it took that 1 to 4 % more time.
__device__ __forceinline__ double add_and_normalise(const float *s, int n, int slots, double *red, double *sum,
                                                 double *out) {
  if (sum) {
#pragma unroll 4
    for (int o = threadIdx.x; o < n; o += blockDim.x) sum[o] = (double)s[o] + out[o];
    __syncthreads();
  }
  auto value = [&](int o) { return sum ? sum[o] : (double)s[o] + out[o]; };
  double norm = sqrt(norm2_by_slots(n, slots, red, value));
  if (norm < 1.0e-5) norm = 1.0;
  const double inv = 1.0 / norm;
  for (int o = threadIdx.x; o < n; o += blockDim.x) out[o] = value(o) * inv;
  return norm;
}

// ------------------------------------------------------------ descriptor
// One CTA of a few warps per site; a thread owns one k = (l, m) and NH of the
// radial indices of every species block (warp w: k = 32 (w % kw) + lane, radial
// indices from NH (w / kw)).
//  entries    the (pair, species) entries the expansion applies to, by species,
//             then in CSR order, found with ballots by every warp for itself
//  staging    a round of at most 64 entries: the rows' first part and R_n, a
//             warp per row, with 16-byte asynchronous copies
//  c_nlm      FP32 partial sums over groups of four entries flushed into FP64;
//             two radial indices per fma.rn.f32x2.  A species' sums stay in
//             registers from its first entry to its last.  Rounds are those of
//             `chunk` pairs' entries cut at multiples of min(chunk / 2, 64): the
//             groups do not depend on the launch shape.
//  spectrum   one dot product per kept component, the components ordered by
//             l (P.ps_order) so that a warp's dot products are equally long
// What bounds it: instructions, and the latency of a warp's chain: per site of 52 pairs and
// three species 14.0 k with four radial indices a thread, issued at 60 % of the rate (39.6
// us at 1679 sites), 8.7 k with eight, at 46 % (227 us at 13092); the products are a tenth
// of them.  One CTA of 128 threads that staged, sorted and summed behind barriers took
// 15 k: 55 and 338 us.
struct DescLayout {
  size_t list, base, X, P, S, total;
};
__host__ __device__ constexpr int desc_head(int LC) { return (row_p(LC) + (LC + 1) * (LC + 2) / 2 + 3) / 4 * 4; }
// a staged entry: the row's first part, then its species' R_n
__host__ __device__ constexpr int desc_stride(int AMAX, int LC) { return desc_head(LC) + AMAX; }
__host__ __device__ inline DescLayout desc_layout(const DevParams &P, int chunk, int AMAX, int LC) {
  DescLayout L{};
  size_t o = align_up((size_t)P.n_max * (size_t)(P.k_max | 1) * sizeof(float2), 16);  // c_nlm, (n, KS), at 0
  L.base = o; o += 16 * sizeof(int);
  L.list = o; o = align_up(o + (size_t)chunk * P.n_species * sizeof(unsigned short), 16);
  // the staged round; after c_nlm the components and the compressed descriptor
  L.X = L.P = o;
  const size_t x = o + (size_t)(chunk / 2 < 64 ? chunk / 2 : 64) * desc_stride(AMAX, LC) * sizeof(float);
  L.S = o + (P.cmap_identity ? 0 : (size_t)P.n_kept * sizeof(float));
  const size_t y = L.S + (size_t)P.n_soap * sizeof(float);
  L.total = align_up(x > y ? x : y, 16);
  return L;
}

// resident CTAs the register count is held to (the staged round allows seven)
__host__ __device__ constexpr int desc_min_ctas(int AMAX, int NH, int groups) {
  if (groups) return 768 / groups;
  return AMAX == 8 ? (NH == 8 ? 7 : NH == 4 ? 6 : 3) : 3;
}

// Threads per site: those of one species' sums; with GROUPS more, in groups of warps
// each of which sums another species (launch parameter groups)
template <int AMAX, int LC, int NH, int GROUPS>
constexpr int kDescThreads = GROUPS ? GROUPS : ((LC + 1) * (LC + 2) / 2 + 31) / 32 * 32 * (AMAX / NH);

// ACC: the components are added to the caller's rows
template <int AMAX, int LC, int NH, int GROUPS, bool ACC>
__global__ void __launch_bounds__(kDescThreads<AMAX, LC, NH, GROUPS>,
                                  desc_min_ctas(AMAX, NH, GROUPS))
    k_descriptor(const DevParams P, const DevBatch B, int chunk, int kw, int groups, double *__restrict__ soap_out,
                 float *__restrict__ keep_c, double *__restrict__ keep_norm, int keep) {
  // keep: whether c_nlm and the norm are kept for the contract
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int AW = row_len(LC), ST = desc_stride(AMAX, LC), HD = desc_head(LC);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x, nw = nt >> 5;
  const DescLayout Ly = desc_layout(P, chunk, AMAX, LC);
  float2 *sC = (float2 *)smem;
  float *sX = (float *)(smem + Ly.X), *sP = (float *)(smem + Ly.P), *sS = (float *)(smem + Ly.S);
  int *sBase = (int *)(smem + Ly.base);
  unsigned short *list = (unsigned short *)(smem + Ly.list);
  const int KS = P.k_max | 1, nsp = P.n_species;
  if constexpr (GROUPS == 0) groups = 1;
  const int group = GROUPS ? warp * groups / nw : 0, wg = GROUPS ? warp - group * (nw / groups) : warp;
  const int k_of = 32 * (wg % kw) + lane, n0 = NH * (wg / kw);
  const bool own = k_of < P.k_max;
  const int kk = own ? k_of : P.k_max - 1;  // the last lanes repeat the last k and store nothing
  const int lm = __ldg((const int *)(P.blob + P.off_klm) + kk), l = lm & 0xff, m = lm >> 8;
  const int rounds = min(chunk / 2, 64);
  const int4 it0 = tid < P.n_kept ? __ldg(P.ps_order + tid) : make_int4(0, 0, 0, 0);
  // the 16-byte pieces of an entry that the lane stages: of the row's head, then of R_n
  constexpr int NC = (HD / 4 + AMAX / 4 + 31) / 32;
  const int n_head = (row_p(LC) + P.k_max + 3) / 4;
  struct {
    bool on, rad;
    int first, dst;
    unsigned per_pair, per_species;
  } piece[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int t = lane + 32 * c, r = t - n_head;
    piece[c].on = r < AMAX / 4;
    piece[c].rad = r >= 0;
    piece[c].first = 4 * (r >= 0 ? r : t);
    piece[c].dst = r >= 0 ? HD + 4 * r : 4 * t;
    piece[c].per_pair = r >= 0 ? nsp * 2 * AMAX : AW;
    piece[c].per_species = r >= 0 ? 2 * AMAX : 0;
  }

  const int site = B.order ? B.order[blockIdx.x] : B.site_lo + (int)blockIdx.x;
  const int p_begin = B.off[site], p_end = min(B.off[site + 1], B.n_pairs);
  // the species whose sums the thread holds, its rounds so far, their sums but
  // for the last, and that of the last
  int cs = group, n_rounds = 0;
  double tr[NH], ti[NH], dr[NH], di[NH];
  float2 *kc = (float2 *)(keep_c + (keep ? (size_t)site * keep_stride(P) : 0)) + kk;
  auto finish = [&]() {  // species cs is complete
    const int a = P.rad[cs].alpha, nb = P.rad[cs].nbeg;
    if (n_rounds != 1)
#pragma unroll
      for (int n = 0; n < NH; ++n) {
        dr[n] = n_rounds ? tr[n] + dr[n] : 0.0;
        di[n] = n_rounds ? ti[n] + di[n] : 0.0;
      }
    // poly3gauss central-atom term (src/soap_turbo.f90:646-662)
    if (P.basis == 1 && kk == 0) {
      const int mult = B.species_mult[site];
      for (int mm = 0; mm < mult; ++mm)
        if (B.species[(size_t)site * B.max_mult + mm] - 1 == cs)
#pragma unroll
          for (int n = 0; n < NH; ++n)
            if (n0 + n < a) dr[n] += P.central[nb + n0 + n];
    }
    float2 *cc = sC + (nb + n0) * KS + kk;
    if (own)
#pragma unroll
      for (int n = 0; n < NH; ++n)
        if (n0 + n < a) cc[n * KS] = make_float2((float)dr[n], (float)di[n]);
    if (own && keep) {
      float2 *kr = kc + (nb + n0) * KS;
#pragma unroll
      for (int n = 0; n < NH; ++n)
        if (n0 + n < a) kr[n * KS] = make_float2((float)dr[n], (float)di[n]);
    }
    cs += groups;
    n_rounds = 0;
  };
  // a site of one chunk takes all its species at once; else a species per group at a time
  const bool multi = p_end - p_begin > chunk;
  for (int s_lo = 0; s_lo < nsp; s_lo += multi ? groups : nsp) {
    const int s_hi = multi ? min(nsp, s_lo + groups) : nsp;
    for (int c0 = p_begin; c0 < p_end; c0 += chunk) {
      const int c1 = min(p_end, c0 + chunk);
      const unsigned long long valid = valid_species(P, B, p_begin, c0, c1, false);
      // the place of species s_lo among the chunk's entries, which fixes the rounds
      const int e0 = __reduce_add_sync(0xffffffffu, __popcll(valid & (0x0101010101010101ull * ((1u << s_lo) - 1u))));
      if (multi) __syncthreads();  // the previous chunk's list is read
      int e = e0;
      for (int s = s_lo; s < s_hi; ++s) {
        if (lane == 0) sBase[s] = e;
        e = list_species(valid, s, c1 - c0, e, list - e0);
      }
      if (lane == 0) sBase[s_hi] = e;
      __syncwarp();
      const int e1 = e;
      const float *src[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c)
        src[c] = piece[c].rad ? B.rad + (size_t)c0 * nsp * 2 * AMAX + piece[c].first
                              : B.ang + (size_t)c0 * AW + piece[c].first;
      for (int w0 = e0, w1; w0 < e1; w0 = w1) {
        w1 = min(e1, w0 + rounds - (w0 & (rounds - 1)));
        float *dst = sX + warp * ST;
#pragma unroll 4
        for (int q = w0 + warp; q < w1; q += nw, dst += nw * ST) {
          const unsigned code = list[q - e0], j = code & 0xffu, sp = code >> 8;
#pragma unroll
          for (int c = 0; c < NC; ++c)
            if (piece[c].on)
              cp_async16(dst + piece[c].dst, src[c] + (j * piece[c].per_pair + sp * piece[c].per_species));
        }
        cp_async_wait_all();
        __syncthreads();
        for (int s = s_lo + group; s < s_hi; s += groups) {
          const int lo = max(w0, sBase[s]), hi = min(w1, sBase[s + 1]);
          if (lo >= hi) continue;
          while (cs < s) finish();
          if (n0 >= P.rad[s].alpha) continue;
          // the central pair carries central_weight (:638-646): the pair kernel
          // expanded every pair as a neighbour
          const bool weighted = P.rad[s].cw != 1.0 && c0 == p_begin && lo == sBase[s] && (list[lo - e0] & 0xff) == 0;
          const float cw = (float)P.rad[s].cw;
          if (n_rounds > 0)
#pragma unroll
            for (int n = 0; n < NH; ++n) {
              tr[n] = n_rounds > 1 ? tr[n] + dr[n] : dr[n];
              ti[n] = n_rounds > 1 ? ti[n] + di[n] : di[n];
            }
          ++n_rounds;
          f32x2 pr[NH / 2], pi[NH / 2];
          const float *A = sX + (lo - w0) * ST;
          const float *aP = A + row_p(LC) + kk, *aL = A + row_il(LC) + l, *aE = A + row_e(LC) + 2 * m,
                      *aR = A + HD + n0;
          auto add = [&](int o, bool first, bool opens) {  // the round's first entry, its group's first
            // u_k = (preflm_k P_k) (amp i_l) (src/soap_turbo_angular.f90:590-594)
            const float u = aP[o] * aL[o];
            const float2 e2 = *(const float2 *)(aE + o);
            const float ar = u * e2.x, ai = u * e2.y;
            const f32x2 ar2 = pack2(ar, ar), ai2 = pack2(ai, ai);
            f32x2 r[NH / 2];
            if constexpr (NH % 4 == 0) {
#pragma unroll
              for (int n = 0; n < NH / 4; ++n) {
                const ulonglong2 v = *(const ulonglong2 *)(aR + o + 4 * n);
                r[2 * n] = v.x;
                r[2 * n + 1] = v.y;
              }
            } else {
#pragma unroll
              for (int n = 0; n < NH / 2; ++n) r[n] = *(const f32x2 *)(aR + o + 2 * n);
            }
            if (first && weighted)
#pragma unroll
              for (int n = 0; n < NH / 2; ++n) {
                const float2 v = unpack2(r[n]);
                r[n] = pack2(v.x * cw, v.y * cw);
              }
#pragma unroll
            for (int n = 0; n < NH / 2; ++n) {
              pr[n] = opens ? fmul2(r[n], ar2) : ffma2(r[n], ar2, pr[n]);
              pi[n] = opens ? fmul2(r[n], ai2) : ffma2(r[n], ai2, pi[n]);
            }
          };
          auto flush = [&](bool first) {  // the round's first group
#pragma unroll
            for (int n = 0; n < NH / 2; ++n) {
              const float2 vr = unpack2(pr[n]), vi = unpack2(pi[n]);
              dr[2 * n] = first ? (double)vr.x : dr[2 * n] + (double)vr.x;
              dr[2 * n + 1] = first ? (double)vr.y : dr[2 * n + 1] + (double)vr.y;
              di[2 * n] = first ? (double)vi.x : di[2 * n] + (double)vi.x;
              di[2 * n + 1] = first ? (double)vi.y : di[2 * n + 1] + (double)vi.y;
            }
          };
          int i = lo;
          for (; i + 4 <= hi; i += 4) {
#pragma unroll
            for (int q = 0; q < 4; ++q) add(q * ST, q == 0 && i == lo, q == 0);
            if (i == lo) flush(true);
            else flush(false);
            aP += 4 * ST;
            aL += 4 * ST;
            aE += 4 * ST;
            aR += 4 * ST;
          }
          if (i < hi) {
            const int n_last = hi - i;
            add(0, i == lo, true);
            if (n_last > 1) add(ST, false, false);
            if (n_last > 2) add(2 * ST, false, false);
            if (i == lo) flush(true);
            else flush(false);
          }
        }
        __syncthreads();  // the round's rows are read
      }
    }
  }
  while (cs < nsp) finish();
  __syncthreads();
  // power spectrum of the kept components (src/soap_turbo.f90:750-795)
  float *pout = P.cmap_identity ? sS : sP;
  int4 it = it0;
  for (int t = tid; t < P.n_kept; t += nt) {
    const int4 nx = t + nt < P.n_kept ? __ldg(P.ps_order + t + nt) : it;  // a round trip ahead
    const float2 *cn = sC + it.x, *cp = sC + it.y;
    const int lq = it.w & 0xff;
    const float acc0 = cn[0].x * cp[0].x + cn[0].y * cp[0].y;
    float acc = 0.f;
#pragma unroll 4
    for (int q = 1; q <= lq; ++q) acc += cn[q].x * cp[q].x + cn[q].y * cp[q].y;
    const float base = it.w < 0 ? 1.41421356237309504880f : 1.f;
    const float v = base * (acc0 + 2.f * acc);
    pout[it.z] = v;
    it = nx;
  }
  __syncthreads();
  if (!P.cmap_identity) {
    // compression through the map (:798-802)
    for (int o = tid; o < P.n_soap; o += nt) {
      float v = 0.f;
      for (int t = P.pi_off[o]; t < P.pi_off[o + 1]; ++t) v += P.pi_el[t] * sP[P.pi_q[t]];
      sS[o] = v;
    }
    __syncthreads();
  }
  double *out = soap_out + (size_t)site * P.n_soap, norm;
  if constexpr (ACC) {
    const size_t at = align_up(Ly.S + (size_t)P.n_soap * sizeof(float), 8);
    const bool room = at + (size_t)P.n_soap * sizeof(double) <= Ly.total;
    norm = add_and_normalise(sS, P.n_soap, chunk, (double *)(smem + Ly.base), room ? (double *)(smem + at) : nullptr, out);
  } else {
    norm = sqrt(chunk == 128 ? norm2_by_warp(sS, P.n_soap)
                             : norm2_by_slots(P.n_soap, chunk, (double *)(smem + Ly.base), [&](int o) { return (double)sS[o]; }));
    if (norm < 1.0e-5) norm = 1.0;
    const double inv = 1.0 / norm;
    for (int o = tid; o < P.n_soap; o += nt) out[o] = (double)sS[o] * inv;
  }
  if (keep && tid == 0) keep_norm[site] = norm;
}

// ------------------------------------------------------------ descriptor on tensor cores
// get_soap's c_nlm (src/soap_turbo.f90:619-664) as a tcgen05 product per site:
// D[2 k + re/im][n] = sum_e A_e(k, re/im) R_e(n), with A_e(k) = u_k e^{-i m phi}
// of entry e (u_k = (preflm_k P_k)(amp i_l), the same FP32 products as the
// CUDA-core kernel) and R_e its species' 4 pi R_n (zero in the other species'
// columns).  M = 128 rows (2 k_max <= 128), N = 32 columns (n_max <= 32), K =
// the entries, 16 at a time (two K-steps of 3xTF32 MMAs); each group's FP32
// partial sums are read from TMEM by the thread that owns the row and added to
// its FP64 accumulators (fixed order, no atomics) -- the accuracy of the
// CUDA-core kernel's FP32 groups flushed into FP64.  Then the poly3gauss
// central term, and k_descriptor's power spectrum, norm and output.
constexpr int kTdGroup = 16;   // entries per group (two K-steps)
constexpr int kTdCols = 32;    // D columns (n)
constexpr int kTdTmemCols = 128;  // c_nlm's 32 columns, then the power spectrum's up to 128

struct TdLayout {
  size_t red, ent, wcnt, misc, mbar, tmem, Ahi, Alo, Bhi, Blo, Phi, Plo, X, R, A, C, P, S, Pl, total;
};
constexpr int kPsTcK = 32;  // K columns of a power-spectrum tile (the host's groups agree)
__host__ __device__ inline TdLayout make_td_layout(const DevParams &P, int NT, int AMAX, int LC) {
  TdLayout L{};
  const size_t KS = (size_t)(P.k_max | 1), nsp = (size_t)P.n_species;
  size_t o = site_blob_bytes(P, 0);
  L.red = o;  o += 40 * sizeof(double);
  L.ent = o;  o += (size_t)NT * nsp * sizeof(int);
  L.wcnt = o; o += (size_t)SOAPB_MAX_SPECIES * (NT / 32) * sizeof(int);
  L.misc = o; o += 64 * sizeof(int);
  L.mbar = align_up(o, 8); o = L.mbar + 8;
  L.tmem = o; o += 8;
  o = align_up(o, 1024);
  // the c_nlm tiles, and afterwards the power-spectrum tiles, in one region
  const size_t tcb = o;
  L.Ahi = o; o += 128 * kTdGroup * 4;
  L.Alo = o; o += 128 * kTdGroup * 4;
  L.Bhi = o; o += kTdCols * kTdGroup * 4;
  L.Blo = o; o += kTdCols * kTdGroup * 4;
  if (P.ps_ng > 0) {
    L.Phi = tcb;
    L.Plo = tcb + 128 * kPsTcK * 4;
    const size_t pe = tcb + 2 * 128 * kPsTcK * 4;
    o = o > pe ? o : pe;
  }
  o = align_up(o, 16);
  L.X = o;
  size_t x = o;
  L.R = x; x += kTdGroup * AMAX * sizeof(float);
  L.A = x; x += kTdGroup * (size_t)stage_stride(LC) * sizeof(float);
  const size_t end_stage = x;
  x = o;
  L.C = x; x += 2 * (size_t)P.n_max * KS * sizeof(float);
  L.P = x; x += (size_t)P.n_kept * sizeof(float);
  L.S = x; x += (size_t)P.n_soap * sizeof(float);
  if (P.ps_mt > 0) {
    x = align_up(x, 16);
    L.Pl = x; x += (size_t)(P.l_max + 1) * 16 * P.ps_mt * 8 * P.ps_nt * sizeof(float);
  }
  L.total = align_up(end_stage > x ? end_stage : x, 16);
  return L;
}

template <int NT, int AMAX, int LC>
__global__ void __launch_bounds__(NT) k_descriptor_tc(const DevParams P, const DevBatch B,
                                                      double *__restrict__ soap_out, float *__restrict__ keep_c,
                                                      double *__restrict__ keep_norm, int keep) {
  static_assert(NT == 128, "one thread per TMEM lane");
  extern __shared__ __align__(16) unsigned char smem[];  // no-swizzle operand tiles need 16-byte alignment
  const int AS = stage_stride(LC);
  const TdLayout Ly = make_td_layout(P, NT, AMAX, LC);
  const int *klm = (const int *)SBLOB(off_klm);
  const int *kept = (const int *)SBLOB(off_kept);
  const double *central = (const double *)SBLOB(off_central);
  double *sRed = (double *)(smem + Ly.red);
  float *sR = (float *)(smem + Ly.R);
  float *sA = (float *)(smem + Ly.A);
  float *sC = (float *)(smem + Ly.C);
  float *sP = (float *)(smem + Ly.P);
  float *sS = (float *)(smem + Ly.S);
  unsigned char *sAhi = smem + Ly.Ahi, *sAlo = smem + Ly.Alo, *sBhi = smem + Ly.Bhi, *sBlo = smem + Ly.Blo;
  uint64_t *mbar = (uint64_t *)(smem + Ly.mbar);
  uint32_t *tmem_slot = (uint32_t *)(smem + Ly.tmem);
  int *sEnt = (int *)(smem + Ly.ent);
  int *sW_cnt = (int *)(smem + Ly.wcnt);
  int *sMisc = (int *)(smem + Ly.misc);
  int *sBase = sMisc, *sCnt = sMisc + SOAPB_MAX_SPECIES, *sNent = sMisc + 2 * SOAPB_MAX_SPECIES;
  int *sSite = sMisc + 3 * SOAPB_MAX_SPECIES;

  const int tid = threadIdx.x, warp = tid >> 5;
  const int KS = P.k_max | 1;
  const int n_max = P.n_max, nsp = P.n_species, k_max = P.k_max;
  const uint32_t idesc = tc::idesc_tf32(128, kTdCols);
  copy_site_blob<NT>(P, smem, 0);
  if (warp == 0) tc::tmem_alloc(tmem_slot, kTdTmemCols);
  if (tid == 0) tc::mbar_init(mbar);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  // this thread's row of D: (k, re/im)
  const int my_k = tid >> 1, my_ri = tid & 1;
  const int my_l = my_k < k_max ? (klm[my_k] & 0xff) : 0, my_m = my_k < k_max ? (klm[my_k] >> 8) : 0;
  const uint32_t tmem = *tmem_slot;
  uint32_t phase = 0;
  bool failed = false;
  int col_s = -1, col_n = 0;  // (tid < 32) the species and local index of D column tid
  if (tid < kTdCols)
    for (int s = 0; s < nsp; ++s) {
      const RadSp &RS = rad_of(smem, P, s);
      if (tid >= RS.nbeg && tid < RS.nbeg + RS.alpha) {
        col_s = s;
        col_n = tid - RS.nbeg;
      }
    }

  first_site(B, B.ticket, sSite);
  for (;;) {
    const int site = sSite[0];
    if (site >= B.site_hi || failed) break;
    const int p_begin = sSite[1];
    const int p_end = min(sSite[2], B.n_pairs);
    int nx = 0, nx0 = 0, nx1 = 0;
    if (tid == 0) nx = take_ticket(B, B.ticket);
    double acc[kTdCols];
#pragma unroll
    for (int n = 0; n < kTdCols; ++n) acc[n] = 0.0;

    for (int chunk = p_begin; chunk < p_end && !failed; chunk += NT) {
      int slot[SOAPB_MAX_SPECIES];
      unsigned my_bits;
      double my_r;
      const int n_ent = build_entries<NT>(P, B, p_begin, chunk, p_end, false, sEnt, sW_cnt, sBase, sCnt, sNent,
                                          slot, my_bits, my_r);
      for (int ebase = 0; ebase < n_ent; ebase += kTdGroup) {
        const int n_g = min(kTdGroup, n_ent - ebase);
        // ---- the group's rows (angular and radial) into shared memory
        stage_entries<NT, AMAX, LC>(P, B, sEnt, chunk, ebase, n_g, sA, sR);
        __syncthreads();
        // the central pair's entries carry central_weight (:638-646)
        if (chunk == p_begin) {
          for (int el = tid; el < n_g; el += NT) {
            const int code = sEnt[ebase + el];
            const double cw = rad_of(smem, P, code >> 24).cw;
            if ((code & 0xffffff) == 0 && cw != 1.0)
#pragma unroll
              for (int n = 0; n < AMAX; ++n) sR[(size_t)el * AMAX + n] *= (float)cw;
          }
          __syncthreads();
        }
        // ---- A operand: row (k, re/im) of this thread, 16 entries
        {
          float v[kTdGroup];
#pragma unroll
          for (int e = 0; e < kTdGroup; ++e) {
            v[e] = 0.f;
            if (e < n_g && my_k < k_max) {
              const float *Ae = sA + (size_t)e * AS;
              // u_k = (preflm_k P_k)(amp i_l) (src/soap_turbo_angular.f90:590-594)
              const float u = Ae[row_p(LC) + my_k] * Ae[row_il(LC) + my_l];
              v[e] = u * Ae[row_e(LC) + 2 * my_m + my_ri];
            }
          }
#pragma unroll
          for (int e4 = 0; e4 < kTdGroup / 4; ++e4) {
            uint4 h, lo;
            tc::split(v[4 * e4], h.x, lo.x);
            tc::split(v[4 * e4 + 1], h.y, lo.y);
            tc::split(v[4 * e4 + 2], h.z, lo.z);
            tc::split(v[4 * e4 + 3], h.w, lo.w);
            const uint32_t off = tc::kmajor_off(tid, 4 * e4, kTdGroup);
            *(uint4 *)(sAhi + off) = h;
            *(uint4 *)(sAlo + off) = lo;
          }
        }
        // ---- B operand: row n, the entries' R_n of their species (else 0)
        if (tid < kTdCols) {
          float v[kTdGroup];
#pragma unroll
          for (int e = 0; e < kTdGroup; ++e) {
            v[e] = 0.f;
            if (e < n_g && col_s >= 0 && (sEnt[ebase + e] >> 24) == col_s) v[e] = sR[(size_t)e * AMAX + col_n];
          }
#pragma unroll
          for (int e4 = 0; e4 < kTdGroup / 4; ++e4) {
            uint4 h, lo;
            tc::split(v[4 * e4], h.x, lo.x);
            tc::split(v[4 * e4 + 1], h.y, lo.y);
            tc::split(v[4 * e4 + 2], h.z, lo.z);
            tc::split(v[4 * e4 + 3], h.w, lo.w);
            const uint32_t off = tc::kmajor_off(tid, 4 * e4, kTdGroup);
            *(uint4 *)(sBhi + off) = h;
            *(uint4 *)(sBlo + off) = lo;
          }
        }
        tc::fence_proxy_async();
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        if (tid == 0) {
          const uint32_t ahi = tc::smem_addr(sAhi), alo = tc::smem_addr(sAlo);
          const uint32_t bhi = tc::smem_addr(sBhi), blo = tc::smem_addr(sBlo);
          for (int k0 = 0; k0 < kTdGroup; k0 += 8)
            tc::mma3_step(tmem, ahi, alo, kTdGroup, bhi, blo, kTdGroup, k0, idesc, k0 > 0);
          tc::commit(mbar);
        }
        const int ok = tc::mbar_wait(mbar, phase, tc::kMaxTries);
        phase ^= 1u;
        if (__syncthreads_or(!ok)) {
          if (tid == 0) prep_error(B, kErrTc);
          tc::mbar_wait(mbar, phase ^ 1u, tc::kMaxTries);
          failed = true;
          break;
        }
        tc::fence_after_sync();
        // ---- the group's FP32 partial sums into the FP64 accumulators
#pragma unroll
        for (int j = 0; j < kTdCols / 16; ++j) {
          float v[16];
          tc::ld16(tc::taddr(tmem, 32 * warp, 16 * j), v);
#pragma unroll
          for (int q = 0; q < 16; ++q) acc[16 * j + q] += (double)v[q];
        }
        tc::fence_before_sync();
        __syncthreads();
      }
    }
    if (failed) break;
    ahead_bounds(B, nx, nx0, nx1);
    // ---- poly3gauss central-atom term (src/soap_turbo.f90:646-662), row (k = 0, re)
    if (P.basis == 1 && tid == 0) {
      const int mult = B.species_mult[site];
      for (int mm = 0; mm < mult; ++mm) {
        const int s = B.species[(size_t)site * B.max_mult + mm] - 1;
        if (s < 0 || s >= nsp) continue;
        const RadSp &RS = rad_of(smem, P, s);
#pragma unroll
        for (int n = 0; n < kTdCols; ++n)
          if (n >= RS.nbeg && n < RS.nbeg + RS.alpha) acc[n] += central[n];
      }
    }
    // ---- c_nlm to FP32 in sC (re/im, n, KS); the padding column k_max stays 0
    if (my_k < KS)
#pragma unroll
      for (int n = 0; n < kTdCols; ++n)
        if (n < n_max) sC[(size_t)(my_ri * n_max + n) * KS + my_k] = my_k < k_max ? (float)acc[n] : 0.f;
    __syncthreads();
    // ---- power spectrum on the tensor cores (src/soap_turbo.f90:750-795): per
    // group of l, A = rows (l, n) with X_l[n] = (Re c_nl0, r2 Re c_nl1 .., Im
    // c_nl0, r2 Im c_nl1 ..) in l's block of K (zero elsewhere), the J rows
    // first; B = A's first rows, so D[(l, n)][(l, j)] = P_l[n, J_j] (the other
    // blocks of D are zero and unread).  Written to sPl as ps_tensor writes it.
    const bool ps_tc = P.ps_ng > 0;
    if (ps_tc) {
      float *sPl = (float *)(smem + Ly.Pl);
      const int *psrow = (const int *)SBLOB(off_psrow);
      unsigned char *sPhi = smem + Ly.Phi, *sPlo = smem + Ly.Plo;
      const int MR = 16 * P.ps_mt, JP = 8 * P.ps_nt, nJ = P.ps_nj;
      for (int g = 0; g < P.ps_ng && !failed; ++g) {
        const int K = P.ps_gk[g], NB = P.ps_gnb[g];
        int l = -1, n = 0, cb = 0;
        if (tid < P.ps_grows[g]) {
          const int code = psrow[P.ps_grow[g] + tid];
          n = code & 0xff;
          l = (code >> 8) & 0xff;
          cb = code >> 16;
        }
        const int ko = l >= 0 ? P.ps_ko[l] : 0, kb = l * (l + 1) / 2;
        for (int k4 = 0; k4 < K; k4 += 4) {
          float v[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int c = k4 + q - ko;
            v[q] = 0.f;
            if (l >= 0 && c >= 0 && c < 2 * (l + 1)) {
              const int im = c > l, m = im ? c - l - 1 : c;
              const float x = sC[(size_t)(im ? n_max + n : n) * KS + kb + m];
              v[q] = m ? 1.41421356237309504880f * x : x;
            }
          }
          uint4 h, lo;
          tc::split(v[0], h.x, lo.x);
          tc::split(v[1], h.y, lo.y);
          tc::split(v[2], h.z, lo.z);
          tc::split(v[3], h.w, lo.w);
          const uint32_t off = tc::kmajor_off(tid, k4, K);
          *(uint4 *)(sPhi + off) = h;
          *(uint4 *)(sPlo + off) = lo;
        }
        tc::fence_proxy_async();
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        if (tid == 0) {
          const uint32_t phi = tc::smem_addr(sPhi), plo = tc::smem_addr(sPlo);
          const uint32_t id = tc::idesc_tf32(128, NB);
          for (int k0 = 0; k0 < K; k0 += 8) tc::mma3_step(tmem, phi, plo, K, phi, plo, K, k0, id, k0 > 0);
          tc::commit(mbar);
        }
        const int ok = tc::mbar_wait(mbar, phase, tc::kMaxTries);
        phase ^= 1u;
        if (__syncthreads_or(!ok)) {
          if (tid == 0) prep_error(B, kErrTc);
          tc::mbar_wait(mbar, phase ^ 1u, tc::kMaxTries);
          failed = true;
          break;
        }
        tc::fence_after_sync();
        for (int j = 0; j < NB / 16; ++j) {
          float v[16];
          tc::ld16(tc::taddr(tmem, 32 * warp, 16 * j), v);
          if (l >= 0)
#pragma unroll
            for (int q = 0; q < 16; ++q) {
              const int jc = 16 * j + q - cb;
              if (jc >= 0 && jc < nJ) sPl[(size_t)(l * MR + n) * JP + jc] = v[q];
            }
        }
        tc::fence_before_sync();
        __syncthreads();
      }
      if (failed) break;
    }
    site_output<NT>(P, smem, sC, sP, sS, (float *)(smem + Ly.Pl), kept, sRed, site, soap_out, keep_c, keep_norm,
                    keep, P.ps_mt > 0, ps_tc);
    ahead_publish(sSite, nx, nx0, nx1);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, kTdTmemCols);
}

// ------------------------------------------------------------ contract
// One CTA of a few warps per site.
//  G -> Gp -> Gu -> H  as the reference (src/soap_turbo.f90:1783-1835); H(n, k) to
//             shared memory as (re, im) pairs
//  entries    (pair, species) by species, two at a time to a warp, a half-warp
//             each, lane hl over k = hl + 16 j; the rows come two entries ahead
//             into the warp's own buffer by asynchronous copies, so that no barrier
//             stands between the entries
//  contraction  U = sum_n R'_n H(n, k), V = sum_n R_n H(n, k), H in registers from a
//             species' first entry to its last where they hold it (AMAX 8, three k a
//             lane); the k summed over the lanes
//  pairs      their entries added, rotated to Cartesian; the self pair minus their sum
// What bounds it: instructions (13.7 k per site of 58 pairs and one species, 16.7 k of
// three species), issued at 66 and 48 % of the rate by 16 warps per SM.  One CTA of 128
// threads with 32 staged entries behind barriers and H read from shared memory for every
// entry took 439 us at 16384 sites of one species and 66 at 1679 of three; this one 313
// and 57.
struct ContractLayout {
  size_t H, base, list, slot, red, X, C, Gu, Gp, F, stage, total;
};
constexpr int kContractChunk = 128;  // pairs whose entries are listed at a time
// a staged entry: the row, then R_n and dR_n/dr, padded so that the two half-warps'
// rows lie in disjoint halves of the banks
__host__ __device__ constexpr int contract_stride(int AMAX, int LC) {
  return (row_len(LC) + 2 * AMAX + 15) / 32 * 32 + 16;
}
// row of H: the species' blocks of AMAX (re, im) and a pad that spreads the k rows over the banks
__host__ __device__ inline int contract_h_stride(const DevParams &P, int AMAX) { return P.n_species * AMAX + 2; }
__host__ __device__ inline ContractLayout contract_layout(const DevParams &P, int threads, int AMAX, int LC) {
  ContractLayout L{};
  const size_t KS = (size_t)(P.k_max | 1), nsp = (size_t)P.n_species;
  size_t o = 0;
  L.H = o;    o += KS * (size_t)contract_h_stride(P, AMAX) * sizeof(float2);
  o = align_up(o, 16);
  L.red = o;  o += 40 * sizeof(double);
  L.base = o; o += 16 * sizeof(int);
  L.list = o; o += kContractChunk * nsp * sizeof(unsigned short);
  L.slot = o; o += kContractChunk * nsp * sizeof(short);
  o = align_up(o, 16);
  // the site's c_nlm, Gp and Gu; then the entries' rows and sums
  L.X = L.C = o;
  size_t x = o + ((size_t)P.n_max * KS + 2) * sizeof(float2);  // H items read up to two values past the end
  L.Gp = x;   x += (size_t)P.n_soap * sizeof(float);
  L.Gu = x;   x += (P.cmap_identity ? 0 : (size_t)P.n_kept) * sizeof(float);
  L.stage = o;
  size_t y = o + (size_t)(threads / 32) * 4 * contract_stride(AMAX, LC) * sizeof(float);
  L.F = y;    y += kContractChunk * nsp * 3 * sizeof(float);
  L.total = align_up(x > y ? x : y, 16);
  return L;
}

constexpr int kHM = 3;  // m values per H item (the host's items must agree)

template <int AMAX, int LC>
__global__ void __launch_bounds__(256, 2)
    k_contract(const DevParams P, const DevBatch B, int slots, const double *__restrict__ soap_in,
               const double *__restrict__ G, int g_layout, double sgn, const float *__restrict__ keep_c,
               const double *__restrict__ keep_norm, double *__restrict__ pair_out) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int AW = row_len(LC), ST = contract_stride(AMAX, LC);
  constexpr int KC = (LC + 1) * (LC + 2) / 2, KJ = (KC + 15) / 16;
  constexpr bool HREG = AMAX * KJ <= 24;  // the lane's H of a species fits its registers
  constexpr int GPT = 5;  // G values a thread holds while the norm dot product is reduced
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x, nw = nt >> 5;
  const int half = lane >> 4, hl = lane & 15;
  // the first `wide` threads take the slots, two apiece where they are fewer than the slots
  const int wide = min(nt, slots), t0 = tid < wide ? tid : P.n_soap;
  const bool two = slots > nt;
  const ContractLayout Ly = contract_layout(P, nt, AMAX, LC);
  float2 *sH = (float2 *)(smem + Ly.H);
  double *sRed = (double *)(smem + Ly.red);
  int *sBase = (int *)(smem + Ly.base);
  unsigned short *list = (unsigned short *)(smem + Ly.list);
  short *slot = (short *)(smem + Ly.slot);
  float2 *sC = (float2 *)(smem + Ly.C);
  float *sGp = (float *)(smem + Ly.Gp), *sGu = P.cmap_identity ? sGp : (float *)(smem + Ly.Gu);
  float *sF = (float *)(smem + Ly.F), *stage = (float *)(smem + Ly.stage) + (size_t)warp * 4 * ST;
  const int KS = P.k_max | 1, HS = contract_h_stride(P, AMAX);
  const int n_max = P.n_max, k_max = P.k_max, n_soap = P.n_soap, nsp = P.n_species, n_sites = B.n_sites;
  const int *klm = (const int *)(P.blob + P.off_klm);
  const int *hitem = (const int *)(P.blob_c + P.off_hitem), *nmap = (const int *)(P.blob_c + P.off_nmap);

  // the lane's k: where its values stand in a row, and the derivative forms'
  // coefficients (src/soap_turbo_angular.f90:194-246; a form that an (l, m) lacks has
  // coefficient 0 and reads a neighbouring value)
  int oP[KJ], oX[KJ], oL[KJ], oE[KJ];
  float4 cf[KJ];
#pragma unroll
  for (int j = 0; j < KJ; ++j) {
    const int k = hl + 16 * j, kk = k < k_max ? k : 0, lm = __ldg(klm + kk), l = lm & 0xff, m = lm >> 8;
    oP[j] = row_p(LC) + kk;
    oX[j] = row_p(LC) + kk + (m ? -1 : 1);
    oL[j] = l;
    oE[j] = row_e(LC) + 2 * m;
    cf[j] = k < k_max ? __ldg((const float4 *)(P.blob_c + P.off_kcoef) + kk) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  // the pieces (16 bytes) of two entries' rows that the lane stages
  constexpr int NPC = (AW + 2 * AMAX) / 4, NC = (2 * NPC + 31) / 32;
  struct {
    bool on, rad;
    int second, first, dst;
    unsigned per_pair, per_species;
  } piece[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int t = lane + 32 * c, p = t >= NPC ? t - NPC : t;
    piece[c].on = t < 2 * NPC;
    piece[c].second = t >= NPC ? 1 : 0;
    piece[c].rad = p >= AW / 4;
    piece[c].first = 4 * (p >= AW / 4 ? p - AW / 4 : p);
    piece[c].dst = piece[c].second * ST + 4 * p;
    piece[c].per_pair = p >= AW / 4 ? nsp * 2 * AMAX : AW;
    piece[c].per_species = p >= AW / 4 ? 2 * AMAX : 0;
  }

  const int site = B.order ? B.order[blockIdx.x] : B.site_lo + (int)blockIdx.x;
  const int p_begin = B.off[site], p_end = min(B.off[site + 1], B.n_pairs);
  const double knorm = keep_norm[site];
  const double *q = soap_in + (size_t)site * n_soap;
  const double *g = g_layout == 0 ? G + site : G + (size_t)site * n_soap;
  const size_t gs = g_layout == 0 ? (size_t)n_sites : 1;
  double gv[GPT], qv[GPT];
#pragma unroll
  for (int j = 0; j < GPT; ++j) {
    const int o = t0 + j * wide;
    gv[j] = qv[j] = 0.0;
    if (o < n_soap) {
      gv[j] = g[o * gs];
      qv[j] = q[o];
    }
  }
  {
    const float *kc = keep_c + (size_t)site * keep_stride(P);
    const int n4 = (2 * n_max * KS) / 4;
    for (int t = tid; t < n4; t += nt) cp_async16((float *)sC + 4 * t, kc + 4 * t);
    for (int t = 4 * n4 + tid; t < 2 * n_max * KS; t += nt) ((float *)sC)[t] = kc[t];
  }
  // ---- back through the normalisation (src/soap_turbo.f90:1783-1790)
  double qg0 = 0.0, qg1 = 0.0;
#pragma unroll
  for (int j = 0; j < GPT; ++j) {
    if (two && (j & 1)) qg1 = fma(qv[j], gv[j], qg1);
    else qg0 = fma(qv[j], gv[j], qg0);
  }
#pragma unroll 4
  for (int o = t0 + GPT * wide, j = GPT; o < n_soap; o += wide, ++j) {
    const double gj = g[o * gs], qj = q[o];
    if (two && (j & 1)) qg1 = fma(qj, gj, qg1);
    else qg0 = fma(qj, gj, qg0);
  }
  if (tid < wide) {
    qg0 = warp_sum(qg0);
    if (lane == 0) sRed[warp] = qg0;
    if (two) {
      qg1 = warp_sum(qg1);
      if (lane == 0) sRed[warp + nw] = qg1;
    }
  }
  __syncthreads();
  const double qg = slot_tree(sRed, slots), inv = 1.0 / knorm;
#pragma unroll
  for (int j = 0; j < GPT; ++j) {
    const int o = t0 + j * wide;
    if (o < n_soap) sGp[o] = (float)((gv[j] - qv[j] * qg) * inv);
  }
#pragma unroll 4
  for (int o = t0 + GPT * wide; o < n_soap; o += wide) sGp[o] = (float)((g[o * gs] - q[o] * qg) * inv);
  cp_async_wait_all();
  __syncthreads();
  // ---- back through the compression (:1791-1798), unless it is one-to-one
  if (!P.cmap_identity) {
    for (int t = tid; t < P.n_kept; t += nt) {
      float v = 0.f;
      for (int e = P.pj_off[t]; e < P.pj_off[t + 1]; ++e) v += P.pj_el[e] * sGp[P.pj_o[e]];
      sGu[t] = v;
    }
    __syncthreads();
  }
  // ---- H(k,n) = w(m) sum_np Y(n,np,l) c(k,np) over the non-zero Y (:1800-1835); an
  // item per (n, l, m0) walks its Y list once for up to kHM values of m, the
  // longest lists first
  for (int it = tid; it < P.n_hitem; it += nt) {
    const int code = __ldg(hitem + it), n = code & 0xff, l = (code >> 8) & 0xff, m0 = code >> 16;
    const int kb = l * (l + 1) / 2 + m0, mn = min(kHM, l + 1 - m0), li = l * n_max + n;
    const int t1 = __ldg(P.hl_off + li + 1);
    float2 h[kHM];
#pragma unroll
    for (int j = 0; j < kHM; ++j) h[j] = make_float2(0.f, 0.f);
    const float2 *cb = sC + kb;
#pragma unroll 2
    for (int t = __ldg(P.hl_off + li); t < t1; ++t) {
      const int e = __ldg(P.hl_packed + t);
      const float y = (e < 0 ? 2.f : 1.41421356237309504880f) * sGu[(e >> 8) & 0xffff];
      // past the last m the values belong to the next l, or to the next array: read, not stored
      const float2 *c = cb + (e & 0xff) * KS;
#pragma unroll
      for (int j = 0; j < kHM; ++j) {
        h[j].x = fmaf(y, c[j].x, h[j].x);
        h[j].y = fmaf(y, c[j].y, h[j].y);
      }
    }
    const int nm = __ldg(nmap + n);
    float2 *o = sH + kb * HS + (nm & 0xff) * AMAX + (nm >> 8);
#pragma unroll
    for (int j = 0; j < kHM; ++j)
      if (j < mn) {
        const float w = (m0 + j == 0) ? 1.f : 2.f;
        o[j * HS] = make_float2(w * h[j].x, w * h[j].y);
      }
  }
  // what no item writes: the columns past a species' alpha, and of empty lists
  for (int t = tid; t < P.n_hzero; t += nt) {
    const int code = __ldg(P.h_zero + t);
    sH[(code >> 16) * HS + (code & 0xffff)] = make_float2(0.f, 0.f);
  }

  // the thread's slots of the central pair between two chunks of the row (volatile: in
  // local memory, and not in registers while H fills them)
  volatile double held[6];
  for (int c0 = p_begin; c0 < p_end; c0 += kContractChunk) {
    const int c1 = min(p_end, c0 + kContractChunk);
    if (c0 > p_begin) __syncthreads();  // the chunk before is read
    // entries by species, and per (pair, species) its entry or -1, by the last warp
    // (which has the shortest of H's lists)
    if (warp == nw - 1) {
      const unsigned long long valid = valid_species(P, B, p_begin, c0, c1, true);
      const unsigned lt = (1u << lane) - 1u;
      int e = 0;
      for (int s = 0; s < nsp; ++s) {
        if (lane == 0) sBase[s] = e;
        for (int c = 0; c0 + 32 * c < c1; ++c) {
          const bool on = (valid >> (8 * c + s)) & 1ull;
          const unsigned m = __ballot_sync(0xffffffffu, on);
          const int at = e + __popc(m & lt);
          if (on) list[at] = (unsigned short)(32 * c + lane);
          slot[s * kContractChunk + 32 * c + lane] = (short)(on ? at : -1);
          e += __popc(m);
        }
      }
      if (lane == 0) sBase[nsp] = e;
    }
    __syncthreads();  // H and the lists are complete; c_nlm and Gp under the rows are read
    const float *src[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c)
      src[c] = piece[c].rad ? B.rad + (size_t)c0 * nsp * 2 * AMAX + piece[c].first
                            : B.ang + (size_t)c0 * AW + piece[c].first;
    // a unit: two entries of a species.  The units go round the warps, from one
    // species on to the next; s, e: this warp's next unit, turn: the warp to which
    // the species' first unit falls
    int s = 0, turn = 0, e = sBase[0] + 2 * warp;
    auto settle = [&]() {  // past the species' last unit: on to the next species
      while (s < nsp && e >= sBase[s + 1]) {
        turn = (turn + ((sBase[s + 1] - sBase[s] + 1) >> 1)) & (nw - 1);
        ++s;
        if (s < nsp) e = sBase[s] + 2 * ((warp - turn) & (nw - 1));
      }
    };
    auto copy = [&](float *dst) {
      const int last = sBase[s + 1] - 1;
      const unsigned j0 = list[e], j1 = list[min(e + 1, last)];
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (piece[c].on)
          cp_async16(dst + piece[c].dst,
                     src[c] + ((piece[c].second ? j1 : j0) * piece[c].per_pair + s * piece[c].per_species));
    };
    float2 H[HREG ? KJ * AMAX : 1];
    int hs = -1;  // the species H holds
    settle();
    if (s < nsp) copy(stage);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    for (int buf = 0; s < nsp; buf ^= 1) {
      const int us = s, ue = e, u_end = sBase[s + 1];
      e += 2 * nw;
      settle();
      if (s < nsp) copy(stage + (buf ^ 1) * 2 * ST);
      asm volatile("cp.async.commit_group;\ncp.async.wait_group 1;\n" ::: "memory");
      const float2 *Hs = sH + us * AMAX;
      if constexpr (HREG)
        if (us != hs) {
          hs = us;
#pragma unroll
          for (int j = 0; j < KJ; ++j) {
            const int k = hl + 16 * j;
#pragma unroll
            for (int n = 0; n < AMAX; n += 2) {
              float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
              if (k < k_max) v = *(const float4 *)(Hs + k * HS + n);
              H[j * AMAX + n] = make_float2(v.x, v.y);
              H[j * AMAX + n + 1] = make_float2(v.z, v.w);
            }
          }
        }
      __syncwarp();
      const float *A = stage + (2 * buf + half) * ST;
      const bool act = ue + half < u_end;
      float R[AMAX], Rd[AMAX];
#pragma unroll
      for (int n4 = 0; n4 < AMAX / 4; ++n4) {
        const float4 a = ((const float4 *)(A + AW))[n4], d = ((const float4 *)(A + AW + AMAX))[n4];
        R[4 * n4] = a.x; R[4 * n4 + 1] = a.y; R[4 * n4 + 2] = a.z; R[4 * n4 + 3] = a.w;
        Rd[4 * n4] = d.x; Rd[4 * n4 + 1] = d.y; Rd[4 * n4 + 2] = d.z; Rd[4 * n4 + 3] = d.w;
      }
      const float sfac = A[row_sf(LC)];
      float f_rad = 0.f, f_azi = 0.f, f_pol = 0.f;
#pragma unroll
      for (int j = 0; j < KJ; ++j) {
        if (16 * j >= k_max) break;
        float Ur = 0.f, Ui = 0.f, Vr = 0.f, Vi = 0.f;
        const int kj = hl + 16 * j;
        const float2 *h = Hs + (kj < k_max ? kj : 0) * HS;
#pragma unroll
        for (int n = 0; n < AMAX; n += 2) {
          float4 v;
          if constexpr (HREG)
            v = make_float4(H[j * AMAX + n].x, H[j * AMAX + n].y, H[j * AMAX + n + 1].x, H[j * AMAX + n + 1].y);
          else
            v = *(const float4 *)(h + n);
          Ur = fmaf(Rd[n], v.x, Ur); Ui = fmaf(Rd[n], v.y, Ui);
          Vr = fmaf(R[n], v.x, Vr); Vi = fmaf(R[n], v.y, Vi);
          Ur = fmaf(Rd[n + 1], v.z, Ur); Ui = fmaf(Rd[n + 1], v.w, Ui);
          Vr = fmaf(R[n + 1], v.z, Vr); Vi = fmaf(R[n + 1], v.w, Vi);
        }
        if (!HREG && kj >= k_max) Ur = Ui = Vr = Vi = 0.f;
        // rows hold amp i_l, amp di_l/dr and preflm_k P_k; cf carries the
        // preflm ratios of the derivative combinations
        const float Pk = A[oP[j]], il = A[row_il(LC) + oL[j]], ild = A[row_ild(LC) + oL[j]];
        const float2 ee = *(const float2 *)(A + oE[j]);
        const float *Pl = A + oP[j] + oL[j];
        const float dms = cf[j].x * A[oX[j]] + cf[j].y * A[oP[j] + 1];
        const float dvs = cf[j].z * Pl[0] + cf[j].w * Pl[2];
        const float er = ee.x, ei = ee.y;
        const float uu = Pk * il;
        const float ur = Pk * ild - sfac * uu;
        const float ua = dvs * il;
        const float up = dms * il;
        const float reU = er * Ur + ei * Ui;
        const float reV = er * Vr + ei * Vi;
        const float imV = ei * Vr - er * Vi;
        f_rad = fmaf(uu, reU, fmaf(ur, reV, f_rad));
        f_azi = fmaf(-ua, imV, f_azi);
        f_pol = fmaf(up, reV, f_pol);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        f_rad += __shfl_xor_sync(0xffffffffu, f_rad, o);
        f_azi += __shfl_xor_sync(0xffffffffu, f_azi, o);
        f_pol += __shfl_xor_sync(0xffffffffu, f_pol, o);
      }
      if (act && hl == 0) {
        float *F = sF + 3 * (ue + half);
        F[0] = f_rad;
        F[1] = f_azi;
        F[2] = f_pol;
      }
      __syncwarp();  // the rows are read: the buffer is free for the unit after next
    }
    __syncthreads();
    // ---- per pair: sum its entries, rotate to Cartesian (:1864-1875)
    // and add it to the central pair's slot (the pair's place in the row, modulo
    // slots): tid's, and tid + nt's with two apiece
    const int n_k = c1 - c0;
    double x0 = 0.0, y0 = 0.0, z0 = 0.0, x1 = 0.0, y1 = 0.0, z1 = 0.0;
    if (c0 > p_begin) {
      x0 = held[0]; y0 = held[1]; z0 = held[2];
      x1 = held[3]; y1 = held[4]; z1 = held[5];
    }
    for (int k = tid - (slots > kContractChunk ? (c0 - p_begin) & (slots - 1) : 0); k < n_k; k += nt) {
      if (k < 0 || c0 + k <= p_begin) continue;
      double px = 0.0, py = 0.0, pz = 0.0, fr = 0.0, fa = 0.0, fp = 0.0;
      bool any = false;
      for (int s = 0; s < nsp; ++s) {
        const int e = slot[s * kContractChunk + k];
        if (e >= 0) {
          any = true;
          fr += sF[3 * e];
          fa += sF[3 * e + 1];
          fp += sF[3 * e + 2];
        }
      }
      if (any) {
        const float *A = B.ang + (size_t)(c0 + k) * AW;
        const double ct = A[row_x(LC)], st = A[row_sq(LC)], cf_ = A[row_e(LC) + 2], sf = -A[row_e(LC) + 3];
        const double ir = 1.0 / B.rjs[c0 + k];
        px = sgn * (st * cf_ * fr - ct * cf_ * ir * fp - sf * ir * fa);
        py = sgn * (st * sf * fr - ct * sf * ir * fp + cf_ * ir * fa);
        pz = sgn * (ct * fr + st * ir * fp);
      }
      double *po = pair_out + (size_t)3 * (c0 + k);
      po[0] = px;
      po[1] = py;
      po[2] = pz;
      if (two && k >= nt) {
        x1 -= px;
        y1 -= py;
        z1 -= pz;
      } else {
        x0 -= px;
        y0 -= py;
        z0 -= pz;
      }
    }
    if (c1 < p_end) {
      held[0] = x0; held[1] = y0; held[2] = z0;
      held[3] = x1; held[4] = y1; held[5] = z1;
      continue;
    }
    // the central pair is minus the sum of the others (:1875)
    auto fold = [&](double x, double y, double z, int w) {  // the slots 32 w + lane
      if (32 * w < p_end - p_begin) {  // the row reaches them
        x = warp_sum(x);
        y = warp_sum(y);
        z = warp_sum(z);
      }
      if (lane == 0) {
        double *r = sRed + 8 + 3 * w;
        r[0] = x;
        r[1] = y;
        r[2] = z;
      }
    };
    if (tid < slots) fold(x0, y0, z0, warp);
    if (two) fold(x1, y1, z1, warp + nw);
    __syncthreads();
    if (tid < 3) pair_out[(size_t)3 * p_begin + tid] = slot_tree<3>(sRed + 8 + tid, slots);
  }
}

// ------------------------------------------------------------ contract on tensor cores
// soap_contract (src/soap_turbo.f90:1723-1884) with the per-entry contraction
// on the tensor cores.  Per site, as k_contract: Gp, Gu and H(k, n) on the CUDA
// cores.  H becomes the B operand of a tcgen05 MMA, [96 columns c = 2k + re/im
// (k < 48, beyond k_max zero) x KB = n_species * AMAX] (K-major, split into
// TF32 head and tail).  The site's entries go in rounds of 64: the A operand
// is [128 x KB], row e < 64 the entry's dR_n/dr and row 64 + e its R_n, each
// in its species' AMAX columns (zero elsewhere), so that one 3xTF32 product
// D = A B^T (9 MMAs of 128 x 96 x 8) gives every entry's
//   U(k) = sum_n dR_n/dr H(k, n)  (rows < 64),   V(k) = sum_n R_n H(k, n)  (rows >= 64)
// in TMEM (the reference's four dot products per n, src/soap_turbo.f90:
// 1842-1866, reassociated over n).  Thread t < 64 then takes U of entry t and
// forms u Re(e conj U); thread 64 + t takes V of entry t and forms the rest of
// the radial, azimuthal and polar sums, each over k in a fixed order, from the
// entry's angular row (read from global memory, where the descriptor's pair
// kernel left it).  The per-pair rotation and the self pair are k_contract's.
constexpr int kTcEntries = 64;   // entries per round
constexpr int kTcCols = 96;      // U / V columns: 2 k + re/im for k < 48
constexpr int kTcTmemCols = 128; // TMEM columns a CTA holds

__host__ __device__ inline int tc_kb(const DevParams &P, int AMAX) { return (P.n_species * AMAX + 7) / 8 * 8; }

struct TcLayout {
  size_t red, ent, wcnt, misc, H, Rot, F, Fu, Bhi, Blo, X, Ahi, Alo, AT, C, Gu, Gp, mbar, tmem, total;
};
__host__ __device__ inline TcLayout make_tc_layout(const DevParams &P, int NT, int AMAX) {
  TcLayout L{};
  const size_t KS = (size_t)(P.k_max | 1), nsp = (size_t)P.n_species, KB = (size_t)tc_kb(P, AMAX);
  size_t o = site_blob_bytes(P, 1);
  L.red = o;  o += 40 * sizeof(double);
  L.ent = o;  o += (size_t)NT * nsp * sizeof(int);
  L.wcnt = o; o += (size_t)SOAPB_MAX_SPECIES * (NT / 32) * sizeof(int);
  L.misc = o; o += 64 * sizeof(int);
  L.mbar = align_up(o, 8); o = L.mbar + 8;
  L.tmem = o; o += 8;
  o = align_up(o, 16);
  L.H = o;   o += 2 * KS * (size_t)h_stride(P.n_species, AMAX) * sizeof(float);
  L.Rot = o; o += (size_t)NT * 4 * sizeof(float);
  L.F = o;   o += (size_t)NT * nsp * 3 * sizeof(float);
  L.Fu = o;  o += (size_t)NT * nsp * sizeof(float);
  o = align_up(o, 1024);
  L.Bhi = o; o += (size_t)kTcCols * KB * 4;
  L.Blo = o; o += (size_t)kTcCols * KB * 4;
  o = align_up(o, 1024);
  L.X = o;
  // per round: the A tiles; per site (before H is built): c_nlm, Gu, Gp
  size_t x = o;
  L.Ahi = x; x += 128 * KB * 4;
  L.Alo = x; x += 128 * KB * 4;
  L.AT = x;  x += (size_t)row_len(AMAX == 8 ? 8 : 12) * kTcEntries * 4;  // the round's angular rows, transposed
  const size_t end_round = x;
  x = o;
  L.C = x;  x += 2 * (size_t)P.n_max * KS * sizeof(float);
  L.Gu = x; x += (size_t)P.n_kept * sizeof(float);
  L.Gp = x; x += (size_t)P.n_soap * sizeof(float);
  L.total = align_up(end_round > x ? end_round : x, 16);
  return L;
}

__host__ __device__ constexpr int tc_l_of(int kk) {
  int l = 0;
  while ((l + 1) * (l + 2) / 2 <= kk) ++l;
  return l;
}
__host__ __device__ constexpr int tc_m_of(int kk) { return kk - tc_l_of(kk) * (tc_l_of(kk) + 1) / 2; }

template <int NT, int AMAX, int LC>
__global__ void __launch_bounds__(NT) k_contract_tc(const DevParams P, const DevBatch B,
                                                    const double *__restrict__ soap_in,
                                                    const double *__restrict__ G, int g_layout, double sgn,
                                                    const float *__restrict__ keep_c,
                                                    const double *__restrict__ keep_norm,
                                                    double *__restrict__ pair_out) {
  static_assert(NT == 128, "one thread per TMEM lane");
  constexpr int KC = (LC + 1) * (LC + 2) / 2;
  static_assert(KC <= 2 * kTcCols / 4 && 2 * KC <= kTcCols, "U/V columns");
  constexpr int GPT = 8;
  constexpr int AW = row_len(LC);
  constexpr int O_IL = row_il(LC), O_ILD = row_ild(LC), O_E = row_e(LC),
                O_SF = row_sf(LC), O_X = row_x(LC), O_SQ = row_sq(LC), O_P = row_p(LC);
  extern __shared__ __align__(16) unsigned char smem[];  // no-swizzle operand tiles need 16-byte alignment
  const TcLayout Ly = make_tc_layout(P, NT, AMAX);
  const float4 *kcoef = (const float4 *)SBLOBC(off_kcoef);
  const int *nmap = (const int *)SBLOBC(off_nmap);
  const int *hitem = (const int *)SBLOBC(off_hitem);
  const int *hloff = (const int *)SBLOBC(off_hloff);
  const int *hl = P.hl_in_blob ? (const int *)SBLOBC(off_hl) : P.hl_packed;
  double *sRed = (double *)(smem + Ly.red);
  float *sH = (float *)(smem + Ly.H);
  float *sRot = (float *)(smem + Ly.Rot);
  float *sF = (float *)(smem + Ly.F);
  float *sFu = (float *)(smem + Ly.Fu);
  float *sC = (float *)(smem + Ly.C);
  float *sGu = (float *)(smem + Ly.Gu);
  float *sGp = (float *)(smem + Ly.Gp);
  unsigned char *sAhi = smem + Ly.Ahi, *sAlo = smem + Ly.Alo, *sBhi = smem + Ly.Bhi, *sBlo = smem + Ly.Blo;
  float *sAT = (float *)(smem + Ly.AT);
  uint64_t *mbar = (uint64_t *)(smem + Ly.mbar);
  uint32_t *tmem_slot = (uint32_t *)(smem + Ly.tmem);
  int *sEnt = (int *)(smem + Ly.ent);
  int *sW_cnt = (int *)(smem + Ly.wcnt);
  int *sMisc = (int *)(smem + Ly.misc);
  int *sBase = sMisc, *sCnt = sMisc + SOAPB_MAX_SPECIES, *sNent = sMisc + 2 * SOAPB_MAX_SPECIES;
  int *sSite = sMisc + 3 * SOAPB_MAX_SPECIES;
  int *sFail = sMisc + 3 * SOAPB_MAX_SPECIES + 4;

  const int tid = threadIdx.x, warp = tid >> 5;
  const int KS = P.k_max | 1;
  const int HS = h_stride(P.n_species, AMAX);
  const size_t HPL = (size_t)KS * HS;
  const int n_max = P.n_max, k_max = P.k_max, n_soap = P.n_soap, nsp = P.n_species;
  const int n_sites = B.n_sites;
  const int KB = tc_kb(P, AMAX);
  const uint32_t idesc = tc::idesc_tf32(128, kTcCols);
  float *sGu_eff = P.cmap_identity ? sGp : sGu;

  copy_site_blob<NT>(P, smem, 1);
  for (int t = tid; t < 2 * (int)HPL; t += NT) sH[t] = 0.f;  // entries no item writes stay 0
  if (warp == 0) tc::tmem_alloc(tmem_slot, kTcTmemCols);
  if (tid == 0) {
    tc::mbar_init(mbar);
    *sFail = 0;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  uint32_t phase = 0;
  bool failed = false;

  first_site(B, B.ticket + 1, sSite);
  for (;;) {
    const int site = sSite[0];
    if (site >= B.site_hi || failed) break;
    const int p_begin = sSite[1];
    const int p_end = min(sSite[2], B.n_pairs);
    int nx = 0, nx0 = 0, nx1 = 0;
    if (tid == 0) nx = take_ticket(B, B.ticket + 1);
    // ---- per-site loads, Gp, Gu and H, as k_contract (:1783-1835)
    const double knorm = keep_norm[site];
    const double *q = soap_in + (size_t)site * n_soap;
    double gv[GPT], qv[GPT];
#pragma unroll
    for (int j = 0; j < GPT; ++j) {
      const int o = tid + j * NT;
      gv[j] = qv[j] = 0.0;
      if (o < n_soap) {
        gv[j] = g_layout == 0 ? G[(size_t)o * n_sites + site] : G[(size_t)site * n_soap + o];
        qv[j] = q[o];
      }
    }
    {
      const float *kc = keep_c + (size_t)site * keep_stride(P);
      const int n4 = (2 * n_max * KS) / 4;
      for (int t = tid; t < n4; t += NT) cp_async16(sC + 4 * t, kc + 4 * t);
      for (int t = 4 * n4 + tid; t < 2 * n_max * KS; t += NT) sC[t] = kc[t];
      cp_async_wait_all();
    }
    double qg = 0.0;
#pragma unroll
    for (int j = 0; j < GPT; ++j) qg += qv[j] * gv[j];
    for (int o = tid + GPT * NT; o < n_soap; o += NT) {
      const double g = g_layout == 0 ? G[(size_t)o * n_sites + site] : G[(size_t)site * n_soap + o];
      sGp[o] = (float)g;
      qg += q[o] * g;
    }
    qg = block_sum<NT>(qg, sRed);
    const double inv = 1.0 / knorm;
#pragma unroll
    for (int j = 0; j < GPT; ++j) {
      const int o = tid + j * NT;
      if (o < n_soap) sGp[o] = (float)((gv[j] - qv[j] * qg) * inv);
    }
    for (int o = tid + GPT * NT; o < n_soap; o += NT) sGp[o] = (float)(((double)sGp[o] - q[o] * qg) * inv);
    __syncthreads();
    if (!P.cmap_identity) {
      for (int t = tid; t < P.n_kept; t += NT) {
        float v = 0.f;
        for (int e = P.pj_off[t]; e < P.pj_off[t + 1]; ++e) v += P.pj_el[e] * sGp[P.pj_o[e]];
        sGu[t] = v;
      }
      __syncthreads();
    }
    for (int it = tid; it < P.n_hitem; it += NT) {
      const int code = hitem[it];
      const int n = code & 0xff, l = (code >> 8) & 0xff, m0 = code >> 16;
      const int kb = l * (l + 1) / 2 + m0, mn = min(kHM, l + 1 - m0);
      float hr[kHM], hi[kHM];
#pragma unroll
      for (int j = 0; j < kHM; ++j) hr[j] = hi[j] = 0.f;
      const int li = l * n_max + n;
      for (int t = hloff[li]; t < hloff[li + 1]; ++t) {
        const int e = hl[t];
        const int np = e & 0xff, qq = (e >> 8) & 0xffff;
        const float y = ((e >> 31) ? 2.f : 1.41421356237309504880f) * sGu_eff[qq];
        const float2 *c = (const float2 *)sC + (size_t)np * KS + kb;
#pragma unroll
        for (int j = 0; j < kHM; ++j) {
          if (j < mn) {
            hr[j] = fmaf(y, c[j].x, hr[j]);
            hi[j] = fmaf(y, c[j].y, hi[j]);
          }
        }
      }
      const int nm = nmap[n];
      const int col = (nm & 0xff) * AMAX + (nm >> 8);
#pragma unroll
      for (int j = 0; j < kHM; ++j) {
        if (j < mn) {
          const float w = (m0 + j == 0) ? 1.f : 2.f;
          sH[(size_t)(kb + j) * HS + col] = w * hr[j];
          sH[HPL + (size_t)(kb + j) * HS + col] = w * hi[j];
        }
      }
    }
    __syncthreads();
    // ---- the B operand: H as [96 x KB], column c = 2 k + (re, im); one row per
    // thread, 16 bytes at a time (H rows are 16-byte aligned: HS is a multiple of 4)
    if (tid < kTcCols) {
      const int c = tid, k = c >> 1;
      const float *hrow = sH + (c & 1) * HPL + (size_t)k * HS;
      for (int kk4 = 0; kk4 < KB; kk4 += 4) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k < k_max && kk4 < nsp * AMAX) v = *(const float4 *)(hrow + kk4);
        uint4 h, lo;
        tc::split(v.x, h.x, lo.x);
        tc::split(v.y, h.y, lo.y);
        tc::split(v.z, h.z, lo.z);
        tc::split(v.w, h.w, lo.w);
        const uint32_t off = tc::kmajor_off(c, kk4, KB);
        *(uint4 *)(sBhi + off) = h;
        *(uint4 *)(sBlo + off) = lo;
      }
    }
    ahead_bounds(B, nx, nx0, nx1);
    double self_x = 0.0, self_y = 0.0, self_z = 0.0;

    for (int chunk = p_begin; chunk < p_end; chunk += NT) {
      int slot[SOAPB_MAX_SPECIES];
      unsigned my_bits;
      double my_r;
      // (its barriers also order the B tiles' stores before the first round)
      const int n_ent = build_entries<NT>(P, B, p_begin, chunk, p_end, true, sEnt, sW_cnt, sBase, sCnt, sNent,
                                          slot, my_bits, my_r);
      for (int ebase = 0; ebase < n_ent && !failed; ebase += kTcEntries) {
        const int n_round = min(kTcEntries, n_ent - ebase);
        // ---- A operand: rows e < 64 dR/dr, rows 64 + e R, in the species' columns;
        // row tid per thread: its entry's AMAX values, zero in the other columns
        {
          const int e = tid & (kTcEntries - 1);
          int sp = -1;
          float4 rv[AMAX / 4];
#pragma unroll
          for (int j = 0; j < AMAX / 4; ++j) rv[j] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (e < n_round) {
            const int code = sEnt[ebase + e];
            sp = code >> 24;
            const float4 *src = (const float4 *)(B.rad + ((size_t)(chunk + (code & 0xffffff)) * nsp + sp) * 2 * AMAX +
                                                 (tid < kTcEntries ? AMAX : 0));
#pragma unroll
            for (int j = 0; j < AMAX / 4; ++j) rv[j] = src[j];
          }
          for (int kk4 = 0; kk4 < KB; kk4 += 4) {
            const int blk = kk4 / AMAX, j = (kk4 - blk * AMAX) >> 2;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (blk == sp) {
#pragma unroll
              for (int q = 0; q < AMAX / 4; ++q)
                if (q == j) v = rv[q];
            }
            uint4 h, lo;
            tc::split(v.x, h.x, lo.x);
            tc::split(v.y, h.y, lo.y);
            tc::split(v.z, h.z, lo.z);
            tc::split(v.w, h.w, lo.w);
            const uint32_t off = tc::kmajor_off(tid, kk4, KB);
            *(uint4 *)(sAhi + off) = h;
            *(uint4 *)(sAlo + off) = lo;
          }
        }
        // the round's angular rows, transposed to [field][entry] for the epilogue
        // (thread-per-entry reads then fall in distinct banks); pieces of 16 bytes
        for (int t = tid; t < (AW / 4) * kTcEntries; t += NT) {
          const int j4 = t / kTcEntries, e = t - j4 * kTcEntries;
          if (e < n_round) {
            const float4 v = __ldg((const float4 *)(B.ang + (size_t)(chunk + (sEnt[ebase + e] & 0xffffff)) * AW) + j4);
            sAT[(4 * j4) * kTcEntries + e] = v.x;
            sAT[(4 * j4 + 1) * kTcEntries + e] = v.y;
            sAT[(4 * j4 + 2) * kTcEntries + e] = v.z;
            sAT[(4 * j4 + 3) * kTcEntries + e] = v.w;
          }
        }
        tc::fence_proxy_async();
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        if (tid == 0) {
          const uint32_t ahi = tc::smem_addr(sAhi), alo = tc::smem_addr(sAlo);
          const uint32_t bhi = tc::smem_addr(sBhi), blo = tc::smem_addr(sBlo);
          for (int k0 = 0; k0 < KB; k0 += 8) tc::mma3_step(tmem, ahi, alo, KB, bhi, blo, KB, k0, idesc, k0 > 0);
          tc::commit(mbar);
        }
        const int ok = tc::mbar_wait(mbar, phase, tc::kMaxTries);
        phase ^= 1u;
        if (__syncthreads_or(!ok)) {
          // give up: report, and make sure the MMAs are no longer running
          // before the TMEM is freed
          if (tid == 0) {
            prep_error(B, kErrTc);
            *sFail = 1;
          }
          tc::mbar_wait(mbar, phase ^ 1u, tc::kMaxTries);
          failed = true;
          break;
        }
        tc::fence_after_sync();
        // ---- epilogue: thread tid reads TMEM lane tid
        const bool vrole = tid >= kTcEntries;
        const int e = tid & (kTcEntries - 1);
        const bool act = e < n_round;
        const int code = act ? sEnt[ebase + e] : 0;
        // field f of this entry's row: Ae[f * kTcEntries]
        const float *Ae = sAT + e;
        float il[LC + 1], ild[LC + 1], er[LC + 1], ei[LC + 1], sfac = 0.f;
#pragma unroll
        for (int l = 0; l <= LC; ++l) {
          il[l] = act ? Ae[(O_IL + l) * kTcEntries] : 0.f;
          er[l] = act ? Ae[(O_E + 2 * l) * kTcEntries] : 0.f;
          ei[l] = act ? Ae[(O_E + 2 * l + 1) * kTcEntries] : 0.f;
          ild[l] = (act && vrole) ? Ae[(O_ILD + l) * kTcEntries] : 0.f;
        }
        if (act && vrole) sfac = Ae[O_SF * kTcEntries];
        float f_rad = 0.f, f_azi = 0.f, f_pol = 0.f;
        const float *Pe = Ae + O_P * kTcEntries;
#pragma unroll
        for (int j = 0; j < (2 * KC + 15) / 16; ++j) {
          float v[16];
          tc::ld16(tc::taddr(tmem, 32 * warp, 16 * j), v);
#pragma unroll
          for (int qq = 0; qq < 8; ++qq) {
            const int kk = 8 * j + qq;
            if (kk >= KC) break;
            const int l = tc_l_of(kk), m = tc_m_of(kk);
            if (!act || l > P.l_max) continue;
            const float xr = v[2 * qq], xi = v[2 * qq + 1];
            const float Pk = Pe[kk * kTcEntries];
            const float u = Pk * il[l];
            if (!vrole) {
              f_rad = fmaf(u, er[m] * xr + ei[m] * xi, f_rad);
            } else {
              const float4 cf = kcoef[kk];
              // the derivative forms' P_l^m indices (src/soap_turbo_angular.f90:194-246)
              const int ixx = (m == 0) ? (l > 0 ? l * (l + 1) / 2 + 1 : kk) : kk - 1;
              const int ixy = (m == 0) ? (l > 0 ? l * (l + 1) / 2 + 1 : kk) : (m != l ? kk + 1 : kk);
              const int ixz = (m == 0) ? kk : (l + 1) * (l + 2) / 2 + m - 1;
              const int ixw = (m == 0) ? kk : (l + 1) * (l + 2) / 2 + m + 1;
              const float dms = cf.x * Pe[ixx * kTcEntries] + cf.y * Pe[ixy * kTcEntries];
              const float dvs = cf.z * Pe[ixz * kTcEntries] + cf.w * Pe[ixw * kTcEntries];
              const float ur = Pk * ild[l] - sfac * u;
              const float ua = dvs * il[l];
              const float up = dms * il[l];
              const float reV = er[m] * xr + ei[m] * xi;
              const float imV = ei[m] * xr - er[m] * xi;
              f_rad = fmaf(ur, reV, f_rad);
              f_azi = fmaf(-ua, imV, f_azi);
              f_pol = fmaf(up, reV, f_pol);
            }
          }
        }
        if (act) {
          if (vrole) {
            float *Fe = sF + (size_t)(ebase + e) * 3;
            Fe[0] = f_rad;
            Fe[1] = f_azi;
            Fe[2] = f_pol;
            // the rotation to Cartesian uses the same angles (:1867-1871)
            float *rot = sRot + 4 * (code & 0xffffff);
            rot[0] = Ae[O_X * kTcEntries];
            rot[1] = Ae[O_SQ * kTcEntries];
            rot[2] = er[1];
            rot[3] = -ei[1];
          } else {
            sFu[ebase + e] = f_rad;
          }
        }
        tc::fence_before_sync();
        __syncthreads();
      }
      if (failed) break;
      // ---- per pair: sum its entries, rotate to Cartesian (:1864-1875)
      const int k = chunk + tid;
      if (k < p_end && k > p_begin) {
        double px = 0.0, py = 0.0, pz = 0.0;
        if (my_bits != 0u) {
          double fr = 0.0, fa = 0.0, fp = 0.0;
#pragma unroll
          for (int s = 0; s < SOAPB_MAX_SPECIES; ++s) {
            if (s < nsp && slot[s] >= 0) {
              fr += (double)(sF[3 * slot[s] + 0] + sFu[slot[s]]);
              fa += sF[3 * slot[s] + 1];
              fp += sF[3 * slot[s] + 2];
            }
          }
          const float *rot = sRot + 4 * tid;
          const double ct = rot[0], st = rot[1], cf = rot[2], sf = rot[3];
          const double ir = 1.0 / my_r;
          px = sgn * (st * cf * fr - ct * cf * ir * fp - sf * ir * fa);
          py = sgn * (st * sf * fr - ct * sf * ir * fp + cf * ir * fa);
          pz = sgn * (ct * fr + st * ir * fp);
        }
        double *po = pair_out + (size_t)3 * k;
        po[0] = px;
        po[1] = py;
        po[2] = pz;
        self_x -= px;
        self_y -= py;
        self_z -= pz;
      }
    }
    if (failed) break;
    block_sum3<NT>(self_x, self_y, self_z, sRed);
    if (tid == 0 && p_end > p_begin) {
      double *po = pair_out + (size_t)3 * p_begin;
      po[0] = self_x;
      po[1] = self_y;
      po[2] = self_z;
    }
    ahead_publish(sSite, nx, nx0, nx1);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, kTcTmemCols);
}

// ------------------------------------------------------------ launchers
// What a launch needs from the runtime besides the launch itself -- the
// kernel's dynamic shared memory limit raised, its resident CTAs per SM for a
// persistent grid -- asked once per (kernel, device, CTA size, shared memory)
// and remembered: the drop-in layer launches the same kernels once per site
// chunk, and these queries would otherwise cost it host time on every call.
struct LaunchMemo {
  const void *fn;
  int dev, threads;
  size_t smem;
  int sms, per_sm;
};
struct SmemLimit {
  const void *fn;
  int dev;
  size_t smem;
};
static std::mutex g_launch_mu;
static std::vector<LaunchMemo> g_launch_memo;
static std::vector<SmemLimit> g_smem_limit;

// Raises fn's dynamic shared memory limit on the current device to at least
// smem (never lowers it, so that launches of other sizes stay valid).
template <typename K>
static cudaError_t ensure_smem_limit(K kernel, size_t smem) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const void *fn = (const void *)kernel;
  std::lock_guard<std::mutex> g(g_launch_mu);
  for (auto &x : g_smem_limit)
    if (x.fn == fn && x.dev == dev) {
      if (x.smem >= smem) return cudaSuccess;
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e == cudaSuccess) x.smem = smem;
      return e;
    }
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) g_smem_limit.push_back({fn, dev, smem});
  return e;
}

int sm_count() {
  static std::atomic<int> known[32];
  int dev = 0;
  cudaGetDevice(&dev);
  int n = dev < 32 ? known[dev].load(std::memory_order_relaxed) : 0;
  if (n > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) return 148;
  if (dev < 32) known[dev].store(n, std::memory_order_relaxed);
  return n;
}

template <typename K>
static int persistent_grid_query(K kernel, int threads, size_t smem, int dev, int &sms);

template <typename K>
static int persistent_grid(K kernel, int threads, size_t smem, int n_sites, int max_ctas) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaGetDevice(&dev);
  const void *fn = (const void *)kernel;
  bool found = false;
  {
    std::lock_guard<std::mutex> g(g_launch_mu);
    for (const auto &x : g_launch_memo)
      if (x.fn == fn && x.dev == dev && x.threads == threads && x.smem == smem) {
        sms = x.sms;
        per_sm = x.per_sm;
        found = true;
        break;
      }
  }
  if (!found) {
    per_sm = persistent_grid_query(kernel, threads, smem, dev, sms);
    std::lock_guard<std::mutex> g(g_launch_mu);
    g_launch_memo.push_back({fn, dev, threads, smem, sms, per_sm});
  }
  int g = sms * (per_sm > 0 ? per_sm : 1);
  if (max_ctas > 0 && g > max_ctas) g = max_ctas;
  return g < n_sites ? g : n_sites;
}

template <typename K>
static int persistent_grid_query(K kernel, int threads, size_t smem, int dev, int &sms) {
  int per_sm = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
  // the count from the kernel's registers and shared memory as well: the
  // occupancy query has been seen to answer 1 for CTAs of 66-74 KB that fit
  // three times.  Too many CTAs is harmless here -- a persistent CTA that
  // starts late finds the remaining sites, none waits on another.
  cudaFuncAttributes fa{};
  int sm_per_sm = 0, regs_per_sm = 0;
  if (cudaFuncGetAttributes(&fa, kernel) == cudaSuccess &&
      cudaDeviceGetAttribute(&sm_per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) == cudaSuccess &&
      cudaDeviceGetAttribute(&regs_per_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev) == cudaSuccess) {
    const int by_smem = (int)((size_t)sm_per_sm / (smem + fa.sharedSizeBytes + 1024));
    const int by_regs = fa.numRegs > 0 ? regs_per_sm / (fa.numRegs * threads) : by_smem;
    const int by_threads = 2048 / threads;
    const int est = by_smem < by_regs ? (by_smem < by_threads ? by_smem : by_threads)
                                      : (by_regs < by_threads ? by_regs : by_threads);
    if (est > per_sm) per_sm = est;
  } else {
    cudaGetLastError();
  }
  return per_sm;
}

// The tensor-core descriptor: definitions with alpha <= 8, l_max <= 8 and n_max
// <= 32 (the D tile's 32 columns).
bool descriptor_tc_fits(const DevParams &P) { return P.tc_descriptor && P.amax_t == 8 && P.n_max <= kTdCols; }
size_t descriptor_tc_smem(const DevParams &P) { return make_td_layout(P, 128, 8, 8).total; }

static cudaError_t run_descriptor_tc(const DevParams &P, const DevBatch &B, const LaunchCfg &cfg, double *soap,
                                     float *keep_c, double *keep_norm, int keep) {
  const size_t sm = descriptor_tc_smem(P);
  auto kern = k_descriptor_tc<128, 8, 8>;
  cudaError_t e = ensure_smem_limit(kern, sm);
  if (e != cudaSuccess) return e;
  if (B.site_hi > B.site_lo) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int cap = sms * (512 / kTdTmemCols);
    const int grid = persistent_grid(kern, 128, sm, B.site_hi - B.site_lo,
                                     cfg.max_ctas > 0 ? (cfg.max_ctas < cap ? cfg.max_ctas : cap) : cap);
    kern<<<grid, 128, sm, cfg.stream>>>(P, B, soap, keep_c, keep_norm, keep);
  }
  return cudaGetLastError();
}

// Radial indices per thread: the fewer, the more warps share a site and the more
// loads a product takes.  Two where the sites are at most two per SM and a site's
// latency is all, and where four would leave a site one or two warps or products
// with no radial index (alpha 4, or alpha 5 and 6 with every k in one warp: the kernel at
// 300, 1679 and 8000 sites 24.4, 55.6 and 232 us with two, 27.0, 62.6 and 286 with
// four of eight species, alpha 4, l_max 8; 16.7, 35.2 and 133 against 18.8, 39.5 and 155
// of five, alpha 6, l_max 6).  Else four below kDescWideSites sites, and where every k
// fits one warp; eight from there on: 64 sites of one species of alpha 8 12.6, 13.6 and
// 16.8 us with two, four and eight; with four and eight 29.3 and 33.0 at 1679, 47.2 and
// 45.8 at 3000, 61.1 and 60.1 at 4000, 74.0 and 72.7 at 5000, 111 and 108 at 8000; of
// three species 37 and 41, 64 and 64, 82 and 84, 99 and 103, 150 and 154.
constexpr int kDescFewPerSm = 2, kDescWideSites = 4096;

template <int AMAX, int LC, int NH, int GROUPS = 0, bool ACC = false>
static cudaError_t run_descriptor_as(const DevParams &P, const DevBatch &B, const LaunchCfg &cfg, int max_alpha,
                                     double *soap, float *keep_c, double *keep_norm, int keep) {
  const int kw = (P.k_max + 31) / 32, n = B.site_hi - B.site_lo, own = 32 * kw * ((max_alpha + NH - 1) / NH);
  const int room = GROUPS / own, groups = room < 1 ? 1 : room < P.n_species ? room : P.n_species;
  int threads = own * groups;
  // at few sites a small definition gets warps that only stage rows and form components
  if (NH == 2 && GROUPS == 0 && n <= kDescFewPerSm * sm_count() && threads < 128) threads = 128;
  const int chunk = cfg.slots;  // fixes the summation groups
  const size_t sm = desc_layout(P, chunk, AMAX, LC).total;
  auto kern = k_descriptor<AMAX, LC, NH, GROUPS, ACC>;
  cudaError_t e = ensure_smem_limit(kern, sm);
  if (e != cudaSuccess) return e;
  if (n > 0) {
    kern<<<n, threads, sm, cfg.stream>>>(P, B, chunk, kw, groups, soap, keep_c, keep_norm, keep & 1);
  }
  return cudaGetLastError();
}

template <int AMAX, int LC>
static cudaError_t run_descriptor(const DevParams &P, const DevBatch &B, const LaunchCfg &cfg, double *soap,
                                  float *keep_c, double *keep_norm, int keep) {
  if (AMAX == 8 && LC == 8 && descriptor_tc_fits(P))
    return run_descriptor_tc(P, B, cfg, soap, keep_c, keep_norm, keep);
  int max_alpha = 1;
  for (int s = 0; s < P.n_species; ++s) max_alpha = P.rad[s].alpha > max_alpha ? P.rad[s].alpha : max_alpha;
  const int n = B.site_hi - B.site_lo, sms = sm_count();
  // Sums into the caller's rows are the drop-in call's alone, which the copies around
  // bound: one form.
  if (keep & 2)
    return run_descriptor_as<AMAX, LC, AMAX == 8 ? 4 : 8, 0, true>(P, B, cfg, max_alpha, soap, keep_c, keep_norm, keep);
  // Rows of several chunks on average: one species at a time leaves a round few entries.
  // Up to a site per SM every species gets its warps (rows of 340 pairs, 100 sites of
  // eight species of alpha 4 103 -> 48 us, of five of alpha 6 68 -> 41); beyond, where one
  // species' are at most two, two to four species at a time do (with the pair kernel, 290
  // sites 127 -> 89 and 91 -> 81, 600 195 -> 158 and 135 -> 126; 450 sites of five with
  // 256 threads 131, with 128 111, without groups 117).
  if constexpr (AMAX == 8)
    if (P.n_species > 1 && max_alpha > 2 && (long)B.n_pairs > (long)cfg.slots * B.n_sites) {
      if (n <= sms)
        return run_descriptor_as<AMAX, LC, 4, 512>(P, B, cfg, max_alpha, soap, keep_c, keep_norm, keep);
      if (32 * ((P.k_max + 31) / 32) * ((max_alpha + 3) / 4) <= 64) {
        if (n <= 3 * sms)  // its resident CTAs
          return run_descriptor_as<AMAX, LC, 4, 256>(P, B, cfg, max_alpha, soap, keep_c, keep_norm, keep);
        return run_descriptor_as<AMAX, LC, 4, 128>(P, B, cfg, max_alpha, soap, keep_c, keep_norm, keep);
      }
    }
  if constexpr (AMAX == 8) {
    if (n <= kDescFewPerSm * sms || max_alpha <= 4 || (max_alpha <= 6 && P.k_max <= 32))
      return run_descriptor_as<AMAX, LC, 2>(P, B, cfg, max_alpha, soap, keep_c, keep_norm, keep);
    if (n < kDescWideSites || P.k_max <= 32)
      return run_descriptor_as<AMAX, LC, 4>(P, B, cfg, max_alpha, soap, keep_c, keep_norm, keep);
  }
  return run_descriptor_as<AMAX, LC, 8>(P, B, cfg, max_alpha, soap, keep_c, keep_norm, keep);
}

// The tensor-core contract for the alpha <= 8, l_max <= 8 instantiation: a
// persistent grid of at most 4 CTAs per SM, so that the CTAs resident on an SM
// never ask for more than its 512 TMEM columns.
size_t contract_tc_smem(const DevParams &P) { return make_tc_layout(P, 128, 8).total; }

static cudaError_t run_contract_tc(const DevParams &P, const DevBatch &B, const LaunchCfg &cfg,
                                   const double *soap, const double *G, int g_layout, double sgn,
                                   const float *keep_c, const double *keep_norm, double *pair) {
  const size_t sm = contract_tc_smem(P);
  auto kern = k_contract_tc<128, 8, 8>;
  cudaError_t e = ensure_smem_limit(kern, sm);
  if (e != cudaSuccess) return e;
  if (B.site_hi > B.site_lo) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int cap = sms * (512 / kTcTmemCols);
    const int grid = persistent_grid(kern, 128, sm, B.site_hi - B.site_lo,
                                     cfg.max_ctas > 0 ? (cfg.max_ctas < cap ? cfg.max_ctas : cap) : cap);
    kern<<<grid, 128, sm, cfg.stream>>>(P, B, soap, G, g_layout, sgn, keep_c, keep_norm, pair);
  }
  return cudaGetLastError();
}

// Threads per site: with 64 a site costs the least work, with more it is done
// sooner and the last wave wastes less.  Registers hold an SM to 512 threads (128
// apiece by the launch bounds); shared memory, with many species or l_max 12, to fewer
// CTAs of 64 or 128.  A wave of c CTAs an SM takes cost x 512 / threads, whatever c is, a
// site at 128 and 256 threads costing 1.2 and 1.6 of its share at 64; the choice is the
// one with the cheapest waves.  Contracts at 64, 128 and 256 threads, us: 64 sites of one
// species 21, 15 and 13; 1000 of three 38, 39 and 53; 1679 of three 67, 60 and 79; 8000
// of one 157, 181 and 240; of eight (three, three and two CTAs an SM) 700 89, 69 and 64,
// 3000 324, 241 and 242.  It picks the slower of two in sites of 7 or 8 CTAs of 64 that
// leave the L1 too little for the lists of H (l_max 12, 3000 sites: 198 for 168).
constexpr int kSmemPerSm = 228 * 1024, kSmemReserved = 1024;  // B200; of each CTA
template <int AMAX, int LC>
static int contract_threads(const DevParams &P, int n_sites) {
  const double cost[3] = {1.0, 1.2, 1.6};
  int best = 128;
  double least = 0.0;
  for (int i = 0; i < 3; ++i) {
    const int nt = 64 << i, by_smem = kSmemPerSm / ((int)contract_layout(P, nt, AMAX, LC).total + kSmemReserved);
    const int slots = sm_count() * (by_smem < 512 / nt ? by_smem : 512 / nt);
    if (slots == 0) continue;
    const double t = (double)((n_sites + slots - 1) / slots) * cost[i] * (512 / nt);
    if (least == 0.0 || t < least) {
      least = t;
      best = nt;
    }
  }
  return best;
}

int contract_rule_threads(const DevParams &P, int n_sites) {
  return P.amax_t == 8 ? contract_threads<8, 8>(P, n_sites) : contract_threads<16, 12>(P, n_sites);
}

template <int AMAX, int LC>
static cudaError_t run_contract(const DevParams &P, const DevBatch &B, const LaunchCfg &cfg,
                                const double *soap, const double *G, int g_layout, double sgn,
                                const float *keep_c, const double *keep_norm, double *pair) {
  if (AMAX == 8 && LC == 8 && P.tc_contract)
    return run_contract_tc(P, B, cfg, soap, G, g_layout, sgn, keep_c, keep_norm, pair);
  const int n = B.site_hi - B.site_lo, threads = cfg.threads ? cfg.threads : contract_threads<AMAX, LC>(P, n);
  const size_t sm = contract_layout(P, threads, AMAX, LC).total;
  auto kern = k_contract<AMAX, LC>;
  cudaError_t e = ensure_smem_limit(kern, sm);
  if (e != cudaSuccess) return e;
  if (n > 0) {
    kern<<<n, threads, sm, cfg.stream>>>(P, B, cfg.slots, soap, G, g_layout, sgn, keep_c, keep_norm, pair);
  }
  return cudaGetLastError();
}

int prep_err_words(int n_sites) { return 3 + prep_scan_tiles(n_sites); }

unsigned long long prep_error_code(unsigned long long word) {
  return word == 0 ? ~0ull : kErrTop - word;
}

cudaError_t launch_prep(const DevParams &P, const DevBatch &B, cudaStream_t s) {
  const int tiles = prep_scan_tiles(B.n_sites);
  const int blocks = tiles + (B.n_pairs + kPrepThreads - 1) / kPrepThreads;
  if (blocks > 0) k_prep<<<blocks, kPrepThreads, 0, s>>>(B, P.n_species, tiles);
  return cudaGetLastError();
}

template <int AMAX, int LC, bool OP, bool TAB = false>
static cudaError_t run_pair(const DevParams &P, const DevBatch &B, cudaStream_t s, int do_der, int pair_lo,
                            int pair_hi, bool scan) {
  size_t sm = (size_t)P.off_rad + (size_t)P.n_species * SOAPB_RADSP_BYTES +
              (size_t)kPairThreads * pair_stage_stride(LC) * sizeof(float4);
  // scan tiles reuse it: the tile's counts, then the site order's buckets
  if (sm < (kScanTile + kScanOrderBuckets) * sizeof(int)) sm = (kScanTile + kScanOrderBuckets) * sizeof(int);
  auto kern = k_pair<AMAX, LC, OP, TAB>;
  cudaError_t e = ensure_smem_limit(kern, sm);
  if (e != cudaSuccess) return e;
  const int tiles = scan ? prep_scan_tiles(B.n_sites) : 0;
  const int blocks = pair_cta_offset(B, tiles) + (pair_hi - pair_lo + kPairThreads - 1) / kPairThreads;
  if (blocks > 0) kern<<<blocks, kPairThreads, sm, s>>>(P, B, do_der, tiles, pair_lo, pair_hi);
  return cudaGetLastError();
}

cudaError_t launch_pair(const DevParams &P, const DevBatch &B, cudaStream_t s, int do_der, int pair_lo,
                        int pair_hi, bool scan) {
  if (pair_hi < 0) pair_hi = B.n_pairs;
  if (pair_lo < 0 || pair_lo > pair_hi || pair_hi > B.n_pairs) return cudaErrorInvalidValue;
  if (P.basis == kBasisOperator) {
    if (P.amax_t == 8) return run_pair<8, 8, true>(P, B, s, do_der, pair_lo, pair_hi, scan);
    return run_pair<16, 12, true>(P, B, s, do_der, pair_lo, pair_hi, scan);
  }
  if (P.rtab) {
    if (P.amax_t == 8) return run_pair<8, 8, false, true>(P, B, s, do_der, pair_lo, pair_hi, scan);
    return run_pair<16, 12, false, true>(P, B, s, do_der, pair_lo, pair_hi, scan);
  }
  if (P.amax_t == 8) return run_pair<8, 8, false>(P, B, s, do_der, pair_lo, pair_hi, scan);
  return run_pair<16, 12, false>(P, B, s, do_der, pair_lo, pair_hi, scan);
}

// The radial block is fixed by the definition: the host lays the constants
// blob out for amax_t (8 when every alpha <= 8 and l_max <= 8, else 16).
cudaError_t launch_descriptor(const DevParams &P, const DevBatch &B, const LaunchCfg &cfg,
                              double *soap, float *keep_c, double *keep_norm, int keep) {
  if (P.amax_t == 8) return run_descriptor<8, 8>(P, B, cfg, soap, keep_c, keep_norm, keep);
  return run_descriptor<16, 12>(P, B, cfg, soap, keep_c, keep_norm, keep);
}

cudaError_t launch_contract(const DevParams &P, const DevBatch &B, const LaunchCfg &cfg,
                            const double *soap, const double *G, int g_layout, double sgn,
                            const float *keep_c, const double *keep_norm, double *pair) {
  if (P.amax_t == 8) return run_contract<8, 8>(P, B, cfg, soap, G, g_layout, sgn, keep_c, keep_norm, pair);
  return run_contract<16, 12>(P, B, cfg, soap, G, g_layout, sgn, keep_c, keep_norm, pair);
}

size_t keep_floats_per_site(const DevParams &P) { return keep_stride(P); }

}  // namespace soapb
