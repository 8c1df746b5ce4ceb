// Hamiltonian build on the device: neighbour screen, Slater-Condon SEF blocks, full CSR.
//
// Reference path (psociRestart-Cori/):
//   PsociGAhamiltonian.C:2530-2857  build loop: rows of configuration i, columns j <= i
//   PsociGADeterminants.C:2249-2277 orbmap screen (excitation level <= 2)
//   PsociHamiltonian.C:401-558      generateSOCIblocks: excitation analysis and dispatch
//   PsociHamiltonian.C:139-388      double / single / spin-orbit / diagonal integral sums
//   PsociHamiltonian.C:709-858      socig: spin-orbit determinant elements
//   PsociHamiltonian.C:860-1118     generateSEFCIG: spin-free determinant elements
//   PsociHamiltonian.C:1350-1516    ciout / transformCDCt: det -> SEF (double group) transform
//   PsociGAhamiltonian.C:4077-4136  packSefsef: keep |x| >= 1e-8 and the diagonal
//
// Storage.  The reference keeps the lower triangle and runs a symmetric product.  On one
// GPU the full matrix in CSR streams twice the bytes but needs no scattered atomics in
// sigma, so both triangles are stored.  Every off-diagonal element is the reference's
// lower-triangle value: a block (I, J > I) is the block (J, I) in the reference's roles,
// transposed.  Rows are written in ascending column order, deterministically:
//
//   1. screen:  per configuration, the sorted list of configurations within two
//               excitations (XOR + popcount on occupancy bit-planes), then the blocks
//               that the integrals alone make zero are dropped;
//   2. tables:  every pair's coupling table (blocktab.cuh) and integrals;
//   3. count:   the kept elements of each row, from the tables;
//   4. offsets: a scan of the counts;
//   5. fill:    columns and values in order, the FP32 copy.
// The diagonal blocks are evaluated determinant by determinant before the count.
//
// Spaces with 11 open shells take the generic path instead: every block of the full neighbour
// list is evaluated determinant by determinant in a count pass and again in a fill pass.
//
// Floating point follows the reference's operation order; this file is compiled with
// --fmad=false so products and sums round as the reference's do.
#include <algorithm>
#include <chrono>
#include <climits>
#include <cstdio>
#include <functional>
#include <queue>
#include <vector>

#include "blocktab.cuh"
#include "psoci_internal.cuh"

namespace {

enum { K_NONE = 0, K_DIAG = 1, K_SINGLE = 2, K_DOUBLE = 3, K_SO = 4 };

constexpr int WARPS_PER_CTA = 4;
constexpr int MAXK = 1 + PSOCI_MAX_OPEN * (PSOCI_MAX_OPEN - 1) / 2;  // diagonal vnt list

struct PairInfo {
  int64_t detA, detB;   // first determinant of A, B
  int64_t colbase;      // first SEF of the neighbour J
  int kind, swap;       // swap: J > I, element (t, r) of block (J, I)
  int iex0, jex0;       // single excitations: the orbital A -> B
  int nopenA, nopenB, jsA, jsB, nsefJ;
  double v0, v1;
  double X[PSOCI_MAX_OPEN];  // single: (iex0 s|s jex0) over the open shells s of A
  uint64_t SA[PSOCI_MAX_WORDS];  // open shells of A
  // orbital ranges the determinant phases count electrons over, fixed for the pair:
  //   K_DOUBLE: 0-3 strictly between ex_i and jy_j (index 2i + j), 4 between ex0 and ex1,
  //             5 between jy0 and jy1;
  //   K_SINGLE, K_SO: 0 strictly between ie and je, 1 below ie, 2 above je, 3 below je,
  //             4 above ie
  uint64_t bm[6][PSOCI_MAX_WORDS];
};

struct WarpSmem {
  PairInfo pi[PSOCI_SEG];
  int itemoff[PSOCI_SEG + 1];
  double K[MAXK];  // diagonal: K[0] = vnt(1), K[mm] = open-pair exchange (reference order)
};

struct Params {
  int nconf, nbf, nelec, ksym;
  const uint64_t *e1, *e2;
  const int32_t *jsym, *nopen;
  const int64_t *sefoff, *detoff;
  const uint64_t *alpha, *beta;
  const uint8_t *phase, *nalpha;
  const double *one, *eri;
  // screen
  const int64_t *nbroff;
  int32_t *nbr;
  // segments
  int64_t nseg;
  const int32_t *seg_cfg;
  const int64_t *seg_k0;
  const int32_t *seg_n;
  const int64_t *seg_rowoff;
  int64_t *seg_cnt;        // count pass output / fill pass row offsets (local)
  const int64_t *rowptr;
  int32_t *col;
  double *val;
  float *val32;
  double *diag;
  // direct sigma (PASS 2): Y[:, 0:kvec] += H X[:, 0:kvec]; with dx32 (the inputs in FP32,
  // 8 per row) the products are FP32 element x FP32 input with compensated FP32 sums
  const float *dx32;
  const double *dx;
  double *dy;
  int ldx, ldy, kvec;
};

// ------------------------------------------------------------------------------------
// bit helpers over W words
// ------------------------------------------------------------------------------------
template <int W>
__device__ __forceinline__ int popc_range(const uint64_t *x, int lo, int hi) {
  if (lo > hi) return 0;
  int c = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    int l = lo - 64 * w, h = hi - 64 * w;
    if (h < 0 || l > 63) continue;
    if (l < 0) l = 0;
    if (h > 63) h = 63;
    uint64_t m = (h == 63 ? ~0ull : ((1ull << (h + 1)) - 1ull)) & (~0ull << l);
    c += __popcll(x[w] & m);
  }
  return c;
}
template <int W>
__device__ __forceinline__ int popc_w(const uint64_t *x) {
  int c = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) c += __popcll(x[w]);
  return c;
}
template <int W>
__device__ __forceinline__ int lowest_bit(const uint64_t *x) {
#pragma unroll
  for (int w = 0; w < W; ++w)
    if (x[w]) return 64 * w + __ffsll((long long)x[w]) - 1;
  return -1;
}
template <int W>
__device__ __forceinline__ int second_bit(const uint64_t *x) {
  uint64_t y[W];
  bool cleared = false;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    y[w] = x[w];
    if (!cleared && y[w]) { y[w] &= y[w] - 1; cleared = true; }
  }
  return lowest_bit<W>(y);
}
// bits lo..hi inclusive (none when lo > hi) over W words
template <int W>
__device__ __forceinline__ void range_mask(int lo, int hi, uint64_t *m) {
#pragma unroll
  for (int w = 0; w < W; ++w) {
    int l = lo - 64 * w, h = hi - 64 * w;
    if (lo > hi || h < 0 || l > 63) { m[w] = 0ull; continue; }
    if (l < 0) l = 0;
    if (h > 63) h = 63;
    m[w] = (h == 63 ? ~0ull : ((1ull << (h + 1)) - 1ull)) & (~0ull << l);
  }
}
// orbitals strictly between a and b
template <int W>
__device__ __forceinline__ void between_mask(int a, int b, uint64_t *m) {
  range_mask<W>(min(a, b) + 1, max(a, b) - 1, m);
}
template <int W>
__device__ __forceinline__ int popc_and(const uint64_t *x, const uint64_t *m) {
  int c = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) c += __popcll(x[w] & m[w]);
  return c;
}

// register-array forms: word selection by value, so that the arrays stay in registers
template <int W>
__device__ __forceinline__ bool bit_w(const uint64_t (&x)[W], int p) {
  uint64_t v = x[0];
#pragma unroll
  for (int w = 1; w < W; ++w)
    if ((p >> 6) == w) v = x[w];
  return (v >> (p & 63)) & 1ull;
}
template <int W>
__device__ __forceinline__ void sel_w(uint64_t (&d)[W], bool c, const uint64_t (&a)[W], const uint64_t (&b)[W]) {
#pragma unroll
  for (int w = 0; w < W; ++w) d[w] = c ? a[w] : b[w];
}

__device__ __forceinline__ double g2(const Params &P, int i, int j, int k, int l) { return __ldg(P.eri + canon4(i, j, k, l)); }
__device__ __forceinline__ double g1(const Params &P, int i, int j) { return __ldg(P.one + tri64(i, j)); }

// ------------------------------------------------------------------------------------
// excitation screen
// ------------------------------------------------------------------------------------
// Excitation orbitals between occupations A and B, ascending with multiplicity:
// A has more electrons than B in iex, fewer in jex (generateSOCIblocks, PsociHamiltonian.C:496-512).
template <int W>
__device__ __forceinline__ int excitation(const uint64_t *e1A, const uint64_t *e2A, const uint64_t *e1B,
                                          const uint64_t *e2B, int *ex, int *jy) {
  int ni = 0, nj = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    uint64_t i1 = e1A[w] & ~e1B[w], i2 = e2A[w] & ~e2B[w];
    uint64_t j1 = e1B[w] & ~e1A[w], j2 = e2B[w] & ~e2A[w];
    uint64_t u = i1 | i2;
    while (u) {
      int b = __ffsll((long long)u) - 1;
      u &= u - 1;
      int mult = (int)((i1 >> b) & 1ull) + (int)((i2 >> b) & 1ull);
      for (int q = 0; q < mult; ++q) { if (ni < 2) ex[ni] = 64 * w + b; ++ni; }
    }
    u = j1 | j2;
    while (u) {
      int b = __ffsll((long long)u) - 1;
      u &= u - 1;
      int mult = (int)((j1 >> b) & 1ull) + (int)((j2 >> b) & 1ull);
      for (int q = 0; q < mult; ++q) { if (nj < 2) jy[nj] = 64 * w + b; ++nj; }
    }
  }
  return ni;
}

// The same, with the first two positions of each side returned in registers (no local
// arrays): ex0 <= ex1 removed from A, jy0 <= jy1 added in B, -1 where absent.
template <int W>
__device__ __forceinline__ int excitation_r(const uint64_t *e1A, const uint64_t *e2A, const uint64_t *e1B,
                                            const uint64_t *e2B, int &ex0, int &ex1, int &jy0, int &jy1) {
  int ni = 0, nj = 0;
  ex0 = ex1 = jy0 = jy1 = -1;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    const uint64_t i1 = e1A[w] & ~e1B[w], i2 = e2A[w] & ~e2B[w];
    const uint64_t j1 = e1B[w] & ~e1A[w], j2 = e2B[w] & ~e2A[w];
    uint64_t u = i1 | i2;
    while (u) {
      const int b = __ffsll((long long)u) - 1;
      u &= u - 1;
      const int p = 64 * w + b;
      const int both = (int)((i1 >> b) & (i2 >> b) & 1ull);
      if (ni == 0) { ex0 = p; if (both) ex1 = p; }
      else if (ni == 1) ex1 = p;
      ni += 1 + both;
    }
    u = j1 | j2;
    while (u) {
      const int b = __ffsll((long long)u) - 1;
      u &= u - 1;
      const int p = 64 * w + b;
      const int both = (int)((j1 >> b) & (j2 >> b) & 1ull);
      if (nj == 0) { jy0 = p; if (both) jy1 = p; }
      else if (nj == 1) jy1 = p;
      nj += 1 + both;
    }
  }
  return ni;
}

// Screen, stage 1: configurations within two excitations of i (sum |occ_i - occ_j| <= 4,
// the orbmap test of PsociGADeterminants.C:2249-2277).  One thread per row configuration;
// tiles of column configurations are staged in shared memory and read by broadcast, so each
// thread's candidate list comes out sorted.  blockIdx.y selects a contiguous range of
// column configurations [y*chunk, (y+1)*chunk) so small problems still fill the GPU; MODE 0
// counts per (range, row), MODE 1 writes each range's candidates after the earlier ranges'.
constexpr int SCR_THREADS = 256;
constexpr int SCR_TILE = 512;
constexpr int SCR_ROWS = 4;  // row configurations per thread: one shared-memory load serves four tests

template <int W, int MODE>
__global__ void __launch_bounds__(SCR_THREADS) k_screen(Params P, int64_t *cnt, const int64_t *soff, int64_t chunk,
                                                        const int64_t *candoff, int32_t *cand) {
  __shared__ uint64_t t1[SCR_TILE * W], t2[SCR_TILE * W];
  uint64_t a1[SCR_ROWS][W], a2[SCR_ROWS][W];
  int64_t n[SCR_ROWS], out[SCR_ROWS];
  bool act[SCR_ROWS];
#pragma unroll
  for (int q = 0; q < SCR_ROWS; ++q) {
    const int64_t i = (int64_t)blockIdx.x * (SCR_THREADS * SCR_ROWS) + q * SCR_THREADS + threadIdx.x;
    act[q] = i < P.nconf;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      a1[q][w] = act[q] ? P.e1[i * W + w] : ~0ull;  // inactive rows match nothing
      a2[q][w] = act[q] ? P.e2[i * W + w] : ~0ull;
    }
    n[q] = 0;
    out[q] = (MODE == 1 && act[q]) ? candoff[i] + soff[(int64_t)blockIdx.y * P.nconf + i] : 0;
  }
  const int64_t jbeg = (int64_t)blockIdx.y * chunk;
  const int64_t jend = min((int64_t)P.nconf, jbeg + chunk);
  for (int64_t j0 = jbeg; j0 < jend; j0 += SCR_TILE) {
    const int nt = (int)min((int64_t)SCR_TILE, jend - j0);
    __syncthreads();
    for (int e = threadIdx.x; e < nt * W; e += SCR_THREADS) {
      t1[e] = P.e1[j0 * W + e];
      t2[e] = P.e2[j0 * W + e];
    }
    __syncthreads();
    for (int jj = 0; jj < nt; ++jj) {
      uint64_t b1[W], b2[W];
#pragma unroll
      for (int w = 0; w < W; ++w) { b1[w] = t1[jj * W + w]; b2[w] = t2[jj * W + w]; }
#pragma unroll
      for (int q = 0; q < SCR_ROWS; ++q) {
        int d = __popcll(a1[q][0] ^ b1[0]) + __popcll(a2[q][0] ^ b2[0]);
#pragma unroll
        for (int w = 1; w < W; ++w)
          if (d <= 4) d += __popcll(a1[q][w] ^ b1[w]) + __popcll(a2[q][w] ^ b2[w]);
        if (d <= 4 && act[q]) {
          if (MODE == 1) cand[out[q] + n[q]] = (int32_t)(j0 + jj);
          ++n[q];
        }
      }
    }
  }
  if (MODE == 0) {
#pragma unroll
    for (int q = 0; q < SCR_ROWS; ++q) {
      const int64_t i = (int64_t)blockIdx.x * (SCR_THREADS * SCR_ROWS) + q * SCR_THREADS + threadIdx.x;
      if (act[q]) cnt[(int64_t)blockIdx.y * P.nconf + i] = n[q];
    }
  }
}

// A double-excitation block (PsociHamiltonian.C:180-185) has determinant elements +-v0,
// +-v1 or +-(v0 - v1) with v0 = (i0 j0|i1 j1), v1 = (i0 j1|i1 j0), and each SEF element
// combines at most four of them with weights +-1/2, so |element| <= 2 (|v0| + |v1|) (plus
// rounding of a few ulps).  With |v0| + |v1| < 4e-9 every element is below the 1e-8 that
// packSefsef stores (PsociGAhamiltonian.C:4077-4136): the block adds nothing to H and is
// not evaluated.  This includes the blocks the reference skips outright (v0 = v1 = 0).
__device__ __forceinline__ bool double_block_kept(double v0, double v1) { return fabs(v0) + fabs(v1) >= 4e-9; }

// Screen, stage 2: drop candidates whose block stores nothing, judged from its integral
// prefactors alone — double excitations as above and spin-orbit singles with SO_ij = 0
// (PsociHamiltonian.C:227); both tests are symmetric in (i, j).  One warp per row configuration, candidates in order, ballot
// compaction; MODE 0 tests and counts, and marks a dropped candidate by its complement, MODE 1 writes
// (with the tests again it took 98 us for the 4.3 M candidates of 6 electrons in 12 orbitals, 20 now).
template <int W, int MODE>
__global__ void k_prune(Params P, const int64_t *candoff, int32_t *cand, int64_t *cnt) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i = warp; i < P.nconf; i += nwarps) {
    uint64_t a1[W], a2[W];
    int js_i = 0;
    if (MODE == 0) {
#pragma unroll
      for (int w = 0; w < W; ++w) { a1[w] = P.e1[i * W + w]; a2[w] = P.e2[i * W + w]; }
      js_i = P.jsym[i];
    }
    const int64_t c0 = candoff[i], c1 = candoff[i + 1];
    int64_t n = 0;
    const int64_t out = (MODE == 1) ? P.nbroff[i] : 0;
    for (int64_t t0 = c0; t0 < c1; t0 += 32) {
      const int64_t t = t0 + lane;
      bool keep = false;
      int32_t j = 0;
      if (t < c1) {
        j = cand[t];
        keep = j >= 0;
        if (MODE == 0 && j != i) {
          uint64_t b1[W], b2[W];
#pragma unroll
          for (int w = 0; w < W; ++w) { b1[w] = __ldg(P.e1 + (int64_t)j * W + w); b2[w] = __ldg(P.e2 + (int64_t)j * W + w); }
          int ex[2], jy[2];
          int ni = (j <= i) ? excitation<W>(a1, a2, b1, b2, ex, jy) : excitation<W>(b1, b2, a1, a2, ex, jy);
          if (ni == 2) {
            keep = double_block_kept(__ldg(P.eri + canon4(ex[0], jy[0], ex[1], jy[1])),
                                     __ldg(P.eri + canon4(ex[0], jy[1], ex[1], jy[0])));
          } else if (ni == 1 && __ldg(P.jsym + j) != js_i) {
            keep = __ldg(P.one + tri64(ex[0], jy[0])) != 0.0;
          }
          if (!keep) cand[t] = ~j;
        }
      }
      const unsigned b = __ballot_sync(0xffffffffu, keep);
      if (MODE == 1 && keep) P.nbr[out + n + __popc(b & ((1u << lane) - 1u))] = j;
      n += __popc(b);
    }
    if (MODE == 0 && lane == 0) cnt[i] = n;
  }
}

// ------------------------------------------------------------------------------------
// Screen by lookup ("split join").  With the orbitals split at s so that every
// configuration holds at most two electrons in the orbitals >= s, a configuration is a
// (hi pattern g, lo pattern l) pair and its distance to another is d_hi + d_lo.  Any two
// hi patterns of <= 2 electrons are within 4, so the neighbours of i are, for every hi
// pattern h, the configurations T[h][l'] with d_lo(l_i, l') <= 4 - d_hi(g_i, h): one lookup
// when the hi patterns are disjoint, a short list otherwise — work in proportion to the
// neighbours instead of to all pairs.  Configurations are numbered in (g, l) order (checked
// when the tables are built), so scanning h and then l' in ascending order yields sorted
// lists.  The integral-based pruning of k_prune is applied to each candidate on the spot.
// One warp per row configuration, one lane per hi pattern; MODE 0 counts (kept and all
// candidates), MODE 1 writes the kept neighbours at off[i].
// ------------------------------------------------------------------------------------
struct JoinTabs {
  int s, G, L;
  const int32_t *gid, *lid, *T, *lnoff, *ln, *hdec;
  const uint32_t *lokey;
  const int64_t *goff;    // per hi pattern g: its list of hi patterns h to visit ...
  const uint32_t *glist;  // ... h | d_hi(g, h) << 28, ascending h
  const uint32_t *dkept;  // double_block_kept of (ex0 <= ex1) -> (jy0 <= jy1), bit tri(ex)*NT + tri(jy)
  int64_t nt;             // NT = nbf(nbf+1)/2; at most 128 orbitals, so NT^2 bits have 32-bit places
};

// The pruning decision of every double excitation, as bits: word q holds the pairs
// (a, b), a = tri(ex0, ex1), b = tri(jy0, jy1), with a * NT + b in [32q, 32q + 32).  The
// same integrals and test as the per-candidate form, so the same decisions.
__global__ void k_double_kept(int64_t nt, const int2 *__restrict__ pairs, const double *__restrict__ eri,
                              uint32_t *bits) {
  const int64_t nwords = (nt * nt + 31) / 32;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nwords; q += (int64_t)gridDim.x * blockDim.x) {
    uint32_t w = 0u;
    for (int u = 0; u < 32; ++u) {
      const int64_t e = q * 32 + u;
      if (e >= nt * nt) break;
      const int2 x = pairs[e / nt], y = pairs[e % nt];  // (ex0, ex1), (jy0, jy1), ascending
      const bool k = double_block_kept(__ldg(eri + canon4(x.x, y.x, x.y, y.y)), __ldg(eri + canon4(x.x, y.y, x.y, y.x)));
      w |= (uint32_t)k << u;
    }
    bits[q] = w;
  }
}

template <int W>
__device__ __forceinline__ void set_bit_w(uint64_t (&x)[W], int p) {
#pragma unroll
  for (int w = 0; w < W; ++w)
    if ((p >> 6) == w) x[w] |= 1ull << (p & 63);
}

// occupancy bit-planes of hi pattern code (kind 0: empty, 1: one electron in a, 2: one
// each in a < b, 3: two in a; positions relative to s)
template <int W>
__device__ __forceinline__ void hi_bits(int code, int s, uint64_t (&e1)[W], uint64_t (&e2)[W]) {
#pragma unroll
  for (int w = 0; w < W; ++w) e1[w] = e2[w] = 0ull;
  const int kind = code & 3, a = (code >> 8) & 0xfff, b = (code >> 20) & 0xfff;
  if (kind != 0) set_bit_w<W>(e1, s + a);
  if (kind == 3) set_bit_w<W>(e2, s + a);
  if (kind == 2) set_bit_w<W>(e1, s + b);
}

// electrons of hi pattern code: 0, 1, 2, 2 for kinds 0-3
__device__ __forceinline__ int hi_electrons(int code) { return min(code & 3, 2); }

// Hi-pattern lists.  For d_hi(g, h) = 4 the lo patterns must be equal, so the pair is a
// double excitation between the hi orbitals alone and whether its block survives the
// integral test (double_block_kept) depends on (g, h) only — it is decided here once
// instead of once per configuration pair.  The list of g keeps every h with d_hi < 4 and
// the h with d_hi = 4 whose block survives.  One warp per g, lanes over h; MODE 0 counts,
// MODE 1 writes (ascending h).
template <int W, int MODE>
__global__ void k_group_lists(JoinTabs J, const double *__restrict__ eri, int64_t *gcnt, uint32_t *glist) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t g = warp; g < J.G; g += nwarps) {
    uint64_t g1[W], g2[W];
    hi_bits<W>(J.hdec[g], J.s, g1, g2);
    int64_t n = 0;
    const int64_t out = (MODE == 1) ? J.goff[g] : 0;
    for (int h0 = 0; h0 < J.G; h0 += 32) {
      const int h = h0 + lane;
      bool take = false;
      int d = 0;
      if (h < J.G) {
        uint64_t b1[W], b2[W];
        hi_bits<W>(J.hdec[h], J.s, b1, b2);
#pragma unroll
        for (int w = 0; w < W; ++w) d += __popcll(g1[w] ^ b1[w]) + __popcll(g2[w] ^ b2[w]);
        take = true;
        if (d == 4) {
          int ex[2], jy[2];
          const int ni = excitation<W>(g1, g2, b1, b2, ex, jy);
          take = (ni == 2) && double_block_kept(__ldg(eri + canon4(ex[0], jy[0], ex[1], jy[1])),
                                                __ldg(eri + canon4(ex[0], jy[1], ex[1], jy[0])));
        }
      }
      const unsigned b = __ballot_sync(0xffffffffu, take);
      if (MODE == 1 && take) glist[out + n + __popc(b & ((1u << lane) - 1u))] = (uint32_t)h | ((uint32_t)d << 28);
      n += __popc(b);
    }
    if (MODE == 0 && lane == 0) gcnt[g] = n;
  }
}

// Slab of the single-pass join (MODE 2): each warp appends the neighbour lists of its
// configurations to chunks it takes from a shared counter; a configuration's list stays
// contiguous (a list outgrowing its chunk moves to a fresh one).  Positions at or beyond
// cap are not touched; the host sees the counter and falls back to count + write passes.
struct JoinSlab {
  int32_t *list;
  unsigned long long *counter;
  int64_t cap;
  int64_t *start;  // [nconf] slab position of each configuration's list
};
constexpr int JOIN_CHUNK = 4096, JOIN_ALONE = -1;

// One warp a configuration, lanes over its lookups in (hi pattern, lo pattern) order.  Bound by
// instruction issue (67% of the slots) and the lookups' latency: 1.04 G lookups of mrcisd_6e8o_v48,
// of which 181 M pairs stay, 9.9 -> 7.7 ms with a lookup's run found by ballot instead of a binary
// search, the orbitals of two electrons taken as the lowest and the highest set bit (9.9 -> 8.7), and
// the table T by hi pattern, so that a list's ascending lo patterns share its sectors (8.7 -> 7.7).
template <int W, int MODE>
__global__ void __launch_bounds__(256) k_join(Params P, JoinTabs J, int64_t *cnt, int64_t *ncand, const int64_t *off,
                                              JoinSlab S) {
  // per hi pattern with lo patterns to visit: x, the first of them in J.ln less the first lookup (l_i
  // itself when the hi patterns are disjoint); y, the pattern; z, w, its part of the excitation from
  // i: orbitals, electrons (JOIN_ALONE when the hi patterns are disjoint)
  __shared__ uint4 s_run[8][32];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u, le = lt | (1u << lane);
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const uint32_t lomask = (1u << J.s) - 1u;
  unsigned long long cursor = 0, chunk_end = 0;  // MODE 2: this warp's slab chunk
  for (int64_t i = warp; i < P.nconf; i += nwarps) {
    const int li = J.lid[i], js_i = P.jsym[i], gi = J.gid[i];
    const int ne_i = hi_electrons(J.hdec[gi]);
    // the excitation i -> j splits into its lo part (orbitals < s, from the two lo keys) and
    // its hi part (from the two hi patterns, once per hi pattern); orbitals ascend, so the lo
    // orbitals come first in each list
    uint64_t g1[W], g2[W];
    hi_bits<W>(J.hdec[gi], J.s, g1, g2);
    const uint32_t keyi = J.lokey[li];
    int64_t nk = 0, nc = 0;
    int64_t base = (MODE == 1) ? off[i] : 0;
    unsigned long long lstart = cursor;  // MODE 2: where this configuration's list begins
    const int64_t gl0 = J.goff[gi], gl1 = J.goff[gi + 1];
    for (int64_t h0 = gl0; h0 < gl1; h0 += 32) {
      // this lane's hi pattern h: the lo patterns l' with d_lo <= 4 - d_hi and the electron
      // count that h leaves, as a range of the neighbour list of l_i (or l_i alone when the
      // hi patterns are disjoint: those blocks passed the integral test when the list was
      // built)
      int h = 0;
      int len = 0, q0 = li, hn = JOIN_ALONE;
      uint32_t hx = 0u;
      if (h0 + lane < gl1) {
        const uint32_t ent = J.glist[h0 + lane];
        h = (int)(ent & 0x0fffffffu);
        const int d = (int)(ent >> 28);
        const int tau = 4 - d;
        const int code = J.hdec[h];
        const int k = ne_i - hi_electrons(code) + 2;  // lo electrons of l' minus l_i's, + 2
        if (tau <= 0) len = (k == 2);
        else {
          const int64_t at = (int64_t)(tau - 1) * (5 * (int64_t)J.L + 1) + 5 * (int64_t)li + k;
          q0 = J.lnoff[at];
          len = J.lnoff[at + 1] - q0;
          // hi part: the electrons leaving g_i (the first two, ascending, with multiplicity)
          // and their count, the first two arriving in h; 8 bits per orbital
          uint64_t b1[W], b2[W];
          hi_bits<W>(code, J.s, b1, b2);
          int x0, x1, y0, y1;
          hn = excitation_r<W>(g1, g2, b1, b2, x0, x1, y0, y1);
          hx = (uint32_t)(x0 & 0xff) | ((uint32_t)(x1 & 0xff) << 8) | ((uint32_t)(y0 & 0xff) << 16) |
               ((uint32_t)(y1 & 0xff) << 24);
        }
      }
      int incl = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      const int tot = __shfl_sync(0xffffffffu, incl, 31);
      const int st = incl - len;
      const unsigned runs = __ballot_sync(0xffffffffu, len > 0);
      if (len > 0)
        s_run[wib][__popc(runs & lt)] = make_uint4((uint32_t)(hn == JOIN_ALONE ? q0 : q0 - st), (uint32_t)h, hx, (uint32_t)hn);
      __syncwarp();
      // the chunk's lookups, spread evenly over the lanes in (h, l') order; a lookup's run is the
      // last that starts at or before it
      int started = 0;
      for (int e0 = 0; e0 < tot; e0 += 32) {
        const unsigned bw =
            __reduce_or_sync(0xffffffffu, (len > 0 && (unsigned)(st - e0) < 32u) ? 1u << ((st - e0) & 31) : 0u);
        bool found = false, keep = false;
        int j = -1;
        if (e0 + lane < tot) {
          const uint4 u = s_run[wib][started + __popc(bw & le) - 1];
          const bool alone = (int)u.w == JOIN_ALONE;
          const int lp = alone ? (int)u.x : __ldg(J.ln + (int)u.x + (e0 + lane));
          j = __ldg(J.T + ((int64_t)u.y * J.L + lp));
          found = keep = j >= 0;
          if (found && j != (int)i && !alone) {
            // lo part from the keys (bit q: orbital q occupied; bit s + q: doubly)
            const uint32_t keyj = __ldg(J.lokey + lp), di = keyi & ~keyj, dj = keyj & ~keyi;
            const int lni = __popc(di), ni = lni + (int)u.w;
            if (ni <= 2) {
              // first two orbitals of each list: lo ones (of two electrons the lowest and the highest
              // orbital, the same if they share one), then hi ones
              const uint32_t ui = (di | (di >> J.s)) & lomask, uj = (dj | (dj >> J.s)) & lomask;
              const int lnj = __popc(dj);
              const int ex0 = lni >= 1 ? __ffs(ui) - 1 : (int)(u.z & 0xffu);
              const int jy0 = lnj >= 1 ? __ffs(uj) - 1 : (int)((u.z >> 16) & 0xffu);
              // the tests below are symmetric in the two configurations' roles
              if (ni == 2) {
                const int ex1 = lni >= 2 ? 31 - __clz(ui) : (int)((lni == 1 ? u.z : u.z >> 8) & 0xffu);
                const int jy1 = lnj >= 2 ? 31 - __clz(uj) : (int)((lnj == 1 ? u.z >> 16 : u.z >> 24) & 0xffu);
                const uint32_t at = (uint32_t)(ex1 * (ex1 + 1) / 2 + ex0) * (uint32_t)J.nt +
                                    (uint32_t)(jy1 * (jy1 + 1) / 2 + jy0);
                keep = (__ldg(J.dkept + (at >> 5)) >> (at & 31u)) & 1u;
              } else if (ni == 1 && __ldg(P.jsym + j) != js_i) {
                keep = __ldg(P.one + tri64(ex0, jy0)) != 0.0;
              }
            }
          }
        }
        started += __popc(bw);
        const unsigned kb = __ballot_sync(0xffffffffu, keep);
        if (MODE == 0) {
          nc += __popc(__ballot_sync(0xffffffffu, found));
          nk += __popc(kb);
        } else if (MODE == 1) {
          if (keep) P.nbr[base + __popc(kb & ((1u << lane) - 1u))] = j;
          base += __popc(kb);
        } else {
          nc += __popc(__ballot_sync(0xffffffffu, found));
          if (cursor + 32 > chunk_end) {
            // a fresh chunk; the list written so far moves along
            const unsigned long long len = (unsigned long long)max((int64_t)JOIN_CHUNK, 2 * (nk + 32));
            unsigned long long b = 0;
            if (lane == 0) b = atomicAdd(S.counter, len);
            b = __shfl_sync(0xffffffffu, b, 0);
            __syncwarp();  // the list's earlier entries were written by other lanes
            for (int64_t t = lane; t < nk; t += 32) {
              const unsigned long long from = lstart + t, to = b + t;
              if ((int64_t)from < S.cap && (int64_t)to < S.cap) S.list[to] = S.list[from];
            }
            lstart = b;
            cursor = b + nk;
            chunk_end = b + len;
          }
          const unsigned long long pos = cursor + __popc(kb & ((1u << lane) - 1u));
          if (keep && (int64_t)pos < S.cap) S.list[pos] = j;
          cursor += __popc(kb);
          nk += __popc(kb);
        }
      }
      __syncwarp();
    }
    if (MODE != 1 && lane == 0) { cnt[i] = nk; ncand[i] = nc; }
    if (MODE == 2 && lane == 0) S.start[i] = (int64_t)lstart;
  }
}

// neighbour lists from the join slab to their final, contiguous places
__global__ void k_join_compact(int nconf, const int32_t *__restrict__ slab, const int64_t *__restrict__ start,
                               const int64_t *__restrict__ nbroff, int32_t *__restrict__ nbr) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i = warp; i < nconf; i += nwarps) {
    const int64_t o = nbroff[i], len = nbroff[i + 1] - o, st = start[i];
    for (int64_t t = lane; t < len; t += 32) nbr[o + t] = slab[st + t];
  }
}

// per row configuration: exclusive offsets of its column ranges and its total
__global__ void k_screen_offsets(int nconf, int nsplit, const int64_t *cnt, int64_t *soff, int64_t *tot) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nconf) return;
  int64_t run = 0;
  for (int sp = 0; sp < nsplit; ++sp) {
    int64_t v = cnt[(int64_t)sp * nconf + i];
    soff[(int64_t)sp * nconf + i] = run;
    run += v;
  }
  tot[i] = run;
}

// per configuration: number of segments and segment-row slots over its neighbours
__global__ void k_seg_counts(int nconf, const int64_t *nbroff, const int64_t *sefoff, int64_t *nseg_i,
                             int64_t *nrow_i) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nconf) return;
  int64_t nn = nbroff[i + 1] - nbroff[i];
  int64_t ns = (nn + PSOCI_SEG - 1) / PSOCI_SEG;
  nseg_i[i] = ns;
  nrow_i[i] = ns * (sefoff[i + 1] - sefoff[i]);
}

__global__ void k_seg_init(int nconf, const int64_t *nbroff, const int64_t *sefoff, const int64_t *segoff,
                           const int64_t *rowslot, int32_t *seg_cfg, int64_t *seg_k0,
                           int32_t *seg_n, int64_t *seg_rowoff) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nconf) return;
  int64_t nn = nbroff[i + 1] - nbroff[i];
  int64_t s0 = segoff[i], ns = segoff[i + 1] - s0;
  int64_t nsef = sefoff[i + 1] - sefoff[i];
  for (int64_t s = 0; s < ns; ++s) {
    seg_cfg[s0 + s] = (int32_t)i;
    seg_k0[s0 + s] = nbroff[i] + s * PSOCI_SEG;
    int64_t left = nn - s * PSOCI_SEG;
    seg_n[s0 + s] = (int32_t)(left < PSOCI_SEG ? left : PSOCI_SEG);
    seg_rowoff[s0 + s] = rowslot[i] + s * nsef;
  }
}

// per configuration: exclusive scan over its segments of the per-row counts (in place),
// totals per SEF row into row_nnz
__global__ void k_seg_rowscan(int nconf, const int64_t *sefoff, const int64_t *segoff, const int64_t *seg_rowoff,
                              int64_t *seg_cnt, int64_t *row_nnz) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nconf) return;
  int64_t nsef = sefoff[i + 1] - sefoff[i];
  for (int64_t r = 0; r < nsef; ++r) {
    int64_t run = 0;
    for (int64_t s = segoff[i]; s < segoff[i + 1]; ++s) {
      int64_t *p = seg_cnt + seg_rowoff[s] + r;
      int64_t v = *p;
      *p = run;
      run += v;
    }
    row_nnz[sefoff[i] + r] = run;
  }
}

// ------------------------------------------------------------------------------------
// per-pair set-up (one lane per neighbour)
// ------------------------------------------------------------------------------------
// The first two positions of the multiset m1 + m2 (a position in both counts twice),
// ascending.
template <int W>
__device__ __forceinline__ void two_positions(const uint64_t (&m1)[W], const uint64_t (&m2)[W], int &p0, int &p1) {
  int nd = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    uint64_t u = m1[w] | m2[w];
    while (u && nd < 2) {
      const int b = __ffsll((long long)u) - 1;
      u &= u - 1;
      const int p = 64 * w + b;
      const int mult = (int)((m1[w] >> b) & 1ull) + (int)((m2[w] >> b) & 1ull);
      if (nd == 0) { p0 = p; nd = 1; if (mult == 2) { p1 = p; nd = 2; } }
      else { p1 = p; nd = 2; }
    }
  }
}

// Set up the pair (A, B) in the reference's roles (A = "iconf" of generateSOCIblocks);
// J is the configuration whose SEFs are the CSR columns.
template <int W>
__device__ void pair_setup_ab(const Params &P, int A, int B, int J, int swap, PairInfo &pi, double *Kd) {
  pi.swap = swap;
  pi.detA = P.detoff[A]; pi.detB = P.detoff[B];
  pi.colbase = P.sefoff[J];
  pi.nsefJ = (int)(P.sefoff[J + 1] - P.sefoff[J]);
  pi.nopenA = P.nopen[A]; pi.nopenB = P.nopen[B];
  pi.jsA = P.jsym[A]; pi.jsB = P.jsym[B];
  uint64_t e1A[W], e2A[W], e1B[W], e2B[W], im1[W], im2[W], jm1[W], jm2[W];
#pragma unroll
  for (int w = 0; w < W; ++w) {
    e1A[w] = P.e1[(int64_t)A * W + w]; e2A[w] = P.e2[(int64_t)A * W + w];
    e1B[w] = P.e1[(int64_t)B * W + w]; e2B[w] = P.e2[(int64_t)B * W + w];
    im1[w] = e1A[w] & ~e1B[w]; im2[w] = e2A[w] & ~e2B[w];
    jm1[w] = e1B[w] & ~e1A[w]; jm2[w] = e2B[w] & ~e2A[w];
    pi.SA[w] = e1A[w] & ~e2A[w];
  }
  pi.v0 = 0.0; pi.v1 = 0.0;
  pi.iex0 = pi.jex0 = -1;
  int ni = popc_w<W>(im1) + popc_w<W>(im2);
  if (A == B) {
    pi.kind = K_DIAG;
    // processDiagExcitation (PsociHamiltonian.C:306-388)
    int sing[PSOCI_MAX_OPEN], ns = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      uint64_t s = pi.SA[w];
      while (s && ns < PSOCI_MAX_OPEN) { sing[ns++] = 64 * w + __ffsll((long long)s) - 1; s &= s - 1; }
    }
    int mm = 1;
    for (int a = 1; a < ns; ++a)
      for (int b = 0; b < a; ++b) Kd[mm++] = g2(P, sing[a], sing[b], sing[b], sing[a]);
    double v = 0.0;
#pragma unroll
    for (int wi = 0; wi < W; ++wi) {
      uint64_t oi = e1A[wi];
      while (oi) {
        int ib = 64 * wi + __ffsll((long long)oi) - 1;
        oi &= oi - 1;
        int occi = 1 + (int)bit_w<W>(e2A, ib);
        if (occi == 1) v += g1(P, ib, ib);
        else v += 2.0 * g1(P, ib, ib) + g2(P, ib, ib, ib, ib);
#pragma unroll
        for (int wj = 0; wj < W; ++wj) {
          uint64_t oj = e1A[wj];
          while (oj) {
            int jb = 64 * wj + __ffsll((long long)oj) - 1;
            oj &= oj - 1;
            if (jb >= ib) break;
            int ninj = occi * (1 + (int)bit_w<W>(e2A, jb));
            if (ninj == 1) v += g2(P, ib, ib, jb, jb);
            else {
              double buf = 2.0 * g2(P, ib, ib, jb, jb);
              buf -= g2(P, ib, jb, ib, jb);
              if (ninj == 2) v += buf; else v += 2.0 * buf;
            }
          }
        }
      }
    }
    Kd[0] = v;
    pi.v0 = v;
    return;
  }
  if (ni == 1) {
    uint64_t im[W], jm[W];
#pragma unroll
    for (int w = 0; w < W; ++w) { im[w] = im1[w] | im2[w]; jm[w] = jm1[w] | jm2[w]; }
    int ie = lowest_bit<W>(im), je = lowest_bit<W>(jm);
    pi.iex0 = ie; pi.jex0 = je;
    between_mask<W>(ie, je, pi.bm[0]);
    range_mask<W>(0, ie - 1, pi.bm[1]);
    range_mask<W>(je + 1, 64 * W - 1, pi.bm[2]);
    range_mask<W>(0, je - 1, pi.bm[3]);
    range_mask<W>(ie + 1, 64 * W - 1, pi.bm[4]);
    if (pi.jsA != pi.jsB) {
      // spin-orbit single (PsociHamiltonian.C:223-237): +-SO/2, sign flip if jex > iex
      double v = g1(P, ie, je);
      if (v != 0.0) {
        if (je > ie) v = -v;
        v = v / 2;
        pi.kind = K_SO;
        pi.v0 = v;
      } else {
        pi.kind = K_NONE;
      }
      return;
    }
    // same-symmetry single (PsociHamiltonian.C:239-258)
    double v = g1(P, ie, je) - g2(P, ie, je, ie, ie);
#pragma unroll
    for (int w = 0; w < W; ++w) {
      uint64_t o = e1A[w];
      while (o) {
        int p = 64 * w + __ffsll((long long)o) - 1;
        o &= o - 1;
        double buf = g2(P, ie, je, p, p);
        v += buf;
        bool dA = bit_w<W>(e2A, p);
        if (dA) v += buf;
        if (dA && bit_w<W>(e2B, p)) v -= g2(P, ie, p, p, je);
      }
    }
    if (v == 0.0) { pi.kind = K_NONE; return; }
    pi.kind = K_SINGLE;
    pi.v0 = v;
    int t = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      uint64_t s = pi.SA[w];
      while (s && t < PSOCI_MAX_OPEN) {
        int p = 64 * w + __ffsll((long long)s) - 1;
        s &= s - 1;
        pi.X[t++] = g2(P, ie, p, p, je);
      }
    }
    return;
  }
  if (ni == 2) {
    // ascending with multiplicity: a position in both masks appears twice
    int ex0 = -1, ex1 = -1, jy0 = -1, jy1 = -1;
    two_positions<W>(im1, im2, ex0, ex1);
    two_positions<W>(jm1, jm2, jy0, jy1);
    const int ex[2] = {ex0, ex1}, jy[2] = {jy0, jy1};
    pi.iex0 = ex0; pi.jex0 = jy0;
    between_mask<W>(ex0, jy0, pi.bm[0]);
    between_mask<W>(ex0, jy1, pi.bm[1]);
    between_mask<W>(ex1, jy0, pi.bm[2]);
    between_mask<W>(ex1, jy1, pi.bm[3]);
    between_mask<W>(ex0, ex1, pi.bm[4]);
    between_mask<W>(jy0, jy1, pi.bm[5]);
    // processDoubleExcitation (PsociHamiltonian.C:180-184)
    double v0 = g2(P, ex[0], jy[0], ex[1], jy[1]);
    double v1 = g2(P, ex[0], jy[1], ex[1], jy[0]);
    if (v0 == 0.0 && v1 == 0.0) { pi.kind = K_NONE; return; }
    pi.kind = K_DOUBLE;
    pi.v0 = v0; pi.v1 = v1;
    return;
  }
  pi.kind = K_NONE;
}

template <int W>
__device__ void pair_setup(const Params &P, int I, int J, PairInfo &pi, double *Kd) {
  if (J <= I) pair_setup_ab<W>(P, I, J, J, 0, pi, Kd);
  else pair_setup_ab<W>(P, J, I, J, 1, pi, Kd);
}

// ------------------------------------------------------------------------------------
// determinant element <det a of A | H | det b of B>
// ------------------------------------------------------------------------------------
// One determinant: alpha and beta bit-strings, phase, alpha count.
template <int W>
struct DetBits {
  uint64_t al[W], be[W];
  int ph, na;
};

template <int W>
__device__ __forceinline__ void load_det(DetBits<W> &d, const uint64_t *alpha, const uint64_t *beta,
                                         const uint8_t *phase, const uint8_t *nalpha, int64_t i) {
#pragma unroll
  for (int w = 0; w < W; ++w) { d.al[w] = alpha[i * W + w]; d.be[w] = beta[i * W + w]; }
  d.ph = phase[i];
  d.na = nalpha[i];
}

// Diagonal element of a determinant (processDiagExcitation's vnt list): Kd[0] minus the
// exchange integral of every pair of open shells (io > jo, in the reference's order) whose
// spins agree.  Out of line: it runs for the diagonal blocks only, and keeping its loops out
// of the element code keeps that code compact.
template <int W>
__device__ __noinline__ double diag_det_elem(const uint64_t *SA, const double *Kd, const uint64_t (&aa)[W]) {
  double v = Kd[0];
  int mm = 0, io = 0;
#pragma unroll
  for (int wi = 0; wi < W; ++wi) {
    uint64_t si_bits = SA[wi];
    while (si_bits) {
      const uint64_t lo_i = si_bits & (~si_bits + 1);
      si_bits ^= lo_i;
      const bool si = (aa[wi] & lo_i) != 0ull;
      // open shells below this one, ascending
      int jo = 0;
#pragma unroll
      for (int wj = 0; wj < W; ++wj) {
        uint64_t sj = SA[wj];
        while (sj && jo < io) {
          const uint64_t lo_j = sj & (~sj + 1);
          sj ^= lo_j;
          ++mm;
          if (si == ((aa[wj] & lo_j) != 0ull)) v -= Kd[mm];
          ++jo;
        }
      }
      ++io;
    }
  }
  return v;
}

// <det a of A | H | det b of B> from the loaded determinants.  sef_elem calls it from a
// single site (a loop over the determinant pairs of an SEF element), so the kernels hold
// one copy of this body: several inlined copies overflow their instruction cache.
template <int W>
__device__ __forceinline__ double det_elem(const double *eri, const PairInfo &pi, const double *Kd,
                                           const DetBits<W> &A, const DetBits<W> &B) {
  const uint64_t(&aa)[W] = A.al;
  const uint64_t(&ba)[W] = A.be;
  const uint64_t(&ab)[W] = B.al;
  const uint64_t(&bb)[W] = B.be;
  const int pha = A.ph, phb = B.ph, naa = A.na, nab = B.na;
  uint64_t ua[W], ub[W];
#pragma unroll
  for (int w = 0; w < W; ++w) { ua[w] = ab[w] & ~aa[w]; ub[w] = bb[w] & ~ba[w]; }
  int nmarka = popc_w<W>(ua);
  int nmarkb = nmarka + popc_w<W>(ub);
  const int ie = pi.iex0, je = pi.jex0;

  if (pi.kind == K_SO) {
    // socig (PsociHamiltonian.C:746-855): no spin-projection restriction
    if (nmarka > 1 || nmarkb > 1) return 0.0;
    int ncount = pha + phb;
    if (naa < nab) {
      ncount += popc_and<W>(ba, pi.bm[1]) + popc_and<W>(ab, pi.bm[2]);
      if ((pi.jsA + pi.jsB) % 2 == 0) ++ncount;
      else if (pi.jsA % 2 == 1) ++ncount;
    } else if (naa > nab) {
      ncount += popc_and<W>(aa, pi.bm[4]) + popc_and<W>(bb, pi.bm[3]);
      if ((pi.jsA + pi.jsB) % 2 != 0 && (pi.jsA % 2) == 1) ++ncount;
    } else {
      if (nmarka == 0) ++ncount;
      if (pi.jsA % 2 == 1) ++ncount;
      uint64_t sp[W];
      sel_w<W>(sp, nmarka != 0, aa, ba);
      ncount += popc_and<W>(sp, pi.bm[0]);  // empty unless |ie - je| > 1
    }
    return (ncount & 1) ? -pi.v0 : pi.v0;
  }

  // generateSEFCIG (PsociHamiltonian.C:902-1113): equal spin projection only
  if (naa != nab) return 0.0;
  if (nmarka > 2 || nmarkb > 2) return 0.0;
  if (nmarkb == 0) {
    if (pi.kind != K_DIAG) return 0.0;  // identical determinants occur only on the diagonal
    return diag_det_elem<W>(pi.SA, Kd, aa);
  }
  if (nmarkb == 1) {
    // one spin-orbital excitation within spin (nmarka == 1: alpha, else beta)
    uint64_t sp[W];
    sel_w<W>(sp, nmarka != 0, aa, ba);
    int ncount = pha + phb + popc_and<W>(sp, pi.bm[0]);  // empty unless |ie - je| > 1
    double v = pi.v0;
    // exchange with the open shells of that spin in det a, except the excited orbitals, in
    // ascending orbital order; X is indexed by the rank among A's open shells
    int t = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      uint64_t m = sp[w] & ~(aa[w] & ba[w]);
      if ((ie >> 6) == w) m &= ~(1ull << (ie & 63));
      if ((je >> 6) == w) m &= ~(1ull << (je & 63));
      uint64_t sa = pi.SA[w];
      while (sa) {
        const uint64_t low = sa & (~sa + 1);
        if (m & low) v -= pi.X[t];
        ++t;
        sa ^= low;
      }
    }
    return (ncount & 1) ? -v : v;
  }
  if (nmarka == 1) {
    // alpha single times beta single
    uint64_t xa[W], xb[W];
#pragma unroll
    for (int w = 0; w < W; ++w) { xa[w] = aa[w] & ~ab[w]; xb[w] = ba[w] & ~bb[w]; }
    if (pi.kind == K_DOUBLE) {
      // the alpha electron moves ex_ia -> jy_ja, the beta one the other two orbitals (the
      // same one when a doubly occupied orbital empties or fills); the integral
      // (beta move | alpha move) is then the table entry of v0 (ia == ja) or v1
      const int ia = bit_w<W>(xa, pi.iex0) ? 0 : 1, ja = bit_w<W>(ua, pi.jex0) ? 0 : 1;
      const int ncount = pha + phb + popc_and<W>(aa, pi.bm[2 * ia + ja]) + popc_and<W>(ba, pi.bm[3 - 2 * ia - ja]);
      const double v = (ia == ja) ? pi.v0 : pi.v1;
      return (ncount & 1) ? -v : v;
    }
    int iex2 = lowest_bit<W>(ua), jex2 = lowest_bit<W>(ub);
    int iex3 = lowest_bit<W>(xa), jex3 = lowest_bit<W>(xb);
    int ncount = pha + phb;
    if (abs(iex2 - iex3) > 1) ncount += popc_range<W>(aa, min(iex2, iex3) + 1, max(iex2, iex3) - 1);
    if (abs(jex2 - jex3) > 1) ncount += popc_range<W>(ba, min(jex2, jex3) + 1, max(jex2, jex3) - 1);
    double v = __ldg(eri + canon4(jex2, jex3, iex2, iex3));
    return (ncount & 1) ? -v : v;
  }
  // same-spin double (nmarka == 2: alpha, nmarka == 0: beta)
  if (pi.kind != K_DOUBLE) return 0.0;
  // both electrons of one spin move ex0, ex1 -> jy0, jy1 (distinct orbitals)
  uint64_t spb[W], sa[W];
  sel_w<W>(spb, nmarka == 2, ab, bb);
  sel_w<W>(sa, nmarka != 0, aa, ba);
  int ncount = pha + phb + popc_and<W>(spb, pi.bm[5]) + popc_and<W>(sa, pi.bm[4]);
  double v = pi.v0 - pi.v1;
  return (ncount & 1) ? -v : v;
}

// Where sef_elem finds the determinants of A: the global tables, or a copy of A's own
// determinants in shared memory (rows indexed from A's first determinant).
struct RowDets {
  const uint64_t *al, *be;
  const uint8_t *ph, *na;
};

// SEF element (a, b) of the reference block (A, B): ciout / transformCDCt.  conn bit
// (x << 1 | y) says whether determinant x of SEF a and determinant y of SEF b can couple;
// a determinant element that cannot is exactly zero and is not evaluated (adding the zero
// it would return leaves every partial sum unchanged).  The determinant elements are
// added in the reference's order: t = d00 + mB d01, u = d10 + mB d11, r (r t) + mA r (r u).
template <int W>
__device__ double sef_elem(const Params &PP, const PairInfo &pi, const double *Kd, int a, int b,
                           unsigned conn = 0xFu, const RowDets *rowA = nullptr) {
  if (pi.kind == K_NONE) return 0.0;
  const bool odd = PP.nelec & 1;
  const bool oa = !odd && pi.nopenA != 0, ob = !odd && pi.nopenB != 0;
  const int64_t a0 = odd ? a : (oa ? 2 * a : 0), b0 = pi.detB + (odd ? b : (ob ? 2 * b : 0));
  if (!ob) conn &= 0x5u;
  if (!oa) conn &= 0x3u;
  DetBits<W> A[2] = {}, B[2] = {};
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    if (x == 1 && !oa) break;
    if (rowA) load_det<W>(A[x], rowA->al, rowA->be, rowA->ph, rowA->na, a0 + x);
    else load_det<W>(A[x], PP.alpha, PP.beta, PP.phase, PP.nalpha, pi.detA + a0 + x);
  }
#pragma unroll
  for (int y = 0; y < 2; ++y) {
    if (y == 1 && !ob) break;
    load_det<W>(B[y], PP.alpha, PP.beta, PP.phase, PP.nalpha, b0 + y);
  }
  const double mA = (pi.jsA % 2 != PP.ksym % 2) ? -1.0 : 1.0;
  const double mB = (pi.jsB % 2 != PP.ksym % 2) ? -1.0 : 1.0;
  double t = 0.0, u = 0.0;
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
    if (!((conn >> q) & 1u)) continue;
    const int x = q >> 1, y = q & 1;
    DetBits<W> Ax, By;  // selected by value: the arrays stay in registers
#pragma unroll
    for (int w = 0; w < W; ++w) {
      Ax.al[w] = x ? A[1].al[w] : A[0].al[w];
      Ax.be[w] = x ? A[1].be[w] : A[0].be[w];
      By.al[w] = y ? B[1].al[w] : B[0].al[w];
      By.be[w] = y ? B[1].be[w] : B[0].be[w];
    }
    Ax.ph = x ? A[1].ph : A[0].ph;
    Ax.na = x ? A[1].na : A[0].na;
    By.ph = y ? B[1].ph : B[0].ph;
    By.na = y ? B[1].na : B[0].na;
    const double d = det_elem<W>(PP.eri, pi, Kd, Ax, By);
    if (x == 0) t = (y == 0) ? d : t + mB * d;
    else u = (y == 0) ? d : u + mB * d;
  }
  if (odd) return t;
  const double r = sqrt(0.5);
  const double ds0 = ob ? t * r : t;
  const double ds1 = ob ? u * r : u;
  if (oa) {
    double v = r * ds0;
    v += (mA * r) * ds1;
    return v;
  }
  return ds0;
}

// FP64 sum over the warp of v[0..7], scattered: lanes 4q..4q+3 end with the total of q
__device__ __forceinline__ double reduce_scatter8_f64(const double (&v)[8], int lane) {
  double a[4], b[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool hi = lane & 16;
    a[i] = (hi ? v[i + 4] : v[i]) + __shfl_xor_sync(0xffffffffu, hi ? v[i] : v[i + 4], 16);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const bool hi = lane & 8;
    b[i] = (hi ? a[i + 2] : a[i]) + __shfl_xor_sync(0xffffffffu, hi ? a[i] : a[i + 2], 8);
  }
  const bool hi = lane & 4;
  double c = (hi ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, hi ? b[0] : b[1], 4);
  c += __shfl_xor_sync(0xffffffffu, c, 2);
  c += __shfl_xor_sync(0xffffffffu, c, 1);
  return c;
}

// ------------------------------------------------------------------------------------
// segment kernel over full neighbour lists: PASS 0 counts kept elements per row, PASS 1
// writes them; direct mode: PASS 2 adds H X into Y (atomically: a configuration's rows
// may span several segments), PASS 3 writes the diagonal only
// ------------------------------------------------------------------------------------
template <int W, int PASS>
__global__ void __launch_bounds__(WARPS_PER_CTA * 32) k_hbuild(Params P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WarpSmem *ws = reinterpret_cast<WarpSmem *>(smem_raw) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t s = warp; s < P.nseg; s += nwarps) {
    const int I = P.seg_cfg[s];
    const int64_t k0 = P.seg_k0[s];
    const int n = P.seg_n[s];
    const int nsefI = (int)(P.sefoff[I + 1] - P.sefoff[I]);
    int myJ = -1, myn = 0;
    if (lane < n) {
      myJ = P.nbr[k0 + lane];
      pair_setup<W>(P, I, myJ, ws->pi[lane], ws->K);
      myn = ws->pi[lane].nsefJ;
    }
    // exclusive prefix of nsefJ over the segment
    int incl = myn;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    ws->itemoff[lane + 1] = incl;
    if (lane == 0) ws->itemoff[0] = 0;
    __syncwarp();
    const int T = ws->itemoff[n];
    // PASS 3: the diagonal block (J = I) is in exactly one segment of I
    if (PASS == 3 && lane < n && ws->pi[lane].kind == K_DIAG)
      for (int r = 0; r < nsefI; ++r) P.diag[P.sefoff[I] + r] = sef_elem<W>(P, ws->pi[lane], ws->K, r, r);
    for (int r = 0; r < (PASS == 3 ? 0 : nsefI); ++r) {
      double acc[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[q] = 0.0;
      int64_t base = 0;
      if (PASS == 1) base = P.rowptr[P.sefoff[I] + r] + P.seg_cnt[P.seg_rowoff[s] + r];
      int64_t cnt = 0;
      for (int q0 = 0; q0 < T; q0 += 32) {
        const int q = q0 + lane;
        bool keep = false;
        double v = 0.0;
        int k = 0, t = 0;
        if (q < T) {
          // neighbour k with itemoff[k] <= q < itemoff[k+1]
          int lo = 0, hi = n - 1;
          while (lo < hi) {
            int mid = (lo + hi + 1) >> 1;
            if (ws->itemoff[mid] <= q) lo = mid; else hi = mid - 1;
          }
          k = lo;
          t = q - ws->itemoff[k];
          const PairInfo &pi = ws->pi[k];
          // lower half of a diagonal block as the reference computes it, upper half mirrored;
          // block (J, I) transposed for J > I
          const bool diag_blk = (pi.kind == K_DIAG);
          const bool flip = diag_blk ? (t > r) : (pi.swap != 0);
          v = sef_elem<W>(P, pi, ws->K, flip ? t : r, flip ? r : t);
          keep = (fabs(v) >= PSOCI_MIN_VALUE) || (diag_blk && t == r);
        }
        if (PASS == 2 && keep) {
          const double *xr = P.dx + (int64_t)(ws->pi[k].colbase + t) * P.ldx;
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (q < P.kvec) acc[q] = fma(v, xr[q], acc[q]);
        }
        unsigned b = __ballot_sync(0xffffffffu, keep);
        if (PASS == 1 && keep) {
          int64_t pos = base + cnt + __popc(b & ((1u << lane) - 1u));
          const PairInfo &pi = ws->pi[k];
          P.col[pos] = (int32_t)(pi.colbase + t);
          P.val[pos] = v;
          if (P.val32) P.val32[pos] = (float)v;
          if (pi.kind == K_DIAG && t == r) P.diag[P.sefoff[I] + r] = v;
        }
        cnt += __popc(b);
      }
      if (PASS == 0 && lane == 0) P.seg_cnt[P.seg_rowoff[s] + r] = cnt;
      if (PASS == 2) {
        const double tot = reduce_scatter8_f64(acc, lane);
        const int q = lane >> 2;
        if ((lane & 3) == 0 && q < P.kvec && tot != 0.0) atomicAdd(P.dy + (P.sefoff[I] + r) * P.ldy + q, tot);
      }
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------------------------------
// Elements from coupling tables (blocktab.cuh), for configurations of at most TAB_MAXOPEN open
// shells.  k_pair_slots gives every pair of the neighbour lists its table (and its integrals);
// k_elems then walks each configuration's list, 32 pairs at a time, and
//   MODE 0  counts the kept elements of its rows,
//   MODE 1  writes them, columns ascending, at the rows' places,
//   MODE 2  multiplies them with X (direct mode).
// Both triangles are evaluated: an element costs so little that reading its pair twice is cheaper
// than mirroring it.  mrcisd_6e8o_v48 (2.18 million SEFs, 1.25e9 elements): pair slots, tables and
// diagonal 8.7 ms, count 6.2 ms, fill 17.0 ms (20 GB of CSR: 3 ms at the copy rate), where
// evaluating the lower triangle determinant by determinant, counting its mirror image and
// assembling the rows took 98 + 7 + 27 ms; 31,650 SEFs with up to 8 open shells: 14.6 -> 2.0 ms.
// ------------------------------------------------------------------------------------
template <int W>
__global__ void k_cfg_rec(Params P, CfgRec<W> *__restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < P.nconf; i += (int64_t)gridDim.x * blockDim.x) {
    CfgRec<W> r;
#pragma unroll
    for (int w = 0; w < W; ++w) { r.e1[w] = P.e1[i * W + w]; r.e2[w] = P.e2[i * W + w]; }
    const int js = P.jsym[i];
    r.sef = (uint32_t)P.sefoff[i];
    r.flags = (uint32_t)P.nopen[i] | ((uint32_t)(P.phase[P.detoff[i]] & 1) << 4) |
              ((uint32_t)(psoci_det_class(P.nelec & 1, js, P.ksym) & 1) << 5) | ((uint32_t)(js & 1) << 6) |
              ((uint32_t)(P.sefoff[i + 1] - P.sefoff[i]) << 16);
    r.jsym = js;
    r.pad = 0u;
    out[i] = r;
  }
}

// Rounding to FP32 on the integer pipe (round to nearest even; values outside FP32's normal
// range by the conversion instruction, which shares the narrow FP64 pipe).
__device__ __forceinline__ float f32_of(double v) {
  const uint32_t hi = (uint32_t)__double2hiint(v);
  const uint64_t a = ((uint64_t)(hi & 0x7fffffffu) << 32) | (uint32_t)__double2loint(v);
  const uint64_t r = (a + 0x0fffffffull + ((a >> 29) & 1ull)) >> 29;  // 11 exponent bits, 23 mantissa bits
  const uint64_t f = r - (896ull << 23);
  if (f - 0x00800000ull >= 0x7f000000ull) return (float)v;
  return __uint_as_float((uint32_t)f | (hi & 0x80000000u));
}
// |v| >= PSOCI_MIN_VALUE (not NaN) by its bits, word by word: masking the sign of the 64-bit
// pattern compiles to an FP64 absolute value
__device__ __forceinline__ bool kept_value(double v) {
  const uint64_t a = ((uint64_t)((uint32_t)__double2hiint(v) & 0x7fffffffu) << 32) | (uint32_t)__double2loint(v);
  constexpr uint64_t lo = 0x3e45798ee2308c3aull, inf = 0x7ff0000000000000ull;  // the bits of 1e-8
  return a - lo <= inf - lo;
}

__device__ __forceinline__ bool is_zero(double v) { return ((uint64_t)__double_as_longlong(v) << 1) == 0ull; }

// Integrals of a pair in the reference's roles, times its sign.  Singles: v0 and, for the
// X[t] that the element kernels gather themselves, ie | je << 8 | sign bit in v1.  False when
// they make the whole block zero (the reference's skips).
template <int W>
__device__ __forceinline__ bool pair_values(const Params &P, const CfgRec<W> &A, const CfgRec<W> &B,
                                            const PairShape &s, double &v0, double &v1) {
  v0 = v1 = 0.0;
  bool any = false;
  if (s.kind == K_DOUBLE) {  // processDoubleExcitation (PsociHamiltonian.C:180-184)
    v0 = g2(P, s.ex0, s.jy0, s.ex1, s.jy1);
    v1 = g2(P, s.ex0, s.jy1, s.ex1, s.jy0);
    any = !(is_zero(v0) && is_zero(v1));
  } else if (s.kind == K_SO) {  // PsociHamiltonian.C:223-237: +-SO/2, sign flip if jex > iex
    v0 = g1(P, s.ex0, s.jy0);
    any = !is_zero(v0);
    v0 = flip_sign(v0 * 0.5, s.jy0 > s.ex0 ? 0x80000000u : 0u);
  } else if (s.kind == K_SINGLE) {  // PsociHamiltonian.C:239-258
    const int ie = s.ex0, je = s.jy0;
    double v = g1(P, ie, je) - g2(P, ie, je, ie, ie);
#pragma unroll
    for (int w = 0; w < W; ++w) {
      uint64_t o = A.e1[w];
      while (o) {
        const int b = __ffsll((long long)o) - 1, p = 64 * w + b;
        o &= o - 1;
        const double buf = g2(P, ie, je, p, p);
        v += buf;
        const bool dA = (A.e2[w] >> b) & 1ull;
        if (dA) v += buf;
        if (dA && ((B.e2[w] >> b) & 1ull)) v -= g2(P, ie, p, p, je);
      }
    }
    v0 = v;
    any = !is_zero(v);
    v1 = __longlong_as_double((long long)((uint32_t)ie | ((uint32_t)je << 8) | s.sign));
  }
  v0 = flip_sign(v0, s.sign);
  if (s.kind != K_SINGLE) v1 = flip_sign(v1, s.sign);
  return any;
}

// Slot of every pair (ordered; one warp a configuration, lanes over its list), and with VALS
// its integrals, pairs whose integrals make the block zero getting TAB_NONE.  LOWER: the pairs
// J < I alone (the list's first; the slots of the others are not written).  The sum over occupied
// orbitals of a single's integral is the longest part and one pair in twenty has it, so a
// configuration's singles are set aside and summed by full warps (evaluated where they came up:
// 7.4 ms at mrcisd_6e8o_v48, now 6.5 ms, of it 0.6 ms for the kept-form bits that the count reads; bound by integer issue).
template <int W, bool VALS, bool LOWER>
__global__ void __launch_bounds__(256) k_pair_slots(Params P, const CfgRec<W> *__restrict__ cfg,
                                                    const int64_t *__restrict__ nbroff, const int32_t *__restrict__ nbr,
                                                    uint64_t *keys, uint32_t mask, int *err, uint32_t *list,
                                                    uint32_t *__restrict__ slot, double2 *__restrict__ vals) {
  __shared__ int64_t s_q[8][64];   // singles set aside: place in the lists ...
  __shared__ uint32_t s_m[8][64];  // ... ie | je << 8 | J > I << 16 | sign
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t I = warp; I < P.nconf; I += nwarps) {
    const CfgRec<W> a = cfg[I];
    const int64_t e = nbroff[I + 1];
    int ns = 0;  // singles set aside
    auto sum_singles = [&](int n) {
      __syncwarp();
      if (lane < n) {
        const int64_t q = s_q[wib][lane];
        const uint32_t m = s_m[wib][lane];
        const CfgRec<W> b = cfg[nbr[q]];
        const bool up = (m >> 16) & 1u;
        CfgRec<W> A, B;
#pragma unroll
        for (int w = 0; w < W; ++w) {
          A.e1[w] = up ? b.e1[w] : a.e1[w]; A.e2[w] = up ? b.e2[w] : a.e2[w];
          B.e2[w] = up ? a.e2[w] : b.e2[w];
        }
        const PairShape s{K_SINGLE, (int)(m & 0xffu), -1, (int)((m >> 8) & 0xffu), -1, m & TAB_SIGN};
        double v0, v1;
        if (!pair_values<W>(P, A, B, s, v0, v1)) slot[q] = TAB_NONE;
        vals[q] = make_double2(v0, v1);
      }
      __syncwarp();
      if (lane < ns - n) {  // the rest moves up (at most 32)
        const int64_t q = s_q[wib][lane + n];
        const uint32_t m = s_m[wib][lane + n];
        s_q[wib][lane] = q;
        s_m[wib][lane] = m;
      }
      ns -= n;
      __syncwarp();
    };
    for (int64_t q0 = nbroff[I]; q0 < e; q0 += 32) {
      const int64_t q = q0 + lane;
      const int J = q < e ? nbr[q] : INT_MAX;
      const bool in = LOWER ? J < (int)I : q < e;
      if (LOWER && __ballot_sync(0xffffffffu, in) == 0u) break;
      bool single = false;
      uint32_t meta = 0u;
      if (in) {
      uint32_t sl = TAB_NONE;
      double v0 = 0.0, v1 = 0.0;
      if (J == (int)I) {
        sl = TAB_DIAG;
      } else {
        const CfgRec<W> b = cfg[J];
        const bool up = J > (int)I;  // block (J, I): A = J, rows are B's SEFs
        CfgRec<W> A, B;
#pragma unroll
        for (int w = 0; w < W; ++w) {
          A.e1[w] = up ? b.e1[w] : a.e1[w]; A.e2[w] = up ? b.e2[w] : a.e2[w];
          B.e1[w] = up ? a.e1[w] : b.e1[w]; B.e2[w] = up ? a.e2[w] : b.e2[w];
        }
        A.flags = up ? b.flags : a.flags; A.jsym = up ? b.jsym : a.jsym;
        B.flags = up ? a.flags : b.flags; B.jsym = up ? a.jsym : b.jsym;
        const PairShape s = pair_shape<W>(A, B);
        bool any = s.kind != K_NONE;
        single = VALS && s.kind == K_SINGLE;
        meta = (uint32_t)s.ex0 | ((uint32_t)s.jy0 << 8) | ((uint32_t)up << 16) | s.sign;
        if (VALS && any && !single) any = pair_values<W>(P, A, B, s, v0, v1);
        if (any) {
          sl = tab_insert(keys, mask, pair_key<W>(A, B, s.kind, up), err, list);
          if (sl != TAB_NONE) sl |= s.sign;
          if (VALS && !single && sl != TAB_NONE) {
            const uint32_t oa = A.flags & 15u, ob = B.flags & 15u;
            const uint32_t fc = (P.nelec & 1) ? 0u : ((oa ? 2u : 0u) | (ob ? 1u : 0u)) << TAB_FACTORS;
            sl |= (kept_value(tab_scale(v0, fc)) ? 1u : 0u) << TAB_KEPT;
            if (s.kind == K_DOUBLE)
              sl |= ((kept_value(tab_scale(v1, fc)) ? 2u : 0u) | (kept_value(tab_scale(v0 - v1, fc)) ? 4u : 0u)) << TAB_KEPT;
          }
        }
      }
      slot[q] = sl;
      if (VALS && !single) vals[q] = make_double2(v0, v1);
      }
      if (VALS) {
        const unsigned sb = __ballot_sync(0xffffffffu, single);
        if (sb) {
          if (single) {
            const int at = ns + __popc(sb & ((1u << lane) - 1u));
            s_q[wib][at] = q;
            s_m[wib][at] = meta;
          }
          ns += __popc(sb);
          if (ns >= 32) sum_singles(32);
        }
      }
    }
    if (VALS && ns > 0) sum_singles(ns);
  }
}

// Diagonal blocks: D[(sef r) * ldd + t], the lower half as the reference computes it and its
// mirror image, and the diagonal.  One warp a configuration: the diagonal's integral sums with
// their loads spread over the lanes and added in the reference's order, then lanes over the
// elements that can differ from zero (all of them evaluated: 3.2 ms at mrcisd_6e8o_v48, now
// 2.1 ms).
constexpr int DG_WARPS = 4;
template <int W>
__global__ void __launch_bounds__(DG_WARPS * 32) k_diag_blocks(Params P, int ldd, double *__restrict__ D,
                                                               double *__restrict__ diag) {
  __shared__ PairInfo spi[DG_WARPS];
  __shared__ double sK[DG_WARPS][MAXK];
  __shared__ uint16_t list[DG_WARPS][64];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  PairInfo &pi = spi[wib];
  double *Kd = sK[wib];
  for (int64_t I = warp; I < P.nconf; I += nwarps) {
    uint64_t o1[W], o2[W], so[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      o1[w] = P.e1[I * W + w];
      o2[w] = P.e2[I * W + w];
      so[w] = o1[w] & ~o2[w];
    }
    // the p-th lowest set bit of x, or -1
    auto nth = [](const uint64_t(&x)[W], int p) {
#pragma unroll
      for (int w = 0; w < W; ++w) {
        uint64_t u = x[w];
        const int c = __popcll(u);
        if (p < c) {
          for (; p > 0; --p) u &= u - 1;
          return 64 * w + __ffsll((long long)u) - 1;
        }
        p -= c;
      }
      return -1;
    };
    const int nop = popc_w<W>(so), nocc = popc_w<W>(o1);
    // exchange of the open-shell pairs (a > b), in diag_det_elem's order
    for (int mm = lane; mm < nop * (nop - 1) / 2; mm += 32) {
      int a = 1, q = mm;
      while (q >= a) { q -= a; ++a; }
      const int oa = nth(so, a), ob = nth(so, q);
      Kd[1 + mm] = g2(P, oa, ob, ob, oa);
    }
    // processDiagExcitation (PsociHamiltonian.C:306-388): per occupied ib its own term, then
    // its pairs jb < ib ascending
    double v = 0.0;
    for (int i = 0; i < nocc; ++i) {
      const int ib = nth(o1, i), occi = 1 + (int)bit_w<W>(o2, ib);
      for (int j0 = -1; j0 < i; j0 += 32) {
        const int j = j0 + lane;
        double x = 0.0;
        if (j < 0) {
          x = occi == 1 ? g1(P, ib, ib) : 2.0 * g1(P, ib, ib) + g2(P, ib, ib, ib, ib);
        } else if (j < i) {
          const int jb = nth(o1, j), ninj = occi * (1 + (int)bit_w<W>(o2, jb));
          if (ninj == 1) x = g2(P, ib, ib, jb, jb);
          else {
            double buf = 2.0 * g2(P, ib, ib, jb, jb);
            buf -= g2(P, ib, jb, ib, jb);
            x = ninj == 2 ? buf : 2.0 * buf;
          }
        }
        const int m = min(32, i - j0);
        for (int l = 0; l < m; ++l) v += __shfl_sync(0xffffffffu, x, l);
      }
    }
    const int64_t row0 = P.sefoff[I];
    const int nsef = (int)(P.sefoff[I + 1] - row0);
    if (lane == 0) {
      Kd[0] = v;
      pi.kind = K_DIAG;
      pi.swap = 0;
      pi.detA = pi.detB = P.detoff[I];
      pi.colbase = row0;
      pi.nsefJ = nsef;
      pi.iex0 = pi.jex0 = -1;
      pi.nopenA = pi.nopenB = nop;
      pi.jsA = pi.jsB = P.jsym[I];
      pi.v0 = v;
      pi.v1 = 0.0;
#pragma unroll
      for (int w = 0; w < W; ++w) pi.SA[w] = so[w];
    }
    __syncwarp();
    // elements whose determinants couple (at most one alpha and one beta move apart, equal alpha
    // counts), gathered 32 at a time; the others are zero
    const bool open2 = !(P.nelec & 1) && nop != 0;
    const int64_t d0 = P.detoff[I];
    int n = 0;
    auto eval = [&](int m) {
      __syncwarp();
      if (lane < m) {
        const int r = list[wib][lane] >> 8, t = list[wib][lane] & 255;
        const double x = sef_elem<W>(P, pi, Kd, r, t);
        D[(row0 + r) * ldd + t] = x;
        if (t != r) D[(row0 + t) * ldd + r] = x;
        else diag[row0 + r] = x;
      }
      __syncwarp();
      if (lane < n - m) list[wib][lane] = list[wib][lane + m];
      n -= m;
      __syncwarp();
    };
    const int lg = __ffs(nsef) - 1;  // a power of two
    for (int e0 = 0; e0 < nsef << lg; e0 += 32) {
      const int e = e0 + lane, r = e >> lg, t = e & (nsef - 1);
      bool couple = false;
      if (e < nsef << lg && t <= r) {
        for (int x = 0; x <= (int)open2; ++x) {  // the first column determinant: the second pairs are its flips
          int na = 0, nb = 0, ca = 0;
          const int64_t ia = d0 + (open2 ? 2 * r + x : r), ib = d0 + (open2 ? 2 * t : t);
#pragma unroll
          for (int w = 0; w < W; ++w) {
            const uint64_t aa = P.alpha[ia * W + w], ab = P.alpha[ib * W + w];
            na += __popcll(ab & ~aa);
            ca += __popcll(aa & ~ab);
            nb += __popcll(P.beta[ib * W + w] & ~P.beta[ia * W + w]);
          }
          couple |= na == ca && na <= 1 && nb <= 1;
        }
        if (!couple) {
          D[(row0 + r) * ldd + t] = 0.0;
          D[(row0 + t) * ldd + r] = 0.0;
        }
      }
      const unsigned cb = __ballot_sync(0xffffffffu, couple);
      if (couple) list[wib][n + __popc(cb & ((1u << lane) - 1u))] = (uint16_t)((r << 8) | t);
      n += __popc(cb);
      if (n >= 32) eval(32);
    }
    if (n > 0) eval(n);
    __syncwarp();
  }
}

// Per warp, followed by X (ms doubles a pair) and, MODE 0 and 1, an int32 a row (count, write
// position from the configuration's first), MODE 2 four times eight doubles a row (its
// products).  The pairs that have elements, in order.
struct ElemWarp {
  uint2 run[PSOCI_SEG];        // runs of elements: first entry less first element, pair
  uint4 pair[PSOCI_SEG];       // info, first column, offset of the row indices from the entries
  double F[PSOCI_SEG][4];      // the pair's scaled integrals v0, v1, v0 - v1 (singles: v0, its orbitals)
  float F32[PSOCI_SEG][4];     // and in FP32
};
// in the info of ElemWarp::pair, in place of the number of entries: diagonal block, elements that are sums
// (tab_sum_value), forms above the threshold
constexpr uint32_t EL_DIAG = 1u, EL_SUMS = 2u;
constexpr int EL_KEPT = 4;

// Warps a block: their configurations differ in size by up to 256 times, and a block holds its
// shared memory and registers until its last warp ends (8 warps: 31% of the SM's warps active)
constexpr int EL_WARPS = 2;

template <int W>
struct ElemArgs {
  const CfgRec<W> *cfg;
  const uint32_t *slot;
  const double2 *vals;       // VALS: the pairs' integrals
  const uint4 *hdr;
  const uint32_t *pool;
  const double *D;           // diagonal blocks
  int ldd, ms;               // SEFs / open shells of the largest configuration
  int64_t *row_nnz;          // MODE 0
  unsigned long long *segments;
  int warp_bytes;
};

// One warp per configuration.  Per chunk of 32 pairs the lanes load a pair each (table header,
// integrals; the singles' exchange integrals spread over all lanes), then the pairs' entries are
// laid end to end and lane e % 32 takes element e.  A table lists a row's columns ascending, so
// the elements of one row come in the order in which the matrix holds them: an element's place
// is its row's write position plus the elements of that row on lower lanes.
//   Pair by pair the entries are read coalesced and a pair's kind is uniform over most warps;
// laid out row by row instead (so that the stores coalesce) the bookkeeping of the (row, pair)
// runs took 3,500 instructions a chunk and the kernel 30.5 ms at mrcisd_6e8o_v48 (MODE 1).
// MODE 1 takes four rows of all 32 pairs at a time, so that a warp's elements still fall into few
// runs of the matrix.
// GB300's FP64 pipe takes a warp instruction every 16 clocks an SM, so a double's or spin-orbit
// pair's three values, and their FP32 copies, are formed once a pair, and an element takes one
// with its sign; signs and the threshold are integer operations.
//   MODE 0 reads elements only of singles and two-term forms; a double or spin-orbit pair adds
// the row counts of the forms that pass the threshold.  VALS: integrals read from the pair list
// instead of evaluated here (the list takes 16 bytes a pair; without room for it the kernel
// gathers them itself, to the same values).  SMALL: no configuration of more than 16 SEFs.
template <int W, int MODE, bool VALS, bool SMALL>
__global__ void __launch_bounds__(EL_WARPS * 32) k_elems(Params P, ElemArgs<W> E) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ElemWarp &ws = *reinterpret_cast<ElemWarp *>(smem_raw + (size_t)(threadIdx.x >> 5) * E.warp_bytes);
  double *X = reinterpret_cast<double *>(&ws + 1);
  int *pos = reinterpret_cast<int *>(X + E.ms * PSOCI_SEG);
  double *yacc = reinterpret_cast<double *>(pos);
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u, le = lt | (1u << lane);
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t I = warp; I < P.nconf; I += nwarps) {
    const CfgRec<W> a = E.cfg[I];
    const int nsefI = (int)(a.flags >> 16) & 0x1ff, lgI = __ffs(nsefI) - 1;  // a power of two
    const int64_t row0 = a.sef, b0 = P.nbroff[I], b1 = P.nbroff[I + 1];
    const int64_t first = MODE == 1 ? P.rowptr[row0] : 0;
    if (MODE < 2)
      for (int r = lane; r < nsefI; r += 32) pos[r] = MODE == 0 ? 0 : (int)(P.rowptr[row0 + r] - first);
    else
      for (int r = lane; r < nsefI * 32; r += 32) yacc[r] = 0.0;
    int32_t *col0 = MODE == 1 ? P.col + first : nullptr;
    double *val0 = MODE == 1 ? P.val + first : nullptr;
    float *val320 = (MODE == 1 && P.val32) ? P.val32 + first : nullptr;
    // MODE 0: this lane's row counts, 16 bits a row (cnt[q]: rows q, q + 4, q + 8, q + 12), added to
    // pos before they can carry
    uint64_t cnt[4] = {0ull, 0ull, 0ull, 0ull};
    auto add_counts = [&]() {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint64_t lo = cnt[q] & 0x0000ffff0000ffffull, hi = (cnt[q] >> 16) & 0x0000ffff0000ffffull;
        cnt[q] = 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          lo += __shfl_xor_sync(FULL, lo, o);
          hi += __shfl_xor_sync(FULL, hi, o);
        }
        if (lane == 0) {
          if (q < nsefI) pos[q] += (int)(uint32_t)lo;
          if (q + 8 < nsefI) pos[q + 8] += (int)(lo >> 32);
          if (q + 4 < nsefI) pos[q + 4] += (int)(uint32_t)hi;
          if (q + 12 < nsefI) pos[q + 12] += (int)(hi >> 32);
        }
      }
      __syncwarp();
    };
    for (int64_t k0 = b0; k0 < b1; k0 += 32) {
      const int n = (int)min((int64_t)32, b1 - k0);
      __syncwarp();
      if (MODE == 0 && ((k0 - b0) & (4096 * 32 - 1)) == 4095 * 32) add_counts();
      // this lane's pair
      uint32_t sl = TAB_NONE;
      int J = 0;
      if (lane < n) {
        J = P.nbr[k0 + lane];
        sl = E.slot[k0 + lane];
      }
      bool single = false, two = false;
      int c = 0;           // its elements
      uint4 pr = make_uint4(0u, 0u, 0u, 0u);
      double v0 = 0.0, v1 = 0.0, f0 = 0.0, f1 = 0.0, f2 = 0.0;
      uint64_t sa[W], rows = 0ull;  // open shells of A; entries of each row, 4 bits a row
      uint32_t ent0 = 0u;           // first entry
      if (sl == TAB_DIAG) {
        c = nsefI * nsefI;
        pr.x = EL_DIAG;
        pr.y = (uint32_t)row0;
      } else if (sl != TAB_NONE) {
        const uint4 h = __ldg(E.hdr + 2 * (size_t)(sl & TAB_SLOT));
        single = ((h.y >> TAB_KIND) & 7u) == K_SINGLE;
        two = !single && (h.y >> (TAB_FORMS + 3)) != 0u;
        const bool counted = MODE == 0 && !single && !two && !(h.y & TAB_NOCOUNTS);  // by the table's rows alone
        bool any = true;
#pragma unroll
        for (int w = 0; w < W; ++w) sa[w] = a.e1[w] & ~a.e2[w];
        if (VALS) {
          if (!counted) {
            const double2 v = __ldg(E.vals + k0 + lane);
            v0 = v.x;
            v1 = v.y;
          }
          if (MODE != 0) pr.y = __ldg(&E.cfg[J].sef);
          if (single && J > (int)I) {
#pragma unroll
            for (int w = 0; w < W; ++w) sa[w] = __ldg(&E.cfg[J].e1[w]) & ~__ldg(&E.cfg[J].e2[w]);
          }
        } else {
          const CfgRec<W> b = E.cfg[J];
          const bool up = J > (int)I;
          CfgRec<W> A, B;
#pragma unroll
          for (int w = 0; w < W; ++w) {
            A.e1[w] = up ? b.e1[w] : a.e1[w]; A.e2[w] = up ? b.e2[w] : a.e2[w];
            B.e1[w] = up ? a.e1[w] : b.e1[w]; B.e2[w] = up ? a.e2[w] : b.e2[w];
            sa[w] = A.e1[w] & ~A.e2[w];
          }
          A.flags = up ? b.flags : a.flags; A.jsym = up ? b.jsym : a.jsym;
          B.flags = up ? a.flags : b.flags; B.jsym = up ? a.jsym : b.jsym;
          const PairShape s = pair_shape<W>(A, B);
          any = pair_values<W>(P, A, B, s, v0, v1);  // not: skipped whole, as in the list
          pr.y = b.sef;
        }
        c = any ? (int)(h.y & TAB_ENTRIES) : 0;
        ent0 = h.x;
        rows = any ? (uint64_t)h.z | ((uint64_t)h.w << 32) : 0ull;
        pr.z = 3u * h.x + 4u * (uint32_t)c;  // row indices: a byte each, after the entries
        pr.x = h.y & ((3u << TAB_FACTORS) | (7u << TAB_KIND));
        if (single) {
          pr.x |= EL_SUMS;
        } else {
          uint32_t keep = (sl >> TAB_KEPT) & 7u;
          if (!VALS || !counted) {
            f0 = tab_scale(v0, h.y);
            if ((h.y >> TAB_FORMS) & 0xffeu) {  // more than v0 in use
              f1 = tab_scale(v1, h.y);
              f2 = tab_scale(v0 - v1, h.y);
            }
            if (!VALS) keep = (kept_value(f0) ? 1u : 0u) | (kept_value(f1) ? 2u : 0u) | (kept_value(f2) ? 4u : 0u);
          }
          pr.x |= keep << EL_KEPT;
          if (two) pr.x |= EL_SUMS;
          if (counted) {
            c = 0;
            const uint4 h2 = __ldg(E.hdr + 2 * (size_t)(sl & TAB_SLOT) + 1);
            const uint64_t m = 0x000f000f000f000full;
            const uint64_t n1 = (uint64_t)h2.x | ((uint64_t)h2.y << 32), n2 = (uint64_t)h2.z | ((uint64_t)h2.w << 32);
            const uint64_t nib = ((keep & 1u) ? rows - n1 - n2 : 0ull) + ((keep & 2u) ? n1 : 0ull) + ((keep & 4u) ? n2 : 0ull);
#pragma unroll
            for (int q = 0; q < 4; ++q) cnt[q] += (nib >> (4 * q)) & m;
          }
        }
      }
      const unsigned nz = __ballot_sync(FULL, c > 0);
      const int me = __popc(nz & lt);  // this pair among those with elements
      if (c > 0) {
        ws.pair[me] = pr;
        ws.F[me][0] = single ? v0 : f0;
        ws.F[me][1] = single ? v1 : f1;
        ws.F[me][2] = f2;
        if (MODE == 1) *reinterpret_cast<float4 *>(ws.F32[me]) = make_float4((float)f0, (float)f1, (float)f2, 0.f);
        if (single) {
#pragma unroll
          for (int w = 0; w < W; ++w) X[me * E.ms + w] = __longlong_as_double((long long)sa[w]);
        } else if (two) {
          X[me * E.ms] = v0;
          X[me * E.ms + 1] = v1;
        }
      }
      // exchange integrals of the singles: lane = (single, open shell)
      unsigned sm = __ballot_sync(FULL, single && c > 0);
      __syncwarp();
      while (sm) {
        const int per = 32 / E.ms, g = lane / E.ms, t = lane - g * E.ms;
        unsigned m = sm;
        for (int q = 0; q < g && m; ++q) m &= m - 1;
        const int p = m ? __popc(nz & ((m & (~m + 1u)) - 1u)) : 0;
        double x = 0.0;
        bool have = false;
        if (g < per && m) {
          const uint64_t meta = (uint64_t)__double_as_longlong(ws.F[p][1]);
          const int ie = (int)(meta & 0xffu), je = (int)((meta >> 8) & 0xffu);
          int tt = t, o = -1;
#pragma unroll
          for (int w = 0; w < W; ++w) {
            uint64_t u = (uint64_t)__double_as_longlong(X[p * E.ms + w]);
            const int cc = __popcll(u);
            if (o < 0) {
              if (tt < cc) {
                for (; tt > 0; --tt) u &= u - 1;
                o = 64 * w + __ffsll((long long)u) - 1;
              } else {
                tt -= cc;
              }
            }
          }
          if (o >= 0) {
            have = true;
            x = g2(P, ie, o, o, je);
            x = flip_sign(x, (uint32_t)meta & TAB_SIGN);
          }
        }
        __syncwarp();
        if (have) X[p * E.ms + t] = x;
        for (int q = 0; q < per && sm; ++q) sm &= sm - 1;
        __syncwarp();
      }
      const int ng = (MODE == 1 && SMALL && nsefI > 4) ? nsefI >> 2 : 1;
      for (int g = 0; g < ng; ++g) {
      int cg = c;  // this lane's elements in the rows of the group
      if (ng > 1) {
        const uint32_t x = (uint32_t)(rows >> (16 * g)) & 0xffffu, y = (x & 0x0f0fu) + ((x >> 4) & 0x0f0fu);
        cg = (pr.x & EL_DIAG) ? 4 * nsefI : (int)((y + (y >> 8)) & 0xffu);
      }
      int T = cg;  // elements up to and with this pair's
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(FULL, T, o);
        if (lane >= o) T += u;
      }
      const int st = T - cg;
      T = __shfl_sync(FULL, T, 31);
      const unsigned nzg = __ballot_sync(FULL, cg > 0);
      if (cg > 0) ws.run[__popc(nzg & lt)] = make_uint2(ent0 - (uint32_t)st, (uint32_t)me);
      ent0 += (uint32_t)cg;
      __syncwarp();
      // an element's run (by the runs that start at or below it), pair and entry, fetched a pass ahead
      int started = 0;
      uint2 run_n = make_uint2(0u, 0u);
      uint4 q_n = make_uint4(0u, 0u, 0u, 0u);
      uint32_t ent_n = 0u;
      auto fetch = [&](int e0) {
        const unsigned bw = __reduce_or_sync(FULL, (cg > 0 && (unsigned)(st - e0) < 32u) ? 1u << ((st - e0) & 31) : 0u);
        if (e0 + lane < T) {
          run_n = ws.run[started + __popc(bw & le) - 1];
          q_n = ws.pair[run_n.y];
          if (!(q_n.x & EL_DIAG)) ent_n = __ldg(E.pool + (run_n.x + (uint32_t)(e0 + lane)));
        }
        started += __popc(bw);
      };
      if (MODE != 0 && T > 0) fetch(0);
      for (int e0 = 0; e0 < T; e0 += 32) {
        const int e = e0 + lane;
        if (MODE == 0) fetch(e0);  // few passes: not worth the registers
        const uint2 run = run_n;
        const uint4 q = q_n;
        const uint32_t ent = ent_n;
        if (MODE != 0 && e0 + 32 < T) fetch(e0 + 32);
        bool keep = false;
        double v = 0.0;
        float v32 = 0.f;
        int r = 0;
        uint32_t col = 0u;
        if (e < T) {
          const int p = (int)run.y;
          const uint32_t at = run.x + (uint32_t)e;
          if (q.x & EL_DIAG) {
            const int b = (int)at, t = b & (nsefI - 1);
            r = b >> lgI;
            v = __ldg(E.D + (row0 + r) * E.ldd + t);
            v32 = f32_of(v);
            keep = t == r || kept_value(v);
            col = q.y + (uint32_t)t;
          } else {
            const int f = (int)(ent >> 8) & 15;
            col = q.y + (ent & 0xffu);
            r = (int)(ent >> 12) & 0xff;
            if ((q.x & EL_SUMS) && (f > 2 || ((q.x >> TAB_KIND) & 7u) == K_SINGLE)) {
              v = tab_sum_value(ent, q.x, ws.F[p][0], X + p * E.ms);
              v32 = f32_of(v);
              keep = kept_value(v);
              if (((q.x >> TAB_KIND) & 7u) == K_SINGLE)
                r = __ldg(reinterpret_cast<const uint8_t *>(E.pool) + (size_t)(q.z + at));
            } else {
              v = flip_sign(ws.F[p][f], ent & 0x80000000u);
              if (MODE == 1) v32 = __int_as_float(__float_as_int(ws.F32[p][f]) ^ (int)(ent & 0x80000000u));
              keep = (q.x >> (EL_KEPT + f)) & 1u;
            }
          }
        }
        if (MODE < 2) {
          unsigned same = __ballot_sync(FULL, keep);  // the kept elements of this one's row
#pragma unroll
          for (int b = 0; b < (SMALL ? (MODE == 1 ? 2 : 4) : 8); ++b) {
            const unsigned B = __ballot_sync(FULL, (r >> b) & 1);
            same &= ((r >> b) & 1) ? B : ~B;
          }
          int at = 0;
          if (keep) at = pos[r] + __popc(same & lt);
          if (MODE == 1 && keep) {
            col0[(uint32_t)at] = (int32_t)col;
            val0[(uint32_t)at] = v;
            if (val320) val320[(uint32_t)at] = v32;
          }
          __syncwarp();
          if (keep && (same & ~le) == 0u) pos[r] = at + 1;
          __syncwarp();
        } else {
          // lanes = (element slot, vector); a slot has its own sums of each row
          const int s4 = lane >> 3, q = lane & 7;
          if (!keep) col = 0xffffffffu;
          const int m = min(32, T - e0);
          double *ya = yacc + (s4 * nsefI) * 8 + q;
          for (int x0 = 0; x0 < m; x0 += 16) {
            double vv[4], xx[4];
            int rr[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int l = x0 + 4 * u + s4;
              vv[u] = __shfl_sync(FULL, v, l);
              rr[u] = __shfl_sync(FULL, r, l);
              const uint32_t cc = __shfl_sync(FULL, col, l);
              const bool ok = cc != 0xffffffffu && q < P.kvec;
              if (!ok) vv[u] = 0.0;
              xx[u] = ok ? __ldg(P.dx + (int64_t)cc * P.ldx + q) : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              double *y = ya + rr[u] * 8;
              *y = fma(vv[u], xx[u], *y);
            }
          }
        }
      }
      __syncwarp();
      }
    }
    __syncwarp();
    if (MODE == 0) {
      add_counts();
      for (int r = lane; r < nsefI; r += 32) E.row_nnz[row0 + r] = pos[r];
      if (lane == 0) atomicAdd(E.segments, (unsigned long long)((b1 - b0 + 31) / 32));
    }
    if (MODE == 2)
      for (int r = lane; r < nsefI * 8; r += 32) {
        double y[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) y[u] = yacc[u * nsefI * 8 + r];
        if ((r & 7) < P.kvec) P.dy[(row0 + (r >> 3)) * P.ldy + (r & 7)] = (y[0] + y[1]) + (y[2] + y[3]);
      }
    __syncwarp();
  }
}

// generateSOCIblocks for an explicit list of (A, B) pairs: the full nsef_A x nsef_B block,
// row-major, at out + outoff[p] (reference roles, no transposition or mirroring)
template <int W>
__global__ void __launch_bounds__(WARPS_PER_CTA * 32) k_blocks(Params P, int npairs, const int32_t *pa,
                                                               const int32_t *pb, const int64_t *outoff,
                                                               double *out) {
  __shared__ PairInfo spi[WARPS_PER_CTA];
  __shared__ double sK[WARPS_PER_CTA][MAXK];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t q = warp; q < npairs; q += nwarps) {
    const int A = pa[q], B = pb[q];
    if (lane == 0) pair_setup_ab<W>(P, A, B, B, 0, spi[wib], sK[wib]);
    __syncwarp();
    const int na = (int)(P.sefoff[A + 1] - P.sefoff[A]), nb = (int)(P.sefoff[B + 1] - P.sefoff[B]);
    for (int e = lane; e < na * nb; e += 32) {
      int a = e / nb, b = e - a * nb;
      out[outoff[q] + e] = sef_elem<W>(P, spi[wib], sK[wib], a, b);
    }
    __syncwarp();
  }
}

template <int W>
psoci_status run_blocks(psoci_ctx *c, int npairs, const int32_t *hA, const int32_t *hB, double *hout) {
  std::vector<int64_t> off(npairs + 1, 0);
  for (int q = 0; q < npairs; ++q) {
    if (hA[q] < 0 || hA[q] >= c->nconf || hB[q] < 0 || hB[q] >= c->nconf)
      return psoci_fail(c, PSOCI_ERR_INVALID_ARG, "blocks: configuration index out of range");
    int64_t na = c->h_sefoff[hA[q] + 1] - c->h_sefoff[hA[q]], nb = c->h_sefoff[hB[q] + 1] - c->h_sefoff[hB[q]];
    off[q + 1] = off[q] + na * nb;
  }
  Params P = {};
  P.nconf = c->nconf; P.nbf = c->nbf; P.nelec = c->nelec; P.ksym = c->ksym;
  P.e1 = c->d_e1; P.e2 = c->d_e2; P.jsym = c->d_jsym; P.nopen = c->d_nopen;
  P.sefoff = c->d_sefoff; P.detoff = c->d_detoff;
  P.alpha = c->d_alpha; P.beta = c->d_beta; P.phase = c->d_phase; P.nalpha = c->d_nalpha;
  P.one = c->d_one; P.eri = c->d_eri;
  int32_t *dA = nullptr, *dB = nullptr;
  int64_t *doff = nullptr;
  double *dout = nullptr;
  psoci_status s;
  if ((s = psoci_alloc(c, &dA, npairs)) || (s = psoci_alloc(c, &dB, npairs)) || (s = psoci_alloc(c, &doff, npairs + 1)) ||
      (s = psoci_alloc(c, &dout, off[npairs]))) {
    psoci_free(dA); psoci_free(dB); psoci_free(doff); psoci_free(dout);
    return s;
  }
  cudaStream_t st = c->stream;
  cudaMemcpyAsync(dA, hA, sizeof(int32_t) * npairs, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(dB, hB, sizeof(int32_t) * npairs, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(doff, off.data(), sizeof(int64_t) * (npairs + 1), cudaMemcpyHostToDevice, st);
  int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((npairs + WARPS_PER_CTA - 1) / WARPS_PER_CTA, 152 * 16));
  psoci_note_launch();
  k_blocks<W><<<blocks, WARPS_PER_CTA * 32, 0, st>>>(P, npairs, dA, dB, doff, dout);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(hout, dout, sizeof(double) * off[npairs], cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  psoci_free(dA); psoci_free(dB); psoci_free(doff); psoci_free(dout);
  if (e != cudaSuccess) return psoci_cuda_fail(c, e, "blocks");
  return PSOCI_OK;
}

// Neighbour lists of every configuration: the configurations within two excitations (sorted),
// less the pairs whose block the integral tables prune_one / prune_eri make zero (the build
// passes the Hamiltonian's own tables; a table of ones keeps every pair).  Lookup screen for
// MRCI-type spaces, all-pairs test otherwise.  d_nbroff [nconf+1] and d_nbr [npairs] are
// allocated here and owned by the caller.
template <int W>
psoci_status screen_pairs(psoci_ctx *c, const Params &P0, const double *prune_one, const double *prune_eri,
                          int64_t *&d_nbroff, int32_t *&d_nbr, int64_t &ncand, int64_t &npairs, int &nsplit) {
  cudaStream_t st = c->stream;
  const int n = c->nconf;
  Params P = P0;
  P.one = prune_one;
  P.eri = prune_eri;
  psoci_status s;
  int64_t *d_cnt = nullptr, *d_soff = nullptr, *d_tot = nullptr, *d_candoff = nullptr;
  int32_t *d_cand = nullptr;
  int64_t *d_gcnt = nullptr, *d_goff = nullptr;
  uint32_t *d_glist = nullptr;
  unsigned long long *d_counter = nullptr;
  int32_t *d_jslab = nullptr;
  int64_t *d_jstart = nullptr;
  int2 *d_tpairs = nullptr;
  uint32_t *d_dkept = nullptr;
  ncand = npairs = 0;
  nsplit = 0;
  auto cleanup = [&]() {
    psoci_free(d_cnt); psoci_free(d_soff); psoci_free(d_tot); psoci_free(d_candoff); psoci_free(d_cand);
    psoci_free(d_gcnt); psoci_free(d_goff); psoci_free(d_glist); psoci_free(d_counter); psoci_free(d_jslab);
    psoci_free(d_jstart); psoci_free(d_tpairs); psoci_free(d_dkept);
  };
  auto fail = [&]() {
    cleanup();
    psoci_free(d_nbroff);
    psoci_free(d_nbr);
  };
#define TRY(x)                 \
  do {                         \
    s = (x);                   \
    if (s != PSOCI_OK) {       \
      fail();                  \
      return s;                \
    }                          \
  } while (0)
#define TRYC(x)                                  \
  do {                                          \
    cudaError_t _e = (x);                       \
    if (_e != cudaSuccess) {                    \
      s = psoci_cuda_fail(c, _e, #x);           \
      fail();                                   \
      return s;                                 \
    }                                           \
  } while (0)
  if (c->join_ok) {
    // by lookup, with the integral pruning fused
    JoinTabs J = {c->join_s, c->join_G, c->join_L, c->d_jgid, c->d_jlid, c->d_jT, c->d_jlnoff, c->d_jln,
                  c->d_jhdec, c->d_jlokey, nullptr, nullptr, nullptr, 0};
    // hi-pattern lists (depend on the integrals, so built here)
    const int G = c->join_G;
    TRY(psoci_alloc(c, &d_gcnt, G + 1));
    TRY(psoci_alloc(c, &d_goff, G + 1));
    const int gblocks = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)G * 32 + 255) / 256, 152 * 32));
    psoci_note_launch();
    k_group_lists<W, 0><<<gblocks, 256, 0, st>>>(J, prune_eri, d_gcnt, nullptr);
    TRYC(cudaGetLastError());
    int64_t nglist = 0;
    TRY(psoci_scan_i64(c, d_gcnt, d_goff, G, &nglist));
    TRY(psoci_alloc(c, &d_glist, nglist));
    J.goff = d_goff;
    psoci_note_launch();
    k_group_lists<W, 1><<<gblocks, 256, 0, st>>>(J, prune_eri, nullptr, d_glist);
    TRYC(cudaGetLastError());
    J.glist = d_glist;
    {
      // pruning bits of all double excitations (depend on the integrals)
      const int64_t nt = (int64_t)c->nbf * (c->nbf + 1) / 2;
      std::vector<int2> pairs((size_t)nt);
      for (int a = 0; a < c->nbf; ++a)
        for (int b = 0; b <= a; ++b) pairs[(size_t)a * (a + 1) / 2 + b] = make_int2(b, a);  // (low, high)
      TRY(psoci_alloc(c, &d_tpairs, nt));
      TRY(psoci_alloc(c, &d_dkept, (nt * nt + 31) / 32));
      TRYC(cudaMemcpyAsync(d_tpairs, pairs.data(), sizeof(int2) * nt, cudaMemcpyHostToDevice, st));
      psoci_note_launch();
      k_double_kept<<<152 * 8, 256, 0, st>>>(nt, d_tpairs, prune_eri, d_dkept);
      TRYC(cudaGetLastError());
      TRYC(cudaStreamSynchronize(st));  // pairs is a host buffer
      J.dkept = d_dkept;
      J.nt = nt;
    }
    TRY(psoci_alloc(c, &d_cnt, n + 1));
    TRY(psoci_alloc(c, &d_tot, n + 1));
    TRY(psoci_alloc(c, &d_candoff, n + 1));
    TRY(psoci_alloc(c, &d_nbroff, n + 1));
    const int jblocks = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)n * 32 + 255) / 256, 152 * 32));
    // single pass into a slab sized from the last build of this space (or 1024 neighbours
    // a configuration plus the warps' chunk tails), then a compaction copy; the count and
    // write passes remain for a slab that turns out too small
    JoinSlab S = {};
    bool single = false;
    {
      size_t freeb = 0;
      TRYC(psoci_mem_free(c, &freeb));
      const int64_t tails = (int64_t)jblocks * 8 * 2 * JOIN_CHUNK;
      int64_t cap = std::max<int64_t>(c->join_hint + c->join_hint / 8, 1024 * (int64_t)n) + tails;
      cap = std::min<int64_t>(cap, (int64_t)(freeb * 0.4) / 4);
      if (psoci_alloc(c, &d_jslab, cap) == PSOCI_OK && psoci_alloc(c, &d_jstart, n + 1) == PSOCI_OK &&
          psoci_alloc(c, &d_counter, 1) == PSOCI_OK) {
        TRYC(cudaMemsetAsync(d_counter, 0, sizeof(unsigned long long), st));
        S = {d_jslab, d_counter, cap, d_jstart};
        psoci_note_launch();
        k_join<W, 2><<<jblocks, 256, 0, st>>>(P, J, d_cnt, d_tot, nullptr, S);
        TRYC(cudaGetLastError());
        unsigned long long used = 0;
        TRYC(cudaMemcpyAsync(&used, d_counter, sizeof(used), cudaMemcpyDeviceToHost, st));
        TRYC(cudaStreamSynchronize(st));
        if ((int64_t)used <= cap) {
          TRY(psoci_scan_i64(c, d_tot, d_candoff, n, &ncand));
          TRY(psoci_scan_i64(c, d_cnt, d_nbroff, n, &npairs));
          TRY(psoci_alloc(c, &d_nbr, npairs));
          psoci_note_launch();
          k_join_compact<<<jblocks, 256, 0, st>>>(n, d_jslab, d_jstart, d_nbroff, d_nbr);
          TRYC(cudaGetLastError());
          single = true;
        }
        c->join_hint = (int64_t)used;
      } else {
        cudaGetLastError();  // no room for the slab: the two passes below
      }
      TRYC(cudaStreamSynchronize(st));
      psoci_free(d_jslab);
      psoci_free(d_jstart);
      psoci_free(d_counter);
    }
    if (!single) {
      psoci_note_launch();
      k_join<W, 0><<<jblocks, 256, 0, st>>>(P, J, d_cnt, d_tot, nullptr, S);
      TRYC(cudaGetLastError());
      TRY(psoci_scan_i64(c, d_tot, d_candoff, n, &ncand));
      TRY(psoci_scan_i64(c, d_cnt, d_nbroff, n, &npairs));
      TRY(psoci_alloc(c, &d_nbr, npairs));
      P.nbroff = d_nbroff; P.nbr = d_nbr;
      psoci_note_launch();
      k_join<W, 1><<<jblocks, 256, 0, st>>>(P, J, nullptr, nullptr, d_nbroff, S);
      TRYC(cudaGetLastError());
    }
    P.nbroff = d_nbroff; P.nbr = d_nbr;
  } else {
  const int scr_rows = (n + SCR_THREADS * SCR_ROWS - 1) / (SCR_THREADS * SCR_ROWS);
  nsplit = (int)std::max<int64_t>(1, std::min<int64_t>(64, (152 * 8 + scr_rows - 1) / scr_rows));
  int64_t chunk = ((int64_t)n + nsplit - 1) / nsplit;
  chunk = std::max<int64_t>(chunk, SCR_TILE);
  nsplit = (int)((n + chunk - 1) / chunk);
  TRY(psoci_alloc(c, &d_cnt, (size_t)nsplit * n + 1));
  TRY(psoci_alloc(c, &d_soff, (size_t)nsplit * n + 1));
  TRY(psoci_alloc(c, &d_tot, n + 1));
  TRY(psoci_alloc(c, &d_candoff, n + 1));
  TRY(psoci_alloc(c, &d_nbroff, n + 1));
  dim3 scr_grid(scr_rows, nsplit);
  psoci_note_launch();
  k_screen<W, 0><<<scr_grid, SCR_THREADS, 0, st>>>(P, d_cnt, nullptr, chunk, nullptr, nullptr);
  TRYC(cudaGetLastError());
  psoci_note_launch();
  k_screen_offsets<<<(n + 255) / 256, 256, 0, st>>>(n, nsplit, d_cnt, d_soff, d_tot);
  TRYC(cudaGetLastError());
  TRY(psoci_scan_i64(c, d_tot, d_candoff, n, &ncand));
  TRY(psoci_alloc(c, &d_cand, ncand));
  psoci_note_launch();
  k_screen<W, 1><<<scr_grid, SCR_THREADS, 0, st>>>(P, nullptr, d_soff, chunk, d_candoff, d_cand);
  TRYC(cudaGetLastError());
  const int prune_blocks = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)n * 32 + 255) / 256, 152 * 32));
  psoci_note_launch();
  k_prune<W, 0><<<prune_blocks, 256, 0, st>>>(P, d_candoff, d_cand, d_tot);
  TRYC(cudaGetLastError());
  TRY(psoci_scan_i64(c, d_tot, d_nbroff, n, &npairs));
  TRY(psoci_alloc(c, &d_nbr, npairs));
  P.nbroff = d_nbroff; P.nbr = d_nbr;
  psoci_note_launch();
  k_prune<W, 1><<<prune_blocks, 256, 0, st>>>(P, d_candoff, d_cand, nullptr);
  TRYC(cudaGetLastError());
  psoci_free(d_cand);
  }
  cleanup();
  return PSOCI_OK;
#undef TRY
#undef TRYC
}

// A coupling table set and what its kernels read beside it (freed by free()).
template <int W>
struct TabSet {
  BlockTab t;
  CfgRec<W> *cfg = nullptr;
  uint32_t *slot = nullptr;   // [npairs]
  double2 *vals = nullptr;    // [npairs] or null
  double *D = nullptr;        // diagonal blocks, ldd columns
  int ldd = 0;
  void free() {
    psoci_free(t.keys); psoci_free(t.list); psoci_free(t.hdr); psoci_free(t.pool); psoci_free(t.counter);
    psoci_free(cfg); psoci_free(slot); psoci_free(vals); psoci_free(D);
  }
};

// Whether a space goes by coupling tables: every configuration within TAB_MAXOPEN open shells
// and room for the diagonal blocks (N rows of the largest configuration's SEFs).
bool tab_usable(psoci_ctx *c, bool want_diag) {
  if (c->max_ndet > TAB_MAXDET) return false;
  if (!want_diag) return true;
  size_t freeb = 0;
  if (psoci_mem_free(c, &freeb) != cudaSuccess) return false;
  return (double)c->nsef_total * c->max_nsef * 8.0 <= 0.25 * ((double)freeb + (double)c->pool_bytes);
}

int max_open_of(const psoci_ctx *c) {
  int no = 1;
  while (no < PSOCI_MAX_OPEN && (1 << (no - 1)) < c->max_ndet) ++no;
  return no;
}

// Tables of the pairs whose slots `slots_of(S)` writes (a launch on the stream): with own S.slot and
// with vals S.vals for npairs pairs.  grad: with the tables' programs.  ok = false: the patterns do
// not fit the tables and nothing is left allocated; the generic kernels take the space.
template <int W, class F>
psoci_status tab_prepare(psoci_ctx *c, const Params &P, int64_t npairs, bool own, bool vals, bool grad, TabSet<W> &S,
                         bool &ok, F &&slots_of) {
  int64_t &hint = c->tab_words_hint[!grad ? 0 : own ? 1 : 2];
  cudaStream_t st = c->stream;
  const int n = c->nconf;
  psoci_status s = PSOCI_OK;
  ok = false;
  if ((s = psoci_alloc(c, &S.cfg, n)) || (own && (s = psoci_alloc(c, &S.slot, npairs))) ||
      (vals && (s = psoci_alloc(c, &S.vals, npairs))) || (s = psoci_alloc(c, &S.t.counter, 2))) {
    S.free();
    return s;
  }
  S.t.err = reinterpret_cast<int *>(S.t.counter + 1);
  cudaError_t e = cudaSuccess;
  psoci_note_launch();
  k_cfg_rec<W><<<(int)std::min<int64_t>((n + 255) / 256, 152 * 16), 256, 0, st>>>(P, S.cfg);
  // Key slots and pool words that hold the spaces measured, full CI of 2 to 8 electrons and reference
  // spaces with singles and doubles: 0.56 patterns a pair at 32 pairs, 0.12 at 10^4, 5 * 10^4 at
  // most; the density 10 to 800.  Words a pair: up to 1.5 with 16 SEFs; tables of more than 6 open shells take
  // hundreds to thousands, and few configurations of them hardly share any; the density 35,000 words
  // with 16 SEFs, 180,000 with 64.  Few pairs take little: an allocation of a megabyte or more costs 30 to
  // 70 us, and the first density of 1,001 SEFs took 490 us with 2^14 slots and 2^20 words.  A full
  // table grows, and a pool that was too small, whose keys and slots stay.
  const bool den = grad && !own;
  const int64_t most = den ? 1 << 12 : 1 << 18, wide = c->max_nsef <= 16 ? 2 : 32 * c->max_nsef;
  int64_t slots = 1 << 11;
  while (slots < npairs / 4 && slots < most) slots <<= 1;
  int64_t cap = den ? std::max(1 << 14, c->max_nsef << 12)
                    : std::min<int64_t>(std::max<int64_t>(1 << 12, wide * npairs), 1 << 20);
  cap = std::max<int64_t>(cap, hint + hint / 8);
  bool keyed = false;
  for (int attempt = 0; attempt < 6 && e == cudaSuccess; ++attempt) {
    if ((!keyed && ((s = psoci_alloc(c, &S.t.keys, slots)) || (s = psoci_alloc(c, &S.t.list, slots)) ||
                    (s = psoci_alloc(c, &S.t.hdr, 2 * slots)))) ||
        (s = psoci_alloc(c, &S.t.pool, cap))) {
      S.free();
      return s;
    }
    S.t.slots = slots;
    S.t.cap = cap;
    e = cudaMemsetAsync(S.t.counter, 0, (keyed ? 1 : 2) * sizeof(unsigned long long), st);
    if (e == cudaSuccess && !keyed) e = cudaMemsetAsync(S.t.keys, 0, sizeof(uint64_t) * slots, st);
    if (e != cudaSuccess) break;
    if (!keyed) {
      psoci_note_launch();
      slots_of(S);
    }
    const TabBuildArgs B = {S.t.keys, S.t.list, c->d_tmpl, c->d_tmpl_off, c->nelec, c->ksym & 1,
                            S.t.hdr, S.t.pool, S.t.counter, cap, S.t.err};
    psoci_note_launch();
    k_tab_build<<<(unsigned)std::min<int64_t>(slots / TABB_WARPS, 152 * 16), TABB_WARPS * 32, 0, st>>>(B);
    if (grad) {
      psoci_note_launch();
      k_tab_program<<<(unsigned)std::min<int64_t>(slots / 4, 152 * 16), 128, 0, st>>>(
          S.t.list, S.t.err, den ? 1 : TAB_LISTS, S.t.hdr, S.t.pool, S.t.counter, cap);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) break;
    unsigned long long back[2] = {0, 0};  // words used; error bits
    e = cudaMemcpyAsync(back, S.t.counter, sizeof(back), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) break;
    const int err = (int)(uint32_t)back[1];
    if (err & 2) break;  // a pattern outside the tables' form
    keyed = !(err & 1);
    if (keyed) hint = (int64_t)back[0];
    if (!(err & 1) && (int64_t)back[0] <= cap) {
      ok = true;
      break;
    }
    if (err & 1) slots <<= 2;
    cap = std::max(cap, (int64_t)back[0] + (int64_t)back[0] / 8);
    if (slots > ((int64_t)1 << 24) || cap > ((int64_t)1 << 30)) break;
  }
  if (e != cudaSuccess) {
    S.free();
    return psoci_cuda_fail(c, e, "coupling tables");
  }
  if (!ok) S.free();
  return PSOCI_OK;
}

// The same for the pairs of neighbour lists (grad: the lower pairs alone).
template <int W>
psoci_status tab_prepare_lists(psoci_ctx *c, const Params &P, const int64_t *nbroff, const int32_t *nbr, int64_t npairs,
                               bool vals, bool grad, TabSet<W> &S, bool &ok) {
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)c->nconf * 32 + 255) / 256, 1 << 20));
  auto k = grad ? k_pair_slots<W, false, true> : vals ? k_pair_slots<W, true, false> : k_pair_slots<W, false, false>;
  return tab_prepare<W>(c, P, npairs, true, vals, grad, S, ok, [&](TabSet<W> &T) {
    k<<<blocks, 256, 0, c->stream>>>(P, T.cfg, nbroff, nbr, T.t.keys, (uint32_t)(T.t.slots - 1), T.t.err, T.t.list, T.slot,
                                     T.vals);
  });
}

// The diagonal blocks and the diagonal of H.
template <int W>
psoci_status tab_diagonal(psoci_ctx *c, const Params &P, TabSet<W> &S, double *diag) {
  psoci_status s;
  S.ldd = c->max_nsef;
  if ((s = psoci_alloc(c, &S.D, (size_t)c->nsef_total * S.ldd))) return s;
  psoci_note_launch();
  k_diag_blocks<W><<<(unsigned)std::min<int64_t>((c->nconf + DG_WARPS - 1) / DG_WARPS, 1 << 20), DG_WARPS * 32, 0,
                     c->stream>>>(P, S.ldd, S.D, diag);
  PSOCI_CUDA(c, cudaGetLastError());
  return PSOCI_OK;
}

// One launch of k_elems: EL_WARPS warps a block, one where two do not fit.
template <int W, int MODE, bool VALS, bool SMALL>
psoci_status elems_launch_as(psoci_ctx *c, const Params &P, ElemArgs<W> &E) {
  const size_t per = (sizeof(ElemWarp) + (size_t)E.ms * PSOCI_SEG * 8 + (size_t)E.ldd * (MODE < 2 ? 4 : 256) + 15) & ~(size_t)15;
  E.warp_bytes = (int)per;
  const int warps = per * EL_WARPS <= (size_t)200 * 1024 ? EL_WARPS : 1;
  const size_t smem = per * warps;
  auto k = k_elems<W, MODE, VALS, SMALL>;
  PSOCI_CUDA(c, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  PSOCI_CUDA(c, cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
  psoci_note_launch();
  k<<<(unsigned)std::min<int64_t>((c->nconf + warps - 1) / warps, 1 << 20), warps * 32, smem, c->stream>>>(P, E);
  PSOCI_CUDA(c, cudaGetLastError());
  return PSOCI_OK;
}
template <int W, int MODE, bool VALS>
psoci_status elems_launch(psoci_ctx *c, const Params &P, ElemArgs<W> &E) {
  return E.ldd <= 16 ? elems_launch_as<W, MODE, VALS, true>(c, P, E) : elems_launch_as<W, MODE, VALS, false>(c, P, E);
}

template <int W>
ElemArgs<W> elem_args(const psoci_ctx *c, const TabSet<W> &S) {
  ElemArgs<W> E = {};
  E.cfg = S.cfg; E.slot = S.slot; E.vals = S.vals; E.hdr = S.t.hdr; E.pool = S.t.pool; E.D = S.D;
  E.ldd = S.ldd;
  E.ms = std::max(2, max_open_of(c));  // X also holds a two-word mask, or two integrals
  return E;
}

// What a direct-mode build keeps of its tables (psoci_ctx::dir_tabs).
struct DirTabs {
  TabSet<1> s1;
  TabSet<2> s2;
};
template <int W>
TabSet<W> &dir_set(DirTabs *d) {
  if constexpr (W == 1) return d->s1;
  else return d->s2;
}

// Kernels of a build: by coupling tables with the pairs' integrals listed or evaluated in the element
// launches, or the generic ones.  `form` comes in as the first that may be taken and leaves as the
// one that was; each needs less memory than the one before.
enum { FORM_LISTED, FORM_UNLISTED, FORM_GENERIC };

template <int W>
psoci_status run_build(psoci_ctx *c, psoci_hmode mode, int &form, int64_t *nnz_out) {
  const int first = form;
  form = FORM_GENERIC;
  cudaStream_t st = c->stream;
  const int n = c->nconf;
  Params P = {};
  P.nconf = n; P.nbf = c->nbf; P.nelec = c->nelec; P.ksym = c->ksym;
  P.e1 = c->d_e1; P.e2 = c->d_e2; P.jsym = c->d_jsym; P.nopen = c->d_nopen;
  P.sefoff = c->d_sefoff; P.detoff = c->d_detoff;
  P.alpha = c->d_alpha; P.beta = c->d_beta; P.phase = c->d_phase; P.nalpha = c->d_nalpha;
  P.one = c->d_one; P.eri = c->d_eri;

  psoci_status s;
  int64_t *d_nbroff = nullptr, *d_nseg = nullptr, *d_nrow = nullptr, *d_segoff = nullptr, *d_rowslot = nullptr,
          *d_segk0 = nullptr, *d_segrow = nullptr, *d_segcnt = nullptr, *d_rownnz = nullptr;
  int32_t *d_nbr = nullptr, *d_segcfg = nullptr, *d_segn = nullptr;
  TabSet<W> T;
  cudaEvent_t ev[6] = {};
  auto cleanup = [&]() {
    for (auto &e : ev)
      if (e) cudaEventDestroy(e);
    T.free();
    psoci_free(d_nbroff); psoci_free(d_nseg); psoci_free(d_nrow); psoci_free(d_segoff);
    psoci_free(d_rowslot); psoci_free(d_segk0); psoci_free(d_segrow); psoci_free(d_segcnt); psoci_free(d_rownnz);
    psoci_free(d_nbr); psoci_free(d_segcfg); psoci_free(d_segn);
  };
#define TRY(x)                 \
  do {                         \
    s = (x);                   \
    if (s != PSOCI_OK) {       \
      cleanup();               \
      return s;                \
    }                          \
  } while (0)
#define TRYC(x)                                  \
  do {                                          \
    cudaError_t _e = (x);                       \
    if (_e != cudaSuccess) {                    \
      s = psoci_cuda_fail(c, _e, #x);           \
      cleanup();                                \
      return s;                                 \
    }                                           \
  } while (0)

  auto tnow = [&]() {
    if (c->verbose) cudaStreamSynchronize(st);
    return std::chrono::steady_clock::now();
  };
  for (auto &e : ev) TRYC(cudaEventCreate(&e));
  TRYC(cudaEventRecord(ev[0], st));
  auto t_a = tnow();
  // 1. screen
  int64_t ncand = 0, npairs = 0;
  int nsplit = 0;
  TRY(screen_pairs<W>(c, P, c->d_one, c->d_eri, d_nbroff, d_nbr, ncand, npairs, nsplit));
  P.nbroff = d_nbroff; P.nbr = d_nbr;
  c->ncand = ncand;
  c->npairs = npairs;
  TRYC(cudaEventRecord(ev[1], st));
  auto t_b = tnow();

  // coupling tables for configurations of at most TAB_MAXOPEN open shells; the generic kernels
  // for others, and for patterns the tables do not hold
  const bool direct = (mode == PSOCI_HMODE_DIRECT);
  const int64_t N = c->nsef_total;
  bool fast = first < FORM_GENERIC && tab_usable(c, true), vals = false;
  if (fast) {
    // the pairs' integrals in a list (16 bytes a pair) when it takes at most a quarter of the
    // memory there is, evaluated in each element launch otherwise
    size_t freeb = 0;
    TRYC(psoci_mem_free(c, &freeb));
    vals = first == FORM_LISTED && (double)npairs * 16.0 <= 0.25 * ((double)freeb + (double)c->pool_bytes);
    form = vals ? FORM_LISTED : FORM_UNLISTED;
    TRYC(cudaEventRecord(ev[2], st));
    TRY(tab_prepare_lists<W>(c, P, d_nbroff, d_nbr, npairs, vals, false, T, fast));
    if (!fast) form = FORM_GENERIC;
  }
  auto t_c = tnow();

  // 2. segments of the generic kernels, which direct mode may come to at any time (psoci_give_back),
  // and of its FP32 products (<= 32 neighbours of a configuration, one warp each)
  int64_t nseg = 0, nslots = 0;
  const bool segs = !fast || direct;
  if (segs) {
    TRY(psoci_alloc(c, &d_nseg, n + 1));
    TRY(psoci_alloc(c, &d_nrow, n + 1));
    TRY(psoci_alloc(c, &d_segoff, n + 1));
    TRY(psoci_alloc(c, &d_rowslot, n + 1));
    psoci_note_launch();
    k_seg_counts<<<(n + 255) / 256, 256, 0, st>>>(n, d_nbroff, c->d_sefoff, d_nseg, d_nrow);
    TRYC(cudaGetLastError());
    TRY(psoci_scan_i64(c, d_nseg, d_segoff, n, &nseg));
    TRY(psoci_scan_i64(c, d_nrow, d_rowslot, n, &nslots));
    TRY(psoci_alloc(c, &d_segcfg, nseg));
    TRY(psoci_alloc(c, &d_segk0, nseg));
    TRY(psoci_alloc(c, &d_segn, nseg));
    TRY(psoci_alloc(c, &d_segrow, nseg));
    if (!fast) TRY(psoci_alloc(c, &d_segcnt, nslots));
    psoci_note_launch();
    k_seg_init<<<(n + 255) / 256, 256, 0, st>>>(n, d_nbroff, c->d_sefoff, d_segoff, d_rowslot, d_segcfg, d_segk0,
                                                d_segn, d_segrow);
    TRYC(cudaGetLastError());
    P.nseg = nseg; P.seg_cfg = d_segcfg; P.seg_k0 = d_segk0; P.seg_n = d_segn; P.seg_rowoff = d_segrow;
    P.seg_cnt = d_segcnt;
  }
  c->nseg = nseg;

  // 3. evaluate
  const int hb_blocks = (int)std::max<int64_t>(1, std::min<int64_t>((nseg + WARPS_PER_CTA - 1) / WARPS_PER_CTA, 152 * 16));
  int64_t nnz = 0;
  auto t_d = t_c, t_e = t_c;
  if (direct) {
    // direct mode: the diagonal now, the other elements in every sigma; the neighbour lists
    // and tables (or segments) move to the context
    TRY(psoci_alloc(c, &c->d_diag, N));
    P.diag = c->d_diag;
    if (fast) {
      TRY(tab_diagonal<W>(c, P, T, c->d_diag));
    } else {
      const size_t smem = sizeof(WarpSmem) * WARPS_PER_CTA;
      TRYC(cudaFuncSetAttribute(k_hbuild<W, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      TRYC(cudaEventRecord(ev[2], st));
      psoci_note_launch();
      k_hbuild<W, 3><<<hb_blocks, WARPS_PER_CTA * 32, smem, st>>>(P);
      TRYC(cudaGetLastError());
    }
    TRYC(cudaEventRecord(ev[3], st));
    TRYC(cudaEventRecord(ev[4], st));
    TRYC(cudaEventRecord(ev[5], st));
    TRYC(cudaStreamSynchronize(st));
    c->dir_nbroff = d_nbroff; d_nbroff = nullptr;
    c->dir_nbr = d_nbr; d_nbr = nullptr;
    if (fast) {
      DirTabs *d = new DirTabs();
      dir_set<W>(d) = T;
      T = TabSet<W>();
      c->dir_tabs = d;
    }
    c->dir_segcfg = d_segcfg; d_segcfg = nullptr;
    c->dir_segk0 = d_segk0; d_segk0 = nullptr;
    c->dir_segn = d_segn; d_segn = nullptr;
    c->direct = true;
  } else if (fast) {
    TRY(psoci_alloc(c, &c->d_diag, N));
    TRY(tab_diagonal<W>(c, P, T, c->d_diag));
    TRY(psoci_alloc(c, &d_rownnz, N + 1));
    ElemArgs<W> E = elem_args<W>(c, T);
    E.row_nnz = d_rownnz;
    E.segments = T.t.counter;
    TRYC(cudaMemsetAsync(T.t.counter, 0, sizeof(unsigned long long), st));
    // 3. count the kept elements of each row
    if (vals) TRY((elems_launch<W, 0, true>(c, P, E)));
    else TRY((elems_launch<W, 0, false>(c, P, E)));
    TRYC(cudaEventRecord(ev[3], st));
    t_d = tnow();
    unsigned long long segs = 0;
    TRYC(cudaMemcpyAsync(&segs, T.t.counter, sizeof(segs), cudaMemcpyDeviceToHost, st));
    // 4. row offsets
    TRY(psoci_alloc(c, &c->d_rowptr, N + 1));
    TRY(psoci_scan_i64(c, d_rownnz, c->d_rowptr, N, &nnz));
    c->nseg = nseg = (int64_t)segs;
    TRYC(cudaEventRecord(ev[4], st));
    if (nnz < N) TRY(psoci_fail(c, PSOCI_ERR_CUDA, "H build: rows without their diagonal element"));
    TRY(psoci_alloc(c, &c->d_col, nnz));
    TRY(psoci_alloc(c, &c->d_val, nnz));
    if (mode == PSOCI_HMODE_CSR_BOTH) TRY(psoci_alloc(c, &c->d_val32, nnz));
    P.rowptr = c->d_rowptr; P.col = c->d_col; P.val = c->d_val; P.val32 = c->d_val32;
    t_e = tnow();
    // 5. write them
    if (vals) TRY((elems_launch<W, 1, true>(c, P, E)));
    else TRY((elems_launch<W, 1, false>(c, P, E)));
    TRYC(cudaEventRecord(ev[5], st));
    TRYC(cudaStreamSynchronize(st));
  } else {
    const size_t smem = sizeof(WarpSmem) * WARPS_PER_CTA;
    TRYC(cudaFuncSetAttribute(k_hbuild<W, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    TRYC(cudaFuncSetAttribute(k_hbuild<W, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // 3. count
    TRYC(cudaEventRecord(ev[2], st));
    psoci_note_launch();
    k_hbuild<W, 0><<<hb_blocks, WARPS_PER_CTA * 32, smem, st>>>(P);
    TRYC(cudaGetLastError());
    TRYC(cudaEventRecord(ev[3], st));
    t_d = tnow();
    // 4. offsets
    TRY(psoci_alloc(c, &d_rownnz, N + 1));
    psoci_note_launch();
    k_seg_rowscan<<<(n + 127) / 128, 128, 0, st>>>(n, c->d_sefoff, d_segoff, d_segrow, d_segcnt, d_rownnz);
    TRYC(cudaGetLastError());
    TRY(psoci_alloc(c, &c->d_rowptr, N + 1));
    TRY(psoci_scan_i64(c, d_rownnz, c->d_rowptr, N, &nnz));
    TRYC(cudaEventRecord(ev[4], st));
    TRY(psoci_alloc(c, &c->d_col, nnz));
    TRY(psoci_alloc(c, &c->d_val, nnz));
    if (mode == PSOCI_HMODE_CSR_BOTH) TRY(psoci_alloc(c, &c->d_val32, nnz));
    TRY(psoci_alloc(c, &c->d_diag, N));
    P.rowptr = c->d_rowptr; P.col = c->d_col; P.val = c->d_val; P.val32 = c->d_val32; P.diag = c->d_diag;
    t_e = tnow();
    // 5. fill
    psoci_note_launch();
    k_hbuild<W, 1><<<hb_blocks, WARPS_PER_CTA * 32, smem, st>>>(P);
    TRYC(cudaGetLastError());
    TRYC(cudaEventRecord(ev[5], st));
    TRYC(cudaStreamSynchronize(st));
  }
  auto t_f = std::chrono::steady_clock::now();
  if (c->verbose) {
    auto d = [](auto a, auto b) { return std::chrono::duration<double>(b - a).count(); };
    fprintf(stderr,
            "psoci: H build phases (%s%s, %s screen): screen %.4f s, tables %.4f s, evaluate %.4f s, "
            "offsets %.4f s, fill %.4f s\n",
            fast ? "coupling tables" : "generic kernels", vals ? ", pair integrals listed" : "",
            nsplit ? "all-pairs" : "lookup", d(t_a, t_b), d(t_b, t_c), d(t_c, t_d), d(t_d, t_e), d(t_e, t_f));
  }
  {
    psoci_build_info &b = c->binfo;
    b = psoci_build_info{};
    b.candidates = ncand; b.pairs = npairs; b.segments = nseg; b.nnz = nnz; b.nnz_lower = direct ? 0 : (nnz + N) / 2;
    b.evaluations = direct ? 0 : 1; b.fast = (fast && !direct) ? 1 : 0;
    b.lookup_screen = c->join_ok ? 1 : 0;
    b.eval_launches = (fast && !direct) ? (vals ? 2 : 1) : 0;
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, ev[0], ev[1]) == cudaSuccess) b.screen_ms = ms;
    if (cudaEventElapsedTime(&ms, ev[2], ev[3]) == cudaSuccess) b.evaluate_ms = ms;
    if (cudaEventElapsedTime(&ms, ev[3], ev[4]) == cudaSuccess) b.rows_ms = ms;
    if (cudaEventElapsedTime(&ms, ev[4], ev[5]) == cudaSuccess) b.assemble_ms = ms;
    if (cudaEventElapsedTime(&ms, ev[0], ev[5]) == cudaSuccess) b.total_ms = ms;
  }
  cleanup();
  c->nnz = nnz;
  *nnz_out = nnz;
  return PSOCI_OK;
#undef TRY
#undef TRYC
}

// ------------------------------------------------------------------------------------
// Direct mode with FP32 elements and inputs (configurations of at most 32 determinants, <= 6 open
// shells with an even electron count, <= 5 with an odd one; at most 16 SEFs).  The compensated FP32
// sums of a lane round by the order of its products, so they keep the order of the determinants:
// a lane owns a neighbour and marks, per row SEF r of I, the column SEFs t whose determinants are
// within two spin-orbital substitutions with the same spin projection (one, any spin, for spin-orbit
// pairs); a row's marked elements, by pair kind, neighbour and column, go to the lanes in turn.
// Elements from the coupling tables, in the order of k_elems, took 46 us for 118 and 85 for 442 at two
// small spaces, but agreed with these sums to 3e-8 only.  FP64 products (k_elems MODE 2) are the
// faster choice in direct mode, and what its solves use.
// ------------------------------------------------------------------------------------
constexpr int FAST_MAXDET = 32;
constexpr int FAST_MAXSEF = 16;
constexpr int FAST_MAXOPEN = 6;  // 2^(6-1) = 32 determinants
constexpr int FAST_MAXK = 1 + FAST_MAXOPEN * (FAST_MAXOPEN - 1) / 2;  // diagonal list, <= 6 open shells

__device__ __forceinline__ bool tbit(const uint64_t *x, int p) { return (x[p >> 6] >> (p & 63)) & 1ull; }

template <int W>
struct FastSmem {
  PairInfo pi[PSOCI_SEG];
  double K[FAST_MAXK];
  uint64_t ra[FAST_MAXDET * W], rb[FAST_MAXDET * W];
  uint8_t rna[FAST_MAXDET], rph[FAST_MAXDET];
  // of a row: connectivity of the marked elements of each slot (the marked columns are its four
  // 16-bit quarters or-ed) and their exclusive prefix
  uint64_t cm[PSOCI_SEG];
  int16_t pre[PSOCI_SEG];
  int8_t perm[PSOCI_SEG];  // evaluation order: slot -> neighbour lane, grouped by pair kind
};

template <int W>
__global__ void __launch_bounds__(WARPS_PER_CTA * 32) k_direct_mixed(Params P) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FastSmem<W> *ws = reinterpret_cast<FastSmem<W> *>(smem_raw) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const bool odd = P.nelec & 1;
  for (int64_t s = warp; s < P.nseg; s += nwarps) {
    const int I = P.seg_cfg[s];
    const int64_t k0 = P.seg_k0[s];
    const int n = P.seg_n[s];
    const int nsefI = (int)(P.sefoff[I + 1] - P.sefoff[I]);
    const int64_t d0I = P.detoff[I];
    const int ndI = (int)(P.detoff[I + 1] - d0I);
    const int nopI = P.nopen[I];
    if (lane < n) pair_setup<W>(P, I, P.nbr[k0 + lane], ws->pi[lane], ws->K);
    for (int d = lane; d < ndI; d += 32) {
#pragma unroll
      for (int w = 0; w < W; ++w) {
        ws->ra[d * W + w] = P.alpha[(d0I + d) * W + w];
        ws->rb[d * W + w] = P.beta[(d0I + d) * W + w];
      }
      ws->rna[d] = P.nalpha[d0I + d];
      ws->rph[d] = P.phase[d0I + d];
    }
    __syncwarp();
    // phase 1: connectivity masks C[r] for this lane's neighbour, bit-parallel over the
    // row determinants.  With m_a the alpha pattern of row det a on I's open shells, a column
    // det b (alpha ab, beta bb) differs from a in
    //   c(a) = F + #{p in x : p not in m_a} + #{p in y : p in m_a}
    // spin-orbitals of b, where x, y are b's alpha / beta patterns on I's open shells and F
    // counts b's electrons in orbitals empty in I.  Non-spin-orbit pairs need c(a) <= 2 and
    // equal alpha counts, spin-orbit pairs c(a) <= 1 (the tests det_elem starts with).  The sets
    // {a : p in m_a} and {a : |m_a| = k} are warp ballots; c(a) is kept as a saturating
    // bit-sliced counter over all row dets at once.
    uint32_t Ap[FAST_MAXOPEN], Nk[FAST_MAXOPEN + 1];
    int sI[FAST_MAXOPEN];
    uint64_t occI[W];
    {
      uint64_t SI[W];
#pragma unroll
      for (int w = 0; w < W; ++w) {
        occI[w] = P.e1[(int64_t)I * W + w];
        SI[w] = occI[w] & ~P.e2[(int64_t)I * W + w];
      }
      // open shells of I, ascending (fixed-size loops keep these arrays in registers)
#pragma unroll
      for (int p = 0; p < FAST_MAXOPEN; ++p) {
        sI[p] = lowest_bit<W>(SI);
        bool done = false;
#pragma unroll
        for (int w = 0; w < W; ++w)
          if (!done && SI[w]) { SI[w] &= SI[w] - 1; done = true; }
      }
      uint32_t ma = 0u;
      if (lane < ndI)
#pragma unroll
        for (int p = 0; p < FAST_MAXOPEN; ++p)
          if (p < nopI) ma |= (uint32_t)tbit(&ws->ra[lane * W], sI[p]) << p;
#pragma unroll
      for (int p = 0; p < FAST_MAXOPEN; ++p) Ap[p] = __ballot_sync(0xffffffffu, (lane < ndI) && ((ma >> p) & 1u));
#pragma unroll
      for (int k = 0; k <= FAST_MAXOPEN; ++k) Nk[k] = __ballot_sync(0xffffffffu, (lane < ndI) && __popc(ma) == k);
    }
    const int ndblI = P.nelec - nopI;  // electrons in I's doubly occupied orbitals
    // C[r]: for row SEF r and column SEF t, bit t + 16 (x << 1 | y) says that determinant x
    // of SEF r and determinant y of SEF t can couple; the SEF element is marked when any can.
    uint64_t C[FAST_MAXSEF];
    for (int r = 0; r < FAST_MAXSEF; ++r) C[r] = 0ull;
    if (lane < n) {
      const PairInfo &pi = ws->pi[lane];
      if (pi.kind != K_NONE) {
        const bool so = (pi.kind == K_SO);
        const int64_t d0J = pi.swap ? pi.detA : pi.detB;
        const int nopJ = pi.swap ? pi.nopenA : pi.nopenB;
        const int ndJ = 1 << (nopJ > 1 ? nopJ - 1 : 0);
        const int thr = so ? 1 : 2;
        const uint32_t rows_valid = (ndI >= 32) ? 0xffffffffu : ((1u << ndI) - 1u);
        for (int b = 0; b < ndJ; ++b) {
          uint64_t ja[W], jb[W];
#pragma unroll
          for (int w = 0; w < W; ++w) { ja[w] = __ldg(P.alpha + (d0J + b) * W + w); jb[w] = __ldg(P.beta + (d0J + b) * W + w); }
          int F = 0;
#pragma unroll
          for (int w = 0; w < W; ++w) F += __popcll(ja[w] & ~occI[w]) + __popcll(jb[w] & ~occI[w]);
          if (F > thr) continue;
          uint32_t ok = 0u;
          {
            // saturating counter over the row dets: S0 (c'=0), S1, S2, S3 (>= 3)
            uint32_t S0 = 0xffffffffu, S1 = 0u, S2 = 0u;
#pragma unroll
            for (int p = 0; p < FAST_MAXOPEN; ++p) {
              if (p >= nopI) break;
              const bool xa = bit_w<W>(ja, sI[p]), yb = bit_w<W>(jb, sI[p]);
              if (xa) {  // mismatch where row det has beta on p
                const uint32_t T = ~Ap[p];
                S2 = (S2 & ~T) | (S1 & T);
                S1 = (S1 & ~T) | (S0 & T);
                S0 &= ~T;
              }
              if (yb) {  // mismatch where row det has alpha on p
                const uint32_t T = Ap[p];
                S2 = (S2 & ~T) | (S1 & T);
                S1 = (S1 & ~T) | (S0 & T);
                S0 &= ~T;
              }
            }
            ok = (thr - F >= 2) ? (S0 | S1 | S2) : (thr - F == 1) ? (S0 | S1) : S0;
          }
          int na = 0;
#pragma unroll
          for (int w = 0; w < W; ++w) na += __popcll(ja[w]);
          const int need = na - (ndblI / 2);  // alpha open shells a row det needs for equal counts
          ok &= rows_valid;
          if (!so) {
            uint32_t nk = 0u;
#pragma unroll
            for (int k = 0; k <= FAST_MAXOPEN; ++k)
              if (k == need) nk = Nk[k];
            ok &= (need >= 0 && need <= nopI) ? nk : 0u;
          }
          const int t = odd ? b : (nopJ ? (b >> 1) : 0);
          const int y = (!odd && nopJ) ? (b & 1) : 0;
          while (ok) {
            const int a = __ffs(ok) - 1;
            ok &= ok - 1;
            const int x = (!odd && nopI) ? (a & 1) : 0;
            C[odd ? a : (nopI ? (a >> 1) : 0)] |= 1ull << (t + 16 * ((x << 1) | y));
          }
        }
      }
    }
    const RowDets rowA = {ws->ra, ws->rb, ws->rph, ws->rna};  // I's determinants (A = I)
    // evaluation order of the neighbours: grouped by pair kind (doubles, singles, spin-orbit,
    // diagonal), ascending within a kind, so that neighbouring lanes mostly run the same
    // branch of the element code.  With the marked elements' numbers it fixes the order of the sums.
    {
      const int kd = (lane < n) ? ws->pi[lane].kind : -1;
      const int key = (kd == K_DOUBLE) ? 0 : (kd == K_SINGLE) ? 1 : (kd == K_SO) ? 2 : (kd == K_DIAG) ? 3
                                                                                         : (kd == K_NONE) ? 4 : 5;
      int rank = 0, base = 0;
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const unsigned m = __ballot_sync(0xffffffffu, key == k);
        if (key == k) rank = base + __popc(m & ((1u << lane) - 1u));
        base += __popc(m);
      }
      ws->perm[rank] = (int8_t)lane;
      __syncwarp();
    }
    const int src = ws->perm[lane];  // the neighbour lane at evaluation slot `lane`
    for (int r = 0; r < nsefI; ++r) {
      // marked columns of each slot and their exclusive prefix
      const uint64_t cr = __shfl_sync(0xffffffffu, (lane < n) ? C[r] : 0ull, src);
      const int cm = __popc((uint32_t)((cr | (cr >> 16) | (cr >> 32) | (cr >> 48)) & 0xffffull));
      int inclm = cm;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inclm, o);
        if (lane >= o) inclm += v;
      }
      ws->pre[lane] = (int16_t)(inclm - cm);
      ws->cm[lane] = cr;
      const int T = __shfl_sync(0xffffffffu, inclm, 31);
      double acc[8];
      float accs[8], accc[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) { accs[q] = 0.f; accc[q] = 0.f; }
      __syncwarp();
      for (int e = lane; e < T; e += 32) {
        int o = 0;  // the slot owning element e: last slot whose prefix is <= e
#pragma unroll
        for (int step = 16; step > 0; step >>= 1)
          if (ws->pre[o + step] <= e) o += step;
        const uint64_t cw = ws->cm[o];
        uint32_t m = (uint32_t)((cw | (cw >> 16) | (cw >> 32) | (cw >> 48)) & 0xffffull);
        for (int q = e - ws->pre[o]; q > 0; --q) m &= m - 1;
        const int t = __ffs(m) - 1;
        const PairInfo &pi = ws->pi[ws->perm[o]];
        // reference roles: the lower half of a diagonal block, block (J, I) for J > I
        const bool diag_blk = (pi.kind == K_DIAG);
        const bool flip = diag_blk ? (t > r) : (pi.swap != 0);
        const uint64_t co = cw >> t;
        unsigned conn = (unsigned)((co & 1ull) | ((co >> 15) & 2ull) | ((co >> 30) & 4ull) | ((co >> 45) & 8ull));
        // a diagonal block is symmetric: the transposed element swaps the determinant roles
        if (flip) conn = (conn & 9u) | ((conn & 2u) << 1) | ((conn & 4u) >> 1);
        // A's determinants come from shared memory when A = I (a pair J > I has A = J, read from the
        // tables)
        const double v = sef_elem<W>(P, pi, ws->K, flip ? t : r, flip ? r : t, conn, pi.swap ? nullptr : &rowA);
        if (fabs(v) >= PSOCI_MIN_VALUE || (diag_blk && t == r)) {
          const float vf = (float)v;
          const float4 *xr = reinterpret_cast<const float4 *>(P.dx32 + (pi.colbase + t) * 8);
          const float4 xa = __ldg(xr), xb = __ldg(xr + 1);
          const float xv[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            // Kahan: the rounding error of each addition is carried in accc and fed back
            const float yv = __fsub_rn(__fmul_rn(vf, xv[q]), accc[q]);
            const float tt = __fadd_rn(accs[q], yv);
            accc[q] = __fsub_rn(__fsub_rn(tt, accs[q]), yv);
            accs[q] = tt;
          }
        }
      }
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[q] = (double)accs[q] - (double)accc[q];
      const double tot = reduce_scatter8_f64(acc, lane);
      const int q = lane >> 2;
      if ((lane & 3) == 0 && q < P.kvec && tot != 0.0) atomicAdd(P.dy + (P.sefoff[I] + r) * P.ldy + q, tot);
      __syncwarp();
    }
    __syncwarp();
  }
}

// X (FP64, leading dim ldx, k <= 8 columns) -> X32 (FP32, row stride 8, zero padded)
__global__ void k_direct_x32(int64_t n, int k, const double *__restrict__ x, int ldx, float *__restrict__ x32) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    float f[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) f[q] = (q < k) ? (float)x[r * ldx + q] : 0.f;
    float4 *d = reinterpret_cast<float4 *>(x32 + r * 8);
    d[0] = make_float4(f[0], f[1], f[2], f[3]);
    d[1] = make_float4(f[4], f[5], f[6], f[7]);
  }
}

template <int W>
psoci_status run_direct_sigma(psoci_ctx *c, int k, const double *dX, int ldx, double *dY, int ldy, psoci_prec prec,
                              float *x32) {
  cudaStream_t st = c->stream;
  Params P = {};
  P.nconf = c->nconf; P.nbf = c->nbf; P.nelec = c->nelec; P.ksym = c->ksym;
  P.e1 = c->d_e1; P.e2 = c->d_e2; P.jsym = c->d_jsym; P.nopen = c->d_nopen;
  P.sefoff = c->d_sefoff; P.detoff = c->d_detoff;
  P.alpha = c->d_alpha; P.beta = c->d_beta; P.phase = c->d_phase; P.nalpha = c->d_nalpha;
  P.one = c->d_one; P.eri = c->d_eri;
  P.nbroff = c->dir_nbroff; P.nbr = c->dir_nbr;
  P.nseg = c->nseg; P.seg_cfg = c->dir_segcfg; P.seg_k0 = c->dir_segk0; P.seg_n = c->dir_segn;
  const int64_t N = c->nsef_total;
  psoci_status s;
  const bool fast = c->dir_tabs != nullptr;
  const size_t smem = sizeof(WarpSmem) * WARPS_PER_CTA;
  ElemArgs<W> E = {};
  if (fast) {
    E = elem_args<W>(c, dir_set<W>(static_cast<DirTabs *>(c->dir_tabs)));
  } else {
    PSOCI_CUDA(c, cudaMemset2DAsync(dY, sizeof(double) * ldy, 0, sizeof(double) * k, N, st));
    if (P.nseg == 0) return PSOCI_OK;
    PSOCI_CUDA(c, cudaFuncSetAttribute(k_hbuild<W, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  }
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((P.nseg + WARPS_PER_CTA - 1) / WARPS_PER_CTA, 152 * 16));
  // MIXED (spaces of at most 32 determinants a configuration): FP32 element x FP32 input
  // products; beyond them direct mode is FP64 whatever the precision asked for
  const bool mixed = c->max_ndet <= FAST_MAXDET && prec == PSOCI_PREC_MIXED && x32 && P.nseg > 0;
  const size_t fsmem = sizeof(FastSmem<W>) * WARPS_PER_CTA;
  if (mixed) {
    PSOCI_CUDA(c, cudaFuncSetAttribute(k_direct_mixed<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fsmem));
    if (fast) PSOCI_CUDA(c, cudaMemset2DAsync(dY, sizeof(double) * ldy, 0, sizeof(double) * k, N, st));
  }
  for (int q0 = 0; q0 < k; q0 += 8) {
    P.dx = dX + q0; P.dy = dY + q0; P.ldx = ldx; P.ldy = ldy; P.kvec = std::min(8, k - q0);
    P.dx32 = nullptr;
    if (mixed) {
      psoci_note_launch();
      k_direct_x32<<<(unsigned)std::min<int64_t>((N + 255) / 256, 152 * 16), 256, 0, st>>>(N, P.kvec, P.dx, ldx, x32);
      P.dx32 = x32;
      psoci_note_launch();
      k_direct_mixed<W><<<blocks, WARPS_PER_CTA * 32, fsmem, st>>>(P);
      PSOCI_CUDA(c, cudaGetLastError());
    } else if (fast) {
      if ((s = E.vals ? elems_launch<W, 2, true>(c, P, E) : elems_launch<W, 2, false>(c, P, E))) return s;
    } else {
      psoci_note_launch();
      k_hbuild<W, 2><<<blocks, WARPS_PER_CTA * 32, smem, st>>>(P);
      PSOCI_CUDA(c, cudaGetLastError());
    }
  }
  return PSOCI_OK;
}

}  // namespace

psoci_status psoci_direct_sigma(psoci_ctx *c, int k, const double *dX, int ldx, double *dY, int ldy, psoci_prec prec,
                                float *x32) {
  if (!c->direct) return psoci_fail(c, PSOCI_ERR_STATE, "direct sigma: no direct-mode build");
  return (c->words == 1) ? run_direct_sigma<1>(c, k, dX, ldx, dY, ldy, prec, x32)
                         : run_direct_sigma<2>(c, k, dX, ldx, dY, ldy, prec, x32);
}

void psoci_join_release(psoci_ctx *c) {
  psoci_free(c->d_jgid);
  psoci_free(c->d_jlid);
  psoci_free(c->d_jT);
  psoci_free(c->d_jlnoff);
  psoci_free(c->d_jln);
  psoci_free(c->d_jhdec);
  psoci_free(c->d_jlokey);
  c->join_ok = false;
}

// Tables of the lookup screen (see k_join).  The space qualifies when some split s <= 12
// leaves every configuration at most two electrons in the orbitals >= s, the
// configurations are numbered in ascending (hi pattern, lo pattern) order with lo patterns
// numbered by first appearance, and the tables stay small; otherwise the all-pairs screen
// is used.  Not qualifying is not an error.
namespace {
// the configuration of each (lo pattern, hi pattern) cell; the pairs are unique
__global__ void k_fill_T(int n, const int32_t *__restrict__ gid, const int32_t *__restrict__ lid, int64_t L,
                         int32_t *__restrict__ T) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    T[(int64_t)gid[i] * L + lid[i]] = i;
}

// lo patterns within tau = 1..4 of each lo pattern (itself included), ascending inside each of five
// groups: the lo electron count minus l's, -2..2 (a hi pattern holds 0-2 electrons, so a partner lo
// pattern differs by at most 2; the others never make a configuration and are left out).  Lists
// tau-major, then by pattern, then by group.  One warp a pattern, lanes over the others; MODE 0
// counts to out[((tau - 1) * L + l) * 5 + k], MODE 1 writes the lists.  (On the host's cores the L^2
// distances took 2 of the 4.6 ms of psoci_set_configs at mrcis_6e8o_v40.)
constexpr int LN_GRP = 5, LN_TAU = 4;
template <int MODE>
__global__ void __launch_bounds__(256) k_lo_lists(int L, const uint32_t *__restrict__ key, const int32_t *__restrict__ off,
                                                  int32_t *__restrict__ out) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  for (int l = warp; l < L; l += nwarps) {
    const uint32_t kl = key[l];
    const int nel = __popc(kl);
    // lane LN_GRP (tau - 1) + k: this list's entries, or its next place
    const int t = lane / LN_GRP, g = lane - LN_GRP * t;
    const int64_t own = t < LN_TAU ? (int64_t)t * LN_GRP * L + (int64_t)LN_GRP * l + g : 0;
    int n = (MODE == 1 && t < LN_TAU) ? off[own + t] : 0;
    for (int m0 = 0; m0 < L; m0 += 32) {
      const int m = m0 + lane;
      int d = LN_TAU + 1, k = 0;
      if (m < L) {
        const uint32_t km = key[m];
        k = __popc(km) - nel + 2;
        d = (k < 0 || k >= LN_GRP) ? LN_TAU + 1 : max(__popc(kl ^ km), 1);
      }
      if (!__any_sync(FULL, d <= LN_TAU)) continue;
#pragma unroll
      for (int tt = 0; tt < LN_TAU; ++tt)
#pragma unroll
        for (int kk = 0; kk < LN_GRP; ++kk) {
          const bool in = d <= tt + 1 && k == kk;
          const unsigned b = __ballot_sync(FULL, in);
          if (MODE == 1) {
            const int at = __shfl_sync(FULL, n, LN_GRP * tt + kk);
            if (in) out[at + __popc(b & ((1u << lane) - 1u))] = m;
          }
          if (lane == LN_GRP * tt + kk) n += __popc(b);
        }
    }
    if (MODE == 0 && t < LN_TAU) out[own] = n;
  }
}
}  // namespace

psoci_status psoci_join_prepare(psoci_ctx *c) {
  psoci_join_release(c);
  const int n = c->nconf, nbf = c->nbf;
  const uint8_t *occ = c->h_occ.data();
  // split: orbitals >= s hold at most two electrons in every configuration
  // (the configuration loops run on the host's cores; only the numbering of lo patterns by
  // first appearance is sequential)
  std::vector<int> smax(std::max<unsigned>(1u, std::thread::hardware_concurrency()), 0);
  const int nthr = psoci_parallel_ranges(n, [&](int64_t lo, int64_t hi, int t) {
    int sm = 0;
    for (int64_t i = lo; i < hi; ++i) {
      const uint8_t *o = occ + (size_t)i * nbf;
      int e = 0, si = 0;
      for (int q = nbf - 1; q >= 0; --q) {
        e += o[q];
        if (e >= 3) { si = q + 1; break; }
      }
      sm = std::max(sm, si);
    }
    smax[t] = sm;
  });
  int s = 0;
  for (int t = 0; t < nthr; ++t) s = std::max(s, smax[t]);
  const int nh = nbf - s;
  if (s > 12 || nh < 1) return PSOCI_OK;
  const int64_t G = 1 + nh + (int64_t)nh * (nh + 1) / 2;
  std::vector<int32_t> gid(n), lid(n), keyid((size_t)1 << (2 * s), -1);
  std::vector<uint32_t> lokey, keys(n);
  psoci_parallel_ranges(n, [&](int64_t lo, int64_t hi, int) {
    for (int64_t i = lo; i < hi; ++i) {
      const uint8_t *o = occ + (size_t)i * nbf;
      uint32_t key = 0;
      for (int q = 0; q < s; ++q) {
        if (o[q] >= 1) key |= 1u << q;
        if (o[q] == 2) key |= 1u << (s + q);
      }
      int pa = -1, pb = -1, kind = 0;
      for (int q = s; q < nbf; ++q) {
        if (o[q] == 0) continue;
        if (o[q] == 2) { kind = 3; pa = q - s; }
        else if (pa < 0) { kind = 1; pa = q - s; }
        else { kind = 2; pb = q - s; }
      }
      gid[i] = (kind == 0) ? 0 : (kind == 1) ? 1 + pa
               : (int32_t)(1 + nh + (kind == 3 ? (int64_t)pa * (pa + 1) / 2 + pa : (int64_t)pb * (pb + 1) / 2 + pa));
      keys[i] = key;
    }
  });
  for (int i = 0; i < n; ++i) {
    const uint32_t key = keys[i];
    if (keyid[key] < 0) { keyid[key] = (int32_t)lokey.size(); lokey.push_back(key); }
    lid[i] = keyid[key];
    if (i > 0 && gid[i] < gid[i - 1]) return PSOCI_OK;  // hi patterns must ascend
  }
  const int64_t L = (int64_t)lokey.size();
  // Number the lo patterns so that they ascend inside every hi pattern: each group's order
  // is a chain of constraints; a topological order of all of them (ties broken by first
  // appearance) exists unless two groups order some patterns differently.
  {
    // constraint edges lid[i-1] -> lid[i] within a hi pattern, as a compressed adjacency
    std::vector<int32_t> indeg((size_t)L, 0), eoff((size_t)L + 1, 0), next;
    for (int i = 1; i < n; ++i)
      if (gid[i] == gid[i - 1]) {
        if (lid[i] == lid[i - 1]) return PSOCI_OK;  // repeated configuration
        ++eoff[lid[i - 1] + 1];
        ++indeg[lid[i]];
      }
    for (int64_t l = 0; l < L; ++l) eoff[l + 1] += eoff[l];
    next.resize((size_t)eoff[L]);
    {
      std::vector<int32_t> fill(eoff.begin(), eoff.end() - 1);
      for (int i = 1; i < n; ++i)
        if (gid[i] == gid[i - 1]) next[fill[lid[i - 1]]++] = lid[i];
    }
    std::vector<int32_t> order;
    order.reserve((size_t)L);
    std::priority_queue<int32_t, std::vector<int32_t>, std::greater<int32_t>> ready;
    for (int64_t l = 0; l < L; ++l)
      if (indeg[l] == 0) ready.push((int32_t)l);
    while (!ready.empty()) {
      const int32_t l = ready.top();
      ready.pop();
      order.push_back(l);
      for (int32_t e = eoff[l]; e < eoff[l + 1]; ++e)
        if (--indeg[next[e]] == 0) ready.push(next[e]);
    }
    if ((int64_t)order.size() != L) return PSOCI_OK;  // contradictory orders
    std::vector<int32_t> rank((size_t)L);
    std::vector<uint32_t> key2((size_t)L);
    for (int64_t r = 0; r < L; ++r) { rank[order[r]] = (int32_t)r; key2[r] = lokey[order[r]]; }
    for (int i = 0; i < n; ++i) lid[i] = rank[lid[i]];
    lokey.swap(key2);
    for (int i = 1; i < n; ++i)
      if (gid[i] == gid[i - 1] && lid[i] <= lid[i - 1]) return PSOCI_OK;
  }
  if (G * L > ((int64_t)1 << 26)) return PSOCI_OK;
  std::vector<int32_t> hdec((size_t)G);
  hdec[0] = 0;
  for (int a = 0; a < nh; ++a) hdec[1 + a] = 1 | (a << 8);
  for (int b = 0; b < nh; ++b)
    for (int a = 0; a <= b; ++a)
      hdec[1 + nh + (size_t)b * (b + 1) / 2 + a] = (a == b) ? (3 | (a << 8)) : (2 | (a << 8) | (b << 20));
  // lists of lo patterns (k_lo_lists): counted, their places summed here, then written
  std::vector<int32_t> lnoff((size_t)LN_TAU * (LN_GRP * L + 1)), lcnt((size_t)LN_TAU * LN_GRP * L);
  cudaStream_t q = c->stream;
  psoci_status st;
  int32_t *d_cnt = nullptr;
  const int lblocks = (int)std::min<int64_t>((L + 7) / 8, 152 * 8);
  auto fail = [&](psoci_status r) {
    psoci_free(d_cnt);
    psoci_join_release(c);
    return r;
  };
  if ((st = psoci_alloc(c, &c->d_jlokey, lokey.size())) || (st = psoci_alloc(c, &d_cnt, lcnt.size()))) return fail(st);
  cudaError_t e = cudaMemcpyAsync(c->d_jlokey, lokey.data(), 4 * lokey.size(), cudaMemcpyHostToDevice, q);
  if (e == cudaSuccess) {
    psoci_note_launch();
    k_lo_lists<0><<<lblocks, 256, 0, q>>>((int)L, c->d_jlokey, nullptr, d_cnt);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(lcnt.data(), d_cnt, 4 * lcnt.size(), cudaMemcpyDeviceToHost, q);
  if (e == cudaSuccess) e = cudaStreamSynchronize(q);
  if (e != cudaSuccess) return fail(psoci_cuda_fail(c, e, "lookup screen"));
  psoci_free(d_cnt);
  int64_t nln = 0;
  for (int tau = 1; tau <= LN_TAU; ++tau) {
    for (int64_t g = 0; g < LN_GRP * L; ++g) {
      lnoff[(tau - 1) * (LN_GRP * L + 1) + g] = (int32_t)nln;
      nln += lcnt[(size_t)(tau - 1) * LN_GRP * L + g];
    }
    lnoff[(tau - 1) * (LN_GRP * L + 1) + LN_GRP * L] = (int32_t)nln;
    if (nln > INT32_MAX) {
      psoci_join_release(c);
      return PSOCI_OK;
    }
  }
  if ((st = psoci_alloc(c, &c->d_jgid, n)) || (st = psoci_alloc(c, &c->d_jlid, n)) ||
      (st = psoci_alloc(c, &c->d_jT, (size_t)(G * L))) || (st = psoci_alloc(c, &c->d_jlnoff, lnoff.size())) ||
      (st = psoci_alloc(c, &c->d_jln, (size_t)nln)) || (st = psoci_alloc(c, &c->d_jhdec, hdec.size())))
    return fail(st);
  PSOCI_CUDA(c, cudaMemcpyAsync(c->d_jgid, gid.data(), 4 * gid.size(), cudaMemcpyHostToDevice, q));
  PSOCI_CUDA(c, cudaMemcpyAsync(c->d_jlid, lid.data(), 4 * lid.size(), cudaMemcpyHostToDevice, q));
  // T[hi pattern][lo pattern] = configuration (or -1), filled on the device
  PSOCI_CUDA(c, cudaMemsetAsync(c->d_jT, 0xff, sizeof(int32_t) * (size_t)(G * L), q));
  psoci_note_launch();
  k_fill_T<<<(n + 255) / 256, 256, 0, q>>>(n, c->d_jgid, c->d_jlid, L, c->d_jT);
  PSOCI_CUDA(c, cudaGetLastError());
  PSOCI_CUDA(c, cudaMemcpyAsync(c->d_jlnoff, lnoff.data(), 4 * lnoff.size(), cudaMemcpyHostToDevice, q));
  psoci_note_launch();
  k_lo_lists<1><<<lblocks, 256, 0, q>>>((int)L, c->d_jlokey, c->d_jlnoff, c->d_jln);
  PSOCI_CUDA(c, cudaGetLastError());
  PSOCI_CUDA(c, cudaMemcpyAsync(c->d_jhdec, hdec.data(), 4 * hdec.size(), cudaMemcpyHostToDevice, q));
  PSOCI_CUDA(c, cudaStreamSynchronize(q));
  c->join_s = s; c->join_nh = nh; c->join_G = (int)G; c->join_L = (int)L;
  c->join_ok = true;
  return PSOCI_OK;
}

static void dir_tabs_release(psoci_ctx *c) {
  if (!c->dir_tabs) return;
  DirTabs *d = static_cast<DirTabs *>(c->dir_tabs);
  d->s1.free();
  d->s2.free();
  delete d;
  c->dir_tabs = nullptr;
}

bool psoci_give_back(psoci_ctx *c) {
  if (c->den_tabs && !(c->keep & PSOCI_KEEP_DENSITY)) {
    psoci_density_release(c);
  } else if (c->grad_nbroff && !(c->keep & PSOCI_KEEP_GRAD)) {
    psoci_grad_release(c);
  } else if (c->dir_tabs && !(c->keep & PSOCI_KEEP_DIRECT)) {
    DirTabs *d = static_cast<DirTabs *>(c->dir_tabs);
    if (d->s1.vals || d->s2.vals) {
      psoci_free(d->s1.vals);
      psoci_free(d->s2.vals);
    } else {
      dir_tabs_release(c);
    }
  } else {
    return false;
  }
  return true;
}

void psoci_h_release(psoci_ctx *c) {
  psoci_grad_release(c);
  c->sigma_variant = PSOCI_SIGMA_DEFAULT;
  c->sigma_tuned = false;
  psoci_free(c->dir_nbroff);
  psoci_free(c->dir_nbr);
  psoci_free(c->dir_segcfg);
  psoci_free(c->dir_segk0);
  psoci_free(c->dir_segn);
  dir_tabs_release(c);
  c->direct = false;
  psoci_free(c->d_rowptr);
  psoci_free(c->d_col);
  psoci_free(c->d_val);
  psoci_free(c->d_val32);
  psoci_free(c->d_diag);
  c->have_h = false;
  c->nnz = 0;
  c->binfo = psoci_build_info{};
}

psoci_status psoci_h_blocks(psoci_ctx *c, int npairs, const int32_t *A, const int32_t *B, double *out) {
  if (!c->have_ints) return psoci_fail(c, PSOCI_ERR_STATE, "blocks: no integrals set");
  if (!c->have_dets) return psoci_fail(c, PSOCI_ERR_STATE, "blocks: determinants not built");
  if (npairs < 0 || (npairs > 0 && (!A || !B || !out))) return psoci_fail(c, PSOCI_ERR_INVALID_ARG, "blocks: bad arguments");
  if (npairs == 0) return PSOCI_OK;
  return (c->words == 1) ? run_blocks<1>(c, npairs, A, B, out) : run_blocks<2>(c, npairs, A, B, out);
}

psoci_status psoci_h_build(psoci_ctx *c, psoci_hmode mode, int64_t *nnz) {
  if (!c->have_ints) return psoci_fail(c, PSOCI_ERR_STATE, "psoci_build_hamiltonian: no integrals set");
  if (!c->have_dets) return psoci_fail(c, PSOCI_ERR_STATE, "psoci_build_hamiltonian: determinants not built");
  if (c->nbf != 0 && c->n1 != (int64_t)c->nbf * (c->nbf + 1) / 2)
    return psoci_fail(c, PSOCI_ERR_INVALID_ARG, "integral and configuration orbital counts differ");
  psoci_h_release(c);
  auto t0 = std::chrono::steady_clock::now();
  int form = c->eval_launches == 1 ? FORM_UNLISTED : FORM_LISTED;
  psoci_status s;
  for (bool again = false;; again = true) {
    s = (c->words == 1) ? run_build<1>(c, mode, form, nnz) : run_build<2>(c, mode, form, nnz);
    if (s == PSOCI_OK) {
      if (again) c->err.clear();
      break;
    }
    psoci_h_release(c);
    if (s != PSOCI_ERR_NOMEM || form == FORM_GENERIC) return s;
    ++form;  // no room: the next form
  }
  c->build_seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  c->have_h = true;
  if (c->verbose)
    fprintf(stderr, "psoci: H build N=%lld nnz=%lld candidates=%lld pairs=%lld segments=%lld %.3f s\n",
            (long long)c->nsef_total, (long long)c->nnz, (long long)c->ncand, (long long)c->npairs, (long long)c->nseg,
            c->build_seconds);
  return PSOCI_OK;
}

// ------------------------------------------------------------------------------------
// Energy gradient with respect to the integral tables: the adjoint of the element
// evaluation.  For a CI vector c, E = c^T H c and every element of H is a sum of entries of
// the packed tables with fixed coefficients (once the reference's zero-prefactor skips are
// left out), so dE / d table[t] is the transposed evaluation: every coupling of a
// determinant pair (x of I, y of J) adds its weight w_xy = cd_I[x] cd_J[y] (cd = the vector in
// the determinant basis, CDC^T's transpose) to the entries its element reads, with the
// element's sign and coefficient.  dE/d one[pq] is the spin-free 1-RDM (equal irreps) or the
// spin-orbit density (unequal irreps), dE/d eri[canon(pq,rs)] the 2-RDM in the reference's
// 8-fold packed layout (Hellmann-Feynman).
//
// Work: one warp per row configuration I over its lower neighbours J <= I (pairs J < I
// count twice, as H_JI = H_IJ^T), 32 pairs set up at a time (a lane each); lanes over the
// determinant pairs of one configuration pair classify each coupling (det_adj mirrors
// det_elem's branches) and add its weights to the pair's terms: v0, v1 (double, SO and
// single prefactors, or the diagonal's Kd[0]) in registers, the exchange terms X[t] /
// Kd[mm] in a per-warp shared array; the pair's terms are then scattered to the tables.
// ------------------------------------------------------------------------------------
namespace {

constexpr int ADJ_WARPS = 4;
constexpr int ADJ_MAXR = 8;                                        // roots per pass
constexpr int ADJ_NT = 2 + PSOCI_MAX_OPEN * (PSOCI_MAX_OPEN - 1) / 2;  // v0, v1, X[t] or Kd[mm]

enum { T_NONE = 0, T_V0, T_V1, T_V0MV1, T_SGL, T_X, T_DIAG, T_K, T_DIRECT };

template <int W>
struct AdjPair {
  int64_t detA, detB;
  int A, B, kind;
  int iex0, iex1, jex0, jex1;
  int jsA, jsB, nopenA, ndetA, ndetB;
  uint64_t SA[W];
  uint64_t bm[6][W];
};

// The structure of the pair (A, B) in the reference's roles, from the occupations and the
// symmetries alone: diagonal, same-symmetry single, spin-orbit single, double or none
// (more than two excitations).
template <int W>
__device__ void adj_pair_setup(const Params &P, int A, int B, AdjPair<W> &pi) {
  pi.A = A; pi.B = B;
  pi.detA = P.detoff[A]; pi.detB = P.detoff[B];
  pi.ndetA = (int)(P.detoff[A + 1] - P.detoff[A]);
  pi.ndetB = (int)(P.detoff[B + 1] - P.detoff[B]);
  pi.jsA = P.jsym[A]; pi.jsB = P.jsym[B];
  pi.nopenA = P.nopen[A];
  uint64_t e1A[W], e2A[W], e1B[W], e2B[W], im1[W], im2[W], jm1[W], jm2[W];
#pragma unroll
  for (int w = 0; w < W; ++w) {
    e1A[w] = P.e1[(int64_t)A * W + w]; e2A[w] = P.e2[(int64_t)A * W + w];
    e1B[w] = P.e1[(int64_t)B * W + w]; e2B[w] = P.e2[(int64_t)B * W + w];
    im1[w] = e1A[w] & ~e1B[w]; im2[w] = e2A[w] & ~e2B[w];
    jm1[w] = e1B[w] & ~e1A[w]; jm2[w] = e2B[w] & ~e2A[w];
    pi.SA[w] = e1A[w] & ~e2A[w];
  }
  pi.iex0 = pi.iex1 = pi.jex0 = pi.jex1 = -1;
  const int ni = popc_w<W>(im1) + popc_w<W>(im2);
  const int nj = popc_w<W>(jm1) + popc_w<W>(jm2);
  if (A == B) { pi.kind = K_DIAG; return; }
  if (ni == 1 && nj == 1) {
    uint64_t im[W], jm[W];
#pragma unroll
    for (int w = 0; w < W; ++w) { im[w] = im1[w] | im2[w]; jm[w] = jm1[w] | jm2[w]; }
    const int ie = lowest_bit<W>(im), je = lowest_bit<W>(jm);
    pi.iex0 = ie; pi.jex0 = je;
    between_mask<W>(ie, je, pi.bm[0]);
    range_mask<W>(0, ie - 1, pi.bm[1]);
    range_mask<W>(je + 1, 64 * W - 1, pi.bm[2]);
    range_mask<W>(0, je - 1, pi.bm[3]);
    range_mask<W>(ie + 1, 64 * W - 1, pi.bm[4]);
    pi.kind = (pi.jsA != pi.jsB) ? K_SO : K_SINGLE;
    return;
  }
  if (ni == 2 && nj == 2) {
    int ex0 = -1, ex1 = -1, jy0 = -1, jy1 = -1;
    two_positions<W>(im1, im2, ex0, ex1);
    two_positions<W>(jm1, jm2, jy0, jy1);
    pi.iex0 = ex0; pi.iex1 = ex1; pi.jex0 = jy0; pi.jex1 = jy1;
    between_mask<W>(ex0, jy0, pi.bm[0]);
    between_mask<W>(ex0, jy1, pi.bm[1]);
    between_mask<W>(ex1, jy0, pi.bm[2]);
    between_mask<W>(ex1, jy1, pi.bm[3]);
    between_mask<W>(ex0, ex1, pi.bm[4]);
    between_mask<W>(jy0, jy1, pi.bm[5]);
    pi.kind = K_DOUBLE;
    return;
  }
  pi.kind = K_NONE;
}

// rank of orbital p among the set bits of S (p must be set in S for a meaningful rank)
template <int W>
__device__ __forceinline__ int rank_in(const uint64_t (&S)[W], int p) {
  int r = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    if (64 * w + 63 < p) r += __popcll(S[w]);
    else if (64 * w <= p) r += __popcll(S[w] & ((1ull << (p & 63)) - 1ull));
  }
  return r;
}

// det_elem's branches, returning what the element is made of instead of its value:
// tag T_V0 / T_V1 / T_V0MV1 (+-v0, +-v1, +-(v0 - v1)); T_SGL: +-(v0 - sum of X[t] over the
// bits of mask); T_X: +-X[term]; T_DIAG: Kd[0] - sum of Kd[mm] over the bits mm of mask;
// T_K: +-Kd[term]; T_DIRECT: +-eri[direct]; T_NONE: zero.  sgn = +1 / -1.
template <int W>
__device__ __forceinline__ int det_adj(const AdjPair<W> &pi, const DetBits<W> &A, const DetBits<W> &B, int &sgn,
                                       uint64_t &mask, int &term, int64_t &direct) {
  const uint64_t(&aa)[W] = A.al;
  const uint64_t(&ba)[W] = A.be;
  const uint64_t(&ab)[W] = B.al;
  const uint64_t(&bb)[W] = B.be;
  const int pha = A.ph, phb = B.ph, naa = A.na, nab = B.na;
  uint64_t ua[W], ub[W];
#pragma unroll
  for (int w = 0; w < W; ++w) { ua[w] = ab[w] & ~aa[w]; ub[w] = bb[w] & ~ba[w]; }
  const int nmarka = popc_w<W>(ua);
  const int nmarkb = nmarka + popc_w<W>(ub);
  const int ie = pi.iex0, je = pi.jex0;
  sgn = 1;
  if (pi.kind == K_NONE) return T_NONE;
  if (pi.kind == K_SO) {
    if (nmarka > 1 || nmarkb > 1) return T_NONE;
    int ncount = pha + phb;
    if (naa < nab) {
      ncount += popc_and<W>(ba, pi.bm[1]) + popc_and<W>(ab, pi.bm[2]);
      if ((pi.jsA + pi.jsB) % 2 == 0) ++ncount;
      else if (pi.jsA % 2 == 1) ++ncount;
    } else if (naa > nab) {
      ncount += popc_and<W>(aa, pi.bm[4]) + popc_and<W>(bb, pi.bm[3]);
      if ((pi.jsA + pi.jsB) % 2 != 0 && (pi.jsA % 2) == 1) ++ncount;
    } else {
      if (nmarka == 0) ++ncount;
      if (pi.jsA % 2 == 1) ++ncount;
      uint64_t sp[W];
      sel_w<W>(sp, nmarka != 0, aa, ba);
      ncount += popc_and<W>(sp, pi.bm[0]);
    }
    sgn = (ncount & 1) ? -1 : 1;
    return T_V0;
  }
  if (naa != nab) return T_NONE;
  if (nmarka > 2 || nmarkb > 2) return T_NONE;
  if (nmarkb == 0) {
    if (pi.kind != K_DIAG) return T_NONE;
    // diag_det_elem: Kd[0] minus Kd[mm] for every pair of open shells with equal spins
    mask = 0ull;
    int mm = 0, io = 0;
#pragma unroll
    for (int wi = 0; wi < W; ++wi) {
      uint64_t si_bits = pi.SA[wi];
      while (si_bits) {
        const uint64_t lo_i = si_bits & (~si_bits + 1);
        si_bits ^= lo_i;
        const bool si = (aa[wi] & lo_i) != 0ull;
        int jo = 0;
#pragma unroll
        for (int wj = 0; wj < W; ++wj) {
          uint64_t sj = pi.SA[wj];
          while (sj && jo < io) {
            const uint64_t lo_j = sj & (~sj + 1);
            sj ^= lo_j;
            ++mm;
            if (si == ((aa[wj] & lo_j) != 0ull)) mask |= 1ull << (mm - 1);
            ++jo;
          }
        }
        ++io;
      }
    }
    return T_DIAG;
  }
  if (nmarkb == 1) {
    if (pi.kind != K_SINGLE) return T_NONE;
    uint64_t sp[W];
    sel_w<W>(sp, nmarka != 0, aa, ba);
    const int ncount = pha + phb + popc_and<W>(sp, pi.bm[0]);
    mask = 0ull;
    int t = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      uint64_t m = sp[w] & ~(aa[w] & ba[w]);
      if ((ie >> 6) == w) m &= ~(1ull << (ie & 63));
      if ((je >> 6) == w) m &= ~(1ull << (je & 63));
      uint64_t sa = pi.SA[w];
      while (sa) {
        const uint64_t low = sa & (~sa + 1);
        if (m & low) mask |= 1ull << t;
        ++t;
        sa ^= low;
      }
    }
    sgn = (ncount & 1) ? -1 : 1;
    return T_SGL;
  }
  if (nmarka == 1) {
    uint64_t xa[W], xb[W];
#pragma unroll
    for (int w = 0; w < W; ++w) { xa[w] = aa[w] & ~ab[w]; xb[w] = ba[w] & ~bb[w]; }
    if (pi.kind == K_DOUBLE) {
      const int ia = bit_w<W>(xa, pi.iex0) ? 0 : 1, ja = bit_w<W>(ua, pi.jex0) ? 0 : 1;
      const int ncount = pha + phb + popc_and<W>(aa, pi.bm[2 * ia + ja]) + popc_and<W>(ba, pi.bm[3 - 2 * ia - ja]);
      sgn = (ncount & 1) ? -1 : 1;
      return (ia == ja) ? T_V0 : T_V1;
    }
    if (pi.kind != K_SINGLE && pi.kind != K_DIAG) return T_NONE;
    const int iex2 = lowest_bit<W>(ua), jex2 = lowest_bit<W>(ub);
    const int iex3 = lowest_bit<W>(xa), jex3 = lowest_bit<W>(xb);
    int ncount = pha + phb;
    if (abs(iex2 - iex3) > 1) ncount += popc_range<W>(aa, min(iex2, iex3) + 1, max(iex2, iex3) - 1);
    if (abs(jex2 - jex3) > 1) ncount += popc_range<W>(ba, min(jex2, jex3) + 1, max(jex2, jex3) - 1);
    sgn = (ncount & 1) ? -1 : 1;
    direct = canon4(jex2, jex3, iex2, iex3);
    if (pi.kind == K_SINGLE) {
      // alpha and beta moves through an open shell p of A: the integral is X[rank of p]
      const int p = (iex3 == ie || iex3 == je) ? iex2 : iex3;
      if (bit_w<W>(pi.SA, p) && canon4(ie, p, p, je) == direct) {
        term = rank_in<W>(pi.SA, p);
        return T_X;
      }
      return T_DIRECT;
    }
    // diagonal: a spin exchange between two open shells p and q, the integral Kd[mm(p, q)]
    const int p = iex3, q = iex2;
    if (bit_w<W>(pi.SA, p) && bit_w<W>(pi.SA, q) && canon4(p, q, q, p) == direct) {
      const int rp = rank_in<W>(pi.SA, p), rq = rank_in<W>(pi.SA, q);
      const int a = max(rp, rq), b = min(rp, rq);
      term = a * (a - 1) / 2 + b;  // Kd[1 + term] in diag_det_elem's order
      return T_K;
    }
    return T_DIRECT;
  }
  if (pi.kind != K_DOUBLE) return T_NONE;
  uint64_t spb[W], sa[W];
  sel_w<W>(spb, nmarka == 2, ab, bb);
  sel_w<W>(sa, nmarka != 0, aa, ba);
  const int ncount = pha + phb + popc_and<W>(spb, pi.bm[5]) + popc_and<W>(sa, pi.bm[4]);
  sgn = (ncount & 1) ? -1 : 1;
  return T_V0MV1;
}

// vectors (k per pass, root-major with stride ldv, FP64) in the determinant basis:
// CD[d * k + r], the transpose of ciout's transform (PsociHamiltonian.C:1457-1516)
template <typename CT>
__global__ void k_sef_to_det(int nconf, int nelec, int ksym, const int64_t *__restrict__ sefoff,
                             const int64_t *__restrict__ detoff, const int32_t *__restrict__ jsym,
                             const int32_t *__restrict__ nopen, const double *__restrict__ V, int64_t ldv, int k,
                             CT *__restrict__ CD) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int i = (int)(t >> 5), lane = threadIdx.x & 31;
  if (i >= nconf) return;
  const int64_t s0 = sefoff[i], d0 = detoff[i];
  const int nsef = (int)(sefoff[i + 1] - s0);
  const bool odd = nelec & 1;
  const bool open = !odd && nopen[i] != 0;
  const double m = (jsym[i] % 2 != ksym % 2) ? -1.0 : 1.0;
  const double r = sqrt(0.5);
  for (int e = lane; e < nsef * k; e += 32) {
    const int a = e / k, q = e - a * k;
    const double c = V[(int64_t)q * ldv + s0 + a];
    if (open) {
      CD[(d0 + 2 * a) * k + q] = (CT)(r * c);
      CD[(d0 + 2 * a + 1) * k + q] = (CT)((m * r) * c);
    } else {
      CD[(d0 + a) * k + q] = (CT)c;
    }
  }
}

template <int W>
struct AdjSmem {
  AdjPair<W> pi[32];
  double acc[ADJ_NT][ADJ_MAXR];
};

// scatter of one pair's terms into the gradient tables G1 [k][n1], G2 [k][n2] (FP64 atomics);
// f = 2 for J < I, 1 on the diagonal.  Lanes split the roots and entries.
template <int W>
__device__ void adj_scatter(const Params &P, const AdjPair<W> &pi, const double (&acc)[ADJ_NT][ADJ_MAXR], int k,
                            double f, double *G1, int64_t n1, double *G2, int64_t n2, int lane) {
  const int A = pi.A;
  if (pi.kind == K_DOUBLE) {
    if (lane < k) {
      atomicAdd(G2 + lane * n2 + canon4(pi.iex0, pi.jex0, pi.iex1, pi.jex1), f * acc[0][lane]);
      atomicAdd(G2 + lane * n2 + canon4(pi.iex0, pi.jex1, pi.iex1, pi.jex0), f * acc[1][lane]);
    }
    return;
  }
  if (pi.kind == K_SO) {
    // v = +-SO(ie, je) / 2, negated when je > ie (processSingleExcitation, PsociHamiltonian.C:223-237)
    if (lane < k) atomicAdd(G1 + lane * n1 + tri64(pi.iex0, pi.jex0), f * (pi.jex0 > pi.iex0 ? -0.5 : 0.5) * acc[0][lane]);
    return;
  }
  uint64_t e1A[W], e2A[W], e2B[W];
#pragma unroll
  for (int w = 0; w < W; ++w) {
    e1A[w] = P.e1[(int64_t)A * W + w]; e2A[w] = P.e2[(int64_t)A * W + w];
    e2B[w] = P.e2[(int64_t)pi.B * W + w];
  }
  if (pi.kind == K_SINGLE) {
    const int ie = pi.iex0, je = pi.jex0;
    // lanes over (root, entry): entry 0 one[ie, je], 1 (ie je|ie ie), 2.. the occupied p,
    // then the X[t] terms
    for (int r = 0; r < k; ++r) {
      const double a0 = f * acc[0][r];
      if (lane == 0) {
        atomicAdd(G1 + r * n1 + tri64(ie, je), a0);
        atomicAdd(G2 + r * n2 + canon4(ie, je, ie, ie), -a0);
      }
      // sum over the occupied orbitals p of A: (ie je|p p) x occ_A(p), and -(ie p|p je) where
      // p is doubly occupied in both
      int pidx = 0;
#pragma unroll
      for (int w = 0; w < W; ++w) {
        uint64_t o = e1A[w];
        while (o) {
          const int p = 64 * w + __ffsll((long long)o) - 1;
          o &= o - 1;
          if ((pidx & 31) == lane) {
            const bool dA = bit_w<W>(e2A, p);
            atomicAdd(G2 + r * n2 + canon4(ie, je, p, p), dA ? 2.0 * a0 : a0);
            if (dA && bit_w<W>(e2B, p)) atomicAdd(G2 + r * n2 + canon4(ie, p, p, je), -a0);
          }
          ++pidx;
        }
      }
      int t = 0;
#pragma unroll
      for (int w = 0; w < W; ++w) {
        uint64_t sa = pi.SA[w];
        while (sa) {
          const int p = 64 * w + __ffsll((long long)sa) - 1;
          sa &= sa - 1;
          if ((t & 31) == lane && acc[2 + t][r] != 0.0) atomicAdd(G2 + r * n2 + canon4(ie, p, p, je), f * acc[2 + t][r]);
          ++t;
        }
      }
    }
    return;
  }
  if (pi.kind == K_DIAG) {
    // Kd[0] = sum over occupied ib of occ h_ii (+ (ii|ii) if doubly) and over pairs jb < ib of
    // Coulomb and exchange terms (processDiagExcitation, PsociHamiltonian.C:306-388); lanes
    // over ib
    for (int r = 0; r < k; ++r) {
      const double a0 = f * acc[0][r];
      int iidx = 0;
#pragma unroll
      for (int wi = 0; wi < W; ++wi) {
        uint64_t oi = e1A[wi];
        while (oi) {
          const int ib = 64 * wi + __ffsll((long long)oi) - 1;
          oi &= oi - 1;
          if ((iidx & 31) == lane) {
            const int occi = 1 + (int)bit_w<W>(e2A, ib);
            if (occi == 1) atomicAdd(G1 + r * n1 + tri64(ib, ib), a0);
            else {
              atomicAdd(G1 + r * n1 + tri64(ib, ib), 2.0 * a0);
              atomicAdd(G2 + r * n2 + canon4(ib, ib, ib, ib), a0);
            }
#pragma unroll
            for (int wj = 0; wj < W; ++wj) {
              uint64_t oj = e1A[wj];
              while (oj) {
                const int jb = 64 * wj + __ffsll((long long)oj) - 1;
                oj &= oj - 1;
                if (jb >= ib) break;
                const int ninj = occi * (1 + (int)bit_w<W>(e2A, jb));
                if (ninj == 1) atomicAdd(G2 + r * n2 + canon4(ib, ib, jb, jb), a0);
                else {
                  const double m = (ninj == 2) ? 1.0 : 2.0;
                  atomicAdd(G2 + r * n2 + canon4(ib, ib, jb, jb), 2.0 * m * a0);
                  atomicAdd(G2 + r * n2 + canon4(ib, jb, ib, jb), -m * a0);
                }
              }
            }
          }
          ++iidx;
        }
      }
      // Kd[mm] = (s_a s_b|s_b s_a) over the open shells a > b, in that order
      int sing[PSOCI_MAX_OPEN], ns = 0;
#pragma unroll
      for (int w = 0; w < W; ++w) {
        uint64_t sb = pi.SA[w];
        while (sb && ns < PSOCI_MAX_OPEN) { sing[ns++] = 64 * w + __ffsll((long long)sb) - 1; sb &= sb - 1; }
      }
      int mm = 0;
      for (int a = 1; a < ns; ++a)
        for (int b = 0; b < a; ++b, ++mm)
          if ((mm & 31) == lane && acc[2 + mm][r] != 0.0)
            atomicAdd(G2 + r * n2 + canon4(sing[a], sing[b], sing[b], sing[a]), f * acc[2 + mm][r]);
    }
  }
}

// Whether determinants A and B of the pair can couple (det_adj's early exits): a cheap
// first pass, so that the classification runs on the coupled pairs only.
template <int W>
__device__ __forceinline__ bool det_coupled(const AdjPair<W> &pi, const DetBits<W> &A, const DetBits<W> &B) {
  int na = 0, nb = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) { na += __popcll(B.al[w] & ~A.al[w]); nb += __popcll(B.be[w] & ~A.be[w]); }
  if (pi.kind == K_SO) return na <= 1 && na + nb <= 1;
  if (A.na != B.na || na + nb > 2) return false;
  if (na + nb == 0) return pi.kind == K_DIAG;
  if (na + nb == 1) return pi.kind == K_SINGLE;
  if (na == 1) return pi.kind != K_NONE;
  return pi.kind == K_DOUBLE;
}

constexpr int ADJ_RT = 15;    // exchange terms held in registers (Kd[mm] of <= 6 open shells)
constexpr int ADJ_CONN = 128; // coupled determinant pairs collected per round

// A coupled determinant pair of the pair being processed, classified: its determinants
// (x << 16 | y), the det_adj tag, sign and term, and the exchange-term mask.
struct AdjRec {
  uint64_t mask;
  uint32_t xy;
  int32_t info;  // tag | (sgn < 0) << 4 | term << 8
};

// One warp per row configuration I (grid-stride); its lower neighbours J <= I in chunks of 32
// set up by the lanes.  Per pair: (1) lanes over the determinant pairs (x, y) test them for
// coupling and classify the coupled ones (det_adj), collecting the records in shared memory;
// (2) lanes = (slot, root) take the records, slots over the records and roots over the lanes
// of a slot, and add s * cd_I[x] * cd_J[y] to register accumulators of the pair's terms (v0,
// v1, and the exchange terms X[t] / Kd[mm]; terms beyond ADJ_RT, only on diagonals of 7+ open
// shells, go to shared-memory atomics); (3) the slots' sums are reduced by shuffles and the
// root lanes scatter the pair's terms to the tables.  CT/ACC: the type of the determinant-
// basis vectors and of the sums within a pair (FP64, or FP32 for the FP32-bulk variant).
template <int W, typename CT, typename ACC>
__global__ void __launch_bounds__(ADJ_WARPS * 32) k_energy_grad(Params P, const int64_t *__restrict__ nbroff,
                                                                const int32_t *__restrict__ nbr,
                                                                const CT *__restrict__ CD, int k, double *G1,
                                                                int64_t n1, double *G2, int64_t n2) {
  __shared__ AdjSmem<W> sm[ADJ_WARPS];
  __shared__ AdjRec recs[ADJ_WARPS][ADJ_CONN];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  AdjSmem<W> &S = sm[wib];
  AdjRec *rec = recs[wib];
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  // lanes of one slot hold consecutive roots: kp (a power of two >= k) roots per slot
  const int kp = (k <= 1) ? 1 : (k <= 2) ? 2 : (k <= 4) ? 4 : 8;
  const int nslot = 32 / kp, slot = lane / kp, r = lane % kp;
  const bool rok = r < k;
  for (int e = lane; e < ADJ_NT * ADJ_MAXR; e += 32) (&S.acc[0][0])[e] = 0.0;
  __syncwarp();
  for (int64_t I = warp; I < P.nconf; I += nwarps) {
    const int64_t b0 = nbroff[I], b1 = nbroff[I + 1];
    for (int64_t c0 = b0; c0 < b1; c0 += 32) {
      const int64_t q = c0 + lane;
      const int J = (q < b1) ? nbr[q] : INT_MAX;
      const bool lower = J <= (int)I;
      if (lower) adj_pair_setup<W>(P, (int)I, J, S.pi[lane]);
      const unsigned lm = __ballot_sync(0xffffffffu, lower);
      __syncwarp();
      const int np = __popc(lm);  // lower pairs come first within the chunk
      for (int u = 0; u < np; ++u) {
        const AdjPair<W> &pi = S.pi[u];
        if (pi.kind == K_NONE) continue;
        const double fpair = (pi.A == pi.B) ? 1.0 : 2.0;
        const int nterm = (pi.kind == K_SINGLE) ? pi.nopenA
                          : (pi.kind == K_DIAG) ? min(ADJ_RT, pi.nopenA * (pi.nopenA - 1) / 2) : 0;
        ACC a0 = 0, a1 = 0, aT[ADJ_RT];
#pragma unroll
        for (int t = 0; t < ADJ_RT; ++t) aT[t] = 0;
        const int nd = pi.ndetA * pi.ndetB;
        for (int e0 = 0; e0 < nd;) {
          // (1) classify the determinant pairs, one a lane; keep the coupled ones
          int nc = 0;
          while (e0 < nd && nc + 32 <= ADJ_CONN) {
            const int e = e0 + lane;
            int tag = T_NONE, sgn = 1, term = 0, x = 0, y = 0;
            uint64_t mask = 0ull;
            if (e < nd) {
              x = e / pi.ndetB;
              y = e - x * pi.ndetB;
              DetBits<W> Ad, Bd;
              load_det<W>(Ad, P.alpha, P.beta, P.phase, P.nalpha, pi.detA + x);
              load_det<W>(Bd, P.alpha, P.beta, P.phase, P.nalpha, pi.detB + y);
              if (det_coupled<W>(pi, Ad, Bd)) {
                int64_t direct = 0;
                tag = det_adj<W>(pi, Ad, Bd, sgn, mask, term, direct);
                if (tag == T_DIRECT) {
                  // an integral outside the pair's terms (not met in practice): added here
                  for (int rr = 0; rr < k; ++rr)
                    atomicAdd(G2 + (int64_t)rr * n2 + direct,
                              fpair * sgn * (double)CD[(pi.detA + x) * k + rr] * (double)CD[(pi.detB + y) * k + rr]);
                  tag = T_NONE;
                }
              }
            }
            const bool keep = tag != T_NONE;
            const unsigned cb = __ballot_sync(0xffffffffu, keep);
            if (keep) {
              AdjRec &R = rec[nc + __popc(cb & ((1u << lane) - 1u))];
              R.mask = mask;
              R.xy = ((uint32_t)x << 16) | (uint32_t)y;
              R.info = tag | ((sgn < 0) ? 16 : 0) | (term << 8);
            }
            nc += __popc(cb);
            e0 += 32;
          }
          __syncwarp();
          // (2) accumulate, slots over the records, roots over the lanes of a slot
          if (rok) {
            for (int cq = slot; cq < nc; cq += nslot) {
              const AdjRec R = rec[cq];
              const int x = (int)(R.xy >> 16), y = (int)(R.xy & 0xffffu);
              const int tag = R.info & 15, term = R.info >> 8;
              ACC w = (ACC)__ldg(CD + (pi.detA + x) * k + r) * (ACC)__ldg(CD + (pi.detB + y) * k + r);
              if (R.info & 16) w = -w;
              if (tag == T_V0) a0 += w;
              else if (tag == T_V1) a1 += w;
              else if (tag == T_V0MV1) { a0 += w; a1 -= w; }
              else if (tag == T_SGL || tag == T_DIAG) {
                a0 += w;
#pragma unroll
                for (int t = 0; t < ADJ_RT; ++t) {
                  if (t >= nterm) break;  // uniform over the warp
                  if ((R.mask >> t) & 1ull) aT[t] -= w;
                }
                uint64_t m = R.mask >> ADJ_RT;
                while (m) {
                  const int t = ADJ_RT + __ffsll((long long)m) - 1;
                  m &= m - 1;
                  atomicAdd(&S.acc[2 + t][r], -(double)w);
                }
              } else {  // T_X, T_K
                if (term < ADJ_RT) {
#pragma unroll
                  for (int t = 0; t < ADJ_RT; ++t) {
                    if (t >= nterm) break;
                    if (t == term) aT[t] += w;
                  }
                } else {
                  atomicAdd(&S.acc[2 + term][r], (double)w);
                }
              }
            }
          }
          __syncwarp();
        }
        // (3) sums over the slots (lanes r, r + kp, r + 2kp, ...): lanes of slot 0 hold them
        double s0 = (double)a0, s1 = (double)a1, sT[ADJ_RT];
#pragma unroll
        for (int t = 0; t < ADJ_RT; ++t) sT[t] = (double)aT[t];
        for (int o = kp; o < 32; o <<= 1) {
          s0 += __shfl_xor_sync(0xffffffffu, s0, o);
          s1 += __shfl_xor_sync(0xffffffffu, s1, o);
#pragma unroll
          for (int t = 0; t < ADJ_RT; ++t)
            if (t < nterm) sT[t] += __shfl_xor_sync(0xffffffffu, sT[t], o);
        }
        __syncwarp();  // the shared-memory terms (spilled atomics) are complete
        if (lane < k) {
          S.acc[0][lane] = s0;
          S.acc[1][lane] = s1;
#pragma unroll
          for (int t = 0; t < ADJ_RT; ++t)
            if (t < nterm) S.acc[2 + t][lane] = sT[t];
        }
        __syncwarp();
        adj_scatter<W>(P, pi, S.acc, k, fpair, G1, n1, G2, n2, lane);
        __syncwarp();
        const int used = 2 + ((pi.kind == K_DIAG) ? pi.nopenA * (pi.nopenA - 1) / 2 : pi.nopenA);
        for (int e = lane; e < used * ADJ_MAXR; e += 32) (&S.acc[0][0])[e] = 0.0;
        __syncwarp();
      }
      __syncwarp();
      if (np < 32) break;  // past the diagonal
    }
  }
}

// ------------------------------------------------------------------------------------
// The same from coupling tables (at most TAB_MAXOPEN open shells), pairs J < I and diagonal
// blocks apart.
// ------------------------------------------------------------------------------------
// vectors (k per pass, root-major with stride ldv) side by side, KP a SEF (zero padded)
template <int KP>
__global__ void k_grad_rows(int64_t n, const double *__restrict__ V, int64_t ldv, int k, double *__restrict__ C) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int q = 0; q < KP; ++q) C[i * KP + q] = q < k ? V[(int64_t)q * ldv + i] : 0.0;
  }
}

// G[q * n + i] = T[i * KP + q], zero where tab is (with tab).  Bound by memory: of 13.8 M integrals (102
// orbitals) and 8 roots T is cleared and read and G written once.  The gradient of 203 SEFs takes
// 0.57 ms, 0.53 with tab (with G cleared, added to and masked apart 0.89 and 1.29).
template <int KP>
__global__ void k_grad_out(int64_t n, int k, const double *__restrict__ T, const double *__restrict__ tab,
                           double *__restrict__ G) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const bool zero = tab && tab[i] == 0.0;
#pragma unroll
    for (int q = 0; q < KP; ++q)
      if (q < k) G[(int64_t)q * n + i] = zero ? 0.0 : T[i * KP + q];
  }
}

__device__ __forceinline__ double with_sign(double v, uint32_t x) { return flip_sign(v, x & 0x80000000u); }

constexpr int GT_WARPS = 4;
struct GradPair {
  double f;          // sign, 2 (the pair's two places in H) and the pattern's constants
  uint32_t prog;     // its program: first word
  int lists, kind;
  int ie, je, ex1, jy1;
  uint32_t sefJ;
  int B;
};

// One warp per configuration, 32 lower pairs set up at a time, KP lanes (a root each) to a pair:
// the lists of its table's program give one sum of products c_I[row] c_J[column] an integral,
// which goes to that integral's place in the gradient.  The sums are FP64
// and the places take FP64 atomics, the KP roots of one side by side (T1, T2:
// KP a table entry).  Bound by the FP64 pipe, one FMA an entry of a list (16 clocks a warp
// instruction an SM, whatever its active lanes): mrcisd_6e8o_v16, 8 roots, 2.5 ms (3.2 with the
// pairs in their lists' order, 19 of 32 lanes active; determinant pair by determinant pair the lower
// blocks took 52 ms).
template <int W, int KP>
__global__ void __launch_bounds__(GT_WARPS * 32) k_grad_tab(Params P, const CfgRec<W> *__restrict__ cfg,
                                                            const int64_t *__restrict__ nbroff,
                                                            const int32_t *__restrict__ nbr,
                                                            const uint32_t *__restrict__ slot,
                                                            const uint4 *__restrict__ hdr,
                                                            const uint32_t *__restrict__ pool,
                                                            const double *__restrict__ C, double *T1, double *T2) {
  __shared__ GradPair pairs[GT_WARPS][PSOCI_SEG];
  GradPair *gp = pairs[threadIdx.x >> 5];
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, q = lane % KP, grp = lane / KP;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t I = warp; I < P.nconf; I += nwarps) {
    const CfgRec<W> a = cfg[I];
    const double *cI = C + (int64_t)a.sef * KP + q;
    const int64_t b1 = nbroff[I + 1];
    for (int64_t k0 = nbroff[I]; k0 < b1; k0 += 32) {
      const int J = (k0 + lane < b1) ? nbr[k0 + lane] : INT_MAX;
      const bool low = J < (int)I;
      const int np = __popc(__ballot_sync(FULL, low));  // they come first
      if (np == 0) break;
      uint32_t key = 0xffffffe0u | lane;
      GradPair g;
      if (low) {
        const CfgRec<W> b = cfg[J];
        const PairShape s = pair_shape<W>(a, b);
        g.kind = s.kind;
        g.ie = s.ex0; g.je = s.jy0; g.ex1 = s.ex1; g.jy1 = s.jy1;
        g.sefJ = b.sef;
        g.B = J;
        g.lists = 0;
        g.prog = 0;
        uint32_t len = 0;
        const uint32_t sl = slot[k0 + lane];
        if (sl != TAB_NONE) {
          const uint4 h0 = __ldg(hdr + 2 * (size_t)(sl & TAB_SLOT)), h1 = __ldg(hdr + 2 * (size_t)(sl & TAB_SLOT) + 1);
          g.prog = h1.x;
          g.lists = (int)h1.y;
          g.f = tab_scale(s.sign ? -2.0 : 2.0, h0.y);
          if (g.lists > 0) len = __ldg(reinterpret_cast<const uint16_t *>(pool + g.prog) + g.lists - 1);
        }
        key = ((uint32_t)(s.kind & 3) << 30) | (min(len, 1023u) << 20) | ((g.prog & 0x7fffu) << 5) | lane;
      }
      // pairs of one kind and similar programs go together: a warp's groups take as long as the longest
      int rank = 0;
#pragma unroll
      for (int j = 0; j < 32; ++j) rank += __shfl_sync(FULL, key, j) < key;
      if (low) gp[rank] = g;
      __syncwarp();
      for (int u = grp; u < np; u += 32 / KP) {
        const GradPair &g = gp[u];
        const double *cJ = C + (int64_t)g.sefJ * KP + q;
        const uint16_t *ends = reinterpret_cast<const uint16_t *>(pool + g.prog);
        const uint32_t *pw = pool + g.prog + (TAB_LISTS + 1) / 2;
        int e = 0;
        for (int l = 0; l < g.lists; ++l) {
          const int end = (int)__ldg(ends + l);
          if (e == end) continue;
          double sum = 0;
          for (; e + 2 <= end; e += 2) {
            const uint32_t x0 = __ldg(pw + e), x1 = __ldg(pw + e + 1);
            const double i0 = __ldg(cI + (int)((x0 >> 8) & 0xffu) * KP), i1 = __ldg(cI + (int)((x1 >> 8) & 0xffu) * KP);
            const double j0 = __ldg(cJ + (int)(x0 & 0xffu) * KP), j1 = __ldg(cJ + (int)(x1 & 0xffu) * KP);
            sum = fma(with_sign(i0, x0), j0, sum);
            sum = fma(with_sign(i1, x1), j1, sum);
          }
          if (e < end) {
            const uint32_t x0 = __ldg(pw + e);
            sum = fma(with_sign(__ldg(cI + (int)((x0 >> 8) & 0xffu) * KP), x0), __ldg(cJ + (int)(x0 & 0xffu) * KP), sum);
            ++e;
          }
          const double w = g.f * sum;
          if (g.kind == K_DOUBLE) {
            atomicAdd(T2 + (l == 0 ? canon4(g.ie, g.je, g.ex1, g.jy1) : canon4(g.ie, g.jy1, g.ex1, g.je)) * KP + q, w);
          } else if (g.kind == K_SO) {
            // v = +-SO(ie, je) / 2, negated when je > ie (PsociHamiltonian.C:223-237)
            atomicAdd(T1 + tri64(g.ie, g.je) * KP + q, flip_sign(0.5 * w, g.je > g.ie ? 0x80000000u : 0u));
          } else if (l > 0) {  // X[l - 1]
            int t = l - 1, o = 0;
#pragma unroll
            for (int x = 0; x < W; ++x) {
              uint64_t m = a.e1[x] & ~a.e2[x];
              const int n = __popcll(m);
              if (t >= 0 && t < n) {
                for (; t > 0; --t) m &= m - 1;
                o = 64 * x + __ffsll((long long)m) - 1;
                t = -1;
              } else {
                t -= n;
              }
            }
            atomicAdd(T2 + canon4(g.ie, o, o, g.je) * KP + q, w);
          } else {
            // v0 = h(ie, je) - (ie je|ie ie) + sum over A's occupied p of occ (ie je|p p) less
            // (ie p|p je) where p is doubly occupied in both (PsociHamiltonian.C:239-258)
            atomicAdd(T1 + tri64(g.ie, g.je) * KP + q, w);
            const double w2 = w + w, nw = flip_sign(w, 0x80000000u);
            atomicAdd(T2 + canon4(g.ie, g.je, g.ie, g.ie) * KP + q, nw);
#pragma unroll
            for (int x = 0; x < W; ++x) {
              uint64_t m = a.e1[x];
              const uint64_t both = a.e2[x] & __ldg(&cfg[g.B].e2[x]);
              while (m) {
                const int bit = __ffsll((long long)m) - 1, o = 64 * x + bit;
                m &= m - 1;
                atomicAdd(T2 + canon4(g.ie, g.je, o, o) * KP + q, ((a.e2[x] >> bit) & 1ull) ? w2 : w);
                if ((both >> bit) & 1ull) atomicAdd(T2 + canon4(g.ie, o, o, g.je) * KP + q, nw);
              }
            }
          }
        }
      }
      __syncwarp();
      if (np < 32) break;
    }
  }
}

// Diagonal blocks.  The determinants of a configuration are spin patterns of its open shells, and two
// of them couple only by exchanging the spins of two shells a > b, with the sign of their phases and
// of the a - b - 1 shells between.  So with c' the coefficients times their phases the integral
// (ab|ba) gets, over the patterns x of equal spins in a and b and the pairs x, y that differ by the
// exchange (PsociHamiltonian.C:306-388),
//   -sum c'x^2 + sum 2 s c'x c'y = -sum over all of c'x^2 + sum over the pairs of (c'x + s c'y)^2 ,
// 2^(n-2) squares instead of a test of every determinant with every other.  One warp a configuration,
// KP lanes (a root each) to a shell pair or an integral.  Of 2.4 ms at mrcisd_6e8o_v16, 8 roots,
// 0.14 ms remain.
template <int W, int KP>
__global__ void __launch_bounds__(GT_WARPS * 32) k_grad_diag(Params P, const double *__restrict__ C, double *T1, double *T2) {
  // of a spin pattern: SEF in the block, bit 15 the sign of c'; NO_DET without a determinant
  __shared__ uint16_t maps[GT_WARPS][1 << TAB_MAXOPEN];
  constexpr unsigned FULL = 0xffffffffu, NO_DET = 0x7fffu;
  uint16_t *map = maps[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31, q = lane % KP, grp = lane / KP, ngrp = 32 / KP;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t I = warp; I < P.nconf; I += nwarps) {
    uint64_t o1[W], o2[W], so[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      o1[w] = P.e1[I * W + w];
      o2[w] = P.e2[I * W + w];
      so[w] = o1[w] & ~o2[w];
    }
    auto nth = [](const uint64_t(&x)[W], int p) {  // the p-th lowest set bit of x
#pragma unroll
      for (int w = 0; w < W; ++w) {
        uint64_t u = x[w];
        const int c = __popcll(u);
        if (p < c) {
          for (; p > 0; --p) u &= u - 1;
          return 64 * w + __ffsll((long long)u) - 1;
        }
        p -= c;
      }
      return 0;
    };
    const int nop = popc_w<W>(so), nocc = popc_w<W>(o1);
    const int64_t s0 = P.sefoff[I], d0 = P.detoff[I];
    const int nsef = (int)(P.sefoff[I + 1] - s0), ndet = (int)(P.detoff[I + 1] - d0);
    const bool open2 = !(P.nelec & 1) && nop != 0;
    const bool flip = open2 && P.jsym[I] % 2 != P.ksym % 2;  // second determinants with the other sign
    const double *c = C + s0 * KP + q;
    for (int m = lane; m < 1 << nop; m += 32) map[m] = NO_DET;
    __syncwarp();
    if (nop > 1)
      for (int d = lane; d < ndet; d += 32) {
        int m = 0, b = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const uint64_t al = P.alpha[(d0 + d) * W + w];
          for (uint64_t u = so[w]; u; u &= u - 1, ++b) m |= (int)((al >> (__ffsll((long long)u) - 1)) & 1ull) << b;
        }
        const int neg = (P.phase[d0 + d] & 1) ^ (int)(flip && (d & 1));
        map[m] = (uint16_t)((open2 ? d >> 1 : d) | (neg << 15));
      }
    __syncwarp();
    double n0 = 0;
    for (int s = grp; s < nsef; s += ngrp) {
      const double v = __ldg(c + s * KP);
      n0 = fma(v, v, n0);
    }
    double a0 = n0;
#pragma unroll
    for (int o = KP; o < 32; o <<= 1) a0 += __shfl_xor_sync(FULL, a0, o);
    // exchange integrals of the open-shell pairs
    for (int mm = grp; mm < nop * (nop - 1) / 2; mm += ngrp) {
      int a = 1, b = mm;
      while (b >= a) { b -= a; ++a; }
      const uint32_t between = (uint32_t)(a - b - 1) << 31;
      double sum = 0;
      for (int i = 0; i < 1 << (nop - 2); ++i) {
        // bits a and b put into i: a set, b clear
        int m = (i & ((1 << b) - 1)) | ((i >> b) << (b + 1));
        m = (m & ((1 << a) - 1)) | ((m >> a) << (a + 1)) | (1 << a);
        const uint32_t x = map[m], y = map[m ^ (1 << a) ^ (1 << b)];
        if (x == NO_DET && y == NO_DET) continue;
        const double cx = x == NO_DET ? 0 : __ldg(c + (int)(x & 0x7fffu) * KP);
        const double cy = y == NO_DET ? 0 : __ldg(c + (int)(y & 0x7fffu) * KP);
        const double v = cx + with_sign(cy, ((x ^ y) << 16) ^ between);
        sum = fma(v, v, sum);
      }
      const int oa = nth(so, a), ob = nth(so, b);
      atomicAdd(T2 + canon4(oa, ob, ob, oa) * KP + q, (open2 ? 0.5 : 1.0) * sum - a0);
    }
    // orbital energies and the other pairs of occupied orbitals j < i; j = i: the orbital itself
    for (int e = grp; e < nocc * (nocc + 1) / 2; e += ngrp) {
      int i = 0, j = e;
      while (j > i) { j -= i + 1; ++i; }
      const int ib = nth(o1, i), occi = 1 + (int)bit_w<W>(o2, ib);
      if (j == i) {
        atomicAdd(T1 + tri64(ib, ib) * KP + q, occi * a0);
        if (occi == 2) atomicAdd(T2 + canon4(ib, ib, ib, ib) * KP + q, a0);
        continue;
      }
      const int jb = nth(o1, j), ninj = occi * (1 + (int)bit_w<W>(o2, jb));
      atomicAdd(T2 + canon4(ib, ib, jb, jb) * KP + q, ninj * a0);
      if (ninj > 1) atomicAdd(T2 + canon4(ib, jb, ib, jb) * KP + q, ninj == 2 ? -a0 : -2.0 * a0);
    }
    __syncwarp();
  }
}

__global__ void k_fill(double *p, int64_t n, double v) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) p[i] = v;
}
__global__ void k_nonzero(const double *__restrict__ src, double *__restrict__ dst, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = (src[i] != 0.0) ? 1.0 : 0.0;
}
// entries of zero integrals reported as zero (mode: derivatives of the non-zero integrals)
__global__ void k_mask_zero(const double *__restrict__ tab, int64_t n, int k, double *G) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if (tab[i] == 0.0)
      for (int r = 0; r < k; ++r) G[(int64_t)r * n + i] = 0.0;
}

void grad_tabs_release(psoci_ctx *c) {
  if (c->grad_tabs) {
    DirTabs *d = static_cast<DirTabs *>(c->grad_tabs);
    d->s1.free();
    d->s2.free();
    delete d;
    c->grad_tabs = nullptr;
  }
  c->grad_generic = false;
}

// one pass of kk <= KP roots to G1 [kk][n1] and G2 [kk][n2] (mode 1: zero where the integral is), summed
// in T1 [n1 + n2][KP]; a single root's sums in G itself
template <int W, int KP>
cudaError_t grad_pass(psoci_ctx *c, const Params &P, const TabSet<W> &S, int kk, const double *V, int64_t ldv,
                      int mode, double *CS, double *T1, double *G1, double *G2) {
  cudaStream_t st = c->stream;
  const int64_t N = c->nsef_total, n1 = c->n1, n2 = c->n2;
  double *T2 = T1 + n1 * KP;
  cudaError_t e = cudaSuccess;
  if (KP == 1) {
    T1 = G1;
    T2 = G2;
    e = cudaMemsetAsync(G1, 0, sizeof(double) * n1, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(G2, 0, sizeof(double) * n2, st);
  } else {
    e = cudaMemsetAsync(T1, 0, sizeof(double) * (n1 + n2) * KP, st);
  }
  if (e != cudaSuccess) return e;
  const unsigned rb = (unsigned)std::min<int64_t>((N + 255) / 256, 152 * 16);
  const unsigned gb = (unsigned)std::min<int64_t>((c->nconf + GT_WARPS - 1) / GT_WARPS, 1 << 20);
  psoci_note_launch();
  psoci_note_launch();
  psoci_note_launch();
  k_grad_rows<KP><<<rb, 256, 0, st>>>(N, V, ldv, kk, CS);
  k_grad_tab<W, KP><<<gb, GT_WARPS * 32, 0, st>>>(P, S.cfg, c->grad_nbroff, c->grad_nbr, S.slot, S.t.hdr, S.t.pool, CS,
                                                  T1, T2);
  k_grad_diag<W, KP><<<gb, GT_WARPS * 32, 0, st>>>(P, CS, T1, T2);
  if (KP > 1) {
    psoci_note_launch();
    psoci_note_launch();
    k_grad_out<KP><<<(unsigned)std::min<int64_t>((n1 + 255) / 256, 152 * 8), 256, 0, st>>>(
        n1, kk, T1, mode == 1 ? c->d_one : nullptr, G1);
    k_grad_out<KP><<<(unsigned)std::min<int64_t>((n2 + 255) / 256, 152 * 8), 256, 0, st>>>(
        n2, kk, T2, mode == 1 ? c->d_eri : nullptr, G2);
  } else if (mode == 1) {
    psoci_note_launch();
    psoci_note_launch();
    k_mask_zero<<<152 * 4, 256, 0, st>>>(c->d_one, n1, 1, G1);
    k_mask_zero<<<152 * 8, 256, 0, st>>>(c->d_eri, n2, 1, G2);
  }
  return cudaGetLastError();
}

template <int W>
psoci_status run_energy_grad(psoci_ctx *c, int k, const double *dV, int64_t ldv, int mode, psoci_prec prec,
                             double *dG1, double *dG2) {
  const PsociKeep own(c, PSOCI_KEEP_GRAD);
  cudaStream_t st = c->stream;
  const int n = c->nconf;
  Params P = {};
  P.nconf = n; P.nbf = c->nbf; P.nelec = c->nelec; P.ksym = c->ksym;
  P.e1 = c->d_e1; P.e2 = c->d_e2; P.jsym = c->d_jsym; P.nopen = c->d_nopen;
  P.sefoff = c->d_sefoff; P.detoff = c->d_detoff;
  P.alpha = c->d_alpha; P.beta = c->d_beta; P.phase = c->d_phase; P.nalpha = c->d_nalpha;
  P.one = c->d_one; P.eri = c->d_eri;
  psoci_status s;
  const int64_t n1 = c->n1, n2 = c->n2;
  // neighbour lists: every pair within two excitations (mode 0), or those whose integral
  // prefactors are not all zero (mode 1); kept in the context for later calls
  if (!c->grad_nbroff || c->grad_mode != mode) {
    psoci_free(c->grad_nbroff);
    psoci_free(c->grad_nbr);
    grad_tabs_release(c);
    double *t1 = nullptr, *t2 = nullptr;
    if ((s = psoci_alloc(c, &t1, n1)) || (s = psoci_alloc(c, &t2, n2))) {
      psoci_free(t1);
      psoci_free(t2);
      return s;
    }
    psoci_note_launch();
    if (mode == 0) k_fill<<<152 * 4, 256, 0, st>>>(t1, n1, 1.0);
    else k_nonzero<<<152 * 4, 256, 0, st>>>(c->d_one, t1, n1);
    psoci_note_launch();
    if (mode == 0) k_fill<<<152 * 8, 256, 0, st>>>(t2, n2, 1.0);
    else k_nonzero<<<152 * 8, 256, 0, st>>>(c->d_eri, t2, n2);
    int64_t ncand = 0, npairs = 0;
    int nsplit = 0;
    s = screen_pairs<W>(c, P, t1, t2, c->grad_nbroff, c->grad_nbr, ncand, npairs, nsplit);
    cudaStreamSynchronize(st);
    psoci_free(t1);
    psoci_free(t2);
    if (s) return s;
    c->grad_mode = mode;
    c->grad_npairs = npairs;
  }
  // coupling tables, kept with the lists; the generic kernel for spaces or patterns that they do
  // not hold, where there is no room for them, and for FP32 sums, whose rounding is that of its order
  // (the tables' agreed to 1e-8)
  if (prec == PSOCI_PREC_FP64 && !c->grad_tabs && !c->grad_generic) {
    const PsociKeep plans(c, PSOCI_KEEP_ALL);
    DirTabs *d = new DirTabs();
    bool ok = tab_usable(c, false);
    s = PSOCI_OK;
    if (ok) s = tab_prepare_lists<W>(c, P, c->grad_nbroff, c->grad_nbr, c->grad_npairs, false, true, dir_set<W>(d), ok);
    if (s == PSOCI_OK && ok) c->grad_tabs = d;
    else delete d;
    if (s != PSOCI_OK && s != PSOCI_ERR_NOMEM) return s;
    if (s != PSOCI_OK) c->err.clear();
    c->grad_generic = !c->grad_tabs;
  }
  bool tabs = prec == PSOCI_PREC_FP64 && c->grad_tabs != nullptr;
  double *CD = nullptr;  // determinant-basis vectors (FP64, or FP32 for the FP32-bulk variant)
  double *CS = nullptr, *T1 = nullptr;  // SEF-basis vectors and gradients, the roots of a pass side by side
  auto done = [&](psoci_status r) {
    psoci_free(CD); psoci_free(CS); psoci_free(T1);
    return r;
  };
  const int kmax = std::min(k, ADJ_MAXR), kpmax = kmax <= 2 ? kmax : kmax <= 4 ? 4 : 8;
  const int64_t N = c->nsef_total;
  if (tabs && ((s = psoci_alloc(c, &CS, (size_t)N * kpmax)) ||
               (kpmax > 1 && (s = psoci_alloc(c, &T1, (size_t)(n1 + n2) * kpmax))))) {
    if (s != PSOCI_ERR_NOMEM) return done(s);
    c->err.clear();
    done(s);
    grad_tabs_release(c);
    c->grad_generic = true;
    tabs = false;
  }
  if (!tabs && (s = psoci_alloc(c, &CD, (size_t)c->ndet_total * kmax))) return done(s);
  float *CD32 = reinterpret_cast<float *>(CD);
  cudaError_t e = cudaSuccess;
  if (!tabs) {
    e = cudaMemsetAsync(dG1, 0, sizeof(double) * n1 * k, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(dG2, 0, sizeof(double) * n2 * k, st);
    if (e != cudaSuccess) return done(psoci_cuda_fail(c, e, "energy_gradient"));
  }
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)n + ADJ_WARPS - 1) / ADJ_WARPS, 152 * 16));
  for (int r0 = 0; r0 < k; r0 += ADJ_MAXR) {
    const int kk = std::min(ADJ_MAXR, k - r0);
    const unsigned sb = (unsigned)(((int64_t)n * 32 + 255) / 256);
    const double *V = dV + (int64_t)r0 * ldv;
    if (tabs) {
      const TabSet<W> &S = dir_set<W>(static_cast<DirTabs *>(c->grad_tabs));
      e = kk <= 1 ? grad_pass<W, 1>(c, P, S, kk, V, ldv, mode, CS, T1, dG1 + r0 * n1, dG2 + r0 * n2)
          : kk <= 2 ? grad_pass<W, 2>(c, P, S, kk, V, ldv, mode, CS, T1, dG1 + r0 * n1, dG2 + r0 * n2)
          : kk <= 4 ? grad_pass<W, 4>(c, P, S, kk, V, ldv, mode, CS, T1, dG1 + r0 * n1, dG2 + r0 * n2)
                    : grad_pass<W, 8>(c, P, S, kk, V, ldv, mode, CS, T1, dG1 + r0 * n1, dG2 + r0 * n2);
    } else {
      psoci_note_launch();
      if (prec == PSOCI_PREC_MIXED)
        k_sef_to_det<float><<<sb, 256, 0, st>>>(n, c->nelec, c->ksym, c->d_sefoff, c->d_detoff, c->d_jsym, c->d_nopen, V,
                                                ldv, kk, CD32);
      else
        k_sef_to_det<double><<<sb, 256, 0, st>>>(n, c->nelec, c->ksym, c->d_sefoff, c->d_detoff, c->d_jsym, c->d_nopen, V,
                                                 ldv, kk, CD);
      psoci_note_launch();
      if (prec == PSOCI_PREC_MIXED)
        k_energy_grad<W, float, float><<<blocks, ADJ_WARPS * 32, 0, st>>>(P, c->grad_nbroff, c->grad_nbr, CD32, kk,
                                                                          dG1 + r0 * n1, n1, dG2 + r0 * n2, n2);
      else
        k_energy_grad<W, double, double><<<blocks, ADJ_WARPS * 32, 0, st>>>(P, c->grad_nbroff, c->grad_nbr, CD, kk,
                                                                            dG1 + r0 * n1, n1, dG2 + r0 * n2, n2);
      e = cudaGetLastError();
    }
    if (e != cudaSuccess) return done(psoci_cuda_fail(c, e, "energy_gradient"));
  }
  if (mode == 1 && !tabs) {
    psoci_note_launch();
    k_mask_zero<<<152 * 4, 256, 0, st>>>(c->d_one, n1, k, dG1);
    psoci_note_launch();
    k_mask_zero<<<152 * 8, 256, 0, st>>>(c->d_eri, n2, k, dG2);
  }
  e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return done(psoci_cuda_fail(c, e, "energy_gradient"));
  return done(PSOCI_OK);
}

}  // namespace

void psoci_grad_release(psoci_ctx *c) {
  psoci_free(c->grad_nbroff);
  psoci_free(c->grad_nbr);
  grad_tabs_release(c);
  c->grad_mode = -1;
  c->grad_npairs = 0;
}

psoci_status psoci_energy_grad_run(psoci_ctx *c, int k, const double *dV, int64_t ldv, int mode, psoci_prec prec,
                                   double *dG1, double *dG2) {
  if (!c->have_ints) return psoci_fail(c, PSOCI_ERR_STATE, "energy_gradient: no integrals set");
  if (!c->have_dets) return psoci_fail(c, PSOCI_ERR_STATE, "energy_gradient: determinants not built");
  if (k < 1 || ldv < c->nsef_total || !dV || !dG1 || !dG2)
    return psoci_fail(c, PSOCI_ERR_INVALID_ARG, "energy_gradient: bad arguments");
  if (mode != 0 && mode != 1) return psoci_fail(c, PSOCI_ERR_INVALID_ARG, "energy_gradient: mode must be 0 or 1");
  if (prec != PSOCI_PREC_FP64 && prec != PSOCI_PREC_MIXED)
    return psoci_fail(c, PSOCI_ERR_INVALID_ARG, "energy_gradient: precision must be FP64 or MIXED");
  return (c->words == 1) ? run_energy_grad<1>(c, k, dV, ldv, mode, prec, dG1, dG2)
                         : run_energy_grad<2>(c, k, dV, ldv, mode, prec, dG1, dG2);
}

// ------------------------------------------------------------------------------------
// 1-particle density from coupling tables (density.cu finds the pairs and holds the plan).  An
// element of a single-excitation block of equal symmetries contains v0 with the coefficient of
// the reference's CIDEN block (PsociHamiltonian.C:572-705), so c_I^T S_IJ c_J is the first list of
// the table's program.
// ------------------------------------------------------------------------------------
namespace {

// Pair t of the groups: its slot and what the density kernel reads of it, {table and sign,
// first SEF of I, first SEF of J, place in the packed triangle}.  One thread a chunk of pairs.
constexpr int DEN_CHUNK = 4;
template <int W>
__global__ void __launch_bounds__(256) k_den_slots(Params P, const CfgRec<W> *__restrict__ cfg, int64_t ng, int64_t np,
                                                   const int64_t *__restrict__ geoff, const int64_t *__restrict__ gpoff,
                                                   const int32_t *__restrict__ gcfg, const uint8_t *__restrict__ gorb,
                                                   uint64_t *keys, uint32_t mask, int *err, uint32_t *list,
                                                   uint4 *__restrict__ recs) {
  const int64_t nchunk = (np + DEN_CHUNK - 1) / DEN_CHUNK;
  for (int64_t ch = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; ch < nchunk; ch += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t0 = ch * DEN_CHUNK;
    int64_t lo = 0, hi = ng - 1;  // group holding pair t0: last g with gpoff[g] <= t0
    while (lo < hi) {
      const int64_t mid = (lo + hi + 1) >> 1;
      if (gpoff[mid] <= t0) lo = mid;
      else hi = mid - 1;
    }
    int64_t g = lo, e0 = geoff[g];
    int m = (int)(geoff[g + 1] - e0);
    int64_t u = t0 - gpoff[g];
    int a = 0;
    while (u >= m - 1 - a) { u -= m - 1 - a; ++a; }
    int b = a + 1 + (int)u;
    const int64_t tend = min(t0 + DEN_CHUNK, np);
    for (int64_t t = t0; t < tend; ++t) {
      const int I = gcfg[e0 + a], J = gcfg[e0 + b], p = gorb[e0 + a], q = gorb[e0 + b];
      const CfgRec<W> A = cfg[I], B = cfg[J];
      uint32_t sl = TAB_NONE;
      const PairShape s = pair_shape<W>(A, B);
      // members of a group share a hash, not always the occupation: only p -> q singles count
      if (s.kind == K_SINGLE && s.ex0 == p && s.jy0 == q) {
        sl = tab_insert(keys, mask, pair_key<W>(A, B, s.kind, false), err, list);
        if (sl != TAB_NONE) sl |= s.sign;
      }
      const int x = max(p, q), y = min(p, q);
      recs[t] = make_uint4(sl, A.sef, B.sef, (uint32_t)(x * (x + 1) / 2 + y));
      if (++b == m) {
        if (++a == m - 1) {
          if (++g >= ng) break;
          e0 = geoff[g];
          m = (int)(geoff[g + 1] - e0);
          a = 0;
        }
        b = a + 1;
      }
    }
  }
}

// Off-diagonal: KP lanes (a root each) to a pair, the signed products of its list added in FP64,
// and to the packed triangle T [place][KP] by FP64 atomics.  Bound by the latency of record, table
// header, list and vectors (FP64 pipe 40%).  mrcisd_6e8o_v24, 8 roots: the whole density 240 us,
// where a warp took the determinants of a pair in float-float sums, four roots a pass, for 1,440 us.
template <int KP>
__global__ void __launch_bounds__(256) k_den_pairs(int64_t np, const uint4 *__restrict__ recs,
                                                   const uint4 *__restrict__ hdr, const uint32_t *__restrict__ pool,
                                                   const double *__restrict__ C, double *T) {
  const int q = threadIdx.x % KP;
  const int64_t ngrp = (int64_t)gridDim.x * blockDim.x / KP;
  for (int64_t u = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / KP; u < np; u += ngrp) {
    const uint4 r = __ldg(recs + u);
    if (r.x == TAB_NONE) continue;
    const uint4 h0 = __ldg(hdr + 2 * (size_t)(r.x & TAB_SLOT)), h1 = __ldg(hdr + 2 * (size_t)(r.x & TAB_SLOT) + 1);
    const double *cI = C + (int64_t)r.y * KP + q, *cJ = C + (int64_t)r.z * KP + q;
    const int end = h1.y ? (int)__ldg(reinterpret_cast<const uint16_t *>(pool + h1.x)) : 0;
    const uint32_t *pw = pool + h1.x + (TAB_LISTS + 1) / 2;
    double s0 = 0.0, s1 = 0.0;
    int e = 0;
#pragma unroll 2
    for (; e + 2 <= end; e += 2) {
      const uint32_t x0 = __ldg(pw + e), x1 = __ldg(pw + e + 1);
      s0 = fma(with_sign(__ldg(cI + (int)((x0 >> 8) & 0xffu) * KP), x0), __ldg(cJ + (int)(x0 & 0xffu) * KP), s0);
      s1 = fma(with_sign(__ldg(cI + (int)((x1 >> 8) & 0xffu) * KP), x1), __ldg(cJ + (int)(x1 & 0xffu) * KP), s1);
    }
    if (e < end) {
      const uint32_t x0 = __ldg(pw + e);
      s0 = fma(with_sign(__ldg(cI + (int)((x0 >> 8) & 0xffu) * KP), x0), __ldg(cJ + (int)(x0 & 0xffu) * KP), s0);
    }
    if (end) atomicAdd(T + (int64_t)r.w * KP + q, flip_sign(tab_scale(s0 + s1, h0.y), r.x & TAB_SIGN));
  }
}

// Diagonal: T[p][p] += occ_p(I) |c_I|^2.  One warp a run of configurations; lane l holds orbitals
// l, l + 32, ... for all KP roots, the norms are summed by lanes (SEF, root).
template <int W, int KP>
__global__ void __launch_bounds__(128) k_den_diag(Params P, const CfgRec<W> *__restrict__ cfg,
                                                  const double *__restrict__ C, double *T) {
  constexpr int NO = 2 * W;
  const int lane = threadIdx.x & 31, q = lane % KP;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const double r2 = sqrt(0.5), ssd = r2 * r2 + r2 * r2;  // (C C^T)_aa of an open-shell SEF, even electron count
  double acc[NO][KP];
#pragma unroll
  for (int w = 0; w < NO; ++w)
#pragma unroll
    for (int u = 0; u < KP; ++u) acc[w][u] = 0.0;
  for (int64_t I = warp; I < P.nconf; I += nwarps) {
    const CfgRec<W> a = cfg[I];
    const int nsef = (int)(a.flags >> 16) & 0x1ff;
    double s = 0.0;
    for (int x = lane / KP; x < nsef; x += 32 / KP) {
      const double c = __ldg(C + ((int64_t)a.sef + x) * KP + q);
      s = fma(c, c, s);
    }
#pragma unroll
    for (int o = KP; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (!(P.nelec & 1) && (a.flags & 15u)) s *= ssd;
    double n2[KP];
#pragma unroll
    for (int u = 0; u < KP; ++u) n2[u] = __shfl_sync(0xffffffffu, s, u);
#pragma unroll
    for (int w = 0; w < NO; ++w) {
      const uint32_t o1 = (uint32_t)(a.e1[w / 2] >> (32 * (w & 1))), o2 = (uint32_t)(a.e2[w / 2] >> (32 * (w & 1)));
      if (o1 == 0u) continue;
      const int occ = (int)((o1 >> lane) & 1u) + (int)((o2 >> lane) & 1u);
      const double f = occ == 0 ? 0.0 : occ == 1 ? 1.0 : 2.0;
#pragma unroll
      for (int u = 0; u < KP; ++u) acc[w][u] = fma(f, n2[u], acc[w][u]);
    }
  }
#pragma unroll
  for (int w = 0; w < NO; ++w) {
    const int64_t p = 32 * w + lane;
    if (p < P.nbf)
#pragma unroll
      for (int u = 0; u < KP; ++u)
        if (acc[w][u] != 0.0) atomicAdd(T + (p * (p + 1) / 2 + p) * KP + u, acc[w][u]);
  }
}

// D[q * n + i] = T[i * KP + q]
template <int KP>
__global__ void k_den_out(int n, int k, const double *__restrict__ T, double *__restrict__ D) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n * k; e += gridDim.x * blockDim.x)
    D[e] = T[(int64_t)(e % n) * KP + e / n];
}

Params den_params(const psoci_ctx *c) {
  Params P = {};
  P.nconf = c->nconf; P.nbf = c->nbf; P.nelec = c->nelec; P.ksym = c->ksym;
  P.e1 = c->d_e1; P.e2 = c->d_e2; P.jsym = c->d_jsym; P.nopen = c->d_nopen;
  P.sefoff = c->d_sefoff; P.detoff = c->d_detoff; P.phase = c->d_phase;
  return P;
}

// den_tabs and den_recs, where the records take at most a quarter of the memory at hand and the
// tables hold the patterns and have room; the generic kernels need neither.
template <int W>
psoci_status den_plan(psoci_ctx *c) {
  const Params P = den_params(c);
  const int64_t np = c->den_npairs;
  if (np == 0) return PSOCI_OK;
  size_t freeb = 0;
  PSOCI_CUDA(c, psoci_mem_free(c, &freeb));
  if ((double)np * sizeof(uint4) > 0.25 * ((double)freeb + (double)c->pool_bytes)) return PSOCI_OK;
  const PsociKeep plans(c, PSOCI_KEEP_ALL);
  DirTabs *d = new DirTabs();
  bool ok = false;
  psoci_status s = psoci_alloc(c, &c->den_recs, np);
  if (s == PSOCI_OK)
    s = tab_prepare<W>(c, P, np, false, false, true, dir_set<W>(d), ok, [&](TabSet<W> &T) {
      k_den_slots<W><<<(unsigned)std::max<int64_t>(1, std::min<int64_t>((np + 1023) / 1024, 152 * 32)), 256, 0, c->stream>>>(
          P, T.cfg, c->den_ng, np, c->den_geoff, c->den_gpoff, c->den_gcfg, c->den_gorb, T.t.keys,
          (uint32_t)(T.t.slots - 1), T.t.err, T.t.list, c->den_recs);
    });
  if (s != PSOCI_OK || !ok) {
    delete d;
    psoci_free(c->den_recs);
    if (s != PSOCI_ERR_NOMEM) return s;
    c->err.clear();
    return PSOCI_OK;
  }
  c->den_tabs = d;
  return PSOCI_OK;
}

template <int W, int KP>
cudaError_t den_pass(psoci_ctx *c, int k, const double *V, int64_t ldv, double *D) {
  cudaStream_t st = c->stream;
  const TabSet<W> &S = dir_set<W>(static_cast<DirTabs *>(c->den_tabs));
  const int64_t N = c->nsef_total, np = c->den_npairs;
  const int ntri = c->nbf * (c->nbf + 1) / 2;
  double *T = c->den_rows + N * KP;  // the packed triangles, the roots of an entry side by side
  cudaError_t e = cudaMemsetAsync(T, 0, sizeof(double) * ntri * KP, st);
  if (e != cudaSuccess) return e;
  for (int q = 0; q < 4; ++q) psoci_note_launch();
  k_grad_rows<KP><<<(unsigned)std::min<int64_t>((N + 255) / 256, 152 * 16), 256, 0, st>>>(N, V, ldv, k, c->den_rows);
  k_den_diag<W, KP><<<(unsigned)std::min<int64_t>((c->nconf + 31) / 32, 152 * 4), 128, 0, st>>>(den_params(c), S.cfg,
                                                                                            c->den_rows, T);
  k_den_pairs<KP><<<(unsigned)std::max<int64_t>(1, std::min<int64_t>((np * KP + 255) / 256, 152 * 32)), 256, 0, st>>>(
        np, c->den_recs, S.t.hdr, S.t.pool, c->den_rows, T);
  k_den_out<KP><<<(ntri * k + 255) / 256, 256, 0, st>>>(ntri, k, T, D);
  return cudaGetLastError();
}

template <int W>
psoci_status den_run(psoci_ctx *c, int k, const double *V, int64_t ldv, double *D) {
  const int ntri = c->nbf * (c->nbf + 1) / 2;
  psoci_status s;
  // for eight roots, so that later calls only launch, unless they take more than 1% of the memory
  int width = k <= 2 ? k : k <= 4 ? 4 : 8;
  if (c->den_width < width) {
    size_t freeb = 0;
    PSOCI_CUDA(c, psoci_mem_free(c, &freeb));
    if ((c->nsef_total + ntri) * 64.0 <= 0.01 * ((double)freeb + (double)c->pool_bytes)) width = 8;
    c->den_width = 0;
    if ((s = psoci_alloc(c, &c->den_rows, (size_t)(c->nsef_total + ntri) * width))) return s;
    c->den_width = width;
  }
  for (int r0 = 0; r0 < k; r0 += 8) {
    const int kk = std::min(8, k - r0);
    const double *v = V + (int64_t)r0 * ldv;
    double *d = D + (int64_t)r0 * ntri;
    const cudaError_t e = kk <= 1 ? den_pass<W, 1>(c, kk, v, ldv, d) : kk <= 2 ? den_pass<W, 2>(c, kk, v, ldv, d)
                        : kk <= 4 ? den_pass<W, 4>(c, kk, v, ldv, d) : den_pass<W, 8>(c, kk, v, ldv, d);
    if (e != cudaSuccess) return psoci_cuda_fail(c, e, "density1");
  }
  return PSOCI_OK;
}

}  // namespace

psoci_status psoci_density_plan(psoci_ctx *c) {
  if (c->max_ndet > TAB_MAXDET) return PSOCI_OK;
  return c->words == 1 ? den_plan<1>(c) : den_plan<2>(c);
}
psoci_status psoci_density_tab_run(psoci_ctx *c, int k, const double *dV, int64_t ldv, double *dD) {
  return c->words == 1 ? den_run<1>(c, k, dV, ldv, dD) : den_run<2>(c, k, dV, ldv, dD);
}
void psoci_density_tabs_release(psoci_ctx *c) {
  if (c->den_tabs) {
    DirTabs *d = static_cast<DirTabs *>(c->den_tabs);
    d->s1.free();
    d->s2.free();
    delete d;
    c->den_tabs = nullptr;
  }
  psoci_free(c->den_recs);
  psoci_free(c->den_rows);
  c->den_width = 0;
}
