// Coupling tables: the SEF block of a configuration pair as a short list of signed table
// entries, shared by every pair with the same relative occupation pattern.
//
// Strip the orbitals that two configurations A, B hold alike with zero or two electrons: what
// is left (the open shells of either and the orbitals the excitation touches, at most 12)
// fixes which determinants couple, with which phases and through which of the pair's
// integrals.  The stripped doubles only multiply the whole block by one sign, because every
// determinant move between two orbitals passes the same parity of them whichever spins it
// takes.  So a pair is a pattern (its key, below), a sign and a few integrals:
//   double excitations   v0 = (i0 j0|i1 j1), v1 = (i0 j1|i1 j0)
//   spin-orbit singles   v0
//   singles              v0 and X[t] = (i p_t|p_t j) over the open shells p_t of A
// and an element of its block is (t f1) f2 with t one or two signed terms of these and f1, f2
// the pattern's constants — the operations, in their order, that ciout / transformCDCt
// (PsociHamiltonian.C:1350-1516) leaves once the terms that are exactly zero are dropped: the
// second determinant of an open-shell SEF is the spin flip of the first, so its half of the
// sum is the first half's, with one sign.
//
// A space of 10^8 pairs has 10^4 - 10^5 patterns (8,074 full-CI configurations of 6 electrons
// in 12 orbitals: 37,000; singles and doubles of 6 electrons in 8 orbitals: 33,000), so the
// determinant work is done once a pattern, and a pair costs its key and its integrals.
#pragma once
#include "psoci_internal.cuh"

constexpr int TAB_MAXOPEN = 10;        // open shells a configuration may have (256 SEFs)
constexpr int TAB_MAXDET = 512;        // determinants of 10 open shells
constexpr int TAB_SYMS = 12;           // orbitals of a pattern
// a pair's slot: the table, the forms v0, v1, v0 - v1 that pass the threshold of storage (listed
// pairs only) and the stripped doubles' sign
constexpr uint32_t TAB_SLOT = 0x01ffffffu;
constexpr int TAB_KEPT = 26;
constexpr uint32_t TAB_SIGN = 0x80000000u;
constexpr uint32_t TAB_DIAG = 0x7ffffffeu;  // slot of a configuration with itself
constexpr uint32_t TAB_NONE = 0x7fffffffu;  // slot of a pair whose block is zero

// One configuration, in one or two sectors for the gathers of the pair kernels.
template <int W>
struct __align__(16) CfgRec {
  uint64_t e1[W], e2[W];
  uint32_t sef;    // first SEF
  uint32_t flags;  // bits 0-3 open shells, 4 phase, 5 template class (low bit), 6 jsym odd, 16-24 SEFs
  int32_t jsym;
  uint32_t pad;
};

// hdr[2 slot]: .x first entry (word of pool), .y info, .z/.w entries of each row, 4 bits a row
// (tables of at most 16 rows); hdr[2 slot + 1]: of these, those of form 1 and of form 2 (doubles).
// info: bits 0-11 entries, 12-13 factors (1: f1 = sqrt(1/2), 2: f2 = 2 sqrt(1/2)), 14-16 kind,
//       17 more than 16 rows, 18-29 forms in use (doubles and spin-orbit)
// entries, ascending column within ascending row: bits 0-7 column, then
//   doubles and spin-orbit: 8-11 form, 12-19 row, 31 sign;
//   singles: two 12-bit terms (sign << 11 | isX << 10 | rank or mask), the second TAB_NOTERM
//            where there is one.
// The entries' row indices follow them, a byte each.
constexpr uint32_t TAB_NOTERM = 0x7ffu;

constexpr int TAB_ENTRIES = 0xfff, TAB_FACTORS = 12, TAB_KIND = 14, TAB_FORMS = 18;
constexpr uint32_t TAB_NOCOUNTS = 1u << 17;

struct BlockTab {
  uint64_t *keys = nullptr;  // [slots], 0 = empty
  uint4 *hdr = nullptr;      // [2 slots]
  uint32_t *pool = nullptr;
  unsigned long long *counter = nullptr;  // words of the pool in use
  // counter + 1: err, bit 0: key table full, bit 1: a pattern outside the tables' form; err + 1: the
  // patterns, whose slots are in list
  int *err = nullptr;
  uint32_t *list = nullptr;  // [slots]
  int64_t slots = 0, cap = 0;
};

// two-term forms of a double: t = a + s b with a, b among v0, v1, w = v0 - v1 (codes 0, 1, 2)
//   form 0-2: a alone; 3-5: a + a; 6/7: v0 +- v1; 8/9: v0 +- w; 10/11: v1 +- w
__host__ __device__ __forceinline__ int tab_form2(int a, int b, int minus) {
  return a == b ? 3 + a : 2 * (a + b) + 4 + minus;
}

// ------------------------------------------------------------------------------------
// patterns
// ------------------------------------------------------------------------------------
// Key of the pair in the reference's roles (A the lower-triangle row): 4 bits an orbital
// (A occupied, A doubly, B occupied, B doubly), ascending from bit 0; bits 48-49 kind (1 double,
// 2 single, 3 spin-orbit), 50 rows are B's SEFs, 51/52 template class of A / B, 53/54 jsym odd.
struct PairShape {
  int kind;                 // K_NONE, K_SINGLE, K_DOUBLE, K_SO
  int ex0, ex1, jy0, jy1;   // orbitals that lose / gain an electron (with multiplicity)
  uint32_t sign;            // parity of the stripped doubles and of the configuration phases
};

template <int W>
__device__ __forceinline__ uint64_t below_word(int p, int w) {
  const int b = p - 64 * w;
  return b <= 0 ? 0ull : b >= 64 ? ~0ull : (1ull << b) - 1ull;
}

// kind, excited orbitals and sign (kinds as in hbuild.cu: 2 single, 3 double, 4 spin-orbit)
template <int W>
__device__ __forceinline__ PairShape pair_shape(const CfgRec<W> &A, const CfgRec<W> &B) {
  PairShape s{0, -1, -1, -1, -1, 0u};
  int ni = 0, nj = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    const uint64_t i1 = A.e1[w] & ~B.e1[w], i2 = A.e2[w] & ~B.e2[w];
    const uint64_t j1 = B.e1[w] & ~A.e1[w], j2 = B.e2[w] & ~A.e2[w];
    uint64_t u = i1 | i2;
    while (u && ni < 3) {
      const int b = __ffsll((long long)u) - 1;
      u &= u - 1;
      const int both = (int)((i1 >> b) & (i2 >> b) & 1ull);
      if (ni == 0) { s.ex0 = 64 * w + b; if (both) s.ex1 = 64 * w + b; }
      else if (ni == 1) s.ex1 = 64 * w + b;
      ni += 1 + both;
    }
    u = j1 | j2;
    while (u && nj < 3) {
      const int b = __ffsll((long long)u) - 1;
      u &= u - 1;
      const int both = (int)((j1 >> b) & (j2 >> b) & 1ull);
      if (nj == 0) { s.jy0 = 64 * w + b; if (both) s.jy1 = 64 * w + b; }
      else if (nj == 1) s.jy1 = 64 * w + b;
      nj += 1 + both;
    }
  }
  if (ni != nj) return s;
  s.kind = ni == 1 ? (A.jsym != B.jsym ? 4 : 2) : ni == 2 ? 3 : 0;
  if (s.kind == 0) return s;
  uint32_t par = ((A.flags ^ B.flags) >> 4) & 1u;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    uint64_t m = below_word<W>(s.ex0, w) ^ below_word<W>(s.jy0, w);
    if (ni == 2) m ^= below_word<W>(s.ex1, w) ^ below_word<W>(s.jy1, w);
    par ^= (uint32_t)__popcll(A.e2[w] & B.e2[w] & m) & 1u;
  }
  s.sign = par ? TAB_SIGN : 0u;
  return s;
}

template <int W>
__device__ __forceinline__ uint64_t pair_key(const CfgRec<W> &A, const CfgRec<W> &B, int kind, bool rowsB) {
  uint64_t key = 0ull;
  int sh = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    const uint64_t a1 = A.e1[w], a2 = A.e2[w], b1 = B.e1[w], b2 = B.e2[w];
    uint64_t u = (a1 & ~a2) | (b1 & ~b2) | (a1 ^ b1) | (a2 ^ b2);
    while (u) {
      const int b = __ffsll((long long)u) - 1;
      u &= u - 1;
      const uint64_t sym = ((a1 >> b) & 1ull) | (((a2 >> b) & 1ull) << 1) | (((b1 >> b) & 1ull) << 2) |
                           (((b2 >> b) & 1ull) << 3);
      key |= sym << sh;
      sh += 4;
    }
  }
  const uint64_t k = kind == 3 ? 1 : kind == 2 ? 2 : 3;
  return key | (k << 48) | ((uint64_t)rowsB << 50) | ((uint64_t)((A.flags >> 5) & 1u) << 51) |
         ((uint64_t)((B.flags >> 5) & 1u) << 52) | ((uint64_t)((A.flags >> 6) & 1u) << 53) |
         ((uint64_t)((B.flags >> 6) & 1u) << 54);
}

// the 64-bit mixer published by degski (invertible_hash_functions.hpp)
__device__ __forceinline__ uint64_t tab_hash(uint64_t x) {
  x ^= x >> 32;
  x *= 0xd6e8feb86659fd93ull;
  x ^= x >> 32;
  x *= 0xd6e8feb86659fd93ull;
  return x ^ (x >> 32);
}

// slot of a key, inserted (and listed) when new; TAB_NONE (and bit 0 of *err) when the table is full
__device__ __forceinline__ uint32_t tab_insert(uint64_t *keys, uint32_t mask, uint64_t key, int *err, uint32_t *list) {
  uint32_t s = (uint32_t)tab_hash(key) & mask;
  for (int probe = 0; probe < 256; ++probe) {
    uint64_t cur = *(volatile uint64_t *)(keys + s);
    if (cur == key) return s;
    if (cur == 0ull) {
      cur = atomicCAS((unsigned long long *)(keys + s), 0ull, (unsigned long long)key);
      if (cur == 0ull) list[atomicAdd(err + 1, 1)] = s;
      if (cur == 0ull || cur == key) return s;
    }
    s = (s + 1) & mask;
  }
  atomicOr(err, 1);
  return TAB_NONE;
}

// ------------------------------------------------------------------------------------
// table construction: one warp per pattern
// ------------------------------------------------------------------------------------
// The pattern's orbitals as bits 0..L-1: what det_elem (hbuild.cu) decides from the full
// strings, from the pattern's.
struct RedPair {
  int kind, ie, je, ex0, ex1, jy0, jy1, nD, jA, jB;
  uint32_t SA;
  bool fold;  // a doubly emptied or filled orbital: v1 is v0's table entry
};

__device__ __forceinline__ uint32_t red_below(int p) { return (1u << p) - 1u; }
__device__ __forceinline__ uint32_t red_between(int p, int q) {
  const int lo = min(p, q), hi = max(p, q);
  return ((1u << hi) - 1u) & ~((2u << lo) - 1u);
}
constexpr uint32_t RED_SET = 0x1000u, RED_NEG = 0x800u;

// 0, or RED_SET | sign << 11 | term: the element of determinants (aa, ba) of A, (ab, bb) of B
__device__ __forceinline__ uint32_t red_code(const RedPair &R, uint32_t aa, uint32_t ba, uint32_t ab, uint32_t bb,
                                             bool &bad) {
  const uint32_t ua = ab & ~aa, ub = bb & ~ba;
  const int na = __popc(ua), nt = na + __popc(ub);
  if (nt > 2) return 0u;
  const int naa = __popc(aa), nab = __popc(ab);
  int n = 0;
  uint32_t term = 0u;
  if (R.kind == 4) {  // socig (PsociHamiltonian.C:746-855)
    if (nt > 1) return 0u;
    if (naa < nab) {
      n = __popc(ba & red_below(R.ie)) + __popc(ab & ~red_below(R.je + 1)) + R.nD;
      n += ((R.jA ^ R.jB) & 1) == 0 ? 1 : R.jA;
    } else if (naa > nab) {
      n = __popc(aa & ~red_below(R.ie + 1)) + __popc(bb & red_below(R.je)) + R.nD;
      n += (R.jA ^ R.jB) & R.jA;
    } else {
      n = (na == 0 ? 1 : 0) + R.jA + __popc((na ? aa : ba) & red_between(R.ie, R.je));
    }
  } else {  // generateSEFCIG (PsociHamiltonian.C:902-1113)
    if (naa != nab || nt == 0) return 0u;
    if (nt == 1) {
      if (R.kind != 2) { bad = true; return 0u; }
      const uint32_t s = na ? aa : ba;
      const uint32_t m = s & ~(aa & ba) & ~(1u << R.ie) & ~(1u << R.je);
      n = __popc(s & red_between(R.ie, R.je));
      int t = 0;
      for (uint32_t sa = R.SA; sa; sa &= sa - 1, ++t)
        if (m & (sa & (~sa + 1u))) term |= 1u << t;
    } else if (na == 1) {
      const uint32_t xa = aa & ~ab, xb = ba & ~bb;
      if (R.kind == 3) {
        const int ia = (xa >> R.ex0) & 1u ? 0 : 1, ja = (ua >> R.jy0) & 1u ? 0 : 1;
        const int i = ia ? R.ex1 : R.ex0, i2 = ia ? R.ex0 : R.ex1, j = ja ? R.jy1 : R.jy0, j2 = ja ? R.jy0 : R.jy1;
        n = __popc(aa & red_between(i, j)) + __popc(ba & red_between(i2, j2));
        term = (ia == ja || R.fold) ? 0u : 1u;
      } else {
        const int i2 = __ffs(ua) - 1, j2 = __ffs(ub) - 1, i3 = __ffs(xa) - 1, j3 = __ffs(xb) - 1;
        n = __popc(aa & red_between(i2, i3)) + __popc(ba & red_between(j2, j3));
        const int p = (i3 == R.ie || i3 == R.je) ? i2 : i3;
        const uint32_t mi = (1u << i2) | (1u << i3), mj = (1u << j2) | (1u << j3);
        const uint32_t me = (1u << R.ie) | (1u << p), mf = (1u << R.je) | (1u << p);
        if (!((R.SA >> p) & 1u) || !((mi == me && mj == mf) || (mi == mf && mj == me))) { bad = true; return 0u; }
        term = 0x400u | (uint32_t)__popc(R.SA & red_below(p));
      }
    } else {
      if (R.kind != 3) return 0u;
      if (R.fold) { bad = true; return 0u; }
      n = __popc((na == 2 ? ab : bb) & red_between(R.jy0, R.jy1)) + __popc((na ? aa : ba) & red_between(R.ex0, R.ex1));
      term = 2u;
    }
  }
  return RED_SET | ((n & 1) ? RED_NEG : 0u) | term;
}

// d0 + m d1 as a canonical pair of codes: larger-coded term last, exact cancellation dropped;
// returns the first code (0: none) and the second in c1 (0: none)
__device__ __forceinline__ uint32_t red_sum(uint32_t d0, uint32_t d1, bool m, uint32_t &c1) {
  if (d1 && m) d1 ^= RED_NEG;
  c1 = 0u;
  if (!d0) return d1;
  if (!d1) return d0;
  const uint32_t t0 = d0 & ~RED_NEG, t1 = d1 & ~RED_NEG;
  if (t0 == t1 && d0 != d1) return 0u;
  const bool sw = t0 > t1;
  c1 = sw ? d0 : d1;
  return sw ? d1 : d0;
}

constexpr int TABB_WARPS = 4, TABB_LIST = 1024;
struct TabBuildSmem {
  uint16_t aA[TAB_MAXDET], bA[TAB_MAXDET], aB[TAB_MAXDET], bB[TAB_MAXDET];
  uint32_t ent[TABB_LIST];  // the first entries and their rows
  uint8_t row[TABB_LIST];
};

struct TabBuildArgs {
  const uint64_t *keys;
  const uint32_t *list;
  const uint32_t *tmpl;
  const int32_t *tmpl_off;
  int nelec, kodd;  // electrons; ksym odd
  uint4 *hdr;
  uint32_t *pool;
  unsigned long long *counter;
  int64_t cap;
  int *err;
};

__device__ inline void tab_strings(uint32_t S, uint32_t D, int cls, int nop, const TabBuildArgs &T, uint16_t *al,
                                   uint16_t *be, int lane) {
  const int run = T.tmpl_off[cls * PSOCI_NOPEN_SLOTS + nop], nd = 1 << (nop > 1 ? nop - 1 : 0);
  for (int d = lane; d < nd; d += 32) {
    const uint32_t ent = T.tmpl[run + d];
    uint32_t a = D, b = D;
    int t = 0;
    for (uint32_t s = S; s; s &= s - 1, ++t) {
      const uint32_t low = s & (~s + 1u);
      if ((ent >> t) & 1u) a |= low;
      if ((ent >> (12 + t)) & 1u) b |= low;
    }
    al[d] = (uint16_t)a;
    be[d] = (uint16_t)b;
  }
}

// Every listed slot's table: lanes over its (row, column) elements, the entries found kept in shared
// memory until their number, and so their place, is known; a table of more than TABB_LIST is
// evaluated once more for its place.  Bound by integer issue; 2 * 10^4 patterns of up to 6 open
// shells take about as long as reading the neighbour lists once.  (All tables evaluated twice: 0.77
// ms for 8 electrons in 10 orbitals, up to 8 open shells; 0.42 ms now.  By the list, so that few large
// tables go to as many warps: with a warp to 32 key slots a direct build of 200 configurations of up to 8
// open shells took 2.5 ms, now 1.25.)
__global__ void __launch_bounds__(TABB_WARPS * 32) k_tab_build(TabBuildArgs T) {
  __shared__ TabBuildSmem sm[TABB_WARPS];
  TabBuildSmem &S = sm[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const bool odd = T.nelec & 1;
  const int npat = T.err[1];
  for (int64_t p = warp; p < npat; p += nwarps) {
    const int64_t slot = T.list[p];
    const uint64_t key = T.keys[slot];
    // the pattern
    uint32_t a1 = 0, a2 = 0, b1 = 0, b2 = 0;
    for (int q = 0; q < TAB_SYMS; ++q) {
      const uint32_t y = (uint32_t)(key >> (4 * q)) & 15u;
      a1 |= (y & 1u) << q; a2 |= ((y >> 1) & 1u) << q; b1 |= ((y >> 2) & 1u) << q; b2 |= ((y >> 3) & 1u) << q;
    }
    const int kc = (int)(key >> 48) & 3;
    const bool rowsB = (key >> 50) & 1ull;
    RedPair R;
    R.kind = kc == 1 ? 3 : kc == 2 ? 2 : 4;
    R.jA = (int)(key >> 53) & 1;
    R.jB = (int)(key >> 54) & 1;
    R.SA = a1 & ~a2;
    const uint32_t SB = b1 & ~b2;
    R.nD = (T.nelec - __popc(a1) - __popc(a2)) / 2;
    const uint32_t i1 = a1 & ~b1, i2 = a2 & ~b2, j1 = b1 & ~a1, j2 = b2 & ~a2;
    R.ex0 = __ffs(i1 | i2) - 1;
    R.ex1 = (i1 & i2) ? R.ex0 : __ffs((i1 | i2) & ((i1 | i2) - 1)) - 1;
    R.jy0 = __ffs(j1 | j2) - 1;
    R.jy1 = (j1 & j2) ? R.jy0 : __ffs((j1 | j2) & ((j1 | j2) - 1)) - 1;
    R.ie = R.ex0;
    R.je = R.jy0;
    R.fold = R.kind == 3 && (R.ex0 == R.ex1 || R.jy0 == R.jy1);
    const int opA = __popc(R.SA), opB = __popc(SB);
    const int cls0 = odd ? CLS_FRAC_P : CLS_EVEN;
    tab_strings(R.SA, a2, cls0 + ((int)(key >> 51) & 1), opA, T, S.aA, S.bA, lane);
    tab_strings(SB, b2, cls0 + ((int)(key >> 52) & 1), opB, T, S.aB, S.bB, lane);
    __syncwarp();
    const bool oa = !odd && opA != 0, ob = !odd && opB != 0;
    const bool mA = (R.jA != T.kodd), mB = (R.jB != T.kodd);  // -1 where true
    const int lA = opA > 1 ? opA - 1 - (oa ? 1 : 0) : 0, lB = opB > 1 ? opB - 1 - (ob ? 1 : 0) : 0;  // log2 SEFs
    const int lr = rowsB ? lB : lA, lc = rowsB ? lA : lB;
    const int nrow = 1 << lr, tot = 1 << (lr + lc);
    const bool counts = nrow <= 16;
    uint32_t forms = 0u, ent0 = 0u;
    bool bad = false, fits = false;
    uint64_t nib[3] = {0ull, 0ull, 0ull};
    int nent = 0;
    for (int pass = 0; pass < 2; ++pass) {
      int n = 0;
      for (int e0 = 0; e0 < tot; e0 += 32) {
        const int e = e0 + lane, r = e >> lc, t = e & ((1 << lc) - 1);
        uint32_t ent = 0u;
        bool have = false;
        if (e < tot) {
          const int a = rowsB ? t : r, b = rowsB ? r : t;
          uint32_t d[2][2] = {{0u, 0u}, {0u, 0u}};
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 2; ++y) {
              if ((x && !oa) || (y && !ob)) continue;
              const int da = oa ? 2 * a + x : (odd ? a : 0), db = ob ? 2 * b + y : (odd ? b : 0);
              d[x][y] = red_code(R, S.aA[da], S.bA[da], S.aB[db], S.bB[db], bad);
            }
          uint32_t t1, u1;
          const uint32_t t0 = red_sum(d[0][0], d[0][1], mB, t1);
          have = t0 != 0u;
          if (oa) {  // the second half, times mA: the same terms, or their negatives (sum zero)
            uint32_t u0 = red_sum(d[1][0], d[1][1], mB, u1);
            if (mA) { if (u0) u0 ^= RED_NEG; if (u1) u1 ^= RED_NEG; }
            if ((u0 ^ t0) & ~RED_NEG || (u1 ^ t1) & ~RED_NEG) bad = true;
            else if (t0 && u0 != t0) {
              if (t1 && u1 == t1) bad = true;
              have = false;
            } else if (t1 && u1 != t1) bad = true;
          }
          if (have) {
            if (R.kind == 2) {
              ent = ((t0 & 0xfffu) << 8) | ((t1 ? (t1 & 0xfffu) : TAB_NOTERM) << 20);
            } else {
              const int f = t1 ? tab_form2((int)(t0 & 3u), (int)(t1 & 3u), (int)(((t0 ^ t1) & RED_NEG) != 0u))
                               : (int)(t0 & 3u);
              forms |= 1u << f;
              ent = ((uint32_t)f << 8) | ((uint32_t)r << 12) | ((t0 & RED_NEG) ? 0x80000000u : 0u);
            }
            ent |= (uint32_t)t;
          }
        }
        const unsigned hb = __ballot_sync(0xffffffffu, have);
        const int at = n + __popc(hb & ((1u << lane) - 1u));
        if (pass == 0) {
          if (have && at < TABB_LIST) {
            S.ent[at] = ent;
            S.row[at] = (uint8_t)r;
          }
          if (have && counts) {  // lanes' shares, summed below
            nib[0] += 1ull << (4 * r);
            const uint32_t f = (ent >> 8) & 15u;
            if (R.kind == 3 && f == 1u) nib[1] += 1ull << (4 * r);
            if (R.kind == 3 && f == 2u) nib[2] += 1ull << (4 * r);
          }
        } else if (fits) {
          if (have) {
            T.pool[ent0 + at] = ent;
            reinterpret_cast<uint8_t *>(T.pool + ent0 + nent)[at] = (uint8_t)r;
          }
        }
        n += __popc(hb);
      }
      if (pass == 0) {
        nent = n;
        const uint32_t words = (uint32_t)nent + (uint32_t)(nent + 3) / 4u;
        unsigned long long o = 0;
        if (lane == 0) o = atomicAdd(T.counter, (unsigned long long)words);
        o = __shfl_sync(0xffffffffu, o, 0);
        fits = (int64_t)(o + words) <= T.cap;
        ent0 = (uint32_t)o;
        // a row has at most 2 + one an open shell (of at most 6), so the 4-bit sums do not carry
#pragma unroll
        for (int o2 = 16; o2 > 0; o2 >>= 1)
#pragma unroll
          for (int u = 0; u < 3; ++u) nib[u] += __shfl_xor_sync(0xffffffffu, nib[u], o2);
        __syncwarp();
        if (nent <= TABB_LIST) {
          if (fits)
            for (int q = lane; q < nent; q += 32) {
              T.pool[ent0 + q] = S.ent[q];
              reinterpret_cast<uint8_t *>(T.pool + ent0 + nent)[q] = S.row[q];
            }
          break;
        }
      }
    }
    __syncwarp();
    if (nent > TAB_ENTRIES) bad = true;
#pragma unroll
    for (int o2 = 16; o2 > 0; o2 >>= 1) forms |= __shfl_xor_sync(0xffffffffu, forms, o2);
    if (__ballot_sync(0xffffffffu, bad) && lane == 0) atomicOr(T.err, 2);
    if (lane == 0) {
      const uint32_t fc = odd ? 0u : (oa && ob) ? 3u : ob ? 1u : oa ? 2u : 0u;
      const uint32_t info = ((uint32_t)nent & TAB_ENTRIES) | (fc << TAB_FACTORS) | ((uint32_t)R.kind << TAB_KIND) |
                            (counts ? 0u : TAB_NOCOUNTS) | (forms << TAB_FORMS);
      T.hdr[2 * slot] = make_uint4(ent0, info, (uint32_t)nib[0], (uint32_t)(nib[0] >> 32));
      T.hdr[2 * slot + 1] =
          make_uint4((uint32_t)nib[1], (uint32_t)(nib[1] >> 32), (uint32_t)nib[2], (uint32_t)(nib[2] >> 32));
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------------------------------
// elements
// ------------------------------------------------------------------------------------
__device__ __forceinline__ double tab_scale(double t, uint32_t info) {
  const double r = sqrt(0.5);
  if (info & (1u << TAB_FACTORS)) t = t * r;
  if (info & (2u << TAB_FACTORS)) t = t * (2.0 * r);
  return t;
}

// v with its sign bit changed by s (0 or 0x80000000), on the integer pipe: a double's negation
// compiles to an FP64 instruction
__device__ __forceinline__ double flip_sign(double v, uint32_t s) {
  return __hiloint2double(__double2hiint(v) ^ (int)s, __double2loint(v));
}
// a term of a single's entry; v0 and X[t] with the pair's sign
__device__ __forceinline__ double tab_single_term(uint32_t c, double v0, const double *X) {
  double d;
  if (c & 0x400u) {
    d = X[c & 0x3ffu];
  } else {
    d = v0;
    for (uint32_t m = c & 0x3ffu; m; m &= m - 1) d -= X[__ffs(m) - 1];
  }
  return flip_sign(d, (c & 0x800u) << 20);
}
// Value of an entry that is a sum: any of a single (v0, X[t]), or a two-term form of a double
// (X[0], X[1]: the bare v0, v1).  Out of line, to keep it out of the other entries' way.
__device__ __noinline__ double tab_sum_value(uint32_t ent, uint32_t info, double v0, const double *X) {
  if (((info >> TAB_KIND) & 7u) != 2u) {
    const int f = (int)(ent >> 8) & 15;
    const double x0 = X[0], x1 = X[1], w = x0 - x1;
    const double a = f == 3 ? x0 : f == 4 ? x1 : f == 5 ? w : f < 10 ? x0 : x1;
    const double b = f == 3 ? x0 : f == 4 ? x1 : f == 5 ? w : f < 8 ? x1 : w;
    return flip_sign(tab_scale(a + (f > 5 ? flip_sign(b, (f & 1u) << 31) : b), info), ent & 0x80000000u);
  }
  double t = tab_single_term((ent >> 8) & 0xfffu, v0, X);
  const uint32_t c1 = ent >> 20;
  if (c1 != TAB_NOTERM) t = t + tab_single_term(c1, v0, X);
  return tab_scale(t, info);
}

// ------------------------------------------------------------------------------------
// adjoint
// ------------------------------------------------------------------------------------
// The derivative of a block's elements with respect to one of the pair's integrals is a list of
// (row, column, sign): the program of a table is these lists end to end — doubles v0, v1;
// spin-orbit v0; singles v0, X[0], X[1], ... (to the last that occurs) — with the lists' ends
// (uint16, two a word) before it.  hdr[2 slot + 1].x: first word, .y: lists.  An entry: bits 0-7
// column, 8-15 row, 31 sign.
constexpr int TAB_LISTS = 1 + TAB_MAXOPEN;

// signed count of integral `a` in an entry (0, +-1, +-2); singles: two terms a list may hold it twice
__device__ __forceinline__ int tab_weight(uint32_t ent, bool single, int a) {
  if (!single) {
    constexpr int c0[12] = {1, 0, 1, 2, 0, 2, 1, 1, 2, 0, 1, -1}, c1[12] = {0, 1, -1, 0, 2, -2, 1, -1, -1, 1, 0, 2};
    const int f = (int)(ent >> 8) & 15;
    int w = 0;
#pragma unroll
    for (int u = 0; u < 12; ++u)
      if (f == u) w = a == 0 ? c0[u] : c1[u];
    return (ent >> 31) ? -w : w;
  }
  int w = 0;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const uint32_t c = u ? ent >> 20 : (ent >> 8) & 0xfffu;
    if (u && c == TAB_NOTERM) continue;
    int x = 0;
    if (c & 0x400u) x = (a > 0 && (c & 0x3ffu) == (uint32_t)(a - 1)) ? 1 : 0;
    else x = a == 0 ? 1 : ((c >> (a - 1)) & 1u) ? -1 : 0;
    w += (c & 0x800u) ? -x : x;
  }
  return w;
}

// Programs of all listed slots, from their entries (at most the first `want` lists); one warp a slot,
// lanes over the entries.
__global__ void __launch_bounds__(128) k_tab_program(const uint32_t *__restrict__ list, const int *__restrict__ err,
                                                     int want, uint4 *hdr, uint32_t *pool, unsigned long long *counter,
                                                     int64_t cap) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int npat = err[1];
  for (int64_t p = warp; p < npat; p += nwarps) {
    const int64_t s = list[p];
    const uint4 h = hdr[2 * s];
    const int nent = (int)(h.y & TAB_ENTRIES);
    // entries that did not fit the pool were not written: the host, which sees the count, repeats
    if ((int64_t)h.x + nent + (nent + 3) / 4 > cap) {
      if (lane == 0) hdr[2 * s + 1] = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    const bool single = ((h.y >> TAB_KIND) & 7u) == 2u;
    const uint8_t *rows = reinterpret_cast<const uint8_t *>(pool + h.x + nent);
    const int most = min(want, single ? TAB_LISTS : 2);
    uint32_t words = 0u, off = 0u;
    int lists = 0;
    bool fits = false;
    for (int pass = 0; pass < 2; ++pass) {
      int n = 0;
      for (int a = 0; a < most; ++a) {
        for (int e0 = 0; e0 < nent; e0 += 32) {
          const int e = e0 + lane;
          const uint32_t ent = e < nent ? pool[h.x + e] : 0u;
          const int w = e < nent ? tab_weight(ent, single, a) : 0;
          const unsigned b1 = __ballot_sync(0xffffffffu, w != 0), b2 = __ballot_sync(0xffffffffu, w == 2 || w == -2);
          if (pass == 1 && fits && w != 0) {
            const unsigned lt = (1u << lane) - 1u;
            const uint32_t r = single ? rows[e] : (ent >> 12) & 0xffu;
            const uint32_t x = (ent & 0xffu) | (r << 8) | (w < 0 ? 0x80000000u : 0u);
            uint32_t *to = pool + off + (TAB_LISTS + 1) / 2 + n + __popc(b1 & lt) + __popc(b2 & lt);
            to[0] = x;
            if (w == 2 || w == -2) to[1] = x;
          }
          n += __popc(b1) + __popc(b2);
          if (b1) lists = a + 1;
        }
        if (pass == 1 && fits && lane == 0) reinterpret_cast<uint16_t *>(pool + off)[a] = (uint16_t)n;
      }
      if (pass == 0) {
        words = (uint32_t)(n + (TAB_LISTS + 1) / 2);
        unsigned long long o = 0;
        if (lane == 0) o = atomicAdd(counter, (unsigned long long)words);
        o = __shfl_sync(0xffffffffu, o, 0);
        fits = (int64_t)(o + words) <= cap;
        off = (uint32_t)o;
      }
    }
    if (lane == 0) hdr[2 * s + 1] = make_uint4(off, (uint32_t)lists, 0u, 0u);
  }
}
