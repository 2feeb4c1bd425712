// Row-driven SpMSpV: the product generated and merged one target alpha string at
// a time, without storing a term.
//
// A determinant is a pair of spin strings (A, B).  All targets with alpha string
// A' form a ROW, and the terms of a row come from few places:
//   * sources whose A is one move from A' (opposite-spin doubles: A -> A' times
//     every move of B; and the spin-0 single of each such source);
//   * sources whose A is two moves from A' (spin-0 doubles, B unchanged);
//   * when A' is itself a source string, the diagonals, spin-1 singles and
//     spin-1 doubles of its own sources.
// So the sources are grouped by alpha string, each row gets the list of groups
// it receives from, and one CTA generates a row's terms and merges them in a
// shared-memory hash table over the beta string: a term is a few loads, one FP64
// multiplication and three to five shared-memory reductions, and nothing of it
// reaches HBM.  (The partitioned pipeline of spmspv.cu writes each term once,
// moves it through two partition levels and reads it again: 16 + 80 + 16 B.)
//
// Beta strings are kept hashed: H = B * odd constant mod 2^32 (2^64), a
// bijection, so a table slot needs only H and the string comes back by the
// inverse constant.  Every list a row reads is bucketed by the top bits of H;
// a row too large for one table is processed as ranges of H, each reading only
// its buckets.
//
// Signs: the phase of a move in the interleaved string is its phase in the
// separated order (all alpha, then all beta) times s(source) s(target), where
// s(A, B) is the parity of the interleaving.  Amplitudes are multiplied by s
// when the sources are grouped and the sums by s when a table is read out, so a
// term's phase is the XOR of one alpha and one beta bit.  Negation is exact,
// so every term has the bits the partitioned pipeline gives it, and so has the
// exact sum (FX_FRAC grid, see common.cuh).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "gen.cuh"
#include "merge.cuh"
#include "prims.cuh"
#include "rows.cuh"
#include "strings.cuh"

namespace sfci {

// mark the ranks with sources in the high word, for one scan of both
__global__ void k_rows_mark(u64* __restrict__ arank, unsigned RA) {
  for (unsigned r = blockIdx.x * blockDim.x + threadIdx.x; r < RA; r += gridDim.x * blockDim.x) {
    const u64 v = arank[r];
    if (v) arank[r] = v | (1ull << 32);
  }
}

// out[0]: 1 where a key is not like the first (left alone otherwise); out[1..]: the first
template <class KT>
__global__ void k_keys_check(const KT* __restrict__ keys, u64 n, int N, int unique, u64* __restrict__ out) {
  const KT k0 = keys[0];
  bool bad = false;
  for (u64 j = (u64)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (u64)gridDim.x * blockDim.x) {
    const KT k = keys[j];
    int da = 0, db = 0;
#pragma unroll
    for (int w = 0; w < (int)(sizeof(KT) / 8); ++w) {
      da += popc64(kword(k, w) & 0x5555555555555555ull) - popc64(kword(k0, w) & 0x5555555555555555ull);
      db += popc64(kword(k, w) & 0xaaaaaaaaaaaaaaaaull) - popc64(kword(k0, w) & 0xaaaaaaaaaaaaaaaaull);
    }
    bad |= da || db || !key_within(k, N) || (unique && j && key_eq(k, keys[j - 1]));
  }
  if (bad) out[0] = 1;
  if (blockIdx.x == 0 && threadIdx.x < sizeof(KT) / 8) out[1 + threadIdx.x] = kword(k0, threadIdx.x);
}

template <int W>
int keys_one_spin(Ctx& c, const typename KeyOf<W>::T* keys, u64 n, bool unique, int* na, int* nb, bool* ok) {
  const bool fresh = !c.scratch.count("keys_check");
  u64* out = (u64*)scratch_get(c, "keys_check", 3 * 8);
  if (!out) return SFCI_ERR_NOMEM;
  if (fresh) SFCI_CUDA(cudaMemsetAsync(out, 0, 8, c.stream));
  const unsigned grid = (unsigned)std::max<u64>(1, std::min<u64>((n + 255) / 256, (u64)c.sm_count * 8));
  SFCI_LAUNCH(c, k_keys_check<typename KeyOf<W>::T>, grid, 256, 0, keys, n, c.N, unique ? 1 : 0, out);
  u64 h[3] = {1, 0, 0};
  int st;
  if ((st = read_words(c, out, (1 + W) * 8, h))) return st;
  if (h[0]) SFCI_CUDA(cudaMemsetAsync(out, 0, 8, c.stream));
  *ok = !h[0];
  *na = *nb = 0;
  for (int w = 0; w < W; ++w) {
    *na += popc64(h[1 + w] & 0x5555555555555555ull);
    *nb += popc64(h[1 + w] & 0xaaaaaaaaaaaaaaaaull);
  }
  return SFCI_OK;
}
template int keys_one_spin<1>(Ctx&, const u64*, u64, bool, int*, int*, bool*);
template int keys_one_spin<2>(Ctx&, const K128*, u64, bool, int*, int*, bool*);

// up to four spans of 32-bit words side by side, for one readback
struct Spans {
  const void* p[4];
  int n[4];
};
__global__ void k_rows_gather(Spans s, uint32_t* __restrict__ out) {
  for (int q = 0; q < 4; out += s.n[q++])
    for (int i = threadIdx.x; i < s.n[q]; i += blockDim.x) out[i] = __ldcg((const uint32_t*)s.p[q] + i);
}

namespace {

constexpr int BINS = 40;                   // row size classes (powers of two of the term count)
constexpr unsigned LIGHT_MAX = 128;        // terms of a row one warp merges (256 slots: never full)
constexpr int LIGHT_WARPS = 8;
constexpr int LIGHT_SLOTS = 256;
// Larger rows: threads and table bits (2^TB slots) of a CTA, for rows of fewer
// than 2^MID_BIN terms and for those above.  A step (one filling of the table)
// costs a look at every group the row receives from, so large rows want large
// tables, two CTAs an SM; small rows want many CTAs, whose barriers overlap.
// Measured, whole calls on 3,001, 20,000 and 120,000 sources of 56 spin orbitals: 3.12,
// 13.0 and 63.7 ms with these, 3.24, 14.8 and 73.5 with 256 threads and 2^11 slots for
// the large rows, 3.73, 17.9 and 94.9 with the small rows' size for all; 9,001 of 68
// spin orbitals (8-byte slots): 20.9 ms with 256 threads and 2^11 slots, 23.0 with 512
// and 2^12 (one CTA an SM).  LOAD 0.45 / 0.65 / 0.85 at 120,000: 69.9 / 63.7 / 68.5 ms.
constexpr int MID_THREADS = 128, MID_TB = 10;
template <int W> struct Big { static constexpr int threads = 512, tb = 12; };
template <> struct Big<2> { static constexpr int threads = 256, tb = 11; };
constexpr float LOAD = 0.65f;               // share of a table's slots a step aims to fill
// terms per distinct target the first step of a unit assumes (later steps follow
// the density seen).  With the previous product's mean (3.2 at 120,000 sources) a
// tenth of the first steps overflowed and were redone, 68.2 ms; with 2, one in two
// thousand, 63.7 (a row has no more distinct targets than there are beta strings, either)
constexpr float FIRST_DUP = 2.0f;
constexpr int MID_BIN = 12;                // MID_MAX = 2^MID_BIN - 1 terms
constexpr unsigned D1_PIECE = 128;         // entries of one source's doubles a warp takes at a time
constexpr unsigned PROBE_MAX = 64;         // probes before a table counts as full
constexpr int NW = 5;                      // accumulator words of a slot
constexpr int ROW_EL_MAX = 16;             // electrons of a spin (single_elems)

// row packing: terms << 28 | groups two moves away << 11 | groups one move away
constexpr int RP_D = 11, RP_RAW = 28;

__host__ __device__ constexpr size_t rows_al16(size_t x) { return (x + 15) & ~(size_t)15; }

// ---- tables of one product ----------------------------------------------------
template <int W>
struct RowArgs {
  typedef typename StrOf<W>::T ST;
  typedef typename KeyOf<W>::T KT;
  HamView h;
  int na, nb, nva, nvb;  // electrons and holes per spin
  unsigned nsa, nsb;     // singles per string
  unsigned nda, ndb;     // same-spin doubles per string
  const unsigned* bin;
  const double *sj, *xk; // integrals of the singles (k_rows_sj)
  const double* os;      // opposite-spin integrals [i][a][j][b], orientation chosen (k_rows_os)
  // sources
  const KT* keys;
  const double* amps;
  u64 ns;
  double lambda, coeff;
  const double* diagE;
  unsigned *ra, *rb;     // ranks of each source's strings
  u64* arank;            // per alpha rank: sources | 1 << 32 when any, then their exclusive scan
  uint32_t* brank;       // per beta rank: 1 when any, then the exclusive scan
  unsigned RA, RB;
  unsigned* flag;        // [0] not eligible, [1] a row's term too large, [2] largest group
  // groups (distinct alpha strings), in rank order
  unsigned nG, nB;
  ST* gstr;
  unsigned *gbase, *gcnt;
  unsigned char *gb0, *gb1;  // bucket bits of the two lists of a group
  u64* goff;             // bucket bases: list 0 | list 1 << 32
  uint2* gi;             // list 0: bucket base, bucket bits
  ST* bstr;
  unsigned char* bocc;   // nb per beta string
  // list 0: the sources of each group, bucketed by H(B)
  uint32_t *c0, *off0;
  unsigned *pg, *pb;     // group, beta string
  ST* pH;
  double *pc, *pa, *pd;  // s * coeff * amp, s * amp, s * (D - lambda) * coeff * amp
  // list 1: every spin-1 move of every source of each group, bucketed by H(B')
  uint32_t *c1, *off1;
  ST* eH;
  uint32_t* ex;          // j * M + b | phase << 12 | position within the group << 13
  // per beta string: its moves, and its same-spin doubles bucketed by H
  ST* sH;
  unsigned short* sx;
  ST* dH;
  double* dV;
  unsigned short* dO;    // (1 << db) + 1 bucket offsets per string
  int db;
  // rows
  u64* rpack;            // per alpha rank
  u64* roff;             // S | D << 32, exclusive
  u64* rcur;
  unsigned *rsg, *rsx;   // S entries: group; i | a << 6 | phase << 12
  unsigned* rdg;         // D entries: group and element
  double* rdv;
  // extra sources of one term each (keys and amplitudes from ns on), by row
  u64 nx;
  unsigned* xra;         // alpha ranks
  uint32_t *xc, *xoff;   // per rank: count, exclusive scan
  ST* xH;
  double* xv;            // s * amplitude
  // units
  unsigned* bins;        // [BINS + 1] counts, then cursors at +64
  u64 unit_raw;
  uint4* units;          // rank, first and last H of the unit
  unsigned* light;
  unsigned nunits, nlight;
  unsigned* ucur;        // work counters
  uint4* redo;
  unsigned* nredo;
  // survivors
  FxCut cut;
  KT* sk;
  double* sa;
  u64* scount;           // [0] survivors, [1] distinct
  u64 soft;              // units stop writing above this many survivors
  u64* dexact;
  unsigned smax;         // connections one move away (shared-memory entries)
  int max_exp;           // terms are below 2^max_exp
};

// a term the accumulators do not take: at least 2^max_exp, or not finite
__device__ __forceinline__ bool term_too_large(double x, int max_exp) {
  return (int)(abs_bits(x) >> 52) >= 1023 + max_exp;
}

// opposite-spin integral of the moves i -> a (alpha) and j -> b (beta): the block
// named by the lower of the two occupied spin orbitals (gen.cuh, term_amp)
__global__ void k_rows_os(HamView h, double* __restrict__ os) {
  const int M = h.M;
  const u64 n = (u64)M * M * M * M;
  for (u64 t = (u64)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (u64)gridDim.x * blockDim.x) {
    const int b = (int)(t % M), j = (int)(t / M % M), a = (int)(t / ((u64)M * M) % M), i = (int)(t / ((u64)M * M * M));
    const unsigned pa = (unsigned)spatial_pair(i, a), pb = (unsigned)spatial_pair(j, b);
    os[t] = i <= j ? vat(h, 1, pa, pb) : vat(h, 2, pb, pa);
  }
}

// integrals of the singles (single_elems), directed so that a row over k is contiguous
__global__ void k_rows_sj(HamView h, double* __restrict__ sj, double* __restrict__ sk) {
  const int M = h.M, MM = M * M * M;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 4 * MM; t += gridDim.x * blockDim.x) {
    const int su = t / MM, r = t - su * MM, i = r / (M * M), a = r / M % M, k = r % M;
    sj[t] = vat(h, su, (unsigned)spatial_pair(i, a), (unsigned)spatial_pair(k, k));
    if (su < 2) sk[t] = vat(h, 3 * su, (unsigned)spatial_pair(a, k), (unsigned)spatial_pair(k, i));
  }
}

template <int W>
__global__ void k_rows_split(RowArgs<W> a) {
  typedef typename StrOf<W>::T ST;
  for (u64 j = (u64)blockIdx.x * blockDim.x + threadIdx.x; j < a.ns; j += (u64)gridDim.x * blockDim.x) {
    ST sa, sb;
    split_key(a.keys[j], sa, sb);
    const unsigned ra = rank_of(a.bin, sa), rb = rank_of(a.bin, sb);
    a.ra[j] = ra;
    a.rb[j] = rb;
    atomicAdd((unsigned*)(a.arank + ra), 1u);  // the low word: at most 2^31 sources
    a.brank[rb] = 1u;
  }
}

// extra sources: each adds one term to the row of its own alpha string (counts,
// then entries; an extra determinant of other spin counts, or too large a term,
// declines the product)
template <int W, bool FILL>
__global__ void k_rows_extra(RowArgs<W> a) {
  typedef typename StrOf<W>::T ST;
  unsigned bad = 0;
  for (u64 j = (u64)blockIdx.x * blockDim.x + threadIdx.x; j < a.nx; j += (u64)gridDim.x * blockDim.x) {
    ST sa, sb;
    split_key(a.keys[a.ns + j], sa, sb);
    if (!FILL) {
      if (spop(sa) != a.na || spop(sb) != a.nb || !key_within(a.keys[a.ns + j], a.h.N) ||
          term_too_large(a.amps[a.ns + j], a.max_exp)) {
        bad = 1;
        a.xra[j] = ~0u;
        continue;
      }
      const unsigned r = rank_of(a.bin, sa);
      a.xra[j] = r;
      atomicAdd(a.xc + r, 1u);
      atomicAdd((unsigned long long*)(a.rpack + r), 1ull << RP_RAW);
    } else {
      const unsigned r = a.xra[j];
      if (r == ~0u) continue;
      const unsigned k = a.xoff[r] + atomicSub(a.xc + r, 1u) - 1u;
      a.xH[k] = hs_of(sb);
      a.xv[k] = signed_by(interleave_par(sa, sb), a.amps[a.ns + j]);
    }
  }
  if (bad) atomicOr(a.flag, 1u);
}

// groups and beta strings from the scanned rank tables
template <int W>
__global__ void k_rows_groups(RowArgs<W> a) {
  typedef typename StrOf<W>::T ST;
  unsigned mx = 0;
  const unsigned t0 = blockIdx.x * blockDim.x + threadIdx.x, st = gridDim.x * blockDim.x;
  for (unsigned r = t0; r < a.RA; r += st) {
    const u64 v = a.arank[r], w = a.arank[r + 1];
    const unsigned g = (unsigned)(v >> 32);
    if (g == (unsigned)(w >> 32)) continue;
    const unsigned n = (unsigned)w - (unsigned)v;
    const ST s = unrank_thread<ST>(a.bin, r, a.na, a.h.M);
    a.gstr[g] = s;
    a.gbase[g] = (unsigned)v;
    a.gcnt[g] = n;
    const int b0 = bucket_bits(n), b1 = bucket_bits((u64)n * a.nsb);
    a.gb0[g] = (unsigned char)b0;
    a.gb1[g] = (unsigned char)b1;
    a.goff[g] = (1ull << b0) | (1ull << (b1 + 32));
    mx = max(mx, n);
  }
  for (unsigned r = t0; r < a.RB; r += st) {
    const unsigned b = a.brank[r];
    if (b == a.brank[r + 1]) continue;
    const ST s = unrank_thread<ST>(a.bin, r, a.nb, a.h.M);
    a.bstr[b] = s;
    ST x = s;
    for (int k = 0; k < a.nb; ++k, x &= x - 1) a.bocc[(u64)b * a.nb + k] = (unsigned char)sffs(x);
  }
  if (mx) atomicMax(a.flag + 2, mx);
}

// rows reached from each group: counts (FILL false) or list entries (FILL true).
// A warp takes a slice of one group's moves.
template <int W, bool FILL>
__global__ void __launch_bounds__(256) k_rows_alpha(RowArgs<W> a, unsigned nslice) {
  typedef typename StrOf<W>::T ST;
  __shared__ unsigned char s_o[8][64], s_v[8][64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const u64 nitem = (u64)a.nG * nslice;
  for (u64 it = (u64)blockIdx.x * 8 + warp; it < nitem; it += (u64)gridDim.x * 8) {
    const unsigned g = (unsigned)(it / nslice), sl = (unsigned)(it - (u64)g * nslice);
    const ST s = a.gstr[g];
    __syncwarp();
    for (int p = lane; p < a.h.M; p += 32) {
      const int o = spop((ST)(s & (sbit<ST>(p) - 1)));
      if ((s >> p) & 1) s_o[warp][o] = (unsigned char)p;
      else s_v[warp][p - o] = (unsigned char)p;
    }
    __syncwarp();
    const u64 n = a.gcnt[g];
    if (!FILL && sl == 0 && lane == 0) {
      const unsigned r = rank_of(a.bin, s);
      atomicAdd((unsigned long long*)(a.rpack + r), (n * (1ull + a.nsb + a.ndb)) << RP_RAW);
    }
    for (unsigned t = sl * 32 + lane; t < a.nsa; t += nslice * 32) {
      const int i = s_o[warp][t / a.nva], p = s_v[warp][t % a.nva];
      const unsigned r = rank_of(a.bin, (ST)(s ^ sbit<ST>(i) ^ sbit<ST>(p)));
      if (!FILL) {
        atomicAdd((unsigned long long*)(a.rpack + r), ((n * (1ull + a.nsb)) << RP_RAW) | 1ull);
      } else {
        const unsigned k = (unsigned)a.roff[r] + (unsigned)atomicAdd((unsigned long long*)(a.rcur + r), 1ull);
        a.rsg[k] = g;
        a.rsx[k] = (unsigned)i | ((unsigned)p << 6) | (move_par(s, i, p) << 12);
      }
    }
    const unsigned nvp = a.nva * (a.nva - 1) / 2;
    for (unsigned t = sl * 32 + lane; t < a.nda; t += nslice * 32) {
      const unsigned op = t / nvp, vp = t - op * nvp;
      unsigned x, y, u, v;
      unrank_pair2(op, x, y);
      unrank_pair2(vp, u, v);
      const int i = s_o[warp][x], j = s_o[warp][y], p = s_v[warp][u], q = s_v[warp][v];
      const unsigned r = rank_of(a.bin, (ST)(s ^ sbit<ST>(i) ^ sbit<ST>(j) ^ sbit<ST>(p) ^ sbit<ST>(q)));
      if (!FILL) {
        atomicAdd((unsigned long long*)(a.rpack + r), (n << RP_RAW) | (1ull << RP_D));
      } else {
        const unsigned k = (unsigned)(a.roff[r] >> 32) +
                           (unsigned)(atomicAdd((unsigned long long*)(a.rcur + r), 1ull << 32) >> 32);
        a.rdg[k] = g;
        a.rdv[k] = double_elem(a.h, 0, s, i, j, p, q);
      }
    }
  }
}

// list lengths of each row, for the scan that places its entries
__global__ void k_rows_lens(const u64* __restrict__ rpack, unsigned RA, u64* __restrict__ roff) {
  for (unsigned r = blockIdx.x * blockDim.x + threadIdx.x; r < RA; r += gridDim.x * blockDim.x) {
    const u64 v = rpack[r];
    roff[r] = (v & ((1u << RP_D) - 1u)) | (((v >> RP_D) & ((1u << (RP_RAW - RP_D)) - 1u)) << 32);
  }
}

// Units of work by size class, largest rows first: a row of more than unit_raw
// terms becomes several ranges of H.  Rows of at most LIGHT_MAX terms (they have
// only two-move entries) form their own list, one warp each.
template <int W, bool FILL>
__global__ void __launch_bounds__(256) k_rows_units(RowArgs<W> a) {
  __shared__ unsigned s_n[BINS + 1], s_b[BINS + 1];
  const unsigned tile = 2048;
  for (u64 base = (u64)blockIdx.x * tile; base < a.RA; base += (u64)gridDim.x * tile) {
    for (int i = threadIdx.x; i <= BINS; i += blockDim.x) s_n[i] = 0;
    __syncthreads();
    unsigned loc[tile / 256], cnt[tile / 256];
    int bin[tile / 256];
#pragma unroll
    for (int q = 0; q < (int)(tile / 256); ++q) {
      const u64 r = base + q * 256 + threadIdx.x;
      bin[q] = -1;
      if (r >= a.RA) continue;
      const u64 v = a.rpack[r], raw = v >> RP_RAW;
      if (!raw) continue;
      if (raw <= LIGHT_MAX && !(v & ((1u << RP_D) - 1u))) {
        // a source string's own row has at least 1 + nsb + ndb terms besides
        const bool own = (unsigned)(a.arank[r] >> 32) != (unsigned)(a.arank[r + 1] >> 32);
        if (!own) {
          bin[q] = BINS;
          cnt[q] = 1;
        }
      }
      if (bin[q] < 0) {
        bin[q] = min(BINS - 1, 63 - __clzll((long long)raw));
        cnt[q] = (unsigned)min((raw + a.unit_raw - 1) / a.unit_raw, (u64)4096);
      }
      loc[q] = atomicAdd(&s_n[bin[q]], cnt[q]);
    }
    __syncthreads();
    if (threadIdx.x <= BINS) {
      const unsigned n = s_n[threadIdx.x];
      if (!FILL) {
        if (n) atomicAdd(a.bins + threadIdx.x, n);
      } else {
        unsigned b = 0;  // classes above this one come first
        if (threadIdx.x < BINS)
          for (int i = (int)threadIdx.x + 1; i < BINS; ++i) b += a.bins[i];
        s_b[threadIdx.x] = b + (n ? atomicAdd(a.bins + 64 + threadIdx.x, n) : 0u);
      }
    }
    __syncthreads();
    if (FILL) {
#pragma unroll
      for (int q = 0; q < (int)(tile / 256); ++q) {
        if (bin[q] < 0) continue;
        const unsigned r = (unsigned)(base + q * 256 + threadIdx.x), k = s_b[bin[q]] + loc[q];
        if (bin[q] == BINS) {
          a.light[k] = r;
        } else {
          for (unsigned u = 0; u < cnt[q]; ++u) {
            const u64 lo = (1ull << 32) * u / cnt[q], hi = (1ull << 32) * (u + 1) / cnt[q] - 1;
            a.units[k + u] = make_uint4(r, (unsigned)lo, (unsigned)hi, 0u);
          }
        }
      }
    }
    __syncthreads();
  }
}

// list 0: bucket counts, then entries
template <int W, bool FILL>
__global__ void k_rows_list0(RowArgs<W> a) {
  typedef typename StrOf<W>::T ST;
  if (!FILL)
    for (u64 g = (u64)blockIdx.x * blockDim.x + threadIdx.x; g < a.nG; g += (u64)gridDim.x * blockDim.x)
      a.gi[g] = make_uint2((unsigned)a.goff[g], a.gb0[g]);
  for (u64 j = (u64)blockIdx.x * blockDim.x + threadIdx.x; j < a.ns; j += (u64)gridDim.x * blockDim.x) {
    const unsigned g = (unsigned)(a.arank[a.ra[j]] >> 32), b = a.brank[a.rb[j]];
    const ST s = a.bstr[b], H = hs_of(s);
    const unsigned k = (unsigned)a.goff[g] + bucket_of(hs_top(H), a.gb0[g]);
    if (!FILL) {
      atomicAdd(a.c0 + k, 1u);
    } else {
      const unsigned p = a.off0[k] + atomicSub(a.c0 + k, 1u) - 1u;
      const unsigned par = interleave_par(a.gstr[g], s);
      const double cc = a.coeff * a.amps[j];
      a.pg[p] = g;
      a.pb[p] = b;
      a.pH[p] = H;
      a.pc[p] = signed_by(par, cc);
      a.pa[p] = signed_by(par, a.amps[j]);
      a.pd[p] = signed_by(par, (a.diagE[j] - a.lambda) * cc);
    }
  }
}

// Diagonal elements.  With H's largest elements on the diagonal, a term out of the
// accumulators' range is first of all a diagonal one: the product is declined here,
// before its lists are built.  Found by the rows alone, after their last term, it
// cost the whole row form: 3,001 sources of 56 spin orbitals, out of range, 9.9 ms,
// now 6.4, the partitioned pipeline alone 6.3.  A term found by the rows ends them
// (20,000 sources 27 ms, the rows 18 and the pipeline 23).
template <int W>
__global__ void k_rows_diag(RowArgs<W> a, double* __restrict__ diagE) {
  const u64 nw = ((u64)gridDim.x * blockDim.x) >> 5;
  for (u64 w = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < a.ns; w += nw) {
    const double D = diag_element_warp(a.keys[w], a.h);
    if ((threadIdx.x & 31) == 0) {
      diagE[w] = D;
      if (term_too_large((D - a.lambda) * (a.coeff * a.amps[w]), a.max_exp)) atomicOr(a.flag, 1u);
    }
  }
}

// moves of each beta string
template <int W>
__global__ void __launch_bounds__(256) k_rows_bsingles(RowArgs<W> a) {
  typedef typename StrOf<W>::T ST;
  const u64 n = (u64)a.nB * a.nsb;
  for (u64 t = (u64)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (u64)gridDim.x * blockDim.x) {
    const unsigned b = (unsigned)(t / a.nsb), k = (unsigned)(t - (u64)b * a.nsb);
    const ST s = a.bstr[b];
    const int j = a.bocc[(u64)b * a.nb + k / a.nvb];
    // the (k mod nvb)-th empty orbital
    int q = (int)(k % a.nvb), p = 0;
    ST e = ~s;
    for (; q; --q) e &= e - 1;
    p = sffs(e);
    a.sH[t] = hs_of((ST)(s ^ sbit<ST>(j) ^ sbit<ST>(p)));
    a.sx[t] = (unsigned short)((unsigned)(j * a.h.M + p) | (move_par(s, j, p) << 12));
  }
}

// list 1: a warp per source
template <int W, bool FILL>
__global__ void __launch_bounds__(256) k_rows_list1(RowArgs<W> a) {
  typedef typename StrOf<W>::T ST;
  const int lane = threadIdx.x & 31;
  const u64 nw = ((u64)gridDim.x * blockDim.x) >> 5;
  for (u64 p = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < a.ns; p += nw) {
    const unsigned g = a.pg[p], b = a.pb[p];
    const unsigned base = (unsigned)(a.goff[g] >> 32);
    const int bits = a.gb1[g];
    const unsigned lp = (unsigned)p - a.gbase[g];
    for (unsigned t = lane; t < a.nsb; t += 32) {
      const ST H = a.sH[(u64)b * a.nsb + t];
      const unsigned k = base + bucket_of(hs_top(H), bits);
      if (!FILL) {
        atomicAdd(a.c1 + k, 1u);
      } else {
        const unsigned e = a.off1[k] + atomicSub(a.c1 + k, 1u) - 1u;
        a.eH[e] = H;
        a.ex[e] = (uint32_t)a.sx[(u64)b * a.nsb + t] | (lp << 13);
      }
    }
  }
}

// same-spin doubles of each beta string, bucketed by H: a CTA per string
template <int W>
__global__ void __launch_bounds__(256) k_rows_bdoubles(RowArgs<W> a) {
  typedef typename StrOf<W>::T ST;
  extern __shared__ __align__(16) unsigned char smem[];
  uint32_t* cnt = reinterpret_cast<uint32_t*>(smem);
  __shared__ unsigned char s_o[64], s_v[64];
  __shared__ uint32_t s_scan[256 / 32 + 1];
  const unsigned nbk = 1u << a.db, per = (nbk + 255) / 256;
  const unsigned nvp = a.nvb * (a.nvb - 1) / 2;
  for (unsigned b = blockIdx.x; b < a.nB; b += gridDim.x) {
    const ST s = a.bstr[b];
    if ((int)threadIdx.x < a.h.M) {
      const int p = threadIdx.x, o = spop((ST)(s & (sbit<ST>(p) - 1)));
      if ((s >> p) & 1) s_o[o] = (unsigned char)p;
      else s_v[p - o] = (unsigned char)p;
    }
    for (unsigned k = threadIdx.x; k < nbk; k += 256) cnt[k] = 0;
    __syncthreads();
    for (int pass = 0; pass < 2; ++pass) {
      for (unsigned t = threadIdx.x; t < a.ndb; t += 256) {
        const unsigned op = t / nvp, vp = t - op * nvp;
        unsigned x, y, u, v;
        unrank_pair2(op, x, y);
        unrank_pair2(vp, u, v);
        const int i = s_o[x], j = s_o[y], p = s_v[u], q = s_v[v];
        const ST H = hs_of((ST)(s ^ sbit<ST>(i) ^ sbit<ST>(j) ^ sbit<ST>(p) ^ sbit<ST>(q)));
        const unsigned k = bucket_of(hs_top(H), a.db);
        if (!pass) {
          atomicAdd(&cnt[k], 1u);
        } else {
          const u64 e = (u64)b * a.ndb + atomicAdd(&cnt[k], 1u);
          a.dH[e] = H;
          a.dV[e] = double_elem(a.h, 1, s, i, j, p, q);
        }
      }
      __syncthreads();
      if (!pass) {
        uint32_t sum = 0;
        for (unsigned k = 0; k < per; ++k)
          if (threadIdx.x * per + k < nbk) sum += cnt[threadIdx.x * per + k];
        uint32_t run = block_excl_scan<uint32_t, 256>(sum, nullptr, s_scan);
        for (unsigned k = 0; k < per; ++k) {
          const unsigned i = threadIdx.x * per + k;
          if (i < nbk) {
            const uint32_t n = cnt[i];
            cnt[i] = run;
            a.dO[(u64)b * (nbk + 1) + i] = (unsigned short)run;
            run += n;
          }
        }
        if (threadIdx.x == 0) a.dO[(u64)b * (nbk + 1) + nbk] = (unsigned short)a.ndb;
        __syncthreads();
      }
    }
  }
}

// ---- the merge ----------------------------------------------------------------
// A slot holds H (0: free; no string of one or more electrons hashes to 0) and
// the exact sum of its terms' FX_FRAC-grid integers as NW words of DB-bit
// digits in sign-magnitude: |digit| < 2^DB, so a word takes 2^(31 - DB) terms.
template <class ST, int DB>
struct RowTable {
  ST* k;
  unsigned* w;
  unsigned n;  // word stride

  // Add (flip ? -x : x) to the sum of slot s (-1: nothing).
  __device__ __forceinline__ void acc(int s, double x, unsigned flip, int max_exp, unsigned& bad) const {
    // x on the FX_FRAC grid, nearest, ties to even, as in fx_addends
    const u64 b = dbl_bits(x);
    const int e = (int)((b >> 52) & 0x7ff);
    const u64 m = (b & 0xfffffffffffffull) | (1ull << 52);
    const int sh = (1075 - FX_FRAC) - e;  // |F| = m * 2^-sh
    if (s >= 0 && sh <= 53 && e != 0) {
      u64 l, hi = 0;
      if (sh > 0) {
        l = (m + ((1ull << (sh - 1)) - 1ull) + ((m >> sh) & 1ull)) >> sh;
      } else {
        if (e >= 1023 + max_exp) bad = 1u;
        l = m << (-sh & 63);  // max_exp is at most 15: a shift below 64 unless bad
        if (sh) hi = m >> ((64 + sh) & 63);
      }
      const unsigned neg = 0u - ((unsigned)(b >> 63) ^ flip);
      unsigned* p = w + s;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const unsigned d = (unsigned)(l >> (DB * q)) & ((1u << DB) - 1u);
        atomicAdd(p + q * n, (d ^ neg) - neg);
      }
      if ((l >> (3 * DB)) | hi) {
        const unsigned d = (unsigned)(l >> (3 * DB)) & ((1u << DB) - 1u);
        atomicAdd(p + 3 * n, (d ^ neg) - neg);
        unsigned t;
        if constexpr (DB == 16) t = (unsigned)hi;
        else t = (unsigned)((l >> (4 * DB)) | (hi << (64 - 4 * DB)));
        if (t) atomicAdd(p + 4 * n, (t ^ neg) - neg);
      }
    }
  }
  // Add to H's sum, for the lanes with `act`; every lane of the warp calls it, so
  // that the lanes that claimed a slot and those that found theirs go on together
  // (left to itself the compiler ran the two groups one after the other through the
  // rounding and the reductions).  False: no free slot.
  __device__ __forceinline__ bool add(bool act, ST H, double x, unsigned flip, int tb, int max_exp,
                                      unsigned& bad) const {
    const int s = slot<true>(act, H, tb);
    acc(s, x, flip, max_exp, bad);
    return !act || s >= 0;
  }
  // two entries a lane: their bucket loads overlap and share the probe loop
  __device__ __forceinline__ bool add2(bool a0, ST H0, double x0, unsigned f0, bool a1, ST H1, double x1, unsigned f1,
                                       int tb, int max_exp, unsigned& bad) const {
    const unsigned mask = (1u << (tb - 2)) - 1u;
    unsigned b0 = hs_slot(H0, tb - 2), b1 = hs_slot(H1, tb - 2);
    int s0 = -1, s1 = -1;
    bool p0 = a0, p1 = a1;
    for (unsigned probe = 0; probe < PROBE_MAX; ++probe) {
      look<true>(p0, H0, b0, s0, mask);
      look<true>(p1, H1, b1, s1, mask);
      if (!__any_sync(0xffffffffu, p0 || p1)) break;
    }
    acc(s0, x0, f0, max_exp, bad);
    acc(s1, x1, f1, max_exp, bad);
    return (!a0 || s0 >= 0) && (!a1 || s1 >= 0);
  }
  static __device__ __forceinline__ uint32_t cas(uint32_t* p, uint32_t v) { return atomicCAS(p, 0u, v); }
  static __device__ __forceinline__ u64 cas(u64* p, u64 v) {
    return atomicCAS((unsigned long long*)p, 0ull, (unsigned long long)v);
  }
  __device__ __forceinline__ void sum(unsigned s, u64& L, u64& Hi) const {
    // digits 0-1 and 2-3 as 64-bit sums, then 128 bits
    const long long x = (long long)(int)w[s] + ((long long)(int)w[n + s] << DB);
    const long long y = (long long)(int)w[2 * n + s] + ((long long)(int)w[3 * n + s] << DB);
    const long long z = (long long)(int)w[4 * n + s];
    const u64 ylo = (u64)y << (2 * DB);
    L = (u64)x + ylo;
    Hi = (u64)(x >> 63) + (u64)(y >> (64 - 2 * DB)) + (L < ylo ? 1ull : 0ull);
    if constexpr (DB == 16) {
      Hi += (u64)z;
    } else {
      const u64 zlo = (u64)z << (4 * DB);
      L += zlo;
      Hi += (u64)(z >> (64 - 4 * DB)) + (L < zlo ? 1ull : 0ull);
    }
  }
  // Slot of H for the lanes with `act`, claimed when CLAIM; -1: not there (or no
  // free slot within the probe limit).  Slots form buckets of four, read with one
  // or two 16-byte loads and filled in order, so a warp rarely needs a second probe: with
  // single-slot probing the slowest of 32 lanes took five or six at the same load.
  template <bool CLAIM>
  __device__ __forceinline__ int slot(bool act, ST H, int tb) const {
    const unsigned mask = (1u << (tb - 2)) - 1u;
    unsigned b = hs_slot(H, tb - 2);
    int s = -1;
    for (unsigned probe = 0; probe < PROBE_MAX; ++probe) {
      look<CLAIM>(act, H, b, s, mask);
      if (!__any_sync(0xffffffffu, act)) break;
    }
    return s;
  }
  // one probe: clears `act` when H was found (s), claimed (s) or, unless CLAIM, is absent
  template <bool CLAIM>
  __device__ __forceinline__ void look(bool& act, ST H, unsigned& b, int& s, unsigned mask) const {
    constexpr int BS = 4;
    if (act) {
      ST v[BS];
      load_bucket(k + b * BS, v);
      int hit = -1, free = -1;
#pragma unroll
      for (int i = BS - 1; i >= 0; --i) {
        if (v[i] == H) hit = i;
        if (v[i] == 0) free = i;
      }
      if (hit >= 0) {
        s = (int)(b * BS) + hit;
        act = false;
      } else if (free >= 0) {
        if (CLAIM) {  // (when another key took it, the bucket is looked at again)
          const ST old = cas(k + b * BS + free, H);
          if (old == 0 || old == H) {
            s = (int)(b * BS) + free;
            act = false;
          }
        } else {
          act = false;
        }
      } else {
        b = (b + 1u + (unsigned)(H & 6u)) & mask;  // (odd: every bucket is reached)
      }
    }
  }
  static __device__ __forceinline__ void load_bucket(const uint32_t* p, uint32_t* v) {
    asm volatile("ld.volatile.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"((unsigned)__cvta_generic_to_shared(p)));
  }
  static __device__ __forceinline__ void load_bucket(const u64* p, u64* v) {
    const unsigned q = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v[0]), "=l"(v[1]) : "r"(q));
    asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2 + 16];" : "=l"(v[2]), "=l"(v[3]) : "r"(q));
  }
};

template <class ST>
__host__ __device__ inline size_t row_table_bytes(unsigned slots) {
  return rows_al16((sizeof(ST) + NW * sizeof(unsigned)) * slots);
}

// read out a table: its sums through the cut into the survivor list, slots cleared
template <int W, int DB>
__device__ __forceinline__ unsigned row_flush(const RowArgs<W>& a, const RowTable<typename StrOf<W>::T, DB>& t,
                                              typename StrOf<W>::T rstr, unsigned tsize, unsigned first,
                                              unsigned step, bool emit) {
  typedef typename StrOf<W>::T ST;
  const int lane = threadIdx.x & 31;
  unsigned used = 0;
  for (unsigned s0 = first; s0 < tsize; s0 += step) {  // first, step and tsize: multiples of 32
    const unsigned s = s0 + lane;
    const ST H = t.k[s];
    bool keep = false;
    double v = 0.0;
    ST B = 0;
    if (H) {
      if (emit) {
        ++used;
        u64 L, Hi;
        t.sum(s, L, Hi);
        keep = fx_survives_value(L, Hi, a.cut, v);
        if (keep) {
          B = hs_inv(H);
          // s(A', B'); a sum of zero has no sign
          if (interleave_par(rstr, B) && v != 0.0) v = -v;
        }
      }
      t.k[s] = 0;
#pragma unroll
      for (int q = 0; q < NW; ++q) t.w[q * t.n + s] = 0u;
    }
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (m) {
      u64 b0 = 0;
      if (lane == 0) b0 = atomicAdd((unsigned long long*)a.scount, (unsigned long long)__popc(m));
      b0 = __shfl_sync(0xffffffffu, b0, 0);
      if (keep) {
        const u64 p = b0 + __popc(m & ((1u << lane) - 1u));
        a.sk[p] = join_key(rstr, B);
        a.sa[p] = v;
      }
    }
  }
  return used;
}

// rows of at most LIGHT_MAX terms: one warp each.  Such a row has only two-move
// entries, and its table of LIGHT_SLOTS slots cannot fill up.
template <int W, int DB>
__global__ void __launch_bounds__(LIGHT_WARPS * 32) k_rows_light(RowArgs<W> a) {
  typedef typename StrOf<W>::T ST;
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  RowTable<ST, DB> t;
  unsigned char* base = smem + row_table_bytes<ST>(LIGHT_SLOTS) * warp;
  t.k = reinterpret_cast<ST*>(base);
  t.w = reinterpret_cast<unsigned*>(base + sizeof(ST) * LIGHT_SLOTS);
  t.n = LIGHT_SLOTS;
  for (unsigned s = lane; s < LIGHT_SLOTS; s += 32) {
    t.k[s] = 0;
#pragma unroll
    for (int q = 0; q < NW; ++q) t.w[q * LIGHT_SLOTS + s] = 0u;
  }
  __syncwarp();
  unsigned bad = 0;
  u64 uq = 0;
  const u64 nw = (u64)gridDim.x * LIGHT_WARPS;
  // (a term was too large: the product is declined)
  if (__shfl_sync(0xffffffffu, *(volatile unsigned*)(a.flag + 1), 0)) return;
  for (u64 i = (u64)blockIdx.x * LIGHT_WARPS + warp; i < a.nlight; i += nw) {
    const unsigned r = a.light[i];
    // (a later launch sees the same survivor count, so a skipped row is never half written)
    const u64 sc = __shfl_sync(0xffffffffu, *(volatile u64*)a.scount, 0);
    if (sc > a.soft) {
      if (lane == 0) a.redo[atomicAdd(a.nredo, 1u)] = make_uint4(r, 0u, 0xffffffffu, 0u);
      continue;
    }
    const u64 o0 = a.roff[r], o1 = a.roff[r + 1];
    const unsigned d0 = (unsigned)(o0 >> 32), d1 = (unsigned)(o1 >> 32);
    const unsigned raw = (unsigned)(a.rpack[r] >> RP_RAW);
    int tb = 5;
    while (tb < 8 && (1u << tb) < 2 * raw) ++tb;
    for (unsigned d = d0; d < d1; d += 32) {
      unsigned st = 0, len = 0;
      double val = 0.0;
      if (d + lane < d1) {
        const unsigned g = a.rdg[d + lane];
        st = a.gbase[g];
        len = a.gcnt[g];
        val = a.rdv[d + lane];
      }
      warp_expand(st, len, val, [&](bool ok, unsigned e, double v) {
        t.add(ok, a.pH[e], a.pc[e] * v, 0u, tb, a.max_exp, bad);
      });
    }
    if (a.nx)
      for (unsigned x0 = a.xoff[r], x1 = a.xoff[r + 1]; x0 < x1; x0 += 32) {
        const unsigned x = min(x0 + lane, x1 - 1);
        t.add(x0 + lane < x1, a.xH[x], a.xv[x], 0u, tb, a.max_exp, bad);
      }
    __syncwarp();
    const ST rstr = unrank_warp<ST>(a.bin, r, a.na, a.h.M);
    uq += row_flush<W, DB>(a, t, rstr, 1u << tb, 0u, 32u, true);
    __syncwarp();
  }
  if (bad) atomicOr(a.flag + 1, 1u);
  uq = warp_sum(uq);
  if (lane == 0 && uq) atomicAdd((unsigned long long*)(a.scount + 1), (unsigned long long)uq);
}

template <int W, int TB>
__host__ __device__ inline size_t row_cta_smem(unsigned smax) {
  return row_table_bytes<typename StrOf<W>::T>(1u << TB) + rows_al16(sizeof(unsigned) * (smax + 1)) * 7;
}

// Larger rows: a CTA per unit.  Bound by instruction issue and by the latency that
// half the warps an SM holds leave open: 10.8 warp instructions a term at 24 of 32
// lanes (0.61e9 terms from 20,000 sources of 56 spin orbitals: hash, two-word
// rounding, three to five 32-bit shared reductions, and the steps' set-up) take 61% of
// the issue slots, the rest goes to waits, barriers and loads; DRAM is idle and L2
// serves the lists.  Whole calls with the result's download, partitioned pipeline
// against this one: 120,000 sources of 56 spin orbitals (3.7e9 terms) 178.5 and 63.4
// ms, 3,001 sources 5.7 and 3.2 ms, 9,001 of 68 spin orbitals 37.2 and 21.8 ms.  The unit's range of H is walked in steps
// that fill the table to LOAD; a step whose table overflows is redone at half its
// width.
template <int W, int DB, int NT, int TB_MAX>
__global__ void __launch_bounds__(NT, (W == 1 ? 1024 : 768) / NT) k_rows_cta(RowArgs<W> a) {
  typedef typename StrOf<W>::T ST;
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int NWARP = NT / 32;
  constexpr int CTA_SLOTS = 1 << TB_MAX;
  RowTable<ST, DB> tab;
  tab.k = reinterpret_cast<ST*>(smem);
  tab.w = reinterpret_cast<unsigned*>(smem + sizeof(ST) * CTA_SLOTS);
  tab.n = CTA_SLOTS;
  unsigned char* cb = smem + row_table_bytes<ST>(CTA_SLOTS);
  const size_t cs = rows_al16(sizeof(unsigned) * (a.smax + 1));
  unsigned* c_g = reinterpret_cast<unsigned*>(cb);            // groups one move away: group,
  unsigned* c_row = reinterpret_cast<unsigned*>(cb + cs);     // integral row of the move | phase << 31,
  unsigned* c_gb = reinterpret_cast<unsigned*>(cb + 2 * cs);  // first source,
  unsigned* c_o1 = reinterpret_cast<unsigned*>(cb + 3 * cs);  // list-1 range start less c_p1,
  unsigned* c_p1 = reinterpret_cast<unsigned*>(cb + 4 * cs);  // list-1 lengths, then their prefix,
  unsigned* c_o0 = reinterpret_cast<unsigned*>(cb + 5 * cs);  // and the same for list 0
  unsigned* c_p0 = reinterpret_cast<unsigned*>(cb + 6 * cs);
  __shared__ uint4 s_unit;
  __shared__ ST s_str;
  __shared__ unsigned s_ovf, s_w1, s_w2, s_w3, s_used, s_stop, s_w4;
  __shared__ u64 s_red[NWARP];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int M = a.h.M;
  for (unsigned s = tid; s < CTA_SLOTS; s += NT) {
    tab.k[s] = 0;
#pragma unroll
    for (int q = 0; q < NW; ++q) tab.w[q * CTA_SLOTS + s] = 0u;
  }
  unsigned bad = 0, dbad = 0;
  u64 uq = 0, dlo = 0, dhi = 0;  // distinct targets; this thread's share of <v|Hv>
  for (;;) {
    if (tid == 0) {
      // (no more units once a term was too large: the product is then declined)
      const unsigned stop = *(volatile unsigned*)(a.flag + 1), u = atomicAdd(a.ucur, 1u);
      s_unit = u < a.nunits && !stop ? a.units[u] : make_uint4(0u, 1u, 0u, 0u);
    }
    __syncthreads();
    const uint4 un = s_unit;
    if (un.y > un.z) break;
    const unsigned r = un.x;
    if (warp == 0) {
      const ST x = unrank_warp<ST>(a.bin, r, a.na, M);
      if (lane == 0) s_str = x;
    }
    const u64 o0 = a.roff[r], o1 = a.roff[r + 1];
    const unsigned sb = (unsigned)o0, nS = (unsigned)o1 - sb;
    const unsigned db = (unsigned)(o0 >> 32), nD = (unsigned)(o1 >> 32) - db;
    const unsigned gs = (unsigned)(a.arank[r] >> 32);
    const bool own = gs != (unsigned)(a.arank[r + 1] >> 32);
    const float raw = (float)(a.rpack[r] >> RP_RAW);
    for (unsigned i = tid; i < nS; i += NT) {
      const unsigned g = a.rsg[sb + i], x = a.rsx[sb + i];
      c_g[i] = g;
      c_row[i] = (((x & 63u) * M + ((x >> 6) & 63u)) * M * M) | ((x >> 12) << 31);
      c_gb[i] = a.gbase[g];
    }
    // step width: distinct targets are at most the terms of the step
    const float target = LOAD * CTA_SLOTS;
    const float guess = fminf(raw * (1.0f / FIRST_DUP), (float)a.RB);  // distinct targets of the row
    u64 width = (u64)fminf(4294967296.0f, fmaxf(1.0f, 4294967296.0f * target / guess));
    bool wide = false;  // a table sized for this row's mean density was too small
    u64 lo = un.y;
    const u64 end = (u64)un.z + 1;
    while (lo < end) {
      const u64 hi = min(end, lo + width);  // this step: tops in [lo, hi)
      const uint32_t tlo = (uint32_t)lo, thi = (uint32_t)(hi - 1), span = thi - tlo;
      const float sraw = raw * (float)(hi - lo) * (1.0f / 4294967296.0f);
      int tb = wide ? TB_MAX : 6;
      while (tb < TB_MAX && (float)(1u << tb) < 2.0f * sraw + 32.0f) ++tb;
      if (tid == 0) {
        s_ovf = 0;
        s_w1 = s_w2 = s_w3 = s_w4 = 0;
        s_used = 0;
        s_stop = *(volatile u64*)a.scount > a.soft;
      }
      // (1) ranges of the groups one move away
      for (unsigned i = tid; i < nS; i += NT) {
        const unsigned g = c_g[i];
        const u64 go = a.goff[g];
        const int b0 = a.gb0[g], b1 = a.gb1[g];
        const uint32_t* f1 = a.off1 + (unsigned)(go >> 32);
        const uint32_t* f0 = a.off0 + (unsigned)go;
        const unsigned s1 = f1[bucket_of(tlo, b1)], e1 = f1[bucket_of(thi, b1) + 1];
        const unsigned s0 = f0[bucket_of(tlo, b0)], e0 = f0[bucket_of(thi, b0) + 1];
        c_o1[i] = s1;
        c_p1[i] = e1 - s1;
        c_o0[i] = s0;
        c_p0[i] = e0 - s0;
      }
      __syncthreads();
      if (s_stop) break;
      // (2) prefixes
      for (int w = warp; w < 2; w += NWARP) {
        unsigned *p = w ? c_p0 : c_p1, *q = w ? c_o0 : c_o1;
        unsigned carry = 0;
        for (unsigned i0 = 0; i0 < nS; i0 += 32) {
          const unsigned i = i0 + lane;
          const unsigned v = i < nS ? p[i] : 0u;
          unsigned x = v;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
          }
          if (i < nS) {
            p[i] = carry + x - v;
            q[i] -= carry + x - v;
          }
          carry += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0) p[nS] = carry;
      }
      __syncthreads();
      bool full = false;
      // The long chains of loads first, the finest-grained work last: the warps
      // share each kind through a counter and meet again at the barrier after (3e).
      // (3a) spin-0 singles of the groups one move away
      {
        const unsigned n = c_p0[nS];
        for (unsigned i0 = warp * 32; i0 < n; i0 += NT) {
          const unsigned i = min(i0 + lane, n - 1);
          unsigned l = 0, h = nS;
          while (h - l > 1) {
            const unsigned m = (l + h) >> 1;
            if (c_p0[m] <= i) l = m; else h = m;
          }
          const unsigned row = c_row[l], ia = (row & 0x7fffffffu) / (M * M), p = c_o0[l] + i;
          const ST H = a.pH[p];
          const bool act = i0 + lane < n && hs_top(H) - tlo <= span;
          const double v = single_elems<ST>(a.sj, a.xk, a.h.h1, M, 0, (int)(ia / M), (int)(ia % M), a.gstr[c_g[l]],
                                            hs_inv(H), a.na, a.nb, act);
          full |= !tab.add(act, H, a.pc[p] * v, row >> 31, tb, a.max_exp, bad);
        }
      }
      // (3b) the row's own sources: spin-1 singles and diagonals
      unsigned p0 = 0, p1 = 0;
      if (own) {
        const u64 go = a.goff[gs];
        const uint32_t* f1 = a.off1 + (unsigned)(go >> 32);
        const uint32_t* f0 = a.off0 + (unsigned)go;
        const int b0 = a.gb0[gs], b1 = a.gb1[gs];
        const unsigned s1 = f1[bucket_of(tlo, b1)], e1 = f1[bucket_of(thi, b1) + 1];
        p0 = f0[bucket_of(tlo, b0)];
        p1 = f0[bucket_of(thi, b0) + 1];
        const unsigned gb = a.gbase[gs];
        for (unsigned i0 = s1 + warp * 32; i0 < e1; i0 += NT) {
          const unsigned e = min(i0 + lane, e1 - 1);
          const ST H = a.eH[e];
          const uint32_t y = a.ex[e];
          const bool act = i0 + lane < e1 && hs_top(H) - tlo <= span;
          const unsigned p = gb + (y >> 13), q = y & 0xfffu;
          const double v = single_elems<ST>(a.sj, a.xk, a.h.h1, M, 1, (int)(q / M), (int)(q % M), s_str,
                                            hs_inv(a.pH[p]), a.na, a.nb, act);
          full |= !tab.add(act, H, a.pc[p] * v, (y >> 12) & 1u, tb, a.max_exp, bad);
        }
        for (unsigned i0 = p0 + warp * 32; i0 < p1; i0 += NT) {
          const unsigned p = min(i0 + lane, p1 - 1);
          const ST H = a.pH[p];
          full |= !tab.add(i0 + lane < p1 && hs_top(H) - tlo <= span, H, a.pd[p], 0u, tb, a.max_exp, bad);
        }
      }
      // extra sources of the row (unbucketed: each step passes over them)
      if (a.nx)
        for (unsigned x0 = a.xoff[r] + warp * 32, x1 = a.xoff[r + 1]; x0 < x1; x0 += NT) {
          const unsigned x = min(x0 + lane, x1 - 1);
          const ST H = a.xH[x];
          full |= !tab.add(x0 + lane < x1 && hs_top(H) - tlo <= span, H, a.xv[x], 0u, tb, a.max_exp, bad);
        }
      // (3c) spin-1 doubles of the row's own sources: pieces of one source's list
      // while those are long enough for a warp, else 32 lists at a time
      if (own && a.ndb) {
        const unsigned n = a.gcnt[gs], gb = a.gbase[gs];
        const float mean = (float)a.ndb * (float)(hi - lo) * (1.0f / 4294967296.0f);
        const bool pieces = mean >= 24.0f;
        const unsigned np = pieces ? (unsigned)(mean * (1.0f / D1_PIECE)) + 1u : 1u;  // the last piece takes the rest
        const unsigned step = pieces ? 1u : 32u, last = pieces ? n * np : n;
        for (;;) {
          unsigned i0 = 0;
          if (lane == 0) i0 = *(volatile unsigned*)&s_ovf ? ~0u : atomicAdd(&s_w3, step);
          i0 = __shfl_sync(0xffffffffu, i0, 0);
          if (i0 >= last) break;
          if (pieces) {
            const unsigned p = gb + i0 / np, j = i0 % np;
            const u64 b = a.pb[p];
            const unsigned short* f = a.dO + b * ((1u << a.db) + 1);
            const u64 e0 = b * a.ndb + f[bucket_of(tlo, a.db)] + j * D1_PIECE;
            const u64 e9 = b * a.ndb + f[bucket_of(thi, a.db) + 1];
            const u64 e1 = j + 1 < np ? min(e9, e0 + D1_PIECE) : e9;
            const double c = a.pc[p];
            for (u64 f0 = e0; f0 < e1; f0 += 32) {
              const u64 e = min(f0 + lane, e1 - 1);
              const ST H = a.dH[e];
              const bool act = f0 + lane < e1 && hs_top(H) - tlo <= span;
              full |= !tab.add(act, H, c * a.dV[e], 0u, tb, a.max_exp, bad);
            }
          } else {
            unsigned st = 0, len = 0;
            double val = 0.0;
            if (i0 + lane < n) {
              const unsigned p = gb + i0 + lane;
              const u64 b = a.pb[p];
              const unsigned short* f = a.dO + b * ((1u << a.db) + 1);
              const unsigned s0 = f[bucket_of(tlo, a.db)];
              st = (unsigned)(b * a.ndb) + s0;
              len = f[bucket_of(thi, a.db) + 1] - s0;
              val = a.pc[p];
            }
            warp_expand(st, len, val, [&](bool ok, unsigned e, double v) {
              const ST H = a.dH[e];
              full |= !tab.add(ok && hs_top(H) - tlo <= span, H, v * a.dV[e], 0u, tb, a.max_exp, bad);
            });
          }
          if (full) s_ovf = 1;
        }
      }
      // (3d) spin-0 doubles: 32 groups' sources at a time
      for (;;) {
        unsigned i0 = 0;
        if (lane == 0) i0 = *(volatile unsigned*)&s_ovf ? ~0u : atomicAdd(&s_w2, 32u);
        i0 = __shfl_sync(0xffffffffu, i0, 0);
        if (i0 >= nD) break;
        unsigned st = 0, len = 0;
        double val = 0.0;
        if (i0 + lane < nD) {
          const uint2 gi = a.gi[a.rdg[db + i0 + lane]];
          const uint32_t* f0 = a.off0 + gi.x;
          st = f0[bucket_of(tlo, (int)gi.y)];
          len = f0[bucket_of(thi, (int)gi.y) + 1] - st;
          val = a.rdv[db + i0 + lane];
        }
        warp_expand(st, len, val, [&](bool ok, unsigned e, double v) {
          const ST H = a.pH[e];
          full |= !tab.add(ok && hs_top(H) - tlo <= span, H, v * a.pc[e], 0u, tb, a.max_exp, bad);
        });
        if (full) s_ovf = 1;
      }
      // (3e) opposite-spin doubles: the groups' move lists as one flat list, of
      // which warps take a chunk at a time (lane 0 decides for the warp: the
      // loops hold warp collectives); each lane follows the group its entry is in
      const unsigned n1 = c_p1[nS];
      const unsigned chunk = min(256u, max(64u, (n1 / (NWARP * 8)) & ~63u));
      for (;;) {
        unsigned t = 0;
        if (lane == 0) t = *(volatile unsigned*)&s_ovf ? ~0u : atomicAdd(&s_w1, chunk);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= n1) break;
        const unsigned te = min(n1, t + chunk);
        // (the entry is clamped before the search: past the end it would find a
        // group that does not hold the clamped entry)
        unsigned l = 0, h = nS;
        const unsigned first = min(t + lane, te - 1);
        while (h - l > 1) {
          const unsigned m = (l + h) >> 1;
          if (c_p1[m] <= first) l = m; else h = m;
        }
        // the lane's group: last entry, entry offset, first source, integral row
        unsigned pe = c_p1[l + 1], o1 = c_o1[l], gb = c_gb[l], row = c_row[l];
        auto entry = [&](unsigned i, ST& H, double& v, unsigned& par) {
          if (i >= pe) {
            do ++l; while (c_p1[l + 1] <= i);
            pe = c_p1[l + 1];
            o1 = c_o1[l];
            gb = c_gb[l];
            row = c_row[l];
          }
          const unsigned e = o1 + i;
          H = a.eH[e];
          const uint32_t y = a.ex[e];
          v = a.pc[gb + (y >> 13)] * SFCI_LDG(a.os + (row & 0x7fffffffu) + (y & 0xfffu));
          par = (row >> 31) ^ ((y >> 12) & 1u);
        };
        for (; t < te; t += 64) {
          ST H0, H1;
          double v0, v1;
          unsigned f0, f1;
          entry(min(t + lane, te - 1), H0, v0, f0);
          entry(min(t + 32 + lane, te - 1), H1, v1, f1);
          const bool a0 = t + lane < te && hs_top(H0) - tlo <= span, a1 = t + 32 + lane < te && hs_top(H1) - tlo <= span;
          full |= !tab.add2(a0, H0, v0, f0, a1, H1, v1, f1, tb, a.max_exp, bad);
        }
        if (full) s_ovf = 1;
      }
      if (full) s_ovf = 1;
      __syncthreads();
      const bool ovf = s_ovf != 0;
      if (own && !ovf) {
        // <v|Hv>: the row's own sources look their merged amplitude up (the
        // interleaving signs of both factors cancel)
        for (unsigned i0 = p0 + warp * 32; i0 < p1; i0 += NT) {
          const unsigned p = min(i0 + lane, p1 - 1);
          const ST H = a.pH[p];
          const int s = tab.template slot<false>(i0 + lane < p1 && hs_top(H) - tlo <= span, H, tb);
          if (s < 0) continue;
          u64 L, Hi, xl, xh;
          tab.sum((unsigned)s, L, Hi);
          fx128_of(fx_to_double(L, Hi) * a.pa[p], xl, xh, dbad);
          dlo += xl;
          dhi += xh + (dlo < xl ? 1ull : 0ull);
        }
        __syncthreads();
      }
      const unsigned used = row_flush<W, DB>(a, tab, s_str, 1u << tb, warp * 32, NWARP * 32, !ovf);
      uq += used;
      if (used) atomicAdd(&s_used, used);
      __syncthreads();
      if (ovf) {
        if (tb == TB_MAX) {
          if (hi - lo == 1) {  // cannot be split further: the product goes to the partitioned pipeline
            bad = 1u;
            lo = hi;
          }
          width = max((hi - lo) >> 1, (u64)1);
        }
        wide = true;
      } else {
        const unsigned n = s_used;
        lo = hi;
        // steer the next step to the target from the density seen
        const float f = n ? target / (float)n : 4.0f;
        width = (u64)fminf(4294967296.0f, fmaxf(1.0f, (float)width * fminf(2.0f, fmaxf(0.5f, f))));
      }
      __syncthreads();  // s_used is reset by the next step
    }
    __syncthreads();
    if (lo < end && tid == 0) a.redo[atomicAdd(a.nredo, 1u)] = make_uint4(r, (unsigned)lo, (unsigned)(end - 1), 0u);
    if (bad | dbad) atomicOr(a.flag + 1, 1u);
  }
  // exact 128-bit sum over the CTA, then one global addition
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const u64 ol = __shfl_xor_sync(0xffffffffu, dlo, o), oh = __shfl_xor_sync(0xffffffffu, dhi, o);
    dlo += ol;
    dhi += oh + (dlo < ol ? 1ull : 0ull);
  }
  if (lane == 0 && (dlo | dhi)) {
    const u64 old = atomicAdd((unsigned long long*)a.dexact, (unsigned long long)dlo);
    const u64 hh = dhi + (old + dlo < old ? 1ull : 0ull);
    if (hh) atomicAdd((unsigned long long*)(a.dexact + 1), (unsigned long long)hh);
  }
  uq = warp_sum(uq);
  if (lane == 0) s_red[warp] = uq;
  __syncthreads();
  if (tid == 0) {
    u64 q = 0;
    for (int w = 0; w < NWARP; ++w) q += s_red[w];
    if (q) atomicAdd((unsigned long long*)(a.scount + 1), (unsigned long long)q);
  }
}

}  // namespace

void rows_free(Ctx& c) {
  if (c.d_row_os) cudaFree(c.d_row_os);
  if (c.d_row_bin) cudaFree(c.d_row_bin);
  c.d_row_os = nullptr;
  c.d_row_bin = nullptr;
}

bool row_tables(Ctx& c, const HamView& h) {
  if (c.d_row_os && c.d_row_bin) return true;
  rows_free(c);
  std::vector<unsigned> bin(64 * 34);
  for (int p = 0; p < 64; ++p)
    for (int k = 0; k < 34; ++k) bin[p * 34 + k] = (unsigned)binom(p, k);
  const size_t n = (size_t)c.M * c.M * c.M * c.M, m3 = (size_t)c.M * c.M * c.M;
  if (cudaMalloc(&c.d_row_bin, bin.size() * sizeof(unsigned)) != cudaSuccess ||
      cudaMalloc(&c.d_row_os, (n + 6 * m3) * sizeof(double)) != cudaSuccess ||
      cudaMemcpyAsync(c.d_row_bin, bin.data(), bin.size() * sizeof(unsigned), cudaMemcpyHostToDevice, c.stream) !=
          cudaSuccess ||
      cudaStreamSynchronize(c.stream) != cudaSuccess) {
    cudaGetLastError();
    rows_free(c);
    return false;
  }
  k_rows_os<<<(unsigned)std::min<size_t>((n + 255) / 256, (size_t)c.sm_count * 8), 256, 0, c.stream>>>(h, c.d_row_os);
  k_rows_sj<<<(unsigned)std::min<size_t>((4 * m3 + 255) / 256, (size_t)c.sm_count * 8), 256, 0, c.stream>>>(
      h, c.d_row_os + n, c.d_row_os + n + 4 * m3);
  c.launches += 2;
  if (cudaGetLastError() != cudaSuccess) {
    rows_free(c);
    return false;
  }
  return true;
}

// Work on the context's second stream: begin() orders it after what the main
// stream holds, and the main stream waits for everything issued there since at
// join() or when the object goes out of scope, whichever way the product returns.
// Medians against one stream: 3,001 sources of 56 spin orbitals 3.21 -> 3.15 ms, a
// Lanczos solve of 5,000 38.4 -> 38.0 ms, 20,000 sources 13.32 -> 13.29 ms.
struct SideWork {
  Ctx& c;
  bool open = false;
  explicit SideWork(Ctx& c_) : c(c_) {}
  ~SideWork() { join(); }
  int begin() {
    if (!c.side) SFCI_CUDA(cudaStreamCreateWithFlags(&c.side, cudaStreamNonBlocking));
    if (!c.ev_fork) SFCI_CUDA(cudaEventCreateWithFlags(&c.ev_fork, cudaEventDisableTiming));
    if (!c.ev_join) SFCI_CUDA(cudaEventCreateWithFlags(&c.ev_join, cudaEventDisableTiming));
    SFCI_CUDA(cudaEventRecord(c.ev_fork, c.stream));
    SFCI_CUDA(cudaStreamWaitEvent(c.side, c.ev_fork, 0));
    open = true;
    return SFCI_OK;
  }
  // an event that cannot be recorded leaves the host to wait instead
  void join() {
    if (open && (cudaEventRecord(c.ev_join, c.side) != cudaSuccess ||
                 cudaStreamWaitEvent(c.stream, c.ev_join, 0) != cudaSuccess))
      cudaStreamSynchronize(c.side);
    open = false;
  }
};

template <int W>
int rows_product(Ctx& c, const typename KeyOf<W>::T* keys, const double* amps, u64 ns, u64 nx, double lambda,
                 double coeff, u64 cap, RowsResult<W>* out, bool* done) {
  typedef typename StrOf<W>::T ST;
  typedef typename KeyOf<W>::T KT;
  *done = false;
  const ListsInUse in_use(c);
  int st;
  // (a repeated key would let a target receive more terms than its accumulator takes).
  // Other keys are declined here: with the check among the rank tables a product of
  // 3,750 determinants of mixed spins on 14 orbitals took 90 us more, now 24, and one
  // of two-word keys 180, now 22 (the partitioned pipeline alone 953 and 7,869).
  int na = 0, nb = 0;
  bool alike = false;
  if ((st = keys_one_spin<W>(c, keys, ns, true, &na, &nb, &alike)) || !alike) return st;
  const int M = c.M, nva = M - na, nvb = M - nb;
  if (na < 1 || nb < 1 || nva < 1 || nvb < 1 || na > ROW_EL_MAX || nb > ROW_EL_MAX) return SFCI_OK;
  const u64 RA = binom(M, na), RB = binom(M, nb);
  if (RA > ROW_RANKS_MAX || RB > ROW_RANKS_MAX) return SFCI_OK;
  const u64 nsa = (u64)na * nva, nsb = (u64)nb * nvb;
  const u64 nda = (u64)(na * (na - 1) / 2) * (nva * (nva - 1) / 2), ndb = (u64)(nb * (nb - 1) / 2) * (nvb * (nvb - 1) / 2);
  const u64 conn = 1 + nsa + nsb + nda + ndb + nsa * nsb;
  const u64 most = conn + (nx ? 2 : 0);  // terms of one target: at most two extra vectors
  const u64 T = ns * conn + nx;
  if (most >= (1ull << 16) || nsa >= (1u << RP_D) || nda >= (1u << (RP_RAW - RP_D)) || ndb >= 65536 ||
      ns * (1 + nsb + ndb) + nx >= (1ull << (64 - RP_RAW)) || nx >= (1ull << 31) || ns * nsb >= (1ull << 31) || ns >= (1ull << 31))
    return SFCI_OK;
  // Where the row form pays: its fixed part sweeps the rank tables and visits every
  // row reached, so its lead starts at more terms the more strings there are
  // (measured crossings, terms: 1.0e6 with 252 strings a spin, 1.4e7 with 1.2e6,
  // 5.3e7 with 1.8e7).
  if ((double)T < 1048576.0 + 9000.0 * std::sqrt((double)(RA + RB))) return SFCI_OK;
  const bool d16 = most <= (1u << 15);
  RowArgs<W> a{};
  a.h.N = c.N;
  a.h.M = M;
  a.h.P = c.P;
  a.h.h1 = c.d_h1;
  a.h.V = c.d_V;
  a.h.ecore = c.ham.ecore;
  a.h.inst = nullptr;
  // device memory: the rank tables, the sources' lists, and (from the distinct
  // strings, known after the first kernels) the pairs of rows and groups
  size_t freeb = 0, totb = 0;
  SFCI_CUDA(cudaMemGetInfo(&freeb, &totb));
  size_t held = 0;
  for (const char* nm : {"sp_l1k", "sp_l1a", "sp_l2k", "sp_l2a"}) {
    auto it = c.scratch.find(nm);
    if (it != c.scratch.end()) held += it->second.bytes;
  }
  size_t mine = 0;
  for (auto& kv : c.scratch)
    if (kv.first.compare(0, 3, "rw_") == 0) mine += kv.second.bytes;
  const size_t avail = (size_t)((freeb + held + mine) * 0.9);
  const u64 margin =
      std::min<u64>(T, c.tune_row_margin ? c.tune_row_margin : std::max<u64>(1ull << 24, avail / 64 / (sizeof(KT) + 8)));
  const u64 slack = (u64)c.sm_count * 10240;  // an SM's shared memory holds fewer table slots than that
  const u64 SC = std::min<u64>(cap, T) + margin + slack;
  size_t need = (nx ? RA * 8 + nx * (sizeof(ST) + 12) : 0) + RA * 40 + RB * 8 + ns * (nsb * (sizeof(ST) + 4 + 6) + 64) + SC * 2 * (sizeof(KT) + 8) + ((size_t)64 << 20);
  if (need > avail) return SFCI_OK;
  if (need > freeb + mine) scratch_release_plan(c);
  if (!row_tables(c, a.h)) return SFCI_OK;
  int tok = phase_begin(c, PH_COUNT);
  // the phase open at a return is closed with it (one already closed is left alone)
  struct ClosePhase {
    Ctx& c;
    const int& tok;
    ~ClosePhase() { phase_end(c, tok); }
  } close_phase{c, tok};
  bool ok = true;
  auto get = [&](const char* nm, size_t bytes) -> void* {
    void* p = scratch_get(c, nm, bytes);
    if (!p) ok = false;
    return p;
  };
  a.na = na;
  a.nb = nb;
  a.nva = nva;
  a.nvb = nvb;
  a.nsa = (unsigned)nsa;
  a.nsb = (unsigned)nsb;
  a.nda = (unsigned)nda;
  a.ndb = (unsigned)ndb;
  a.bin = c.d_row_bin;
  a.os = c.d_row_os;
  a.sj = a.os + (size_t)M * M * M * M;
  a.xk = a.sj + (size_t)4 * M * M * M;
  a.keys = keys;
  a.amps = amps;
  a.ns = ns;
  a.nx = nx;
  a.lambda = lambda;
  a.coeff = coeff;
  a.RA = (unsigned)RA;
  a.RB = (unsigned)RB;
  a.ra = (unsigned*)get("rw_ra", ns * 4);
  a.rb = (unsigned*)get("rw_rb", ns * 4);
  a.arank = (u64*)get("rw_arank", (RA + 1) * 8);
  a.brank = (uint32_t*)get("rw_brank", (RB + 1) * 4);
  a.flag = (unsigned*)get("rw_flag", 256 * 4);
  double* diagE = (double*)get("rw_diag", ns * 8);
  a.diagE = diagE;
  a.max_exp = d16 ? 15 : 10;
  if (!ok) return SFCI_OK;
  a.bins = a.flag + 8;  // 64 counts, 64 cursors
  a.ucur = a.flag + 144;
  a.nredo = a.flag + 146;
  SFCI_CUDA(cudaMemsetAsync(a.arank, 0, (RA + 1) * 8, c.stream));
  SFCI_CUDA(cudaMemsetAsync(a.brank, 0, (RB + 1) * 4, c.stream));
  SFCI_CUDA(cudaMemsetAsync(a.flag, 0, 256 * 4, c.stream));
  const unsigned gmax = (unsigned)c.sm_count * 8;
  auto grid_of = [&](u64 n, unsigned per) { return (unsigned)std::max<u64>(1, std::min<u64>((n + per - 1) / per, gmax)); };
  SFCI_LAUNCH(c, k_rows_split<W>, grid_of(ns, 256), 256, 0, a);
  // the diagonal elements need nothing but the sources: beside the rank tables' scans
  SideWork side(c);
  if ((st = side.begin())) return st;
  k_rows_diag<W><<<(unsigned)std::max<u64>(1, std::min<u64>((ns + 7) / 8, gmax * 2)), 256, 0, c.side>>>(a, diagE);
  c.launches++;
  SFCI_CUDA(cudaGetLastError());
  SFCI_LAUNCH(c, k_rows_mark, grid_of(RA, 256), 256, 0, a.arank, a.RA);
  if ((st = scan_excl(c, a.arank, a.arank, RA))) return st;
  if ((st = scan_excl_u32(c, a.brank, a.brank, RB))) return st;
  side.join();
  // the counts the host sizes the rest from
  u64* tot = (u64*)get("rw_tot", 8 * 8);
  if (!ok) return SFCI_OK;
  u64 th[8];
  SFCI_LAUNCH(c, k_rows_gather, 1, 64, 0, (Spans{{a.arank + RA, a.brank + RB, a.flag, nullptr}, {2, 1, 1, 0}}),
              (uint32_t*)tot);
  if ((st = read_words(c, tot, 2 * 8, th))) return st;
  if (th[1] >> 32) return SFCI_OK;
  a.nG = (unsigned)(th[0] >> 32);
  a.nB = (unsigned)th[1];
  // pairs of groups and the rows they reach: 12 B each (and the same for the
  // beta strings' doubles); with nearly as many strings as sources the lists
  // cost what the partitioned pipeline's terms do
  const u64 nSent = a.nG * nsa, nDent = a.nG * nda;
  int db = 0;
  while (db < 10 && (4ull << db) < ndb) ++db;
  a.db = db;
  need += nSent * 8 + nDent * 12 + a.nB * (nsb * (sizeof(ST) + 2) + ndb * (sizeof(ST) + 8) + ((2ull << db) + 4));
  if (need > avail || nSent >= (1ull << 31) || nDent >= (1ull << 31) || a.nB * ndb >= (1ull << 32)) return SFCI_OK;
  if (need > freeb + mine) scratch_release_plan(c);
  const u64 nb0max = 2 * ns + a.nG, nb1max = ns * nsb + a.nG;  // at most n buckets for n entries
  a.gstr = (ST*)get("rw_gstr", a.nG * sizeof(ST));
  a.gbase = (unsigned*)get("rw_gbase", a.nG * 4);
  a.gcnt = (unsigned*)get("rw_gcnt", a.nG * 4);
  a.gb0 = (unsigned char*)get("rw_gb0", a.nG);
  a.gb1 = (unsigned char*)get("rw_gb1", a.nG);
  a.goff = (u64*)get("rw_goff", ((u64)a.nG + 1) * 8);
  a.gi = (uint2*)get("rw_gi", a.nG * sizeof(uint2));
  a.bstr = (ST*)get("rw_bstr", a.nB * sizeof(ST));
  a.bocc = (unsigned char*)get("rw_bocc", (u64)a.nB * nb);
  a.rpack = (u64*)get("rw_rpack", RA * 8);
  a.roff = (u64*)get("rw_roff", (RA + 1) * 8);
  a.rcur = (u64*)get("rw_rcur", RA * 8);
  a.pg = (unsigned*)get("rw_pg", ns * 4);
  a.pb = (unsigned*)get("rw_pb", ns * 4);
  a.pH = (ST*)get("rw_pH", ns * sizeof(ST));
  a.pc = (double*)get("rw_pc", ns * 8);
  a.pa = (double*)get("rw_pa", ns * 8);
  a.pd = (double*)get("rw_pd", ns * 8);
  a.c0 = (uint32_t*)get("rw_c0", (nb0max + 1) * 4);
  a.off0 = (uint32_t*)get("rw_off0", (nb0max + 1) * 4);
  a.c1 = (uint32_t*)get("rw_c1", (nb1max + 1) * 4);
  a.off1 = (uint32_t*)get("rw_off1", (nb1max + 1) * 4);
  a.eH = (ST*)get("rw_eH", ns * nsb * sizeof(ST));
  a.ex = (uint32_t*)get("rw_ex", ns * nsb * 4);
  a.sH = (ST*)get("rw_sH", a.nB * nsb * sizeof(ST));
  a.sx = (unsigned short*)get("rw_sx", a.nB * nsb * 2);
  a.dH = (ST*)get("rw_dH", std::max<u64>(1, a.nB * ndb) * sizeof(ST));
  a.dV = (double*)get("rw_dV", std::max<u64>(1, a.nB * ndb) * 8);
  a.dO = (unsigned short*)get("rw_dO", (u64)a.nB * ((1u << db) + 1) * 2);
  a.rsg = (unsigned*)get("rw_rsg", nSent * 4);
  a.rsx = (unsigned*)get("rw_rsx", nSent * 4);
  a.rdg = (unsigned*)get("rw_rdg", std::max<u64>(1, nDent) * 4);
  a.rdv = (double*)get("rw_rdv", std::max<u64>(1, nDent) * 8);
  if (nx) {
    a.xra = (unsigned*)get("rw_xra", nx * 4);
    a.xc = (uint32_t*)get("rw_xc", RA * 4);
    a.xoff = (uint32_t*)get("rw_xoff", (RA + 1) * 4);
    a.xH = (ST*)get("rw_xH", nx * sizeof(ST));
    a.xv = (double*)get("rw_xv", nx * 8);
  }
  if (!ok) return SFCI_OK;
  SFCI_CUDA(cudaMemsetAsync(a.rpack, 0, RA * 8, c.stream));
  if (nx) {
    SFCI_CUDA(cudaMemsetAsync(a.xc, 0, RA * 4, c.stream));
    SFCI_LAUNCH(c, (k_rows_extra<W, false>), grid_of(nx, 256), 256, 0, a);
    if ((st = scan_excl_u32(c, a.xc, a.xoff, RA))) return st;
    SFCI_LAUNCH(c, (k_rows_extra<W, true>), grid_of(nx, 256), 256, 0, a);
  }
  SFCI_CUDA(cudaMemsetAsync(a.rcur, 0, RA * 8, c.stream));
  SFCI_LAUNCH(c, k_rows_groups<W>, grid_of(std::max(RA, RB), 256), 256, 0, a);
  // the beta strings' doubles need nothing but the strings: beside the lists below
  if (ndb) {
    if ((st = side.begin())) return st;
    k_rows_bdoubles<W><<<grid_of(a.nB, 1), 256, sizeof(uint32_t) << db, c.side>>>(a);
    c.launches++;
    SFCI_CUDA(cudaGetLastError());
  }
  if ((st = scan_excl(c, a.goff, a.goff, a.nG))) return st;
  // slices per group so that a few thousand warps share the moves
  const unsigned nslice = (unsigned)std::max<u64>(1, std::min<u64>((nda + 31) / 32, 8192 / std::max(1u, a.nG)));
  const unsigned ag = grid_of((u64)a.nG * nslice, 8);
  SFCI_LAUNCH(c, (k_rows_alpha<W, false>), ag, 256, 0, a, nslice);
  SFCI_LAUNCH(c, k_rows_lens, grid_of(RA, 256), 256, 0, (const u64*)a.rpack, a.RA, a.roff);
  if ((st = scan_excl(c, a.roff, a.roff, RA))) return st;
  // units: enough of them to fill the device several times over, large enough to
  // amortise a row's set-up
  a.unit_raw = std::max<u64>(8192, std::min<u64>(1ull << 19, T / ((u64)c.sm_count * 32)));
  SFCI_LAUNCH(c, (k_rows_units<W, false>), grid_of(RA, 2048), 256, 0, a);
  u64* rb = (u64*)get("rw_tot2", 64 * 8);
  if (!ok) return SFCI_OK;
  unsigned bh[64];
  {
    u64 buf[3 + 32];
    SFCI_LAUNCH(c, k_rows_gather, 1, 64, 0, (Spans{{a.goff + a.nG, a.flag, a.bins, nullptr}, {2, 4, 64, 0}}), (uint32_t*)rb);
    if ((st = read_words(c, rb, sizeof buf, buf))) return st;
    memcpy(th, buf, 3 * 8);
    memcpy(bh, buf + 3, sizeof bh);
  }
  const u64 nb0 = th[0] & 0xffffffffull, nb1 = th[0] >> 32;
  const unsigned maxg = (unsigned)th[2];
  u64 nunits = 0;
  for (int i = 0; i < BINS; ++i) nunits += bh[i];
  a.nlight = bh[BINS];
  if ((unsigned)th[1] || maxg >= (1u << 19) || nb0 > nb0max || nb1 > nb1max || nunits + a.nlight >= (1ull << 31))
    return SFCI_OK;
  const u64 nall = nunits + a.nlight;
  a.units = (uint4*)get("rw_units", std::max<u64>(1, nunits) * sizeof(uint4));
  a.light = (unsigned*)get("rw_light", std::max<u64>(1, a.nlight) * 4);
  a.redo = (uint4*)get("rw_redo", std::max<u64>(1, nall) * sizeof(uint4));
  uint4* redo2 = (uint4*)get("rw_redo2", std::max<u64>(1, nall) * sizeof(uint4));
  a.sk = (KT*)get("sp_sk", SC * sizeof(KT));
  a.sa = (double*)get("sp_sa", SC * sizeof(double));
  u64* scount = (u64*)get("rw_scount", 4 * 8);
  if (!ok) return SFCI_OK;
  a.scount = scount;
  a.dexact = scount + 2;
  a.soft = SC - slack;
  a.cut = fx_cut(c.opts.coeff_cut);
  a.smax = (unsigned)nsa;
  SFCI_CUDA(cudaMemsetAsync(scount, 0, 4 * 8, c.stream));
  SFCI_CUDA(cudaMemsetAsync(a.c0, 0, (nb0 + 1) * 4, c.stream));
  SFCI_CUDA(cudaMemsetAsync(a.c1, 0, (nb1 + 1) * 4, c.stream));
  SFCI_LAUNCH(c, (k_rows_list0<W, false>), grid_of(ns, 256), 256, 0, a);
  if ((st = scan_excl_u32(c, a.c0, a.off0, nb0))) return st;
  SFCI_LAUNCH(c, (k_rows_list0<W, true>), grid_of(ns, 256), 256, 0, a);
  SFCI_LAUNCH(c, k_rows_bsingles<W>, grid_of(a.nB * nsb, 256), 256, 0, a);
  SFCI_LAUNCH(c, (k_rows_list1<W, false>), grid_of(ns, 8), 256, 0, a);
  if ((st = scan_excl_u32(c, a.c1, a.off1, nb1))) return st;
  SFCI_LAUNCH(c, (k_rows_list1<W, true>), grid_of(ns, 8), 256, 0, a);
  SFCI_LAUNCH(c, (k_rows_alpha<W, true>), ag, 256, 0, a, nslice);
  SFCI_LAUNCH(c, (k_rows_units<W, true>), grid_of(RA, 2048), 256, 0, a);
  side.join();
  phase_end(c, tok);
  // the rows
  tok = phase_begin(c, PH_MERGE);
  const size_t sml = row_table_bytes<ST>(LIGHT_SLOTS) * LIGHT_WARPS;
  const size_t smb = row_cta_smem<W, Big<W>::tb>(a.smax), smm = row_cta_smem<W, MID_TB>(a.smax);
  typedef void (*Kern)(RowArgs<W>);
  const Kern kb = d16 ? k_rows_cta<W, 16, Big<W>::threads, Big<W>::tb> : k_rows_cta<W, 15, Big<W>::threads, Big<W>::tb>;
  const Kern km = d16 ? k_rows_cta<W, 16, MID_THREADS, MID_TB> : k_rows_cta<W, 15, MID_THREADS, MID_TB>;
  const Kern kl = d16 ? k_rows_light<W, 16> : k_rows_light<W, 15>;
  unsigned gb = 0, gm = 0, gl = 0;
  // (the limit belongs to the kernel, whichever context or thread launches it: always
  // the most that any system takes, so that no other launch finds it lowered)
  constexpr unsigned SMAX = ROW_EL_MAX * ((W == 1 ? 32 : 64) - ROW_EL_MAX);
  auto config = [&](Kern k, int threads, size_t sm, size_t most, unsigned* g) -> int {
    int per = 0;
    SFCI_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    SFCI_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, threads, sm));
    if (per < 1) return set_error(SFCI_ERR_CUDA, "row kernel does not fit an SM");
    *g = (unsigned)(c.sm_count * per);
    return SFCI_OK;
  };
  if ((st = config(kb, Big<W>::threads, smb, row_cta_smem<W, Big<W>::tb>(SMAX), &gb)) ||
      (st = config(km, MID_THREADS, smm, row_cta_smem<W, MID_TB>(SMAX), &gm)) ||
      (st = config(kl, LIGHT_WARPS * 32, sml, sml, &gl)))
    return st;
  u64 nbig = 0;  // units are ordered by size class, the largest first
  for (int i = MID_BIN; i < BINS; ++i) nbig += bh[i];
  u64 nsurv = 0;
  out->units = nall;
  for (;;) {
    // Large rows first; the smaller ones on the second stream, so that their CTAs
    // take the SMs that the last large rows leave.
    const bool both = nbig && (nunits > nbig || a.nlight);
    cudaStream_t small = c.stream;
    if (both) {
      if ((st = side.begin())) return st;
      small = c.side;
    }
    if (nbig) {
      RowArgs<W> q = a;
      q.nunits = (unsigned)nbig;
      SFCI_LAUNCH(c, kb, std::min((unsigned)nbig, gb), Big<W>::threads, smb, q);
    }
    if (nunits > nbig) {
      RowArgs<W> q = a;
      q.units = a.units + nbig;
      q.nunits = (unsigned)(nunits - nbig);
      q.ucur = a.ucur + 1;
      km<<<std::min(q.nunits, gm), MID_THREADS, smm, small>>>(q);
      c.launches++;
      SFCI_CUDA(cudaGetLastError());
    }
    if (a.nlight) {
      kl<<<std::min((a.nlight + LIGHT_WARPS - 1) / LIGHT_WARPS, gl), LIGHT_WARPS * 32, sml, small>>>(a);
      c.launches++;
      SFCI_CUDA(cudaGetLastError());
    }
    side.join();
    // survivors, distinct, <v|Hv>, flags, redo count in one read
    SFCI_LAUNCH(c, k_rows_gather, 1, 64, 0, (Spans{{scount, a.flag, a.nredo, nullptr}, {8, 4, 1, 0}}), (uint32_t*)rb);
    u64 buf[7];
    if ((st = read_words(c, rb, sizeof buf, buf))) return st;
    if ((unsigned)(buf[4] >> 32)) return SFCI_OK;  // a term above 2^max_exp
    nsurv = buf[0];
    out->uniq = buf[1];
    out->dexact[0] = buf[2];
    out->dexact[1] = buf[3];
    const unsigned nredo = (unsigned)buf[6];
    if (!nredo) break;
    // the survivor buffer filled up: keep the output's capacity and go on with
    // the units left over
    phase_end(c, tok);
    tok = phase_begin(c, PH_SELECT);
    if (nsurv <= cap) return set_error(SFCI_ERR_NUMERIC, "row units left over below the survivor limit");
    size_t m = 0;
    if ((st = select_sorted<W>(c, a.sk, a.sa, nsurv, cap, &m))) return st;
    out->pruned = true;
    ++out->rounds;
    const u64 m64 = m;
    SFCI_CUDA(cudaMemcpyAsync(scount, &m64, 8, cudaMemcpyHostToDevice, c.stream));
    SFCI_CUDA(cudaMemsetAsync(a.ucur, 0, 4, c.stream));
    SFCI_CUDA(cudaMemsetAsync(a.nredo, 0, 4, c.stream));
    SFCI_CUDA(cudaStreamSynchronize(c.stream));  // m64 is a stack variable
    phase_end(c, tok);
    tok = phase_begin(c, PH_MERGE);
    std::swap(a.redo, redo2);
    a.units = redo2;
    nbig = nunits = nredo;
    a.nlight = 0;
  }
  phase_end(c, tok);
  out->sk = a.sk;
  out->sa = a.sa;
  out->nsurv = nsurv;
  out->terms = T;
  *done = true;
  return SFCI_OK;
}

template int rows_product<1>(Ctx&, const u64*, const double*, u64, u64, double, double, u64, RowsResult<1>*, bool*);
template int rows_product<2>(Ctx&, const K128*, const double*, u64, u64, double, double, u64, RowsResult<2>*, bool*);

}  // namespace sfci
