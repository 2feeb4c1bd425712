// Matrix elements between two sets of determinants: calc_energy
// (src/functions.cpp:1272-1313) and the dots of the linear solver's product with
// its basis (src/functions.cpp:971-978).
//
// Both need only the terms of H v that land on a known set of determinants (the
// bras).  Generating every term and probing a hash set of the bras (k_gen<ENERGY>,
// k_gen<PROJECT> in spmspv.cu) visits 30,724 targets a source at 56 spin orbitals
// to find a few hundred.  Here the bras are grouped by alpha string, each distinct
// alpha string of the sources (kets) gets the list of bra groups one and two moves
// away, and a warp per ket looks only there: in groups one move away it compares
// beta strings by a population count (two bits apart: an opposite-spin double, none:
// a single), in groups two moves away it looks its beta string up in the group's
// buckets, and in the group of its own alpha string it finds the diagonal, spin-1
// singles and doubles.  Elements and phases are those of rows.cu.
//
// Bound by the latency of the lookups in L2 and by issue.  calc_energy of 20,011
// determinants of 56 spin orbitals takes 1.1 ms against 12.9 ms for the sweep,
// 100,000 take 5.1 ms, 3,000 of 68 spin orbitals 0.9 ms.
#include <algorithm>
#include <cmath>
#include <vector>

#include "merge.cuh"
#include "pairs.cuh"
#include "strings.cuh"

namespace sfci {

__global__ void k_rows_mark(u64* arank, unsigned RA);  // rows.cu

namespace {

// determinants grouped by alpha string, each group bucketed by the hash of the beta string
template <int W>
struct Side {
  typedef typename StrOf<W>::T ST;
  typedef typename KeyOf<W>::T KT;
  const KT* keys;
  u64 n;
  int table;       // the keys are an open-addressing table: empty slots are skipped
  unsigned* ra;    // alpha rank per key
  u64* arank;      // per rank: determinants | 1 << 32 when any, then their exclusive scan
  unsigned nG;
  ST* gstr;
  unsigned *gbase, *gcnt;
  unsigned char* gbits;
  uint32_t* goff;  // first bucket
  uint32_t *c0, *off0;
  ST* pH;
  unsigned *px, *pg;  // index of the key | s(A, B) << 31; group
};

template <int W>
struct PairArgs {
  typedef typename StrOf<W>::T ST;
  HamView h;
  int na, nb, nva;
  unsigned nsa, nda, RA;
  const unsigned* bin;
  const double *os, *sj, *xk;
  unsigned* flag;  // [0] not eligible, [1] out of range
  Side<W> bra, ket;
  // neighbours of each ket group among the bra groups
  u64 *noff, *ncur;  // S | D << 32
  u64* ntest;        // beta strings the kets will be compared with
  unsigned *nsg, *nsx;
  unsigned* ndg;
  double* ndv;
  const double* amps;   // of the kets, by key index
  const double* diagE;  // by key index
  double lambda;
  const double* bamps;  // ENERGY: of the bras
  u64* esum;            // ENERGY: exact 128-bit sum of the products times 4^up
  int up;               // ENERGY: power of two that brings the largest amplitude into [1, 2),
  double up2;           // and 4^up, by which the kets are multiplied
  u64 *plo, *phi;       // PROJECT: exact sums by bra index (split form)
  u64 sum[2];           // ENERGY: *esum, on the host after the run
};

template <int W>
__global__ void k_pair_rank(Side<W> s, int na, int nb, int N, const unsigned* bin, unsigned* flag,
                            const double* __restrict__ amps, u64* __restrict__ amax) {
  typedef typename StrOf<W>::T ST;
  typedef typename KeyOf<W>::T KT;
  unsigned bad = 0;
  u64 mx = 0;  // largest |amplitude|, as an integer
  for (u64 j = (u64)blockIdx.x * blockDim.x + threadIdx.x; j < s.n; j += (u64)gridDim.x * blockDim.x) {
    const KT k = s.keys[j];
    if (amps) mx = max(mx, abs_bits(amps[j]));
    if (s.table && key_eq(k, key_empty<KT>())) {
      s.ra[j] = ~0u;
      continue;
    }
    ST a, b;
    split_key(k, a, b);
    if (spop(a) != na || spop(b) != nb || !key_within(k, N)) {
      bad = 1;
      continue;
    }
    const unsigned r = rank_of(bin, a);
    s.ra[j] = r;
    atomicAdd((unsigned*)(s.arank + r), 1u);
  }
  if (bad) atomicOr(flag, 1u);
  if (amps) {
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0 && mx) atomicMax((unsigned long long*)amax, (unsigned long long)mx);
  }
}

template <int W>
__global__ void k_pair_groups(Side<W> s, unsigned RA, int na, int M, const unsigned* bin) {
  typedef typename StrOf<W>::T ST;
  for (unsigned r = blockIdx.x * blockDim.x + threadIdx.x; r < RA; r += gridDim.x * blockDim.x) {
    const u64 v = s.arank[r], w = s.arank[r + 1];
    const unsigned g = (unsigned)(v >> 32);
    if (g == (unsigned)(w >> 32)) continue;
    const unsigned n = (unsigned)w - (unsigned)v;
    s.gstr[g] = unrank_thread<ST>(bin, r, na, M);
    s.gbase[g] = (unsigned)v;
    s.gcnt[g] = n;
    const int b = bucket_bits(n);
    s.gbits[g] = (unsigned char)b;
    s.goff[g] = 1u << b;
  }
}

template <int W, bool FILL>
__global__ void k_pair_list(Side<W> s) {
  typedef typename StrOf<W>::T ST;
  for (u64 j = (u64)blockIdx.x * blockDim.x + threadIdx.x; j < s.n; j += (u64)gridDim.x * blockDim.x) {
    if (s.ra[j] == ~0u) continue;
    const unsigned g = (unsigned)(s.arank[s.ra[j]] >> 32);
    ST a, b;
    split_key(s.keys[j], a, b);
    const ST H = hs_of(b);
    const unsigned k = s.goff[g] + bucket_of(hs_top(H), s.gbits[g]);
    if (!FILL) {
      atomicAdd(s.c0 + k, 1u);
    } else {
      const unsigned p = s.off0[k] + atomicSub(s.c0 + k, 1u) - 1u;
      s.pH[p] = H;
      s.px[p] = (unsigned)j | (interleave_par(a, b) << 31);
      s.pg[p] = g;
    }
  }
}

template <int W>
__global__ void k_pair_diag(const typename KeyOf<W>::T* keys, u64 n, HamView h, double* __restrict__ diagE) {
  const u64 nw = ((u64)gridDim.x * blockDim.x) >> 5;
  for (u64 w = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n; w += nw) {
    const double D = diag_element_warp(keys[w], h);
    if ((threadIdx.x & 31) == 0) diagE[w] = D;
  }
}

// bra groups one and two moves from each ket group; a warp takes a slice of a
// group's moves (counts, then entries)
template <int W, bool FILL>
__global__ void __launch_bounds__(256) k_pair_nbrs(PairArgs<W> a, unsigned nslice) {
  typedef typename StrOf<W>::T ST;
  __shared__ unsigned char s_o[8][64], s_v[8][64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const u64 nitem = (u64)a.ket.nG * nslice;
  const unsigned nvp = a.nva * (a.nva - 1) / 2;
  for (u64 it = (u64)blockIdx.x * 8 + warp; it < nitem; it += (u64)gridDim.x * 8) {
    const unsigned g = (unsigned)(it / nslice), sl = (unsigned)(it - (u64)g * nslice);
    const ST s = a.ket.gstr[g];
    __syncwarp();
    for (int p = lane; p < a.h.M; p += 32) {
      const int o = spop((ST)(s & (sbit<ST>(p) - 1)));
      if ((s >> p) & 1) s_o[warp][o] = (unsigned char)p;
      else s_v[warp][p - o] = (unsigned char)p;
    }
    __syncwarp();
    u64 cnt = 0, tests = 0;
    if (!FILL && sl == 0 && lane == 0) {
      const unsigned r = rank_of(a.bin, s), gb = (unsigned)(a.bra.arank[r] >> 32);
      if (gb != (unsigned)(a.bra.arank[r + 1] >> 32)) tests = a.bra.gcnt[gb];
    }
    for (unsigned t = sl * 32 + lane; t < a.nsa; t += nslice * 32) {
      const int i = s_o[warp][t / a.nva], p = s_v[warp][t % a.nva];
      const unsigned r = rank_of(a.bin, (ST)(s ^ sbit<ST>(i) ^ sbit<ST>(p)));
      const unsigned gb = (unsigned)(a.bra.arank[r] >> 32);
      if (gb == (unsigned)(a.bra.arank[r + 1] >> 32)) continue;
      if (!FILL) {
        ++cnt;
        tests += a.bra.gcnt[gb];
      } else {
        const unsigned k = (unsigned)a.noff[g] + (unsigned)atomicAdd((unsigned long long*)(a.ncur + g), 1ull);
        a.nsg[k] = gb;
        a.nsx[k] = (unsigned)((i * a.h.M + p) * a.h.M * a.h.M) | (move_par(s, i, p) << 31);
      }
    }
    for (unsigned t = sl * 32 + lane; t < a.nda; t += nslice * 32) {
      const unsigned op = t / nvp, vp = t - op * nvp;
      unsigned x, y, u, v;
      unrank_pair2(op, x, y);
      unrank_pair2(vp, u, v);
      const int i = s_o[warp][x], j = s_o[warp][y], p = s_v[warp][u], q = s_v[warp][v];
      const unsigned r = rank_of(a.bin, (ST)(s ^ sbit<ST>(i) ^ sbit<ST>(j) ^ sbit<ST>(p) ^ sbit<ST>(q)));
      const unsigned gb = (unsigned)(a.bra.arank[r] >> 32);
      if (gb == (unsigned)(a.bra.arank[r + 1] >> 32)) continue;
      if (!FILL) {
        cnt += 1ull << 32;
      } else {
        const unsigned k = (unsigned)(a.noff[g] >> 32) +
                           (unsigned)(atomicAdd((unsigned long long*)(a.ncur + g), 1ull << 32) >> 32);
        a.ndg[k] = gb;
        a.ndv[k] = double_elem(a.h, 0, s, i, j, p, q);
      }
    }
    if (!FILL) {
      cnt = warp_sum(cnt);
      if (lane == 0 && cnt) atomicAdd((unsigned long long*)(a.noff + g), (unsigned long long)cnt);
      tests = warp_sum(tests) * a.ket.gcnt[g];
      if (lane == 0 && tests) atomicAdd((unsigned long long*)a.ntest, (unsigned long long)tests);
    }
  }
}

// A warp per ket.  Sums over the pairs found are exact (ENERGY: 128-bit sum of
// each product c_bra * term rounded once to the FX_FRAC grid of the vector scaled to
// a largest amplitude in [1, 2), so that the energy of a vector times a power of
// two has the same bits; PROJECT: the bras' merge accumulators), so they do not
// depend on the order.
template <int W, bool ENERGY>
__global__ void __launch_bounds__(256) k_pairs(PairArgs<W> a) {
  typedef typename StrOf<W>::T ST;
  const int lane = threadIdx.x & 31, M = a.h.M;
  const Side<W>&k = a.ket, &q = a.bra;
  const u64 nw = ((u64)gridDim.x * blockDim.x) >> 5;
  u64 slo = 0, shi = 0;
  unsigned bad = 0;
  auto emit = [&](unsigned e, double amp, unsigned par) {
    const unsigned x = q.px[e];
    amp = signed_by(par ^ (x >> 31), amp);
    if (ENERGY) {
      u64 l, h;
      fx128_of(amp * a.bamps[x & 0x7fffffffu], l, h, bad);
      slo += l;
      shi += h + (slo < l ? 1ull : 0ull);
    } else {
      u64 l, h;
      fx_addends(amp, l, h, bad);
      if (l) atomicAdd((unsigned long long*)(a.plo + (x & 0x7fffffffu)), (unsigned long long)l);
      if (h) atomicAdd((unsigned long long*)(a.phi + (x & 0x7fffffffu)), (unsigned long long)h);
    }
  };
  for (u64 p = ((u64)blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < k.n; p += nw) {
    const unsigned g = k.pg[p], x = k.px[p];
    const ST A = k.gstr[g], H = k.pH[p], B = hs_inv(H);
    const double c0 = ENERGY ? a.up2 * a.amps[x & 0x7fffffffu] : a.amps[x & 0x7fffffffu];
    const double c = signed_by(x >> 31, c0);
    const u64 o0 = a.noff[g], o1 = a.noff[g + 1];
    // groups one move away
    for (unsigned i0 = (unsigned)o0; i0 < (unsigned)o1; i0 += 32) {
      unsigned st = 0, len = 0, row = 0;
      if (i0 + lane < (unsigned)o1) {
        const unsigned gb = a.nsg[i0 + lane];
        st = q.gbase[gb];
        len = q.gcnt[gb];
        row = a.nsx[i0 + lane];
      }
      warp_expand_own(st, len, [&](bool ok, unsigned e, int own) {
        const unsigned r = __shfl_sync(0xffffffffu, row, own);
        const ST Bq = ok ? hs_inv(q.pH[e]) : (ST)~B, d = B ^ Bq;
        const int pc = spop(d);
        if (ok && pc == 2) {
          const int j = sffs((ST)(d & B)), b = sffs((ST)(d & Bq));
          emit(e, c * SFCI_LDG(a.os + (r & 0x7fffffffu) + j * M + b), (r >> 31) ^ move_par(B, j, b));
        }
        const bool one = ok && pc == 0;
        if (__any_sync(0xffffffffu, one)) {
          const unsigned ia = (r & 0x7fffffffu) / (M * M);
          const double v = single_elems<ST>(a.sj, a.xk, a.h.h1, M, 0, (int)(ia / M), (int)(ia % M), A, B, a.na, a.nb, one);
          if (one) emit(e, c * v, r >> 31);
        }
      });
    }
    // the group of its own alpha string
    const unsigned gs = (unsigned)(q.arank[k.ra[x & 0x7fffffffu]] >> 32);
    if (gs != (unsigned)(q.arank[k.ra[x & 0x7fffffffu] + 1] >> 32)) {
      const unsigned e0 = q.gbase[gs], e1 = e0 + q.gcnt[gs];
      for (unsigned i0 = e0; i0 < e1; i0 += 32) {
        const bool ok = i0 + lane < e1;
        const unsigned e = ok ? i0 + lane : e0;
        const ST Bq = ok ? hs_inv(q.pH[e]) : (ST)~B, d = B ^ Bq;
        const int pc = spop(d);
        if (ok && pc == 0) emit(e, signed_by(x >> 31, (a.diagE[x & 0x7fffffffu] - a.lambda) * c0), 0u);
        const ST dh = d & B, dp = d & Bq;
        if (ok && pc == 4) {
          const int i = sffs(dh), j = sffs((ST)(dh & (dh - 1))), u = sffs(dp), v = sffs((ST)(dp & (dp - 1)));
          emit(e, c * double_elem(a.h, 1, B, i, j, u, v), 0u);
        }
        const bool one = ok && pc == 2;
        if (__any_sync(0xffffffffu, one)) {
          const int j = one ? sffs(dh) : 0, b = one ? sffs(dp) : 0;
          const double v = single_elems<ST>(a.sj, a.xk, a.h.h1, M, 1, j, b, A, B, a.na, a.nb, one);
          if (one) emit(e, c * v, move_par(B, j, b));
        }
      }
    }
    // groups two moves away: the same beta string
    const uint32_t top = hs_top(H);
    for (unsigned i = (unsigned)(o0 >> 32) + lane; i < (unsigned)(o1 >> 32); i += 32) {
      const unsigned gb = a.ndg[i];
      const uint32_t* f = q.off0 + q.goff[gb] + bucket_of(top, q.gbits[gb]);
      for (unsigned e = f[0]; e < f[1]; ++e)
        if (q.pH[e] == H) emit(e, c * a.ndv[i], 0u);
    }
  }
  if (bad) atomicOr(a.flag + 1, 1u);
  if (ENERGY) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      const u64 ol = __shfl_xor_sync(0xffffffffu, slo, o), oh = __shfl_xor_sync(0xffffffffu, shi, o);
      slo += ol;
      shi += oh + (slo < ol ? 1ull : 0ull);
    }
    if (lane == 0 && (slo | shi)) {
      const u64 old = atomicAdd((unsigned long long*)a.esum, (unsigned long long)slo);
      const u64 hh = shi + (old + slo < old ? 1ull : 0ull);
      if (hh) atomicAdd((unsigned long long*)(a.esum + 1), (unsigned long long)hh);
    }
  }
}

// host: scratch of one side, named by prefix
template <int W>
struct Builder {
  Ctx& c;
  bool ok = true;
  unsigned gmax;
  explicit Builder(Ctx& c_) : c(c_), gmax((unsigned)c_.sm_count * 8) {}
  void* get(const std::string& nm, size_t bytes) {
    void* p = scratch_get(c, nm.c_str(), bytes);
    if (!p) ok = false;
    return p;
  }
  unsigned grid(u64 n, unsigned per) const {
    return (unsigned)std::max<u64>(1, std::min<u64>((n + per - 1) / per, gmax));
  }
  // ranks and the scanned rank table
  // (amps: their largest magnitude goes to *amax)
  int rank(Side<W>& s, const std::string& p, unsigned RA, int na, int nb, const unsigned* bin, unsigned* flag,
           const double* amps = nullptr, u64* amax = nullptr) {
    s.ra = (unsigned*)get(p + "ra", s.n * 4);
    s.arank = (u64*)get(p + "arank", ((u64)RA + 1) * 8);
    if (!ok) return SFCI_OK;
    SFCI_CUDA(cudaMemsetAsync(s.arank, 0, ((u64)RA + 1) * 8, c.stream));
    SFCI_LAUNCH(c, k_pair_rank<W>, grid(s.n, 256), 256, 0, s, na, nb, c.N, bin, flag, amps, amax);
    SFCI_LAUNCH(c, k_rows_mark, grid(RA, 256), 256, 0, s.arank, RA);
    return scan_excl(c, s.arank, s.arank, RA);
  }
  // groups and bucketed lists (s.nG and the number of determinants nd known)
  int lists(Side<W>& s, const std::string& p, unsigned RA, int na, const unsigned* bin, u64 nd) {
    typedef typename StrOf<W>::T ST;
    s.gstr = (ST*)get(p + "gstr", s.nG * sizeof(ST));
    s.gbase = (unsigned*)get(p + "gbase", (u64)s.nG * 4);
    s.gcnt = (unsigned*)get(p + "gcnt", (u64)s.nG * 4);
    s.gbits = (unsigned char*)get(p + "gbits", s.nG);
    s.goff = (uint32_t*)get(p + "goff", ((u64)s.nG + 1) * 4);
    s.c0 = (uint32_t*)get(p + "c0", (nd + 1) * 4);  // at most nd buckets for nd determinants
    s.off0 = (uint32_t*)get(p + "off0", (nd + 1) * 4);
    s.pH = (ST*)get(p + "pH", nd * sizeof(ST));
    s.px = (unsigned*)get(p + "px", nd * 4);
    s.pg = (unsigned*)get(p + "pg", nd * 4);
    if (!ok) return SFCI_OK;
    int st;
    SFCI_LAUNCH(c, k_pair_groups<W>, grid(RA, 256), 256, 0, s, RA, na, c.M, bin);
    if ((st = scan_excl_u32(c, s.goff, s.goff, s.nG))) return st;
    SFCI_CUDA(cudaMemsetAsync(s.c0, 0, (nd + 1) * 4, c.stream));
    SFCI_LAUNCH(c, (k_pair_list<W, false>), grid(s.n, 256), 256, 0, s);
    if ((st = scan_excl_u32(c, s.c0, s.off0, nd))) return st;
    SFCI_LAUNCH(c, (k_pair_list<W, true>), grid(s.n, 256), 256, 0, s);
    return SFCI_OK;
  }
};

// the common part: bras and kets grouped, neighbours listed, k_pairs run
template <int W, bool ENERGY>
int run_pairs(Ctx& c, PairArgs<W>& a, u64 T, u64* links, bool* done) {
  typedef typename KeyOf<W>::T KT;
  *done = false;
  const ListsInUse in_use(c);
  int st;
  int na = 0, nb = 0;
  bool alike = false;
  if ((st = keys_one_spin<W>(c, a.ket.keys, a.ket.n, ENERGY, &na, &nb, &alike)) || !alike) return st;
  const int M = c.M, nva = M - na, nvb = M - nb;
  if (na < 1 || nb < 1 || nva < 1 || nvb < 1 || na > 16 || nb > 16) return SFCI_OK;
  const u64 RA = binom(M, na);
  if (!ENERGY && !pairs_project_pays(T, a.bra.n, RA)) return SFCI_OK;
  if (RA > ROW_RANKS_MAX || a.ket.n >= (1ull << 31) || a.bra.n >= (1ull << 31)) return SFCI_OK;
  const u64 nsa = (u64)na * nva, nda = (u64)(na * (na - 1) / 2) * (nva * (nva - 1) / 2);
  // In a space so full that the strings' mean group already gives the sweep fewer
  // targets than the search comparisons (the rule below, on counts), nothing is built:
  // 7,687 determinants of 16 orbitals with 15 and 5 electrons took 1,040 us, the sweep
  // alone 923, now 919.
  if (ENERGY && (double)a.ket.n * (double)(nsa + 1) > 4.0 * (double)RA * (double)det_terms(na, nva, nb, nvb))
    return SFCI_OK;
  // a device budget holds here too: ranks, then lists, then neighbours
  u64 need = (RA + 1) * 8 * (ENERGY ? 1 : 2) + a.bra.n * 4 + a.ket.n * 12;
  auto over = [&](u64 more) { return (need += more) > c.opts.mem_budget && c.opts.mem_budget; };
  if (over(0)) return SFCI_OK;
  a.h.N = c.N;
  a.h.M = M;
  a.h.P = c.P;
  a.h.h1 = c.d_h1;
  a.h.V = c.d_V;
  a.h.ecore = c.ham.ecore;
  a.h.inst = nullptr;
  if (!row_tables(c, a.h)) return SFCI_OK;
  a.na = na;
  a.nb = nb;
  a.nva = nva;
  a.nsa = (unsigned)nsa;
  a.nda = (unsigned)nda;
  a.RA = (unsigned)RA;
  a.bin = c.d_row_bin;
  a.os = c.d_row_os;
  a.sj = a.os + (size_t)M * M * M * M;
  a.xk = a.sj + (size_t)4 * M * M * M;
  Builder<W> b(c);
  u64* tot = (u64*)b.get("pr_tot", 8 * 8);
  double* diagE = (double*)b.get("pr_diag", a.ket.n * 8);
  if (!b.ok) return SFCI_OK;
  a.flag = (unsigned*)(tot + 4);
  a.esum = tot + 6;
  a.ntest = tot + 5;
  a.diagE = diagE;
  SFCI_CUDA(cudaMemsetAsync(tot, 0, 8 * 8, c.stream));
  if ((st = b.rank(a.bra, "pr_b", a.RA, na, nb, a.bin, a.flag, a.bamps, tot + 3)) || !b.ok) return st;
  if (ENERGY) {
    a.ket = a.bra;
  } else if ((st = b.rank(a.ket, "pr_k", a.RA, na, nb, a.bin, a.flag)) || !b.ok) {
    return st;
  }
  SFCI_CUDA(cudaMemcpyAsync(tot, a.bra.arank + RA, 8, cudaMemcpyDeviceToDevice, c.stream));
  if (!ENERGY) SFCI_CUDA(cudaMemcpyAsync(tot + 1, a.ket.arank + RA, 8, cudaMemcpyDeviceToDevice, c.stream));
  u64 th[5], rb[6];
  if ((st = read_words(c, tot, sizeof th, th))) return st;
  if (ENERGY) th[1] = th[0];
  if ((unsigned)th[4]) return SFCI_OK;
  if (ENERGY) {
    a.up = 1023 - (int)(th[3] >> 52);
    if (th[3] && std::abs(a.up) > 500) return SFCI_OK;  // (infinities and NaNs too) left to the sweep
    a.up2 = std::ldexp(1.0, th[3] ? 2 * a.up : 0);
  }
  a.bra.nG = (unsigned)(th[0] >> 32);
  a.ket.nG = (unsigned)(th[1] >> 32);
  if (a.ket.nG * nda >= (1ull << 32)) return SFCI_OK;
  if (over(((u64)(unsigned)th[0] + (ENERGY ? 0 : (u64)(unsigned)th[1])) * (16 + sizeof(typename StrOf<W>::T))))
    return SFCI_OK;
  if ((st = b.lists(a.bra, "pr_b", a.RA, na, a.bin, (unsigned)th[0])) || !b.ok) return st;
  if (ENERGY) a.ket = a.bra;
  else if ((st = b.lists(a.ket, "pr_k", a.RA, na, a.bin, (unsigned)th[1])) || !b.ok) return st;
  a.noff = (u64*)b.get("pr_noff", ((u64)a.ket.nG + 1) * 8);
  a.ncur = (u64*)b.get("pr_ncur", (u64)a.ket.nG * 8);
  if (!b.ok) return SFCI_OK;
  SFCI_CUDA(cudaMemsetAsync(a.noff, 0, ((u64)a.ket.nG + 1) * 8, c.stream));
  SFCI_CUDA(cudaMemsetAsync(a.ncur, 0, (u64)a.ket.nG * 8, c.stream));
  const unsigned nslice = (unsigned)std::max<u64>(1, std::min<u64>((nda + 31) / 32, 8192 / std::max(1u, a.ket.nG)));
  const unsigned ng = b.grid((u64)a.ket.nG * nslice, 8);
  SFCI_LAUNCH(c, (k_pair_nbrs<W, false>), ng, 256, 0, a, nslice);
  if ((st = scan_excl(c, a.noff, a.noff, a.ket.nG))) return st;
  SFCI_LAUNCH(c, k_pair_diag<W>, (unsigned)std::max<u64>(1, std::min<u64>((a.ket.n + 7) / 8, b.gmax * 2)), 256, 0,
              a.ket.keys, a.ket.n, a.h, diagE);
  SFCI_CUDA(cudaMemcpyAsync(tot, a.noff + a.ket.nG, 8, cudaMemcpyDeviceToDevice, c.stream));
  if ((st = read_words(c, tot, 6 * 8, rb))) return st;
  const u64 nt = rb[0];
  // The sweep visits n * conn targets for the pair search's `tests` comparisons.  In
  // small, nearly full spaces groups are large and most targets are bras: measured
  // at 20 spin orbitals 186 against 204 us (0.3 tests a target), 990 against 1114
  // (2.6), 4128 against 3373 (5.9); at 56 the ratio is 0.02 to 0.7 and the search 6
  // to 15 times faster.
  if (rb[5] > 4 * a.ket.n * det_terms(na, nva, nb, nvb)) return SFCI_OK;
  const u64 nS = nt & 0xffffffffull, nD = nt >> 32;
  if (over(nS * 8 + nD * 12)) return SFCI_OK;
  a.nsg = (unsigned*)b.get("pr_nsg", std::max<u64>(1, nS) * 4);
  a.nsx = (unsigned*)b.get("pr_nsx", std::max<u64>(1, nS) * 4);
  a.ndg = (unsigned*)b.get("pr_ndg", std::max<u64>(1, nD) * 4);
  a.ndv = (double*)b.get("pr_ndv", std::max<u64>(1, nD) * 8);
  if (!b.ok) return SFCI_OK;
  SFCI_LAUNCH(c, (k_pair_nbrs<W, true>), ng, 256, 0, a, nslice);
  SFCI_LAUNCH(c, (k_pairs<W, ENERGY>), (unsigned)std::max<u64>(1, std::min<u64>((a.ket.n + 7) / 8, b.gmax)), 256, 0, a);
  if ((st = read_words(c, tot + 4, 4 * 8, rb))) return st;
  if (rb[0] >> 32) return SFCI_OK;  // out of range: the general sweep reports it
  a.sum[0] = rb[2];
  a.sum[1] = rb[3];
  if (links) *links = nS + nD;
  *done = true;
  return SFCI_OK;
}

}  // namespace

template <int W>
int pairs_energy(Ctx& c, const typename KeyOf<W>::T* keys, const double* amps, u64 n, double* E, u64* terms,
                 u64* links, bool* done) {
  PairArgs<W> a{};
  a.bra.keys = a.ket.keys = keys;
  a.bra.n = a.ket.n = n;
  a.amps = a.bamps = amps;
  int st = run_pairs<W, true>(c, a, 0, links, done);
  if (st || !*done) return st;
  *E = fx_to_double(a.sum[0], a.sum[1]) / a.up2;
  *terms = n * det_terms(a.na, a.nva, a.nb, c.M - a.nb);
  return SFCI_OK;
}

template <int W>
int pairs_project(Ctx& c, const typename KeyOf<W>::T* keys, const double* amps, u64 n, u64 T, double lambda,
                  const typename KeyOf<W>::T* table, u64 slots, u64* plo, u64* phi, bool* done) {
  PairArgs<W> a{};
  a.ket.keys = keys;
  a.ket.n = n;
  a.bra.keys = table;
  a.bra.n = slots;
  a.bra.table = 1;
  a.amps = amps;
  a.lambda = lambda;
  a.plo = plo;
  a.phi = phi;
  return run_pairs<W, false>(c, a, T, nullptr, done);
}

template int pairs_energy<1>(Ctx&, const u64*, const double*, u64, double*, u64*, u64*, bool*);
template int pairs_energy<2>(Ctx&, const K128*, const double*, u64, double*, u64*, u64*, bool*);
template int pairs_project<1>(Ctx&, const u64*, const double*, u64, u64, double, const u64*, u64, u64*, u64*, bool*);
template int pairs_project<2>(Ctx&, const K128*, const double*, u64, u64, double, const K128*, u64, u64*, u64*, bool*);

}  // namespace sfci
