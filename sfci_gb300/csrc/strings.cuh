// Spin strings: a determinant as a pair (alpha string, beta string) of occupied
// spatial orbitals, their hashes and ranks, and matrix elements between strings
// (rows.cu, pairs.cu).
#pragma once

#include "gen.cuh"
#include "prims.cuh"

namespace sfci {

constexpr u64 ROW_RANKS_MAX = 1ull << 25;  // strings of one spin the rank tables cover

template <int W> struct StrOf;
template <> struct StrOf<1> { typedef uint32_t T; };
template <> struct StrOf<2> { typedef u64 T; };

// ---- strings ----------------------------------------------------------------
__device__ __forceinline__ uint32_t even_bits(u64 x) {
  x &= 0x5555555555555555ull;
  x = (x | (x >> 1)) & 0x3333333333333333ull;
  x = (x | (x >> 2)) & 0x0f0f0f0f0f0f0f0full;
  x = (x | (x >> 4)) & 0x00ff00ff00ff00ffull;
  x = (x | (x >> 8)) & 0x0000ffff0000ffffull;
  x = (x | (x >> 16)) & 0x00000000ffffffffull;
  return (uint32_t)x;
}
__device__ __forceinline__ u64 spread_bits(uint32_t v) {
  u64 x = v;
  x = (x | (x << 16)) & 0x0000ffff0000ffffull;
  x = (x | (x << 8)) & 0x00ff00ff00ff00ffull;
  x = (x | (x << 4)) & 0x0f0f0f0f0f0f0f0full;
  x = (x | (x << 2)) & 0x3333333333333333ull;
  x = (x | (x << 1)) & 0x5555555555555555ull;
  return x;
}
__device__ __forceinline__ void split_key(const u64& k, uint32_t& a, uint32_t& b) {
  a = even_bits(k);
  b = even_bits(k >> 1);
}
__device__ __forceinline__ void split_key(const K128& k, u64& a, u64& b) {
  a = (u64)even_bits(k.lo) | ((u64)even_bits(k.hi) << 32);
  b = (u64)even_bits(k.lo >> 1) | ((u64)even_bits(k.hi >> 1) << 32);
}
__device__ __forceinline__ u64 join_key(uint32_t a, uint32_t b) { return spread_bits(a) | (spread_bits(b) << 1); }
__device__ __forceinline__ K128 join_key(u64 a, u64 b) {
  K128 k;
  k.lo = spread_bits((uint32_t)a) | (spread_bits((uint32_t)b) << 1);
  k.hi = spread_bits((uint32_t)(a >> 32)) | (spread_bits((uint32_t)(b >> 32)) << 1);
  return k;
}
__device__ __forceinline__ bool key_within(const u64& k, int N) { return N >= 64 || (k >> N) == 0; }
__device__ __forceinline__ bool key_within(const K128& k, int N) {
  return N >= 64 ? (N >= 128 || (k.hi >> (N - 64)) == 0) : (k.hi == 0 && (k.lo >> N) == 0);
}
__device__ __forceinline__ int spop(uint32_t s) { return __popc(s); }
__device__ __forceinline__ int spop(u64 s) { return __popcll(s); }
__device__ __forceinline__ int sffs(uint32_t s) { return __ffs((int)s) - 1; }
__device__ __forceinline__ int sffs(u64 s) { return __ffsll((long long)s) - 1; }
template <class ST>
__device__ __forceinline__ ST sbit(int p) { return (ST)1 << p; }
// orbitals strictly between p and q
template <class ST>
__device__ __forceinline__ ST sbetween(int p, int q) {
  const int lo = p < q ? p : q, hi = p < q ? q : p;
  return (sbit<ST>(hi) - 1) & ~((sbit<ST>(lo) << 1) - 1);
}
template <class ST>
__device__ __forceinline__ unsigned move_par(ST s, int p, int q) { return spop((ST)(s & sbetween<ST>(p, q))) & 1; }
// s(A, B): the parity of moving every alpha operator in front of the beta ones,
// the number of pairs (alpha p, beta q) with q < p
__device__ __forceinline__ unsigned interleave_par(uint32_t a, uint32_t b) {
  uint32_t y = b << 1;  // prefix XOR, exclusive
  y ^= y << 1; y ^= y << 2; y ^= y << 4; y ^= y << 8; y ^= y << 16;
  return __popc(a & y) & 1;
}
__device__ __forceinline__ unsigned interleave_par(u64 a, u64 b) {
  u64 y = b << 1;
  y ^= y << 1; y ^= y << 2; y ^= y << 4; y ^= y << 8; y ^= y << 16; y ^= y << 32;
  return __popcll(a & y) & 1;
}

// hashed strings: multiplication by an odd constant; hs_top: the top 32 bits of
// a hash, in which ranges and buckets are expressed; hs_slot: slot of a table
// of 2^tb slots, a second multiplicative hash
__device__ __forceinline__ uint32_t hs_of(uint32_t s) { return s * 0x9e3779b1u; }
__device__ __forceinline__ u64 hs_of(u64 s) { return s * 0x9e3779b97f4a7c15ull; }
__device__ __forceinline__ uint32_t hs_inv(uint32_t h) { return h * 0x0e8b2f51u; }
__device__ __forceinline__ u64 hs_inv(u64 h) { return h * 0xf1de83e19937733dull; }
__device__ __forceinline__ uint32_t hs_top(uint32_t h) { return h; }
__device__ __forceinline__ uint32_t hs_top(u64 h) { return (uint32_t)(h >> 32); }
__device__ __forceinline__ unsigned hs_slot(uint32_t h, int tb) { return (h * 0x85ebca6bu) >> (32 - tb); }
__device__ __forceinline__ unsigned hs_slot(u64 h, int tb) {
  return (unsigned)((h * 0xd6e8feb86659fd93ull) >> (64 - tb));
}
__device__ __forceinline__ unsigned bucket_of(uint32_t top, int bits) { return bits ? top >> (32 - bits) : 0u; }

// colex rank of a string (bin[p * 34 + k] = C(p, k)); unrank by a whole warp
template <class ST>
__device__ __forceinline__ unsigned rank_of(const unsigned* bin, ST s) {
  unsigned r = 0;
  for (int k = 1; s; ++k) {
    const int p = sffs(s);
    r += bin[p * 34 + k];
    s &= s - 1;
  }
  return r;
}
template <class ST>
__device__ __forceinline__ ST unrank_warp(const unsigned* bin, unsigned r, int n, int M) {
  const int lane = threadIdx.x & 31;
  ST s = 0;
  for (int k = n; k >= 1; --k) {
    const unsigned lo = __ballot_sync(0xffffffffu, lane < M && bin[lane * 34 + k] <= r);
    int p = 31 - __clz((int)lo);
    if (sizeof(ST) == 8) {
      const unsigned hi = __ballot_sync(0xffffffffu, lane + 32 < M && bin[(lane + 32) * 34 + k] <= r);
      if (hi) p = 63 - __clz((int)hi);
    }
    s |= sbit<ST>(p);
    r -= bin[p * 34 + k];
  }
  return s;
}
template <class ST>
__device__ __forceinline__ ST unrank_thread(const unsigned* bin, unsigned r, int n, int M) {
  ST s = 0;
  int p = M - 1;
  for (int k = n; k >= 1; --k) {
    while (bin[p * 34 + k] > r) --p;
    s |= sbit<ST>(p);
    r -= bin[p * 34 + k];
  }
  return s;
}

// packed pair index of a strictly upper pair list: (x < y) of k = y(y-1)/2 + x
__device__ __forceinline__ void unrank_pair2(unsigned k, unsigned& x, unsigned& y) {
  y = (unsigned)((1.0f + sqrtf(1.0f + 8.0f * (float)k)) * 0.5f);
  while (y * (y - 1) / 2 > k) --y;
  while ((y + 1) * y / 2 <= k) ++y;
  x = k - y * (y - 1) / 2;
}

// element of a same-spin double i<j -> a<b (spatial orbitals, spin s) from string
// `str`, with its phase in the separated order: (a,i,b,j) - (b,i,a,j)
template <class ST>
__device__ __forceinline__ double double_elem(const HamView& h, int s, ST str, int i, int j, int a, int b) {
  const double v = vat(h, 3 * s, (unsigned)spatial_pair(i, a), (unsigned)spatial_pair(j, b)) -
                   vat(h, 3 * s, (unsigned)spatial_pair(i, b), (unsigned)spatial_pair(j, a));
  const unsigned par = move_par(str, i, a) ^ move_par((ST)(str ^ sbit<ST>(i) ^ sbit<ST>(a)), j, b);
  return signed_by(par, v);
}

// Elements of 32 singles i -> a of spin s (spatial orbitals), one per lane, of
// determinants (A, B) with at most 16 electrons a spin, without their phase.
// Four lanes work on a single at a time and lane l ends up with its own single's
// element; all lanes of the warp call it.  The sum has the bits single_amp_half
// (gen.cuh) gives it: there lane l of 16 adds the l-th occupied alpha and beta
// orbitals' integrals and the lanes combine at distances 8, 4, 2, 1; here lane q
// of 4 holds lanes q, q + 4, q + 8, q + 12.  sj: Coulomb integrals by spin of the
// single, spin of the occupied orbital, i, a, k; sk: exchange integrals by spin,
// i, a, k (k_rows_sj).
template <class ST>
__device__ __forceinline__ double single_elems(const double* sj, const double* sk, const double* h1, int M, int s,
                                               int i, int a, ST A, ST B, int na, int nb, bool act) {
  const int lane = threadIdx.x & 31, q = lane & 3;
  const int MM = M * M * M;
  double mine = 0.0;
  const unsigned any = __ballot_sync(0xffffffffu, act);
#pragma unroll 1
  for (int r0 = 0; r0 < 4; ++r0) {  // singles of lanes r0, r0 + 4, ...
    if (!(any & (0x11111111u << r0))) continue;
    const int src = (lane & 28) + r0;
    const int i_ = __shfl_sync(0xffffffffu, i, src), a_ = __shfl_sync(0xffffffffu, a, src);
    const ST A_ = __shfl_sync(0xffffffffu, A, src), B_ = __shfl_sync(0xffffffffu, B, src);
    double p[4] = {0.0, 0.0, 0.0, 0.0};
    if ((any >> src) & 1u) {
      const int ia = (i_ * M + a_) * M;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const double* row = sj + (2 * s + u) * MM + ia;
        const double* xrow = sk + s * MM + ia;
        ST o = u ? B_ : A_;
        const int n = u ? nb : na;
        for (int x = 0; x < q; ++x) o &= o - 1;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          if (q + 4 * r < n) {
            const int k = sffs(o);
            if (u != s || k != i_) {
              p[r] += SFCI_LDG(row + k);
              if (u == s) p[r] -= SFCI_LDG(xrow + k);
            }
#pragma unroll
            for (int x = 0; x < 4; ++x) o &= o - 1;
          }
        }
      }
    }
    double v = (p[0] + p[2]) + (p[1] + p[3]);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    if (q == r0) mine = v;
  }
  if (act) mine += SFCI_LDG(h1 + (s * M + a) * M + i);
  return mine;
}

// bucket bits of a list of n entries: about two entries a bucket
__device__ __forceinline__ int bucket_bits(u64 n) {
  int b = 0;
  while (b < 20 && (2ull << b) < n) ++b;
  return b;
}

// Entries of 32 short lists at once: lane l holds list [st, st + len); calls
// f(valid, entry, owner lane) with all lanes.
template <class F>
__device__ __forceinline__ void warp_expand_own(unsigned st, unsigned len, F f) {
  const int lane = threadIdx.x & 31;
  unsigned inc = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  const unsigned tot = __shfl_sync(0xffffffffu, inc, 31);
  const unsigned at = st - (inc - len);  // entry = at + flat index
  for (unsigned t0 = 0; t0 < tot; t0 += 32) {
    const unsigned t = t0 + lane;
    int lo = 0;  // the number of lists that end at or before t
#pragma unroll
    for (int step = 16; step; step >>= 1) {
      const unsigned y = __shfl_sync(0xffffffffu, inc, lo + step - 1);
      if (y <= t) lo += step;
    }
    lo &= 31;
    const unsigned e = __shfl_sync(0xffffffffu, at, lo) + t;
    f(t < tot, t < tot ? e : 0u, lo);
  }
}
// the same with a factor per list: f(valid, entry, factor)
template <class F>
__device__ __forceinline__ void warp_expand(unsigned st, unsigned len, double val, F f) {
  warp_expand_own(st, len, [&](bool ok, unsigned e, int own) { f(ok, e, __shfl_sync(0xffffffffu, val, own)); });
}

// C(n, k), saturated at 2^32 - 1
inline u64 binom(int n, int k) {
  if (k < 0 || k > n) return 0;
  __int128 r = 1;
  for (int i = 1; i <= k; ++i) {
    r = r * (n - k + i) / i;
    if (r > 0xffffffffll) return 0xffffffffull;
  }
  return (u64)r;
}

// Electrons of each spin of n determinants (rows.cu): *ok when all have the same,
// lie within the spin orbitals, and (unique) none repeats the one before it.
template <int W>
int keys_one_spin(Ctx& c, const typename KeyOf<W>::T* keys, u64 n, bool unique, int* na, int* nb, bool* ok);

// per-context tables of rows.cu and pairs.cu: binomials, oriented opposite-spin
// integrals and directed integrals of the singles (false: no memory)
bool row_tables(Ctx& c, const HamView& h);

}  // namespace sfci
