// Device primitives (see prims.cuh).
#include <algorithm>
#include <cstring>

#include "prims.cuh"

namespace sfci {

// ============================================================================
// exclusive scan (reduce-then-scan, recursive over block sums)
// ============================================================================

template <typename T>
__global__ void k_scan_reduce(const T* __restrict__ in, size_t n, T* __restrict__ bsum) {
  __shared__ T sh[SCAN_THREADS / 32 + 1];
  size_t base = (size_t)blockIdx.x * SCAN_TILE;
  T s = 0;
#pragma unroll
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    size_t idx = base + (size_t)i * SCAN_THREADS + threadIdx.x;
    if (idx < n) s += __ldcg(in + idx);  // counts may come from atomics of the previous kernel
  }
  T tot;
  block_excl_scan<T, SCAN_THREADS>(s, &tot, sh);
  if (threadIdx.x == 0) bsum[blockIdx.x] = tot;
}

template <typename T>
__global__ void k_scan_down(const T* in, T* out, size_t n, const T* __restrict__ boff) {
  __shared__ T sh[SCAN_THREADS / 32 + 1];
  size_t base = (size_t)blockIdx.x * SCAN_TILE + (size_t)threadIdx.x * SCAN_ITEMS;
  T v[SCAN_ITEMS];
  T s = 0;
#pragma unroll
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    v[i] = (base + i < n) ? __ldcg(in + base + i) : T(0);
    s += v[i];
  }
  T off = block_excl_scan<T, SCAN_THREADS>(s, nullptr, sh) + (boff ? boff[blockIdx.x] : T(0));
#pragma unroll
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    if (base + i < n) out[base + i] = off;
    off += v[i];
  }
  if (n > 0 && base <= n - 1 && n - 1 < base + SCAN_ITEMS) out[n] = off;
}

template <typename T>
static int scan_impl(Ctx& c, const T* in, T* out, size_t n, int depth) {
  if (n == 0) {
    SFCI_CUDA(cudaMemsetAsync(out, 0, sizeof(T), c.stream));
    return SFCI_OK;
  }
  size_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
  if (nb == 1) {
    SFCI_LAUNCH(c, k_scan_down<T>, 1, SCAN_THREADS, 0, in, out, n, (const T*)nullptr);
    return SFCI_OK;
  }
  char name[32];
  snprintf(name, sizeof name, "scan_%d_%d", (int)sizeof(T), depth);
  T* bs = (T*)scratch_get(c, name, (nb + 1) * sizeof(T));
  if (!bs) return SFCI_ERR_NOMEM;
  SFCI_LAUNCH(c, k_scan_reduce<T>, (unsigned)nb, SCAN_THREADS, 0, in, n, bs);
  int st = scan_impl<T>(c, bs, bs, nb, depth + 1);
  if (st) return st;
  SFCI_LAUNCH(c, k_scan_down<T>, (unsigned)nb, SCAN_THREADS, 0, in, out, n, (const T*)bs);
  return SFCI_OK;
}

int scan_excl(Ctx& c, const u64* in, u64* out, size_t n) { return scan_impl<u64>(c, in, out, n, 0); }
int scan_excl_u32(Ctx& c, const uint32_t* in, uint32_t* out, size_t n) {
  return scan_impl<uint32_t>(c, in, out, n, 0);
}

// ============================================================================
// LSD radix sort, 8-bit digits, 4096-item tiles, stable warp-ordered ranking
// ============================================================================

constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_CHUNKS = 16;
constexpr int RS_TILE = RS_THREADS * RS_CHUNKS;  // 4096

template <class KT>
__global__ void k_rs_hist(const KT* __restrict__ keys, size_t n, int shift, uint32_t* __restrict__ counts,
                          size_t ntiles) {
  __shared__ uint32_t hist[256];
  hist[threadIdx.x] = 0;
  __syncthreads();
  size_t base = (size_t)blockIdx.x * RS_TILE;
#pragma unroll 4
  for (int i = 0; i < RS_CHUNKS; ++i) {
    size_t idx = base + (size_t)i * RS_THREADS + threadIdx.x;
    if (idx < n) atomicAdd(&hist[key_digit(keys[idx], shift)], 1u);
  }
  __syncthreads();
  counts[(size_t)threadIdx.x * ntiles + blockIdx.x] = hist[threadIdx.x];
}

template <class KT>
__global__ void __launch_bounds__(RS_THREADS) k_rs_scatter(const KT* __restrict__ kin, const double* __restrict__ vin,
                                                          KT* __restrict__ kout, double* __restrict__ vout, size_t n,
                                                          int shift, const uint32_t* __restrict__ offs, size_t ntiles) {
  __shared__ uint32_t whist[RS_WARPS][256];
  __shared__ uint32_t base[256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int d = threadIdx.x; d < RS_WARPS * 256; d += RS_THREADS) (&whist[0][0])[d] = 0;
  base[threadIdx.x] = offs[(size_t)threadIdx.x * ntiles + blockIdx.x];
  __syncthreads();
  const size_t wbase = (size_t)blockIdx.x * RS_TILE + (size_t)warp * (RS_CHUNKS * 32);
  KT k[RS_CHUNKS];
  double v[RS_CHUNKS];
  int dg[RS_CHUNKS];
#pragma unroll
  for (int c = 0; c < RS_CHUNKS; ++c) {
    size_t idx = wbase + (size_t)c * 32 + lane;
    bool valid = idx < n;
    if (valid) {
      k[c] = kin[idx];
      v[c] = vin[idx];
      dg[c] = (int)key_digit(k[c], shift);
    } else {
      dg[c] = 256 + lane;
    }
    unsigned peers = __match_any_sync(0xffffffffu, dg[c]);
    if (valid && lane == __ffs(peers) - 1) whist[warp][dg[c]] += __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  {
    int d = threadIdx.x;
    uint32_t run = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
      uint32_t t = whist[w][d];
      whist[w][d] = run;
      run += t;
    }
  }
  __syncthreads();
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int c = 0; c < RS_CHUNKS; ++c) {
    size_t idx = wbase + (size_t)c * 32 + lane;
    bool valid = idx < n;
    unsigned peers = __match_any_sync(0xffffffffu, dg[c]);
    if (valid) {
      uint32_t pos = base[dg[c]] + whist[warp][dg[c]] + __popc(peers & lt);
      kout[pos] = k[c];
      vout[pos] = v[c];
    }
    __syncwarp();
    if (valid && lane == __ffs(peers) - 1) whist[warp][dg[c]] += __popc(peers);
    __syncwarp();
  }
}

// ---- one launch for vectors of up to COOP_MAX entries ---------------------------
// The multi-launch passes above cost five launches a digit, whatever the length.
// Here one cooperative kernel runs every pass: each CTA owns a slice of the input
// and counts it by digit per warp, publishes its counts, and after a grid barrier
// adds up the counts of the slices before it, so a pass needs two barriers.  Bound
// by the latency of its phases (about 17 us a pass at 500,000 entries, of which
// the barriers take 4).  Measured for 56-bit keys, us, launches -> one kernel: 860
// entries 162 -> 30, 50,000 213 -> 67, 500,000 288 -> 119, 2,000,000 533 -> 254,
// 4,000,000 945 -> 655, 6,000,000 1400 -> 1290 (12,000,000: 2490 -> 3660, so longer
// ones keep the launches); 68-bit keys 500,000 391 -> 177.  Digits of 8, 9 and 10 bits
// are within 10% of one another.
constexpr size_t COOP_MAX = 6u << 20;      // sort
constexpr size_t SEL_MAX = 1ull << 31;     // selection: faster at every size (30,000,000 entries 0.44 against 0.97 ms)
constexpr int CO_THREADS = 1024;
constexpr int CO_WARPS = CO_THREADS / 32;
constexpr int CO_DIGIT = 8;
constexpr int CO_BATCH = 2;  // entries a lane loads ahead

// Grid barrier of a cooperative launch (every CTA is resident): true when all
// CTAs arrived, false (and *err set) when they did not within the poll limit.  The
// limit, about 40 s, is there so that nothing waits forever: CTAs that get their
// SMs late, behind another stream's kernel of a few seconds, are waited for.  A CTA
// that gives up says so in the counter, and every other one leaves with it.
constexpr unsigned COOP_GAVE_UP = 1u << 31;
constexpr unsigned COOP_POLLS = 1u << 16, COOP_NAPS = 1u << 24;  // without and with a nap of 2 us between them
__device__ bool coop_barrier(unsigned* bar, unsigned target, unsigned* err) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    int ok = 0;
    for (unsigned spin = 0; spin < COOP_POLLS + COOP_NAPS; ++spin) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if (v & COOP_GAVE_UP) break;
      if (v >= target) {
        ok = 1;
        break;
      }
      if (spin >= COOP_POLLS) __nanosleep(2000);
    }
    if (!ok) {
      atomicOr(bar, COOP_GAVE_UP);
      *(volatile unsigned*)err = 1u;
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  const bool ok = s_ok != 0;
  __syncthreads();
  return ok;
}

__device__ __forceinline__ unsigned key_bits(const u64& k, int shift, unsigned mask) { return (unsigned)(k >> shift) & mask; }
__device__ __forceinline__ unsigned key_bits(const K128& k, int shift, unsigned mask) {
  if (shift >= 64) return (unsigned)(k.hi >> (shift - 64)) & mask;
  return (unsigned)((k.lo >> shift) | (shift ? k.hi << (64 - shift) : 0ull)) & mask;
}
__device__ __forceinline__ u64 ld_key(const u64* p) { return __ldcg(p); }
__device__ __forceinline__ K128 ld_key(const K128* p) {
  K128 k;
  k.lo = __ldcg((const u64*)p);
  k.hi = __ldcg((const u64*)p + 1);
  return k;
}

// (values written by other CTAs in an earlier pass are read through L2)
template <class KT>
__global__ void __launch_bounds__(CO_THREADS, 1) k_rs_coop(KT* ka, double* va, KT* kb, double* vb, unsigned n,
                                                        unsigned slice, int passes, int bits, uint32_t* cnt,
                                                        unsigned* bar, unsigned* err) {
  extern __shared__ __align__(16) unsigned char smem[];
  const unsigned nd = 1u << bits, mask = nd - 1u, G = gridDim.x, b = blockIdx.x;
  uint32_t* whist = reinterpret_cast<uint32_t*>(smem);  // [CO_WARPS][nd]
  uint32_t* base = whist + CO_WARPS * nd;               // [nd]
  __shared__ uint32_t s_scan[CO_WARPS + 1];
  __shared__ uint32_t s_bef[CO_THREADS], s_tot[CO_THREADS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt = (1u << lane) - 1u, ws = slice / CO_WARPS;  // a multiple of 32
  const unsigned w0 = min(n, b * slice + warp * ws), w1 = min(n, w0 + ws);
  uint32_t* wh = whist + warp * nd;
  unsigned target = 0;
  for (int p = 0; p < passes; ++p) {
    const int shift = p * bits;
    for (unsigned d = tid; d < CO_WARPS * nd; d += CO_THREADS) whist[d] = 0;
    __syncthreads();
    for (unsigned i = w0 + lane; i < w1; i += 32) atomicAdd(&wh[key_bits(ld_key(ka + i), shift, mask)], 1u);
    __syncthreads();
    // counts of the slice; each warp's become its offset within the slice
    uint32_t mine = 0;
    if (tid < (int)nd) {
#pragma unroll 8
      for (int w = 0; w < CO_WARPS; ++w) {
        const uint32_t t = whist[w * nd + tid];
        whist[w * nd + tid] = mine;
        mine += t;
      }
    }
    uint32_t before = 0, total = mine;
    if (G > 1) {
      uint32_t* c = cnt + (size_t)(p & 1) * G * nd;  // the previous pass's counts may still be read
      if (tid < (int)nd) __stcg(c + (size_t)b * nd + tid, mine);
      target += G;
      if (!coop_barrier(bar, target, err)) return;
      // thread (part, digit) adds its share of the slices; the parts meet in shared memory
      const unsigned d = tid & mask, part = tid >> bits, parts = CO_THREADS >> bits;
      uint32_t bef = 0, tot = 0;
      for (unsigned q = part; q < G; q += 8 * parts) {
        uint32_t v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = q + u * parts < G ? __ldcg(c + (size_t)(q + u * parts) * nd + d) : 0u;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (q + u * parts < b) bef += v[u];
          tot += v[u];
        }
      }
      s_bef[tid] = bef;
      s_tot[tid] = tot;
      __syncthreads();
      if (tid < (int)nd) {
        total = 0;
        for (unsigned q = 0; q < parts; ++q) {
          before += s_bef[q * nd + tid];
          total += s_tot[q * nd + tid];
        }
      }
    }
    const uint32_t ex = block_excl_scan<uint32_t, CO_THREADS>(tid < (int)nd ? total : 0u, nullptr, s_scan);
    if (tid < (int)nd) base[tid] = ex + before;
    __syncthreads();
    for (unsigned i0 = w0; i0 < w1; i0 += 32 * CO_BATCH) {
      KT k[CO_BATCH];
      double v[CO_BATCH];
#pragma unroll
      for (int q = 0; q < CO_BATCH; ++q) {
        const unsigned i = i0 + q * 32 + lane;
        if (i < w1) {
          k[q] = ld_key(ka + i);
          v[q] = __ldcg(va + i);
        }
      }
#pragma unroll
      for (int q = 0; q < CO_BATCH; ++q) {
        if (i0 + q * 32 >= w1) break;  // (the same for the whole warp)
        const bool ok = i0 + q * 32 + lane < w1;
        const unsigned d = ok ? key_bits(k[q], shift, mask) : nd + lane;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        uint32_t pos = 0;
        if (ok) pos = wh[d] + __popc(peers & lt);
        __syncwarp();
        if (ok) {
          if (lane == __ffs(peers) - 1) wh[d] += __popc(peers);
          pos += base[d];
          kb[pos] = k[q];
          vb[pos] = v[q];
        }
        __syncwarp();
      }
    }
    if (G > 1) {
      target += G;
      if (!coop_barrier(bar, target, err)) return;
    } else {
      __syncthreads();
    }
    KT* tk = ka;
    ka = kb;
    kb = tk;
    double* tv = va;
    va = vb;
    vb = tv;
  }
  if (passes & 1)  // the result is in the second buffers
    for (unsigned i = w0 + lane; i < w1; i += 32) {
      kb[i] = ld_key(ka + i);
      vb[i] = __ldcg(va + i);
    }
}

// Cooperative launch; *ran false when the context's one-launch forms are switched
// off, or when the GPU cannot hold the grid at once (a share of the SMs under MPS, for
// one): the callers then take the multi-launch forms.
static int coop_launch(Ctx& c, const void* kern, unsigned G, void** args, size_t sm, bool* ran) {
  *ran = false;
  if (!c.grid_barrier) return SFCI_OK;
  const cudaError_t e = cudaLaunchCooperativeKernel(kern, dim3(G), dim3(CO_THREADS), args, sm, c.stream);
  if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
    cudaGetLastError();
    return SFCI_OK;
  }
  SFCI_CUDA(e);
  c.launches++;
  *ran = true;
  return SFCI_OK;
}

// entries a CTA takes, for n entries
static unsigned coop_slice(const Ctx& c, size_t n) {
  const size_t s = (n + c.sm_count - 1) / c.sm_count;
  return (unsigned)std::max<size_t>(1024, (s + 1023) / 1024 * 1024);
}

template <int W>
static int radix_sort_coop(Ctx& c, typename KeyOf<W>::T* keys, double* vals, size_t n, int nbits, bool* ran) {
  typedef typename KeyOf<W>::T KT;
  const int nb8 = (nbits + 7) / 8 * 8;  // the bits the 8-bit passes cover
  int passes = (nb8 + CO_DIGIT - 1) / CO_DIGIT, bits = (nb8 + passes - 1) / passes;
  unsigned slice = coop_slice(c, n), un = (unsigned)n;
  const unsigned G = (un + slice - 1) / slice;
  KT* k2 = (KT*)scratch_get(c, "rs_keys", n * sizeof(KT));
  double* v2 = (double*)scratch_get(c, "rs_vals", n * sizeof(double));
  uint32_t* cnt = (uint32_t*)scratch_get(c, "rs_coop", (4 + 2 * ((size_t)c.sm_count << CO_DIGIT)) * sizeof(uint32_t));
  if (!k2 || !v2 || !cnt) return SFCI_ERR_NOMEM;
  unsigned* bar = cnt;
  uint32_t* cm = cnt + 4;
  unsigned* err = coop_error_word(c);
  if (!err) return SFCI_ERR_NOMEM;
  if (G > 1) SFCI_CUDA(cudaMemsetAsync(bar, 0, sizeof(unsigned), c.stream));
  const size_t sm = sizeof(uint32_t) * ((size_t)(CO_WARPS + 1) << bits);
  SFCI_CUDA(cudaFuncSetAttribute(k_rs_coop<KT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(uint32_t) * ((size_t)(CO_WARPS + 1) << CO_DIGIT))));
  void* args[] = {&keys, &vals, &k2, &v2, &un, &slice, &passes, &bits, &cm, &bar, &err};
  return coop_launch(c, (const void*)k_rs_coop<KT>, G, args, sm, ran);
}

template <int W>
int radix_sort_pairs(Ctx& c, typename KeyOf<W>::T* keys, double* vals, size_t n, int nbits) {
  typedef typename KeyOf<W>::T KT;
  if (n <= 1 || nbits <= 0) return SFCI_OK;
  if (n >= (1ull << 32)) return set_error(SFCI_ERR_UNSUPPORTED, "radix sort beyond 2^32 items");
  bool ran = false;
  int st;
  if (n <= COOP_MAX && ((st = radix_sort_coop<W>(c, keys, vals, n, nbits, &ran)) || ran)) return st;
  size_t ntiles = (n + RS_TILE - 1) / RS_TILE;
  KT* k2 = (KT*)scratch_get(c, "rs_keys", n * sizeof(KT));
  double* v2 = (double*)scratch_get(c, "rs_vals", n * sizeof(double));
  uint32_t* cnt = (uint32_t*)scratch_get(c, "rs_cnt", (256 * ntiles + 1) * sizeof(uint32_t));
  if (!k2 || !v2 || !cnt) return SFCI_ERR_NOMEM;
  KT* ka = keys;
  double* va = vals;
  KT* kb = k2;
  double* vb = v2;
  int passes = (nbits + 7) / 8;
  for (int p = 0; p < passes; ++p) {
    int shift = 8 * p;
    SFCI_LAUNCH(c, k_rs_hist<KT>, (unsigned)ntiles, RS_THREADS, 0, ka, n, shift, cnt, ntiles);
    int st = scan_excl_u32(c, cnt, cnt, 256 * ntiles);
    if (st) return st;
    SFCI_LAUNCH(c, k_rs_scatter<KT>, (unsigned)ntiles, RS_THREADS, 0, ka, va, kb, vb, n, shift,
                (const uint32_t*)cnt, ntiles);
    std::swap(ka, kb);
    std::swap(va, vb);
  }
  if (ka != keys) {
    SFCI_CUDA(cudaMemcpyAsync(keys, ka, n * sizeof(KT), cudaMemcpyDeviceToDevice, c.stream));
    SFCI_CUDA(cudaMemcpyAsync(vals, va, n * sizeof(double), cudaMemcpyDeviceToDevice, c.stream));
  }
  return SFCI_OK;
}

template int radix_sort_pairs<1>(Ctx&, u64*, double*, size_t, int);
template int radix_sort_pairs<2>(Ctx&, K128*, double*, size_t, int);

// ============================================================================
// radix select on |amp|
// ============================================================================

__global__ void k_sel_hist(const double* __restrict__ a, size_t n, int shift, int width, u64 prefix,
                           int pshift, uint32_t* __restrict__ hist) {
  __shared__ uint32_t sh[4096];
  const int nb = 1 << width;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const u64 mask = (u64)nb - 1;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    u64 b = abs_bits(a[i]);
    if (pshift >= 64 || (b >> pshift) == prefix) atomicAdd(&sh[(b >> shift) & mask], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nb; i += blockDim.x)
    if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

int select_threshold(Ctx& c, const double* amps, size_t n, size_t k, u64* tau, size_t* gt) {
  if (k == 0 || k >= n) return set_error(SFCI_ERR_ARG, "select_threshold needs 0 < k < n");
  uint32_t* hist = (uint32_t*)scratch_get(c, "sel_hist", 4096 * sizeof(uint32_t));
  if (!hist) return SFCI_ERR_NOMEM;
  std::vector<uint32_t> h(4096);
  // 63 magnitude bits: five 12-bit digits (bits 62..3) then the last 3 bits
  const int shifts[6] = {51, 39, 27, 15, 3, 0};
  const int widths[6] = {12, 12, 12, 12, 12, 3};
  u64 prefix = 0;
  size_t need = k;  // how many still to take from items matching prefix
  size_t above = 0;
  unsigned grid = (unsigned)std::min<size_t>((n + 255) / 256, (size_t)c.sm_count * 8);
  if (grid == 0) grid = 1;
  for (int r = 0; r < 6; ++r) {
    int nb = 1 << widths[r];
    SFCI_CUDA(cudaMemsetAsync(hist, 0, nb * sizeof(uint32_t), c.stream));
    int pshift = shifts[r] + widths[r];
    SFCI_LAUNCH(c, k_sel_hist, grid, 256, 0, amps, n, shifts[r], widths[r], prefix, r == 0 ? 64 : pshift, hist);
    int st = read_words(c, hist, nb * sizeof(uint32_t), h.data());
    if (st) return st;
    size_t acc = 0;
    int b = nb - 1;
    for (; b >= 0; --b) {
      if (acc + h[b] >= need) break;
      acc += h[b];
    }
    if (b < 0) return set_error(SFCI_ERR_NUMERIC, "radix select lost items (NaN amplitudes?)");
    above += acc;
    need -= acc;
    prefix = (prefix << widths[r]) | (u64)b;
  }
  *tau = prefix;
  *gt = above;
  return SFCI_OK;
}

// ============================================================================
// stable compaction (warp-ballot ranking over 4096-item tiles)
// ============================================================================

constexpr int CP_THREADS = 256;
constexpr int CP_CHUNKS = 16;
constexpr int CP_TILE = CP_THREADS * CP_CHUNKS;

// mode 0: keep |a| > cut
// mode 1: keep |a| > tau or (|a| == tau and eq-rank >= eq_skip), then |a| > tiny if tiny >= 0.
// Ties at the threshold are kept from the end of the index order (the largest keys
// of a key-sorted vector), as a stable ascending sort by |a| followed by "keep the
// last k" does.
// The magnitude tests compare the bits of |a| as integers (cut_key: -1 keeps
// everything), which orders finite doubles as their values do and keeps these
// passes off the FP64 pipe.
struct KeepRule {
  int mode;
  u64 tau;
  u64 eq_skip;
  long long cut_key;   // mode 0: keep |a| > cut
  long long tiny_key;  // mode 1: then |a| > tiny (-1: no such filter)
};

__device__ __forceinline__ bool keep_of(const KeepRule& r, double a, u64 eq_rank, bool& is_eq) {
  u64 b = abs_bits(a);
  if (r.mode == 0) {
    is_eq = false;
    return (long long)b > r.cut_key;
  }
  is_eq = (b == r.tau);
  bool k = b > r.tau || (is_eq && eq_rank >= r.eq_skip);
  return k && (long long)b > r.tiny_key;
}

// stage 0: per-tile count of |a| == tau
__global__ void k_cp_eqcount(const double* __restrict__ a, size_t n, u64 tau, u64* __restrict__ eqc) {
  __shared__ u64 sh[CP_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  size_t wb = (size_t)blockIdx.x * CP_TILE + (size_t)warp * (CP_CHUNKS * 32);
  u64 cnt = 0;
  for (int ch = 0; ch < CP_CHUNKS; ++ch) {
    size_t i = wb + (size_t)ch * 32 + lane;
    bool e = i < n && abs_bits(a[i]) == tau;
    cnt += __popc(__ballot_sync(0xffffffffu, e));
  }
  if (lane == 0) sh[warp] = cnt;
  __syncthreads();
  if (threadIdx.x == 0) {
    u64 t = 0;
    for (int w = 0; w < CP_THREADS / 32; ++w) t += sh[w];
    eqc[blockIdx.x] = t;
  }
}

// stage 1 (write=false): per-tile keep counts; stage 2 (write=true): scatter
template <class KT, bool WRITE>
__global__ void k_cp_pass(const KT* __restrict__ ik, const double* __restrict__ ia, size_t n, KeepRule rule,
                          const u64* __restrict__ eqoff, u64* __restrict__ keepc, const u64* __restrict__ keepoff,
                          KT* __restrict__ ok, double* __restrict__ oa) {
  __shared__ u64 sh_eq[CP_THREADS / 32], sh_kp[CP_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  size_t wb = (size_t)blockIdx.x * CP_TILE + (size_t)warp * (CP_CHUNKS * 32);
  // warp-level eq counts (for eq rank) and keep counts
  u64 weq = 0, wkp = 0;
  if (rule.mode == 1) {
    for (int ch = 0; ch < CP_CHUNKS; ++ch) {
      size_t i = wb + (size_t)ch * 32 + lane;
      bool e = i < n && abs_bits(ia[i]) == rule.tau;
      weq += __popc(__ballot_sync(0xffffffffu, e));
    }
  }
  if (lane == 0) sh_eq[warp] = weq;
  __syncthreads();
  u64 eq_run = rule.mode == 1 ? eqoff[blockIdx.x] : 0;
  for (int w = 0; w < warp; ++w) eq_run += sh_eq[w];
  u64 kp_run = 0;
  if (WRITE) {
    // need the keep offsets of earlier warps: recompute counts first
    u64 e2 = eq_run;
    for (int ch = 0; ch < CP_CHUNKS; ++ch) {
      size_t i = wb + (size_t)ch * 32 + lane;
      bool valid = i < n;
      double a = valid ? ia[i] : 0.0;
      bool ise = false;
      unsigned eb = __ballot_sync(0xffffffffu, valid && rule.mode == 1 && abs_bits(a) == rule.tau);
      bool k = valid && keep_of(rule, a, e2 + __popc(eb & lt), ise);
      e2 += __popc(eb);
      wkp += __popc(__ballot_sync(0xffffffffu, k));
    }
    if (lane == 0) sh_kp[warp] = wkp;
    __syncthreads();
    kp_run = keepoff[blockIdx.x];
    for (int w = 0; w < warp; ++w) kp_run += sh_kp[w];
  }
  u64 e2 = eq_run;
  u64 cnt = 0;
  for (int ch = 0; ch < CP_CHUNKS; ++ch) {
    size_t i = wb + (size_t)ch * 32 + lane;
    bool valid = i < n;
    double a = valid ? ia[i] : 0.0;
    bool ise = false;
    unsigned eb = __ballot_sync(0xffffffffu, valid && rule.mode == 1 && abs_bits(a) == rule.tau);
    bool k = valid && keep_of(rule, a, e2 + __popc(eb & lt), ise);
    e2 += __popc(eb);
    unsigned kb = __ballot_sync(0xffffffffu, k);
    if (WRITE) {
      if (k) {
        u64 pos = kp_run + __popc(kb & lt);
        ok[pos] = ik[i];
        oa[pos] = a;
      }
      kp_run += __popc(kb);
    } else {
      cnt += __popc(kb);
    }
  }
  if (!WRITE) {
    if (lane == 0) sh_kp[warp] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
      u64 t = 0;
      for (int w = 0; w < CP_THREADS / 32; ++w) t += sh_kp[w];
      keepc[blockIdx.x] = t;
    }
  }
}

template <int W>
static int compact_rule(Ctx& c, const typename KeyOf<W>::T* ik, const double* ia, size_t n, KeepRule rule,
                        typename KeyOf<W>::T* ok, double* oa, size_t* m) {
  typedef typename KeyOf<W>::T KT;
  if (n == 0) {
    *m = 0;
    return SFCI_OK;
  }
  size_t nt = (n + CP_TILE - 1) / CP_TILE;
  u64* eqo = (u64*)scratch_get(c, "cp_eq", (nt + 1) * sizeof(u64));
  u64* kpo = (u64*)scratch_get(c, "cp_kp", (nt + 1) * sizeof(u64));
  if (!eqo || !kpo) return SFCI_ERR_NOMEM;
  int st;
  if (rule.mode == 1) {
    SFCI_LAUNCH(c, k_cp_eqcount, (unsigned)nt, CP_THREADS, 0, ia, n, rule.tau, eqo);
    if ((st = scan_excl(c, eqo, eqo, nt))) return st;
    // eq_skip arrives as the number of ties to keep; turn it into ties to skip
    u64 tot_eq = 0;
    if ((st = read_words(c, eqo + nt, sizeof(u64), &tot_eq))) return st;
    rule.eq_skip = rule.eq_skip >= tot_eq ? 0 : tot_eq - rule.eq_skip;
  }
  SFCI_LAUNCH(c, (k_cp_pass<KT, false>), (unsigned)nt, CP_THREADS, 0, ik, ia, n, rule, (const u64*)eqo, kpo,
              (const u64*)nullptr, (KT*)nullptr, (double*)nullptr);
  if ((st = scan_excl(c, kpo, kpo, nt))) return st;
  SFCI_LAUNCH(c, (k_cp_pass<KT, true>), (unsigned)nt, CP_THREADS, 0, ik, ia, n, rule, (const u64*)eqo,
              (u64*)nullptr, (const u64*)kpo, ok, oa);
  u64 tot = 0;
  if ((st = read_words(c, kpo + nt, sizeof(u64), &tot))) return st;
  *m = (size_t)tot;
  return SFCI_OK;
}

// ---- selection and compaction in one launch ------------------------------------------
// The launches above read a histogram back after each of six digits and the
// counts after that: eight round trips to the host.  Here the digits, the counts
// and the compaction are one cooperative kernel with a grid barrier in place of
// each round trip: the top 400,000 of 1,400,000 entries take 64 us (270 before),
// of 17,000 38 us (200).  A digit whose bin is taken whole ends the search: the
// threshold is then the bin's lower edge and no tie has to be ranked.
struct SelArgs {
  const double* a;
  unsigned n, slice;
  int mode;            // 0: keep |a| above lb only; 1: the k largest first; 2: with every tie of the k-th
  u64 k;
  long long low_key;   // keep bits above this as well (-1: everything)
  uint32_t* hist;      // [6][4096], zero
  uint32_t* cnt;       // [2][G]
  unsigned *bar, *err;
  u64* m;              // entries kept
};
constexpr int SEL_COPIES = 4;

template <class KT>
__global__ void __launch_bounds__(CO_THREADS, 1) k_sel_coop(SelArgs s, const KT* __restrict__ ik, KT* __restrict__ ok,
                                                         double* __restrict__ oa) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint32_t* sh = reinterpret_cast<uint32_t*>(smem);  // [SEL_COPIES][4096] (mode 1)
  __shared__ uint32_t s_scan[CO_WARPS + 1];
  __shared__ uint32_t s_g[CO_WARPS], s_e[CO_WARPS];
  __shared__ unsigned s_bin, s_acc, s_cnt;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned G = gridDim.x, b = blockIdx.x, ws = s.slice / CO_WARPS;
  const unsigned w0 = min(s.n, b * s.slice + warp * ws), w1 = min(s.n, w0 + ws);
  unsigned target = 0;
  u64 lb = 0, tau = ~0ull, need_eq = 0;  // keep bits >= lb, and need_eq of those equal to tau
  if (s.mode) {
    const int shifts[6] = {51, 39, 27, 15, 3, 0}, widths[6] = {12, 12, 12, 12, 12, 3};
    u64 prefix = 0, need = s.k;
    bool whole = false;
    int r = 0;
    for (; r < 6 && !whole; ++r) {
      const unsigned nb = 1u << widths[r];
      const int shift = shifts[r], pshift = shift + widths[r];
      for (unsigned i = tid; i < SEL_COPIES * 4096; i += CO_THREADS) sh[i] = 0;
      __syncthreads();
      uint32_t* h = sh + (warp & (SEL_COPIES - 1)) * 4096;
      for (unsigned i = w0 + lane; i < w1; i += 32) {
        const u64 x = abs_bits(s.a[i]);
        if (r == 0 || (x >> pshift) == prefix) atomicAdd(&h[(unsigned)(x >> shift) & (nb - 1u)], 1u);
      }
      __syncthreads();
      uint32_t* gh = s.hist + r * 4096;
      for (unsigned i = tid; i < nb; i += CO_THREADS) {
        uint32_t v = 0;
#pragma unroll
        for (int q = 0; q < SEL_COPIES; ++q) v += sh[q * 4096 + i];
        if (v) atomicAdd(gh + i, v);
      }
      target += G;
      if (!coop_barrier(s.bar, target, s.err)) return;
      // the bin that holds the need-th largest: thread t looks at bins from the top
      uint32_t v[4], sum = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const unsigned i = tid * 4 + q;  // i-th bin from the top
        v[q] = i < nb ? __ldcg(gh + (nb - 1u - i)) : 0u;
        sum += v[q];
      }
      uint32_t acc = block_excl_scan<uint32_t, CO_THREADS>(sum, nullptr, s_scan);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (acc < need && need <= (u64)acc + v[q]) {
          s_bin = nb - 1u - (tid * 4 + q);
          s_acc = acc;
          s_cnt = v[q];
        }
        acc += v[q];
      }
      __syncthreads();
      need -= s_acc;
      prefix = (prefix << widths[r]) | s_bin;
      whole = s_cnt == need;
      if (whole) lb = prefix << shift;
      __syncthreads();
    }
    if (!whole) {
      tau = prefix;
      lb = tau + 1;
      need_eq = s.mode == 2 ? ~0ull : need;
    }
  }
  const u64 low = (u64)(s.low_key + 1);
  if (lb < low) lb = low;
  if (need_eq && tau < low) need_eq = 0;
  // counts: kept outright, ties
  uint32_t g = 0, e = 0;
  for (unsigned i0 = w0; i0 < w1; i0 += 32) {
    const u64 x = i0 + lane < w1 ? abs_bits(s.a[i0 + lane]) : 0ull;
    const bool in = i0 + lane < w1;
    g += __popc(__ballot_sync(0xffffffffu, in && x >= lb));
    e += __popc(__ballot_sync(0xffffffffu, in && need_eq && x == tau));
  }
  if (lane == 0) {
    s_g[warp] = g;
    s_e[warp] = e;
  }
  __syncthreads();
  u64 gr = 0, er = 0, gtot = 0, etot = 0;  // before this warp; over all
  {
    uint32_t cg = 0, ce = 0;
    for (int w = 0; w < CO_WARPS; ++w) {
      if (w == warp) {
        gr = cg;
        er = ce;
      }
      cg += s_g[w];
      ce += s_e[w];
    }
    gtot = cg;
    etot = ce;
    if (G > 1) {
      if (tid == 0) {
        __stcg(s.cnt + 2 * b, cg);
        __stcg(s.cnt + 2 * b + 1, ce);
      }
      target += G;
      if (!coop_barrier(s.bar, target, s.err)) return;
      u64 bg = 0, be = 0;
      gtot = etot = 0;
      for (unsigned q = lane; q < G; q += 32) {
        const u64 x = __ldcg(s.cnt + 2 * q), y = __ldcg(s.cnt + 2 * q + 1);
        if (q < b) {
          bg += x;
          be += y;
        }
        gtot += x;
        etot += y;
      }
      bg = warp_sum(bg);
      be = warp_sum(be);
      gtot = warp_sum(gtot);
      etot = warp_sum(etot);
      gr += bg;
      er += be;
    }
  }
  // of the ties, the last need_eq are kept
  const u64 skip = etot > need_eq ? etot - need_eq : 0ull;
  if (b == 0 && tid == 0) *s.m = gtot + (etot - skip);
  const unsigned lt = (1u << lane) - 1u;
  for (unsigned i0 = w0; i0 < w1; i0 += 32) {
    const unsigned i = i0 + lane;
    const bool in = i < w1;
    const double v = in ? s.a[i] : 0.0;
    const u64 x = abs_bits(v);
    const bool kg = in && x >= lb, ke = in && need_eq && x == tau;
    const unsigned mg = __ballot_sync(0xffffffffu, kg), me = __ballot_sync(0xffffffffu, ke);
    const u64 el = er + __popc(me & lt);
    if (kg || (ke && el >= skip)) {
      const u64 pos = gr + __popc(mg & lt) + (el > skip ? el - skip : 0ull);
      ok[pos] = ik[i];
      oa[pos] = v;
    }
    gr += __popc(mg);
    er += __popc(me);
  }
}

// mode 0: entries with bits above low_key; 1: the k largest first; 2: the same with
// every entry tied with the k-th (0 < k < n); *ran false: not done (coop_launch)
template <int W>
static int select_coop(Ctx& c, const typename KeyOf<W>::T* ik, const double* ia, size_t n, int mode, size_t k,
                       long long low_key, typename KeyOf<W>::T* ok, double* oa, size_t* m, bool* ran) {
  typedef typename KeyOf<W>::T KT;
  const size_t words = 6 * 4096 + 2 * (size_t)c.sm_count + 8;
  uint32_t* buf = (uint32_t*)scratch_get(c, "sel_coop", words * sizeof(uint32_t));
  unsigned* err = coop_error_word(c);
  if (!buf || !err) return SFCI_ERR_NOMEM;
  SelArgs s{};
  s.a = ia;
  s.n = (unsigned)n;
  s.slice = coop_slice(c, n);
  s.mode = mode;
  s.k = k;
  s.low_key = low_key;
  s.m = (u64*)buf;
  s.bar = buf + 2;
  s.hist = buf + 4;
  s.cnt = buf + 4 + 6 * 4096;
  s.err = err;
  const unsigned G = (unsigned)((n + s.slice - 1) / s.slice);
  SFCI_CUDA(cudaMemsetAsync(buf, 0, (mode ? 4 + 6 * 4096 : 4) * sizeof(uint32_t), c.stream));
  const size_t sm = mode ? SEL_COPIES * 4096 * sizeof(uint32_t) : 0;
  SFCI_CUDA(cudaFuncSetAttribute(k_sel_coop<KT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(SEL_COPIES * 4096 * sizeof(uint32_t))));
  void* args[] = {&s, &ik, &ok, &oa};
  int st = coop_launch(c, (const void*)k_sel_coop<KT>, G, args, sm, ran);
  if (st || !*ran) return st;
  u64 got = 0;
  if ((st = read_words(c, s.m, sizeof(u64), &got))) return st;
  *m = (size_t)got;
  return SFCI_OK;
}

template <int W>
int compact_top(Ctx& c, const typename KeyOf<W>::T* ik, const double* ia, size_t n, u64 tau, size_t need_eq,
                double tiny, typename KeyOf<W>::T* ok, double* oa, size_t* m) {
  KeepRule r{1, tau, (u64)need_eq, -1ll, cut_key(tiny)};
  return compact_rule<W>(c, ik, ia, n, r, ok, oa, m);
}

template <int W>
int compact_cut(Ctx& c, const typename KeyOf<W>::T* ik, const double* ia, size_t n, double cut,
                typename KeyOf<W>::T* ok, double* oa, size_t* m) {
  bool ran = false;
  int st;
  if (n && n <= SEL_MAX && ((st = select_coop<W>(c, ik, ia, n, 0, 0, cut_key(cut), ok, oa, m, &ran)) || ran)) return st;
  KeepRule r{0, 0, 0, cut_key(cut), -1ll};
  return compact_rule<W>(c, ik, ia, n, r, ok, oa, m);
}

template <int W>
int top_k_stable(Ctx& c, typename KeyOf<W>::T* ik, double* ia, size_t n, size_t k, double tiny,
                 typename KeyOf<W>::T* ok, double* oa, size_t* m) {
  typedef typename KeyOf<W>::T KT;
  bool ran = false;
  int st;
  if (n <= k) {
    if (tiny >= 0.0) {
      // filter only: keep |a| > tiny (all of them pass the selection)
      if (n && n <= SEL_MAX && ((st = select_coop<W>(c, ik, ia, n, 0, 0, cut_key(tiny), ok, oa, m, &ran)) || ran))
        return st;
      // tau = 0 keeping all n ties keeps everything before the tiny filter
      KeepRule r{1, 0ull, (u64)n, -1ll, cut_key(tiny)};
      return compact_rule<W>(c, ik, ia, n, r, ok, oa, m);
    }
    if (ok != ik) {
      SFCI_CUDA(cudaMemcpyAsync(ok, ik, n * sizeof(KT), cudaMemcpyDeviceToDevice, c.stream));
      SFCI_CUDA(cudaMemcpyAsync(oa, ia, n * sizeof(double), cudaMemcpyDeviceToDevice, c.stream));
    }
    *m = n;
    return SFCI_OK;
  }
  // a compaction may not run in place across tiles: it is staged through scratch
  KT* tk = ok;
  double* ta = oa;
  if (ok == ik) {
    tk = (KT*)scratch_get(c, "topk_k", n * sizeof(KT));
    ta = (double*)scratch_get(c, "topk_a", n * sizeof(double));
    if (!tk || !ta) return SFCI_ERR_NOMEM;
  }
  if (n <= SEL_MAX && k > 0 && (st = select_coop<W>(c, ik, ia, n, 1, k, cut_key(tiny), tk, ta, m, &ran))) return st;
  if (!ran) {
    u64 tau;
    size_t gt;
    if ((st = select_threshold(c, ia, n, k, &tau, &gt))) return st;
    if ((st = compact_top<W>(c, ik, ia, n, tau, k - gt, tiny, tk, ta, m))) return st;
  }
  if (ok == ik) {
    SFCI_CUDA(cudaMemcpyAsync(ok, tk, *m * sizeof(KT), cudaMemcpyDeviceToDevice, c.stream));
    SFCI_CUDA(cudaMemcpyAsync(oa, ta, *m * sizeof(double), cudaMemcpyDeviceToDevice, c.stream));
  }
  return SFCI_OK;
}

template <int W>
int select_sorted(Ctx& c, typename KeyOf<W>::T* keys, double* vals, size_t n, size_t k, size_t* m) {
  typedef typename KeyOf<W>::T KT;
  int st;
  if (n > k) {
    KT* tk = (KT*)scratch_get(c, "rs_keys", n * sizeof(KT));
    double* ta = (double*)scratch_get(c, "rs_vals", n * sizeof(double));
    if (!tk || !ta) return SFCI_ERR_NOMEM;
    if (k > 0 && n <= SEL_MAX) {
      // by magnitude first, so that only what is kept is sorted; ties of the k-th
      // all stay until the keys are in order
      size_t kept = 0;
      bool ran = false;
      if ((st = select_coop<W>(c, keys, vals, n, 2, k, -1ll, tk, ta, &kept, &ran))) return st;
      if (ran) {
        SFCI_CUDA(cudaMemcpyAsync(keys, tk, kept * sizeof(KT), cudaMemcpyDeviceToDevice, c.stream));
        SFCI_CUDA(cudaMemcpyAsync(vals, ta, kept * sizeof(double), cudaMemcpyDeviceToDevice, c.stream));
        n = kept;
      }
    }
  }
  if ((st = radix_sort_pairs<W>(c, keys, vals, n, c.N))) return st;
  if (n <= k) {
    *m = n;
    return SFCI_OK;
  }
  KT* tk = (KT*)scratch_get(c, "rs_keys", n * sizeof(KT));
  double* ta = (double*)scratch_get(c, "rs_vals", n * sizeof(double));
  if (!tk || !ta) return SFCI_ERR_NOMEM;
  if ((st = top_k_stable<W>(c, keys, vals, n, k, -1.0, tk, ta, m))) return st;
  SFCI_CUDA(cudaMemcpyAsync(keys, tk, *m * sizeof(KT), cudaMemcpyDeviceToDevice, c.stream));
  SFCI_CUDA(cudaMemcpyAsync(vals, ta, *m * sizeof(double), cudaMemcpyDeviceToDevice, c.stream));
  return SFCI_OK;
}

template int select_sorted<1>(Ctx&, u64*, double*, size_t, size_t, size_t*);
template int select_sorted<2>(Ctx&, K128*, double*, size_t, size_t, size_t*);
template int compact_top<1>(Ctx&, const u64*, const double*, size_t, u64, size_t, double, u64*, double*, size_t*);
template int compact_top<2>(Ctx&, const K128*, const double*, size_t, u64, size_t, double, K128*, double*,
                            size_t*);
template int compact_cut<1>(Ctx&, const u64*, const double*, size_t, double, u64*, double*, size_t*);
template int compact_cut<2>(Ctx&, const K128*, const double*, size_t, double, K128*, double*, size_t*);
template int top_k_stable<1>(Ctx&, u64*, double*, size_t, size_t, double, u64*, double*, size_t*);
template int top_k_stable<2>(Ctx&, K128*, double*, size_t, size_t, double, K128*, double*, size_t*);

// ============================================================================
// deterministic sum of squares
// ============================================================================

constexpr int RED_BLOCKS = 512;

__global__ void k_sumsq_part(const double* __restrict__ a, size_t n, double* __restrict__ part) {
  __shared__ double sh[32];
  double s = 0.0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    s += a[i] * a[i];
  double t = block_sum<256>(s, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// Partial sums added by one CTA.  A dependent FP64 addition takes about 150 cycles
// on this GPU, so a serial chain over 512 partials cost 40 us; the tree takes 3.  It adds in twice the working precision, so no rounding is
// added to the partial sums' but the last.
constexpr int SUM_THREADS = 256;

__global__ void __launch_bounds__(SUM_THREADS) k_sum_parts(const double* __restrict__ p, u64 n, double* __restrict__ out) {
  __shared__ double sh[2 * SUM_THREADS];
  double hi = 0.0, lo = 0.0;
  for (u64 i = threadIdx.x; i < n; i += SUM_THREADS) two_sum(hi, lo, __ldcg(p + i), 0.0);
  const double t = block_sum2<SUM_THREADS>(hi, lo, sh);
  if (threadIdx.x == 0) *out = t;
}

int sum_parts(Ctx& c, const double* p, u64 n, double* out) {
  SFCI_LAUNCH(c, k_sum_parts, 1, SUM_THREADS, 0, p, n, out);
  return SFCI_OK;
}

// The same with the squares, rounding errors and all, added in twice the working
// precision, for vectors short enough that the seven FP64 operations an entry (an
// SM issues two a cycle) stay below the launch and readback: 5 us at 400,000
// entries.  The sum is then that of the squares, rounded once but for rare cases.
constexpr size_t SUMSQ2_MAX = 1u << 20;
constexpr int SUMSQ2_BLOCKS = 152;

__global__ void __launch_bounds__(256) k_sumsq_part2(const double* __restrict__ a, size_t n, double* __restrict__ part) {
  __shared__ double sh[512];
  double hi = 0.0, lo = 0.0;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    two_prod_sum(hi, lo, a[i], a[i]);
  const double t = block_sum2<256>(hi, lo, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
}

int reduce_sum_sq(Ctx& c, const double* a, size_t n, double* out) {
  double* part = (double*)scratch_get(c, "red_part", (RED_BLOCKS + 1) * sizeof(double));
  if (!part) return SFCI_ERR_NOMEM;
  const int nb = n <= SUMSQ2_MAX ? SUMSQ2_BLOCKS : RED_BLOCKS;
  if (n <= SUMSQ2_MAX) {
    SFCI_LAUNCH(c, k_sumsq_part2, SUMSQ2_BLOCKS, 256, 0, a, n, part);
  } else {
    SFCI_LAUNCH(c, k_sumsq_part, RED_BLOCKS, 256, 0, a, n, part);
  }
  int st = sum_parts(c, part, nb, part + RED_BLOCKS);
  if (st) return st;
  return read_words(c, part + RED_BLOCKS, sizeof(double), out);
}

}  // namespace sfci
