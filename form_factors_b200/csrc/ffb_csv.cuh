// ffb_csv.cuh -- the form-factor matrix as the reference's CSV text
// (csv_export::export_csv, import_export/csv_export.cpp:26-46): row i holds
// the n entries of matrix row i, each written by `std::ostream << float`,
// separated by ';' and ended by '\n' (std::endl).  `ostream << float` prints
// the value widened to double with "%g" at precision 6: six significant
// digits of the exact binary value, rounded to nearest with ties to even,
// trailing zeros (and a bare decimal point) removed, exponent form when the
// decimal exponent is below -4 or at least 6.
//
// The conversion below is exact integer arithmetic on the float's mantissa
// and exponent: a 64-bit path for values in [2^-36, 2^24) (every form factor
// count / outgoing with outgoing < 2^31 lands there) and a multi-word path
// for the rest of the finite floats.
#pragma once

#include <stdint.h>

#ifndef __CUDACC__
#ifndef __host__
#define __host__
#endif
#ifndef __device__
#define __device__
#endif
#endif

namespace ffb {
namespace csv {

constexpr int kMaxEntry = 16;  // longest entry with its separator is 13 bytes ("-1.17549e-38;")

// Value m * 2^q (m > 0, m < 2^24) rounded to six significant digits:
// value ~= digits * 10^(exp10 - 5), digits in [100000, 999999].
struct Dec6 {
  uint32_t digits;
  int exp10;
};

__host__ __device__ inline Dec6 round6_from_7(uint64_t n7, bool rest, int exp10)
{
  uint32_t n6 = (uint32_t)(n7 / 10u);
  const uint32_t r = (uint32_t)(n7 % 10u);
  if (r > 5u || (r == 5u && (rest || (n6 & 1u))))
    ++n6;
  if (n6 == 1000000u) {
    n6 = 100000u;
    ++exp10;
  }
  return Dec6{n6, exp10};
}

// Number of decimal digits of v > 0.
__host__ __device__ inline int n_digits(uint64_t v)
{
  int n = 1;
  while (v >= 10u) {
    v /= 10u;
    ++n;
  }
  return n;
}

__host__ __device__ inline uint64_t pow10_u64(int k)
{
  uint64_t p = 1;
  for (int i = 0; i < k; ++i)
    p *= 10u;
  return p;
}

// Fast path: s = -q in [1, 59].  Integer part I = m >> s (< 2^24), fraction
// F / 2^s; fraction digits come from F * 10 (< 2^63).
__host__ __device__ inline Dec6 round6_small(uint32_t m, int s)
{
  const uint64_t mask = (s >= 64) ? ~0ull : ((1ull << s) - 1ull);
  const uint64_t I = s >= 32 ? 0ull : (uint64_t)(m >> s);
  uint64_t F = (uint64_t)m & mask;
  uint64_t n7 = 0;
  int got = 0, exp10;
  if (I > 0) {
    const int nI = n_digits(I);
    exp10 = nI - 1;
    if (nI >= 7) {
      const uint64_t p = pow10_u64(nI - 7);
      return round6_from_7(I / p, (I % p) != 0 || F != 0, exp10);
    }
    n7 = I;
    got = nI;
  } else {
    // leading zeros after the point
    exp10 = -1;
    for (;;) {
      F *= 10u;
      const uint64_t d = F >> s;
      F &= mask;
      if (d) {
        n7 = d;
        got = 1;
        break;
      }
      --exp10;
    }
  }
  while (got < 7) {
    F *= 10u;
    n7 = n7 * 10u + (F >> s);
    F &= mask;
    ++got;
  }
  return round6_from_7(n7, F != 0, exp10);
}

// General path: any finite positive value m * 2^q, with 32-bit limbs
// (little endian).  Integer part m << q has at most 128 bits; a fraction
// F / 2^s has s <= 149 bits and grows by 4 bits per digit.
constexpr int kLimbs = 6;

__host__ __device__ inline bool big_zero(const uint32_t* a)
{
  uint32_t o = 0;
  for (int i = 0; i < kLimbs; ++i)
    o |= a[i];
  return o == 0;
}

// a /= 10, returns the remainder
__host__ __device__ inline uint32_t big_div10(uint32_t* a)
{
  uint64_t r = 0;
  for (int i = kLimbs - 1; i >= 0; --i) {
    const uint64_t cur = (r << 32) | a[i];
    a[i] = (uint32_t)(cur / 10u);
    r = cur % 10u;
  }
  return (uint32_t)r;
}

// a *= 10, then returns and clears the bits at and above bit s
__host__ __device__ inline uint32_t big_mul10_take(uint32_t* a, int s)
{
  uint64_t c = 0;
  for (int i = 0; i < kLimbs; ++i) {
    const uint64_t cur = (uint64_t)a[i] * 10u + c;
    a[i] = (uint32_t)cur;
    c = cur >> 32;
  }
  // digit = a >> s (below 10), then a &= 2^s - 1.  a < 2^(s+4) after the
  // multiplication, so the digit's bits lie in limbs w and (for b > 28) w+1.
  const int w = s >> 5, b = s & 31;
  uint32_t d = a[w] >> b;
  if (b > 28 && w + 1 < kLimbs) {
    d |= a[w + 1] << (32 - b);
    a[w + 1] = 0;
  }
  a[w] &= b ? ((1u << b) - 1u) : 0u;
  return d;
}

__host__ __device__ inline Dec6 round6_general(uint32_t m, int q)
{
  uint32_t a[kLimbs];
  for (int i = 0; i < kLimbs; ++i)
    a[i] = 0;
  if (q >= 0) {
    // integer: m << q (q <= 104), decimal digits by repeated division
    const int w = q >> 5, b = q & 31;
    a[w] = m << b;
    if (b && w + 1 < kLimbs)
      a[w + 1] = m >> (32 - b);
    uint8_t dig[40];
    int n = 0;
    while (!big_zero(a))
      dig[n++] = (uint8_t)big_div10(a);
    // dig[n-1] is the leading digit
    uint64_t n7 = 0;
    const int take = n < 7 ? n : 7;
    for (int i = 0; i < take; ++i)
      n7 = n7 * 10u + dig[n - 1 - i];
    for (int i = take; i < 7; ++i)
      n7 *= 10u;
    bool rest = false;
    for (int i = 0; i < n - 7; ++i)
      rest |= dig[i] != 0;
    return round6_from_7(n7, rest, n - 1);
  }
  // pure fraction (s >= 60, so m >> s == 0): digits of m / 2^s
  const int s = -q;
  a[0] = m;
  int exp10 = -1;
  uint32_t d;
  for (;;) {
    d = big_mul10_take(a, s);
    if (d)
      break;
    --exp10;
  }
  uint64_t n7 = d;
  for (int i = 1; i < 7; ++i)
    n7 = n7 * 10u + big_mul10_take(a, s);
  return round6_from_7(n7, !big_zero(a), exp10);
}


template <class Out>
__host__ __device__ inline void put_text(Out& out, const char* t)
{
  for (int i = 0; t[i]; ++i)
    out.put(t[i]);
}

// Appends "%g" of f (precision 6) to out: at most 12 characters.
template <class Out>
__host__ __device__ inline void format_g6_to(float f, Out& out)
{
  uint32_t bits;
#ifdef __CUDA_ARCH__
  bits = __float_as_uint(f);
#else
  __builtin_memcpy(&bits, &f, 4);
#endif
  const bool neg = bits >> 31;
  const uint32_t ex = (bits >> 23) & 0xFFu, fr = bits & 0x7FFFFFu;
  if (ex == 0xFFu) {
    put_text(out, fr ? (neg ? "-nan" : "nan") : (neg ? "-inf" : "inf"));
    return;
  }
  if (neg)
    out.put('-');
  if (ex == 0 && fr == 0) {
    out.put('0');
    return;
  }
  const uint32_t m = ex ? (fr | 0x800000u) : fr;
  const int q = ex ? (int)ex - 150 : -149;
  const Dec6 d = (q < 0 && q >= -59) ? round6_small(m, -q) : round6_general(m, q);
  // digits of d.digits, most significant first, without trailing zeros
  uint32_t v = d.digits;
  int last = 5;
  while (last > 0 && v % 10u == 0u) {
    v /= 10u;
    --last;
  }
  // v now holds digits 0..last; divisor picks them from the top
  uint32_t div = 1;
  for (int i = 0; i < last; ++i)
    div *= 10u;
  const int X = d.exp10;
  auto next_digit = [&]() {
    const uint32_t dg = v / div;
    v -= dg * div;
    div /= 10u;
    return (char)('0' + dg);
  };
  if (X < -4 || X >= 6) {
    out.put(next_digit());
    if (last > 0) {
      out.put('.');
      for (int i = 1; i <= last; ++i)
        out.put(next_digit());
    }
    out.put('e');
    out.put(X < 0 ? '-' : '+');
    const int ax = X < 0 ? -X : X;
    if (ax >= 100)
      out.put((char)('0' + ax / 100));
    out.put((char)('0' + (ax / 10) % 10));
    out.put((char)('0' + ax % 10));
    return;
  }
  if (X >= 0) {
    // integer digits 0..X (digits past `last` are zeros)
    for (int i = 0; i <= X; ++i)
      out.put(i <= last ? next_digit() : '0');
    if (last > X) {
      out.put('.');
      for (int i = X + 1; i <= last; ++i)
        out.put(next_digit());
    }
    return;
  }
  out.put('0');
  out.put('.');
  for (int i = 0; i < -X - 1; ++i)
    out.put('0');
  for (int i = 0; i <= last; ++i)
    out.put(next_digit());
}

// An entry's text in registers: its first 16 bytes, little endian, and the
// length.  The longest entry has 12 characters.
struct Text {
  uint64_t lo, hi;
  int len;

  __host__ __device__ void put(char c)
  {
    if (len < 8)
      lo |= (uint64_t)(uint8_t)c << (8 * len);
    else
      hi |= (uint64_t)(uint8_t)c << (8 * (len - 8));
    ++len;
  }
};

__host__ __device__ inline int bit_width64(uint64_t v)
{
#ifdef __CUDA_ARCH__
  return 64 - __clzll((long long)v);
#else
  return v ? 64 - __builtin_clzll(v) : 0;
#endif
}

// The general formatter's text (a call of its own on the device: it is rare,
// and its digit arrays would take the other entries' registers).
#ifdef __CUDACC__
__noinline__
#endif
__host__ __device__ inline Text text_g6_general(float f)
{
  Text t{0, 0, 0};
  format_g6_to(f, t);
  return t;
}

// "%g" of f.  Values in [10^-4, 10^6) -- every form factor of a row of up to
// 10 000 rays -- take a few dozen integer operations: with X the decimal
// exponent of the value's binade, value * 10^(6 - X) = (m * 5^(6 - X)) >>
// (s - (6 - X)) is one 64-bit product (m < 2^24, 5^10 < 2^24), whose integer
// part holds seven or eight digits and whose low bits say whether anything
// follows them.  The six rounded digits are laid out as bytes and shifted into
// place.  The rest goes through format_g6_to.
__host__ __device__ inline Text text_g6(float f)
{
  uint32_t bits;
#ifdef __CUDA_ARCH__
  bits = __float_as_uint(f);
#else
  __builtin_memcpy(&bits, &f, 4);
#endif
  const int e2 = (int)((bits >> 23) & 0xFFu) - 127;  // the value's binade [2^e2, 2^(e2 + 1))
  if (e2 < -13 || e2 > 18)
    return text_g6_general(f);
  const uint32_t m = (bits & 0x7FFFFFu) | 0x800000u;
  int X = (e2 * 315653) >> 20;  // floor(e2 * log10(2)): 10^X <= 2^e2
  const int k = 6 - X;          // 1 .. 10
  const uint64_t p5 = (uint64_t)((k & 1 ? 5u : 1u) * (k & 2 ? 25u : 1u) * (k & 4 ? 625u : 1u)) * (k & 8 ? 390625u : 1u);
  const uint64_t prod = (uint64_t)m * p5;
  const int sh = 23 - e2 - k;   // at least 3
  uint32_t n = (uint32_t)(prod >> sh);  // the first 7 digits, or 8
  bool rest = (prod & ((1ull << sh) - 1ull)) != 0;
  if (n >= 10000000u) {
    const uint32_t q = n / 10u;
    rest |= n != q * 10u;
    n = q;
    ++X;
  }
  uint32_t v = n / 10u;
  const uint32_t r = n - v * 10u;
  v += r > 5u || (r == 5u && (rest || (v & 1u)));
  if (v == 1000000u) {
    v = 100000u;
    ++X;
  }
  if (X < -4 || X > 5)
    return text_g6_general(f);
  Text t{0, 0, 0};
  // digits, most significant in the lowest byte
  const uint32_t h = v / 1000u, l = v - h * 1000u;
  const uint32_t h1 = h / 100u, h2 = h / 10u, l1 = l / 100u, l2 = l / 10u;
  const uint64_t digits = (uint64_t)(h1 | (h2 - h1 * 10u) << 8 | (h - h2 * 10u) << 16 | l1 << 24) |
                          (uint64_t)((l2 - l1 * 10u) | (l - l2 * 10u) << 8) << 32;
  const int nd = (bit_width64(digits) + 7) >> 3;  // without trailing zeros
  const uint64_t text = digits + 0x303030303030ull;
  const uint64_t kept = text & ((1ull << (8 * nd)) - 1ull);
  if (X >= 0) {
    const int at = 8 * (X + 1);  // the integer part, zeros included
    t.len = X + 1;
    t.lo = text & ((1ull << at) - 1ull);
    if (nd > X + 1) {
      t.lo |= (uint64_t)'.' << at | (kept >> at) << (at + 8);
      t.len = nd + 1;
    }
  } else {
    const int at = 8 * (1 - X);  // "0." and the zeros after the point
    t.lo = (0x3030302E30ull & ((1ull << at) - 1ull)) | kept << at;
    t.hi = kept >> (64 - at);
    t.len = nd + 1 - X;
  }
  if (bits >> 31) {
    t.hi = t.hi << 8 | t.lo >> 56;
    t.lo = t.lo << 8 | (uint64_t)'-';
    ++t.len;
  }
  return t;
}

// Writes "%g" of f to out (no terminator); returns the length.
__host__ __device__ inline int format_g6(float f, char* out)
{
  const Text t = text_g6(f);
  for (int i = 0; i < t.len; ++i)
    out[i] = (char)((i < 8 ? t.lo >> (8 * i) : t.hi >> (8 * (i - 8))) & 0xFFu);
  return t.len;
}

__host__ __device__ inline int format_g6_len(float f)
{
  return text_g6(f).len;
}

#ifdef __CUDACC__
// ---------------------------------------------------------------------------
// Kernels.  The matrix (row-major entries) is cut into tiles of kTile
// entries, one block each.  A device buffer gets its text from k_csv_fused
// (one pass, below); lengths, host buffers and files use:
//  1. k_csv_len: the text length of every tile.
//  2. k_csv_scan: exclusive prefix sums of the tile lengths (64-bit) and the
//     total.
//  3. k_csv_write: each block lays its tile's text out in shared memory and
//     copies it to its global offset with 16-byte stores (the shared buffer
//     starts at the destination's offset modulo 16, so both sides line up;
//     only the ragged head and tail go byte by byte).
// In both passes an entry that is +0 costs a load and a compare ("0" plus
// separator); the other entries go to a per-block queue and are formatted by
// all threads together, so that a sparse matrix does not leave warps running
// the formatter with one lane.  Per-entry offsets come from a block scan of
// the entry lengths (16-bit: a tile's text is below 64 KB).
// ---------------------------------------------------------------------------
constexpr int kThreads = 256;
constexpr int kPerThread = 16;
constexpr int kTile = kThreads * kPerThread;            // entries per block
constexpr int kTileBytes = kTile * (kMaxEntry - 3) + 16;  // 13 bytes per entry at most, + alignment shift
constexpr size_t kIndexSmem = 2 * sizeof(uint16_t) * kTile;  // offsets + queue of k_csv_write
// Dynamic shared memory of k_csv_write for tiles of at most max_tile bytes.
__host__ __device__ inline size_t write_smem(unsigned long long max_tile)
{
  return (size_t)((max_tile + 16u + 15u) & ~15ull) + kIndexSmem;
}

// The n x n matrix: floats, or counts normalised by their row's outgoing
// rays as ffb_normalise does ((float)count * (1.f / (float)outgoing[row]),
// cpu_system.cpp:193-195).
struct Source {
  const float* __restrict__ ff;
  const uint32_t* __restrict__ counts;
  const int32_t* __restrict__ outgoing;
  int n;
  long long n_entries;
};

__device__ __forceinline__ float row_ratio(const Source& s, int row)
{
  return s.ff ? 1.f : 1.f / (float)__ldg(s.outgoing + row);
}

__device__ __forceinline__ float entry_value(const Source& s, long long e, float ratio)
{
  return s.ff ? __ldg(s.ff + e) : (float)__ldg(s.counts + e) * ratio;
}

// A thread's entries o = k * kThreads + tid of one tile, held in registers
// for both walks of a kernel: the 16 loads are issued together.
struct TileRegs {
  float v[kPerThread];
  int col0;  // column of the first entry
};

__device__ __forceinline__ void load_tile(const Source& s, long long tile, TileRegs& r)
{
  const long long e0 = tile * kTile + threadIdx.x;
  uint32_t raw[kPerThread];
#pragma unroll
  for (int k = 0; k < kPerThread; ++k) {
    const long long e = e0 + (long long)k * kThreads;
    raw[k] = 0u;
    if (e < s.n_entries)
      raw[k] = s.ff ? __float_as_uint(__ldg(s.ff + e)) : __ldg(s.counts + e);
  }
  int row = (int)(e0 / s.n), col = (int)(e0 - (long long)row * s.n);
  r.col0 = col;
  float ratio = (!s.ff && row < s.n) ? row_ratio(s, row) : 1.f;
#pragma unroll
  for (int k = 0; k < kPerThread; ++k) {
    r.v[k] = s.ff ? __uint_as_float(raw[k]) : (float)raw[k] * ratio;
    col += kThreads;
    if (col >= s.n) {
      while (col >= s.n) {
        col -= s.n;
        ++row;
      }
      if (!s.ff && row < s.n)
        ratio = row_ratio(s, row);
    }
  }
}

// fn(o, valid, value, col) for the thread's entries; it runs on every lane
// of the warp each step (callers use warp votes); entries past the matrix end
// come with valid = false.
template <class Fn>
__device__ __forceinline__ void walk_tile(const Source& s, long long tile, const TileRegs& r, Fn fn)
{
  int col = r.col0;
#pragma unroll
  for (int k = 0; k < kPerThread; ++k) {
    const int o = k * kThreads + (int)threadIdx.x;
    fn(o, tile * kTile + o < s.n_entries, r.v[k], col);
    col += kThreads;
    while (col >= s.n)
      col -= s.n;
  }
}

// Value and column of entry o of the tile (queue work, one division).
__device__ __forceinline__ float tile_value(const Source& s, long long tile, int o, int* col)
{
  const long long e = tile * kTile + o;
  const int row = (int)(e / s.n);
  *col = (int)(e - (long long)row * s.n);
  return entry_value(s, e, row_ratio(s, row));
}

__device__ __forceinline__ void enqueue(uint16_t* queue, uint32_t* qn, bool take, int o)
{
  const unsigned mask = __ballot_sync(0xFFFFFFFFu, take);
  if (!mask)
    return;
  const int lane = threadIdx.x & 31;
  uint32_t base = 0;
  if (lane == __ffs(mask) - 1)
    base = atomicAdd(qn, (uint32_t)__popc(mask));
  base = __shfl_sync(0xFFFFFFFFu, base, __ffs(mask) - 1);
  if (take)
    queue[base + __popc(mask & ((1u << lane) - 1u))] = (uint16_t)o;
}

// Stores a text's bytes at any address.
__device__ __forceinline__ void put_bytes(unsigned char* to, const Text& t)
{
#pragma unroll
  for (int i = 0; i < kMaxEntry - 3; ++i)
    if (i < t.len)
      to[i] = (unsigned char)(i < 8 ? t.lo >> (8 * i) : t.hi >> (8 * (i - 8)));
}

__global__ void __launch_bounds__(kThreads, 4) k_csv_len(Source s, unsigned long long* __restrict__ tile_len)
{
  __shared__ uint16_t queue[kTile];
  __shared__ uint32_t qn;
  __shared__ uint32_t warp_sum[kThreads / 32];
  if (threadIdx.x == 0)
    qn = 0;
  __syncthreads();
  uint32_t sum = 0;
  TileRegs r;
  load_tile(s, blockIdx.x, r);
  walk_tile(s, blockIdx.x, r, [&](int o, bool valid, float v, int) {
    const bool zero = __float_as_uint(v) == 0u;
    sum += valid && zero ? 2u : 0u;
    enqueue(queue, &qn, valid && !zero, o);
  });
  __syncthreads();
  const uint32_t n_q = qn;
  for (uint32_t q = threadIdx.x; q < n_q; q += kThreads) {
    int col;
    sum += (uint32_t)format_g6_len(tile_value(s, blockIdx.x, queue[q], &col)) + 1u;
  }
  for (int off = 16; off > 0; off >>= 1)
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, off);
  if ((threadIdx.x & 31) == 0)
    warp_sum[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int w = 0; w < kThreads / 32; ++w)
      t += warp_sum[w];
    tile_len[blockIdx.x] = t;
  }
}

// Exclusive scan of n tile lengths (one block; each thread a contiguous run)
// into out[0..n), the total into out[n] and the longest tile into out[n + 1].
constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads) k_csv_scan(const unsigned long long* __restrict__ in, int n,
                                                           unsigned long long* __restrict__ out)
{
  __shared__ unsigned long long warp_sum[kScanThreads / 32];
  __shared__ unsigned long long warp_max[kScanThreads / 32];
  const int per = (n + kScanThreads - 1) / kScanThreads;
  const int b = (int)threadIdx.x * per, e = min(n, b + per);
  unsigned long long s = 0, mx = 0;
  for (int i = b; i < e; ++i) {
    const unsigned long long x = in[i];
    s += x;
    mx = x > mx ? x : mx;
  }
  for (int off = 16; off > 0; off >>= 1) {
    const unsigned long long y = __shfl_xor_sync(0xFFFFFFFFu, mx, off);
    mx = y > mx ? y : mx;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long incl = s;
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, incl, off);
    if (lane >= off)
      incl += y;
  }
  if (lane == 31)
    warp_sum[warp] = incl;
  if (lane == 0)
    warp_max[warp] = mx;
  __syncthreads();
  unsigned long long before = 0;
  for (int w = 0; w < warp; ++w)
    before += warp_sum[w];
  unsigned long long run = before + incl - s;
  for (int i = b; i < e; ++i) {
    out[i] = run;
    run += in[i];
  }
  if (threadIdx.x == kScanThreads - 1) {
    out[n] = run;
    unsigned long long m = 0;
    for (int w = 0; w < kScanThreads / 32; ++w)
      m = warp_max[w] > m ? warp_max[w] : m;
    out[n + 1] = m;
  }
}

// Writes tiles tile0 + blockIdx.x; their text goes to text + (tile_off[t] -
// base).  The dynamic shared memory is write_smem(longest tile): the text
// region first (text_region bytes), then offsets and queue.
__global__ void __launch_bounds__(kThreads, 4) k_csv_write(Source s, const unsigned long long* __restrict__ tile_off,
                                                        long long tile0, unsigned long long base, uint32_t text_region,
                                                        char* __restrict__ text)
{
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned char* sbuf = smem;                                         // text_region bytes
  uint16_t* off = reinterpret_cast<uint16_t*>(smem + text_region);    // per entry: length, then offset
  uint16_t* queue = off + kTile;
  __shared__ uint32_t qn;
  __shared__ uint32_t warp_sum[kThreads / 32];
  const long long tile = tile0 + blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0)
    qn = 0;
  for (int o = threadIdx.x; o < kTile; o += kThreads)
    off[o] = 0;  // entries past the matrix end
  __syncthreads();
  // 1. lengths: zeros directly, the others through the queue
  TileRegs r;
  load_tile(s, tile, r);
  walk_tile(s, tile, r, [&](int o, bool valid, float v, int) {
    const bool zero = __float_as_uint(v) == 0u;
    if (valid && zero)
      off[o] = 2;
    enqueue(queue, &qn, valid && !zero, o);
  });
  __syncthreads();
  const uint32_t n_q = qn;
  for (uint32_t q = threadIdx.x; q < n_q; q += kThreads) {
    const int o = queue[q];
    int col;
    off[o] = (uint16_t)(format_g6_len(tile_value(s, tile, o, &col)) + 1);
  }
  __syncthreads();
  // 2. offsets: thread t scans entries [16t, 16t + 16)
  char* dst = text + (tile_off[tile] - base);
  const uint32_t shift = (uint32_t)((uintptr_t)dst & 15u);
  uint32_t mine = 0;
  for (int i = 0; i < kPerThread; ++i)
    mine += off[threadIdx.x * kPerThread + i];
  uint32_t incl = mine;
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
    if (lane >= d)
      incl += y;
  }
  if (lane == 31)
    warp_sum[warp] = incl;
  __syncthreads();
  uint32_t before = 0, total = 0;
  for (int w = 0; w < kThreads / 32; ++w) {
    const uint32_t u = warp_sum[w];
    before += w < warp ? u : 0u;
    total += u;
  }
  uint32_t run = shift + before + incl - mine;
  for (int i = 0; i < kPerThread; ++i) {
    const int o = threadIdx.x * kPerThread + i;
    const uint32_t len = off[o];
    off[o] = (uint16_t)run;  // below 64 KB
    run += len;
  }
  __syncthreads();
  // 3. text: zeros, then the queued entries
  walk_tile(s, tile, r, [&](int o, bool valid, float v, int col) {
    if (valid && __float_as_uint(v) == 0u) {
      sbuf[off[o]] = '0';
      sbuf[off[o] + 1] = col == s.n - 1 ? '\n' : ';';
    }
  });
  for (uint32_t q = threadIdx.x; q < n_q; q += kThreads) {
    const int o = queue[q];
    int col;
    const float v = tile_value(s, tile, o, &col);
    Text w = text_g6(v);
    w.put(col == s.n - 1 ? '\n' : ';');
    put_bytes(sbuf + off[o], w);
  }
  __syncthreads();
  // 4. copy [shift, shift + total) of sbuf to dst
  const uint32_t L = total;
  const uint32_t head = min(L, (16u - shift) & 15u);
  const uint32_t body = (L - head) >> 4;
  for (uint32_t i = threadIdx.x; i < head; i += kThreads)
    dst[i] = (char)sbuf[shift + i];
  const uint4* sv = reinterpret_cast<const uint4*>(sbuf + shift + head);
  uint4* dv = reinterpret_cast<uint4*>(dst + head);
  for (uint32_t i = threadIdx.x; i < body; i += kThreads)
    dv[i] = sv[i];
  for (uint32_t i = head + 16u * body + threadIdx.x; i < L; i += kThreads)
    dst[i] = (char)sbuf[shift + i];
}

// ---------------------------------------------------------------------------
// Single pass into a device buffer (decoupled look-back).  Each block takes
// the next tile by ticket, so every tile it waits for already runs and waits
// only for earlier tiles.  A warp works through its 512 (or 128) consecutive entries
// without block barriers: lane l holds entries 32k + l, ballots give the
// nonzero ones, which go to the warp's queue in entry order and are formatted
// by all lanes together; a scan of their lengths gives, for an entry with q
// nonzeros before it, the offset 2 * entry + extra[q] (a +0 entry is "0" and
// the separator).  Neighbouring lanes then stage neighbouring bytes.  The tile
// publishes its length, sums the lengths and prefixes the preceding tiles
// published (bounded polls), publishes its inclusive prefix and stores its
// text with 16-byte writes.  A tile whose text would pass the end of the
// buffer writes nothing and sets kFusedOverflow; the last tile writes the text
// length.
//
// What bounds it: instruction issue (about 80 warp instructions per 32
// entries); 487 M entries of which 4.5 % are nonzero, 1.06 GB of text: 3.34 ms
// with a whole tile per barrier phase, each nonzero formatted twice by digit
// loops and zeros staged by byte stores at a 32-byte stride (eight lanes on a
// bank); 1.73 ms as it is now.  A warp stages 2 KB of text at a time, which
// holds its 512 entries unless over a fifth of them are nonzero: shared memory
// for the longest possible text would leave three blocks per SM.  A matrix
// that would not fill one wave of blocks so takes 128 entries per warp
// (csv_run).
// ---------------------------------------------------------------------------
constexpr unsigned long long kTileAgg = 1ull << 62;     // status: the tile's own length
constexpr unsigned long long kTilePrefix = 2ull << 62;  // status: the inclusive prefix
constexpr unsigned long long kTileValue = (1ull << 62) - 1;
constexpr unsigned kLookbackPolls = 1u << 22;           // polls of one status word before giving up
enum : unsigned { kFusedTimeout = 1u, kFusedOverflow = 2u };
constexpr int kFusedThreads = 256;
constexpr int kFusedWarps = kFusedThreads / 32;

// kEntries: entries per warp, 512 or 128 (csv_run).
template <int kEntries>
struct FusedShape {
  static constexpr int kTile = kEntries * kFusedWarps;  // entries per block
  // staged text per warp, a multiple of 16
  static constexpr int kWindow = kEntries * (kMaxEntry - 3) < 2048 ? kEntries * (kMaxEntry - 3) : 2048;
  // A warp's shared memory.
  struct WarpText {
    __align__(16) unsigned char text[kWindow + 16];  // one word is read past the window
    uint16_t entry[kEntries];                        // nonzero entries, in order
    uint16_t extra[kEntries + 1];                    // sum of (length - 2) of those before
    uint32_t nonzero[kEntries / 32];                 // their lanes in each chunk of 32
  };
  static constexpr size_t kSmem = sizeof(WarpText) * kFusedWarps;
};

struct FusedSink {
  char* text;
  unsigned long long cap;
  unsigned long long* status;  // one word per tile, zero before the launch
  unsigned int* ticket;        // zero before the launch
  unsigned int* err;           // kFused* bits, zero before the launch
  unsigned long long* total;   // the text length, written by the last tile
  long long n_tiles;
};

__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p)
{
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v)
{
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Exclusive prefix of `tile` from the status words of the tiles before it;
// run by one full warp after the tile's own length was published.
__device__ __forceinline__ unsigned long long look_back(const FusedSink& out, long long tile, int lane)
{
  unsigned long long excl = 0;
  for (long long j = tile - 1;; j -= 32) {
    const long long idx = j - lane;
    unsigned long long w = kTilePrefix;  // before the first tile: prefix 0
    if (idx >= 0) {
      unsigned polls = 0;
      do {
        w = ld_relaxed(out.status + idx);
      } while ((w >> 62) == 0 && ++polls < kLookbackPolls);
    }
    if (__any_sync(0xFFFFFFFFu, (w >> 62) == 0)) {  // a tile never published: give up
      if (lane == 0)
        atomicOr(out.err, kFusedTimeout);
      return excl;
    }
    // lane 0 is the nearest tile; stop at the nearest one with a prefix
    const unsigned pm = __ballot_sync(0xFFFFFFFFu, (w >> 62) == 2);
    unsigned long long v = w & kTileValue;
    if (pm && lane > __ffs(pm) - 1)
      v = 0;
    for (int d = 16; d > 0; d >>= 1)
      v += __shfl_xor_sync(0xFFFFFFFFu, v, d);
    excl += v;
    if (pm)
      return excl;
  }
}

// Entries [e0, e0 + kEntries) of one warp: where they lie in the matrix.
template <int kEntries>
struct WarpRows {
  uint32_t e0;
  uint32_t row, col;  // of entry e0
  uint32_t n;
  int valid;          // entries before the matrix end, at most kEntries

  // kEntries entries of one or two rows, every count of zero a +0 entry
  bool simple;
  int row_end;        // simple: the last entry of the first row (past the last if it goes on)
  float ratio0, ratio1;  // simple: of the two rows (counts)

  // Separator after entry o, and entry o as text.
  template <bool kSimple>
  __device__ __forceinline__ char separator(int o) const
  {
    if (kSimple)
      return o == row_end ? '\n' : ';';
    uint32_t r, c;
    locate(o, &r, &c);
    return c == n - 1 ? '\n' : ';';
  }
  template <bool kSimple>
  __device__ __forceinline__ Text text(const Source& s, const uint32_t* words, int o) const
  {
    float v;
    char sep;
    if (kSimple) {
      const uint32_t raw = __ldg(words + o);
      v = s.ff ? __uint_as_float(raw) : (float)raw * (o > row_end ? ratio1 : ratio0);
      sep = separator<true>(o);
    } else {
      uint32_t r, c;
      locate(o, &r, &c);
      v = entry_value(s, (long long)e0 + o, row_ratio(s, (int)r));
      sep = c == n - 1 ? '\n' : ';';
    }
    Text t = text_g6(v);
    t.put(sep);
    return t;
  }

  // row and column of entry o
  __device__ __forceinline__ void locate(int o, uint32_t* r, uint32_t* c) const
  {
    uint32_t k = col + (uint32_t)o;
    *r = row;
    if (k >= n) {
      const uint32_t q = n > (uint32_t)kEntries ? 1u : k / n;
      *r += q;
      k -= q * n;
    }
    *c = k;
  }
};

// Stages the warp's text bytes [w0, w0 + kWindow) at W.text; `first` is the
// text of the lane's first queue entry.  With kAll the whole text fits the
// window.
template <int kEntries, bool kAll, bool kSimple>
__device__ __forceinline__ void stage_text(const Source& s, const WarpRows<kEntries>& at, const uint32_t* words,
                                           typename FusedShape<kEntries>::WarpText& W, int n_q, const Text& first,
                                           int w0, int lane)
{
  constexpr int kChunks = kEntries / 32, kWindow = FusedShape<kEntries>::kWindow;
  const uint32_t below = (1u << lane) - 1u;
  const uint16_t* extra = W.extra;  // of the nonzeros in the chunks before
#pragma unroll 8
  for (int k = 0; k < kChunks; ++k) {
    const uint32_t m = W.nonzero[k];
    const int o = 32 * k + lane;
    if (!((m >> lane) & 1u) && (kSimple || o < at.valid)) {
      const int p = 2 * o + extra[__popc(m & below)] - w0;
      const unsigned char sep = (unsigned char)at.template separator<kSimple>(o);
      if (kAll || (unsigned)p < (unsigned)kWindow)
        W.text[p] = '0';
      if (kAll || (unsigned)(p + 1) < (unsigned)kWindow)
        W.text[p + 1] = sep;
    }
    extra += __popc(m);
  }
  for (int q = lane; q < n_q; q += 32) {
    const int o = W.entry[q];
    const int p = 2 * o + W.extra[q] - w0;
    if (!kAll && (p >= kWindow || p + kMaxEntry < 0))
      continue;
    Text t = first;
    if (q >= 32)
      t = at.template text<kSimple>(s, words, o);
    if (kAll) {
      put_bytes(W.text + p, t);
    } else {
#pragma unroll 1
      for (int i = 0; i < t.len; ++i)
        if ((unsigned)(p + i) < (unsigned)kWindow)
          W.text[p + i] = (unsigned char)(i < 8 ? t.lo >> (8 * i) : t.hi >> (8 * (i - 8)));
    }
  }
}

// The warp's entries: the nonzero ones queued and formatted (`first` is the
// text of the lane's first), their lengths scanned.  Returns their number;
// *len gets the length of the warp's text.
template <int kEntries, bool kSimple>
__device__ __forceinline__ int queue_entries(const Source& s, const WarpRows<kEntries>& at, const uint32_t* words,
                                             const uint32_t (&raw)[kEntries / 32], bool plain,
                                             typename FusedShape<kEntries>::WarpText& W, Text& first, int* len,
                                             int lane)
{
  constexpr int kChunks = kEntries / 32;
  const uint32_t below = (1u << lane) - 1u;
  int n_q = 0;
#pragma unroll
  for (int k = 0; k < kChunks; ++k) {
    const int o = 32 * k + lane;
    bool take = raw[k] != 0u;
    if (!kSimple && !plain && o < at.valid) {
      uint32_t r, c;
      at.locate(o, &r, &c);
      take = __float_as_uint((float)raw[k] * row_ratio(s, (int)r)) != 0u;
    }
    const unsigned m = __ballot_sync(0xFFFFFFFFu, take);
    if (take)
      W.entry[n_q + __popc(m & below)] = (uint16_t)o;
    n_q += __popc(m);
    if (lane == 0)
      W.nonzero[k] = m;
  }
  __syncwarp();
  int extra = 0;
  for (int q0 = 0; q0 < n_q; q0 += 32) {
    const int q = q0 + lane;
    int mine = 0;
    if (q < n_q) {
      const Text t = at.template text<kSimple>(s, words, W.entry[q]);
      mine = t.len - 2;
      if (q0 == 0)
        first = t;
    }
    int incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
      if (lane >= d)
        incl += y;
    }
    if (q < n_q)
      W.extra[q] = (uint16_t)(extra + incl - mine);
    extra += __shfl_sync(0xFFFFFFFFu, incl, 31);
  }
  if (lane == 0)
    W.extra[n_q] = (uint16_t)extra;
  *len = 2 * at.valid + extra;
  return n_q;
}

// Copies `len` staged bytes to dst: bytes up to the first 16-byte boundary,
// then 16-byte stores assembled from 32-bit shared words (funnel shifts by the
// misalignment), then the tail.
__device__ __forceinline__ void copy_text(char* dst, const unsigned char* text, uint32_t len, int lane)
{
  const uint32_t head = min(len, (uint32_t)((16u - ((uintptr_t)dst & 15u)) & 15u));
  const uint32_t body = (len - head) >> 4;
  if (lane < (int)head)
    dst[lane] = (char)text[lane];
  const uint32_t r8 = 8u * (head & 3u);
  const uint32_t* sw = reinterpret_cast<const uint32_t*>(text) + (head >> 2);
  uint4* dv = reinterpret_cast<uint4*>(dst + head);
  for (uint32_t i = lane; i < body; i += 32) {
    const uint32_t* w = sw + 4 * i;
    const uint32_t a0 = w[0], a1 = w[1], a2 = w[2], a3 = w[3], a4 = w[4];
    dv[i] = make_uint4(__funnelshift_r(a0, a1, r8), __funnelshift_r(a1, a2, r8), __funnelshift_r(a2, a3, r8),
                       __funnelshift_r(a3, a4, r8));
  }
  const uint32_t tail = head + 16u * body + lane;
  if (tail < len)
    dst[tail] = (char)text[tail];
}

template <int kEntries>
__global__ void __launch_bounds__(kFusedThreads, 5) k_csv_fused(Source s, FusedSink out)
{
  constexpr int kChunks = kEntries / 32, kWindow = FusedShape<kEntries>::kWindow;
  using WarpText = typename FusedShape<kEntries>::WarpText;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ long long s_tile;
  __shared__ unsigned long long s_prefix;
  __shared__ uint32_t s_len[kFusedWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  WarpText& W = reinterpret_cast<WarpText*>(smem)[warp];
  if (threadIdx.x == 0)
    s_tile = (long long)atomicAdd(out.ticket, 1u);
  __syncthreads();
  const long long tile = s_tile;
  // 1. the warp's entries, the nonzero ones queued.  n <= 65535: an entry
  // index fits 32 bits.
  WarpRows<kEntries> at;
  const long long first_entry = tile * FusedShape<kEntries>::kTile + (long long)warp * kEntries;
  at.valid = (int)max(0ll, min((long long)kEntries, s.n_entries - first_entry));
  at.e0 = at.valid ? (uint32_t)first_entry : 0u;
  at.n = (uint32_t)s.n;
  at.row = at.e0 / at.n;
  at.col = at.e0 - at.row * at.n;
  const uint32_t* words = (s.ff ? reinterpret_cast<const uint32_t*>(s.ff) : s.counts) + at.e0;
  uint32_t raw[kChunks];
  if (at.valid == kEntries) {
#pragma unroll
    for (int k = 0; k < kChunks; ++k)
      raw[k] = __ldg(words + 32 * k + lane);
  } else {
#pragma unroll
    for (int k = 0; k < kChunks; ++k)
      raw[k] = 32 * k + lane < at.valid ? __ldg(words + 32 * k + lane) : 0u;
  }
  // a count of zero is a +0 entry unless its row's ratio is negative,
  // infinite or not a number (no rays, or fewer than none)
  bool plain = true;
  at.ratio0 = at.ratio1 = 1.f;
  if (!s.ff && at.valid) {
    uint32_t r, c;
    at.locate(at.valid - 1, &r, &c);
    int rays = 1;
    for (uint32_t i = at.row + lane; i <= r; i += 32) {
      rays = __ldg(s.outgoing + i);
      plain &= rays > 0;
    }
    plain = __all_sync(0xFFFFFFFFu, plain);
    const float ratio = 1.f / (float)rays;
    at.ratio0 = __shfl_sync(0xFFFFFFFFu, ratio, 0);
    at.ratio1 = __shfl_sync(0xFFFFFFFFu, ratio, 1);
  }
  at.simple = plain && at.valid == kEntries && at.n >= (uint32_t)kEntries;
  at.row_end = (int)(at.n - 1 - at.col);
  // 2. the nonzero ones formatted, lengths scanned
  Text first{0, 0, 0};
  int text_len = 0;
  const int n_q = at.simple ? queue_entries<kEntries, true>(s, at, words, raw, plain, W, first, &text_len, lane)
                            : queue_entries<kEntries, false>(s, at, words, raw, plain, W, first, &text_len, lane);
  const uint32_t len = (uint32_t)text_len;
  if (lane == 0)
    s_len[warp] = len;
  __syncthreads();
  uint32_t before = 0, total = 0;
#pragma unroll
  for (int w = 0; w < kFusedWarps; ++w) {
    const uint32_t u = s_len[w];
    before += w < warp ? u : 0u;
    total += u;
  }
  // 3. publish the tile's length; the text is staged while the tiles before
  // it finish
  if (threadIdx.x == 0)
    st_relaxed(out.status + tile, (tile == 0 ? kTilePrefix : kTileAgg) | total);
  const bool fits = len <= (uint32_t)kWindow;
  if (fits && at.simple)
    stage_text<kEntries, true, true>(s, at, words, W, n_q, first, 0, lane);
  else if (fits)
    stage_text<kEntries, true, false>(s, at, words, W, n_q, first, 0, lane);
  // 4. the tile's place in the text
  if (warp == 0) {
    unsigned long long excl = 0;
    if (tile > 0) {
      excl = look_back(out, tile, lane);
      if (lane == 0)
        st_relaxed(out.status + tile, kTilePrefix | (excl + total));
    }
    if (lane == 0) {
      s_prefix = excl;
      if (tile == out.n_tiles - 1)
        *out.total = excl + total;
    }
  }
  __syncthreads();
  const unsigned long long P = s_prefix;
  if (P + total > out.cap) {
    if (threadIdx.x == 0)
      atomicOr(out.err, kFusedOverflow);
    return;
  }
  char* dst = out.text + P + before;
  if (fits) {
    copy_text(dst, W.text, len, lane);
    return;
  }
  for (uint32_t w0 = 0; w0 < len; w0 += kWindow) {
    stage_text<kEntries, false, false>(s, at, words, W, n_q, first, (int)w0, lane);
    __syncwarp();
    copy_text(dst + w0, W.text, min(len - w0, (uint32_t)kWindow), lane);
    __syncwarp();
  }
}
#endif  // __CUDACC__

}  // namespace csv
}  // namespace ffb
