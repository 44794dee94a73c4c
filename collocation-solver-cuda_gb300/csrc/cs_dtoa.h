// Shortest round-trip decimal text of an IEEE double, as Python's repr(float)
// and "{}".format(float) print it: the fewest significant digits that read
// back as the same double, the one nearest the value among those, positional
// notation for 1e-4 <= |v| < 1e16 ("0.0001", "123.0", "1234567890123456.0")
// and scientific otherwise ("1e-05", "1.5e+16", "5e-324"); "inf", "-inf",
// "nan", "0.0", "-0.0".  The reference writes every number of its solution
// files this way (BVPDAEReadWriteData.py:337-364).
//
// Digits: the free-format algorithm of Steele & White and of Burger & Dybvig
// ("Printing floating-point numbers quickly and accurately", PLDI 1996),
// restated here on exact fixed-size integers.  v = f 2^e is held as r / s with
// the half-gaps to the neighbouring doubles m+ / s and m- / s; digits are
// generated until the remaining interval contains a shorter decimal.  With
// an even mantissa the interval's ends read back as v (round half to even),
// so they count as inside.
//
// Host and device code: the library formats solution files on the GPU with it
// and exports it for the host as cs_format_double.
#pragma once
#include <math.h>
#include <stdint.h>

#if defined(__CUDACC__)
#define CS_HD __host__ __device__ __forceinline__
#define CS_HD_CALL static __host__ __device__ __noinline__
#else
#define CS_HD static inline
#define CS_HD_CALL static
#endif

// longest text: "-1.2345678901234567e-308" (24 characters)
#define CS_DTOA_MAX 24

CS_HD int cs_clz64(uint64_t x) {
#if defined(__CUDA_ARCH__)
  return __clzll((long long)x);
#else
  return __builtin_clzll(x);
#endif
}

// little-endian unsigned integer of up to CS_BN_LIMBS 32-bit limbs
#define CS_BN_LIMBS 40
struct CsBig {
  uint32_t w[CS_BN_LIMBS];
  int n;  // limbs in use (w[n-1] != 0, or n == 0 for zero)
};

CS_HD void cs_bn_set(CsBig& a, uint64_t v) {
  a.n = 0;
  while (v) {
    a.w[a.n++] = (uint32_t)v;
    v >>= 32;
  }
}

CS_HD void cs_bn_mul_small(CsBig& a, uint32_t m) {
  uint64_t c = 0;
  for (int i = 0; i < a.n; ++i) {
    const uint64_t t = (uint64_t)a.w[i] * m + c;
    a.w[i] = (uint32_t)t;
    c = t >> 32;
  }
  if (c) a.w[a.n++] = (uint32_t)c;
}

// a *= 2^k
CS_HD void cs_bn_shl(CsBig& a, int k) {
  if (a.n == 0 || k <= 0) return;
  const int q = k >> 5, b = k & 31;
  if (b) {
    uint32_t c = 0;
    for (int i = 0; i < a.n; ++i) {
      const uint32_t x = a.w[i];
      a.w[i] = (x << b) | c;
      c = x >> (32 - b);
    }
    if (c) a.w[a.n++] = c;
  }
  if (q) {
    for (int i = a.n - 1; i >= 0; --i) a.w[i + q] = a.w[i];
    for (int i = 0; i < q; ++i) a.w[i] = 0;
    a.n += q;
  }
}

// a *= 10^k (k >= 0)
CS_HD void cs_bn_mul_pow10(CsBig& a, int k) {
  while (k >= 9) {
    cs_bn_mul_small(a, 1000000000u);
    k -= 9;
  }
  uint32_t m = 1;
  while (k-- > 0) m *= 10;
  if (m > 1) cs_bn_mul_small(a, m);
}

CS_HD int cs_bn_cmp(const CsBig& a, const CsBig& b) {
  if (a.n != b.n) return a.n < b.n ? -1 : 1;
  for (int i = a.n - 1; i >= 0; --i)
    if (a.w[i] != b.w[i]) return a.w[i] < b.w[i] ? -1 : 1;
  return 0;
}

// compare a + b with c
CS_HD int cs_bn_cmp_sum(const CsBig& a, const CsBig& b, const CsBig& c) {
  const int n = a.n > b.n ? a.n : b.n;
  if (n + 1 < c.n) return -1;
  if (n > c.n) return 1;  // a + b >= 2^(32(n-1)) > c
  // sum limb by limb, then compare from the top
  uint32_t s[CS_BN_LIMBS + 1];
  uint64_t cy = 0;
  for (int i = 0; i < n; ++i) {
    const uint64_t t = (uint64_t)(i < a.n ? a.w[i] : 0u) + (i < b.n ? b.w[i] : 0u) + cy;
    s[i] = (uint32_t)t;
    cy = t >> 32;
  }
  int sn = n;
  if (cy) s[sn++] = (uint32_t)cy;
  while (sn > 0 && s[sn - 1] == 0) --sn;
  if (sn != c.n) return sn < c.n ? -1 : 1;
  for (int i = sn - 1; i >= 0; --i)
    if (s[i] != c.w[i]) return s[i] < c.w[i] ? -1 : 1;
  return 0;
}

// a -= b (a >= b)
CS_HD void cs_bn_sub(CsBig& a, const CsBig& b) {
  int64_t br = 0;
  for (int i = 0; i < a.n; ++i) {
    int64_t t = (int64_t)a.w[i] - (i < b.n ? (int64_t)b.w[i] : 0) - br;
    br = t < 0;
    a.w[i] = (uint32_t)(t + (br << 32));
  }
  while (a.n > 0 && a.w[a.n - 1] == 0) --a.n;
}

// Significant digits of v > 0 (finite) into dig[], returns their count;
// *k10: v = 0.d1 d2 ... x 10^k10.
CS_HD int cs_shortest_digits(double v, char* dig, int* k10) {
  union {
    double d;
    uint64_t u;
  } bits;
  bits.d = v;
  const int be = (int)((bits.u >> 52) & 0x7ff);
  const uint64_t frac = bits.u & ((1ull << 52) - 1);
  const uint64_t f = be ? (frac | (1ull << 52)) : frac;
  const int e = be ? be - 1075 : -1074;
  const bool even = (f & 1) == 0;
  const bool pow2 = be > 1 && frac == 0;  // the gap below is half the gap above
  CsBig r, s, mp, mm;
  // v = r / s, upper half-gap mp / s, lower half-gap mm / s
  if (e >= 0) {
    cs_bn_set(r, f);
    cs_bn_shl(r, e + (pow2 ? 2 : 1));
    cs_bn_set(s, pow2 ? 4 : 2);
    cs_bn_set(mp, 1);
    cs_bn_shl(mp, e + (pow2 ? 1 : 0));
    cs_bn_set(mm, 1);
    cs_bn_shl(mm, e);
  } else {
    cs_bn_set(r, f);
    cs_bn_shl(r, pow2 ? 2 : 1);
    cs_bn_set(s, 1);
    cs_bn_shl(s, -e + (pow2 ? 2 : 1));
    cs_bn_set(mp, pow2 ? 2 : 1);
    cs_bn_set(mm, 1);
  }
  // Scale by 10^-k so that the digits start right after the point: k is the
  // smallest integer with (r + mp) / s < 10^k (<= with an odd mantissa, whose
  // upper end does not read back).  Start from floor(log10 v) + 1, which is
  // off by one at most, and step.
  const int top = 63 - cs_clz64(f);  // v in [2^(top+e), 2^(top+e+1))
  int kexp = (int)floor((double)(top + e) * 0.30102999566398119521) + 1;
  if (kexp >= 0) {
    cs_bn_mul_pow10(s, kexp);
  } else {
    cs_bn_mul_pow10(r, -kexp);
    cs_bn_mul_pow10(mp, -kexp);
    cs_bn_mul_pow10(mm, -kexp);
  }
  for (;;) {  // too small a scale: 10^k itself (or more) is in the interval
    const int c = cs_bn_cmp_sum(r, mp, s);
    if (!(even ? c >= 0 : c > 0)) break;
    cs_bn_mul_small(s, 10);
    ++kexp;
  }
  for (;;) {  // too large a scale: k - 1 would also do
    CsBig t = r, u = mp;
    cs_bn_mul_small(t, 10);
    cs_bn_mul_small(u, 10);
    const int c = cs_bn_cmp_sum(t, u, s);
    if (!(even ? c < 0 : c <= 0)) break;
    r = t;
    mp = u;
    cs_bn_mul_small(mm, 10);
    --kexp;
  }
  *k10 = kexp;
  int n = 0;
  for (;;) {
    cs_bn_mul_small(r, 10);
    cs_bn_mul_small(mp, 10);
    cs_bn_mul_small(mm, 10);
    int d = 0;
    while (cs_bn_cmp(r, s) >= 0) {
      cs_bn_sub(r, s);
      ++d;
    }
    const int cl = cs_bn_cmp(r, mm);
    const bool low = even ? cl <= 0 : cl < 0;
    const int ch = cs_bn_cmp_sum(r, mp, s);
    const bool high = even ? ch >= 0 : ch > 0;
    if (!low && !high) {
      dig[n++] = (char)('0' + d);
      if (n >= 20) break;  // cannot happen for a double; bounds the loop
      continue;
    }
    if (low && high) {
      // both neighbours read back: the nearer one; on a tie the even digit
      const int c2 = cs_bn_cmp_sum(r, r, s);
      if (c2 > 0 || (c2 == 0 && (d & 1))) ++d;
    } else if (high) {
      ++d;
    }
    dig[n++] = (char)('0' + d);
    break;
  }
  return n;
}

// ---------------------------------------------------------------------------
// The same digits without big integers, for 2^-143 <= v < 2^53 (about 1e-43 to
// 9e15: what solutions hold).  With v = c 2^q and 10^k <= 2^q < 10^(k+1) the
// interval that reads back as v is 10^k to 10^(k+1) wide, so the answer is its
// one multiple of 10^(k+1) if it has one (then without trailing zeros), else
// the multiple of 10^k nearest to v (Giulietti, "The Schubfach way to render
// doubles", 2020).  In that paper the products with 10^-k are rounded and
// their error bounded; here p = -k <= 59, so c 10^p 2^q = c 5^p / 2^s is held
// exactly in three 64-bit words and every comparison is exact.  Measured on
// the GPU: 30 G values/s, against 1.0 G values/s by the big integers above.
struct CsDec {
  uint64_t d;  // significant digits, no trailing zero
  int n;       // how many
  int k;       // v = 0.d x 10^k
};

struct CsU192 {
  uint64_t w[3];
};

CS_HD int cs_u192_cmp(const CsU192& a, const CsU192& b) {
  if (a.w[2] != b.w[2]) return a.w[2] < b.w[2] ? -1 : 1;
  if (a.w[1] != b.w[1]) return a.w[1] < b.w[1] ? -1 : 1;
  if (a.w[0] != b.w[0]) return a.w[0] < b.w[0] ? -1 : 1;
  return 0;
}

// a * m (the product fits)
CS_HD CsU192 cs_u192_mul(const CsU192& a, uint64_t m) {
  CsU192 r;
  unsigned __int128 t = (unsigned __int128)a.w[0] * m;
  r.w[0] = (uint64_t)t;
  t = (unsigned __int128)a.w[1] * m + (uint64_t)(t >> 64);
  r.w[1] = (uint64_t)t;
  r.w[2] = a.w[2] * m + (uint64_t)(t >> 64);
  return r;
}

CS_HD CsU192 cs_u192_add(const CsU192& a, const CsU192& b) {
  CsU192 r;
  unsigned __int128 t = (unsigned __int128)a.w[0] + b.w[0];
  r.w[0] = (uint64_t)t;
  t = (unsigned __int128)a.w[1] + b.w[1] + (uint64_t)(t >> 64);
  r.w[1] = (uint64_t)t;
  r.w[2] = a.w[2] + b.w[2] + (uint64_t)(t >> 64);
  return r;
}

CS_HD CsU192 cs_u192_sub(const CsU192& a, const CsU192& b) {
  CsU192 r;
  unsigned __int128 t = (unsigned __int128)a.w[0] - b.w[0];
  r.w[0] = (uint64_t)t;
  t = (unsigned __int128)a.w[1] - b.w[1] - ((uint64_t)(t >> 64) & 1u);
  r.w[1] = (uint64_t)t;
  r.w[2] = a.w[2] - b.w[2] - ((uint64_t)(t >> 64) & 1u);
  return r;
}

// m 2^s (s < 192, the result fits)
CS_HD CsU192 cs_u192_shl(uint64_t m, int s) {
  const int q = s >> 6, b = s & 63;
  const uint64_t lo = m << b, hi = b ? m >> (64 - b) : 0;
  CsU192 r;
  r.w[0] = q == 0 ? lo : 0;
  r.w[1] = q == 0 ? hi : (q == 1 ? lo : 0);
  r.w[2] = q == 1 ? hi : (q == 2 ? lo : 0);
  return r;
}

// 5^0 .. 5^59
struct CsPow5 {
  uint64_t w[60][3];
  constexpr CsPow5() : w() {
    w[0][0] = 1;
    for (int p = 1; p < 60; ++p) {
      unsigned __int128 t = 0;
      for (int q = 0; q < 3; ++q) {
        t = (unsigned __int128)w[p - 1][q] * 5 + (uint64_t)(t >> 64);
        w[p][q] = (uint64_t)t;
      }
    }
  }
};
#if defined(__CUDACC__)
static __device__ const CsPow5 cs_pow5_device;
#endif
static constexpr CsPow5 cs_pow5_host;

CS_HD CsU192 cs_pow5(int p) {
#if defined(__CUDA_ARCH__)
  const uint64_t* w = cs_pow5_device.w[p];
#else
  const uint64_t* w = cs_pow5_host.w[p];
#endif
  CsU192 r = {{w[0], w[1], w[2]}};
  return r;
}

CS_HD int cs_ndigits(uint64_t d) {
  int n = 1;
  if (d >= 10000000000000000ull) return 17;  // at most 17 digits
  if (d >= 100000000ull) { d /= 100000000ull; n += 8; }
  uint32_t x = (uint32_t)d;
  if (x >= 10000u) { x /= 10000u; n += 4; }
  if (x >= 100u) { x /= 100u; n += 2; }
  return n + (x >= 10u);
}

// v > 0 in range (see above): the decimal; false when v is out of range
CS_HD bool cs_decimal_fast(uint64_t bits, CsDec* out) {
  const int be = (int)((bits >> 52) & 0x7ff);
  const uint64_t frac = bits & ((1ull << 52) - 1);
  const int q = be - 1075;
  if (be == 0 || q > 0 || q < -195) return false;
  const uint64_t c = frac | (1ull << 52);
  const bool even = (c & 1) == 0, pow2 = frac == 0 && be > 1;
  // floor(log10(2^q)), or of 3/4 2^q: log10(2) 2^22 = 1262611.08 (checked for every q)
  const int k = (q * 1262611 - (pow2 ? 524031 : 0)) >> 22;
  const int p = -k, s = -(q + p) + 2;  // unit: 10^k 2^-s
  if (p > 59) return false;
  const CsU192 g = cs_pow5(p);
  const CsU192 x = cs_u192_mul(g, 4 * c);
  const CsU192 up = cs_u192_add(g, g), lo = pow2 ? g : up;  // half gaps
  // v / 10^k = i + f 2^-s
  const int sw = s >> 6, sb = s & 63;
  const uint64_t a0 = sw == 0 ? x.w[0] : (sw == 1 ? x.w[1] : x.w[2]);
  const uint64_t a1 = sw == 0 ? x.w[1] : (sw == 1 ? x.w[2] : 0);
  const uint64_t i = sb ? (a0 >> sb) | (a1 << (64 - sb)) : a0;
  CsU192 f = x;
  const uint64_t m = sb ? (1ull << sb) - 1 : 0;
  f.w[0] = sw == 0 ? x.w[0] & m : x.w[0];
  f.w[1] = sw == 0 ? 0 : (sw == 1 ? x.w[1] & m : x.w[1]);
  f.w[2] = sw == 2 ? x.w[2] & m : 0;
  const int in = even ? 0 : -1;  // the interval's ends read back when c is even
  // a multiple of 10^(k+1)
  const uint64_t t = i / 10;
  const CsU192 d = cs_u192_add(cs_u192_shl(i - 10 * t, s), f);
  const bool tl = cs_u192_cmp(d, lo) <= in;
  const bool th = cs_u192_cmp(cs_u192_sub(cs_u192_shl(10, s), d), up) <= in;
  uint64_t dig;
  int e = k;
  if (tl || th) {
    dig = tl ? t : t + 1;
    e += 1;
    while (dig % 100 == 0) { dig /= 100; e += 2; }
    if (dig % 10 == 0) { dig /= 10; e += 1; }
  } else {
    const CsU192 one = cs_u192_shl(1, s);
    const bool bl = cs_u192_cmp(f, lo) <= in;
    const bool bh = cs_u192_cmp(cs_u192_sub(one, f), up) <= in;
    const int half = cs_u192_cmp(cs_u192_add(f, f), one);
    dig = (bl && bh) ? i + ((half > 0 || (half == 0 && (i & 1))) ? 1 : 0) : (bl ? i : i + 1);
  }
  out->d = dig;
  out->n = cs_ndigits(dig);
  out->k = out->n + e;
  return true;
}

// the digits of v > 0 by big integers; n in the low byte of *nk, k above.  Not
// inlined: its registers and stack stay out of the fast path.
CS_HD_CALL uint64_t cs_decimal_slow(double v, int* nk) {
  char dig[24];
  int k = 0;
  const int n = cs_shortest_digits(v, dig, &k);
  uint64_t d = 0;
  for (int i = 0; i < n; ++i) d = d * 10 + (uint64_t)(dig[i] - '0');
  *nk = n + 256 * k;
  return d;
}

// what cs_text_plan found out about a value's text
struct CsText {
  CsDec dec;
  int len;    // characters
  int kind;   // 0 decimal, 1 "0.0", 2 "inf", 3 "nan"
  bool neg;
};

// what cs_text_put will write for v
CS_HD void cs_text_plan(double v, CsText* t) {
  union {
    double d;
    uint64_t u;
  } bits;
  bits.d = v;
  t->neg = (bits.u >> 63) != 0;
  const uint64_t u = bits.u & ~(1ull << 63);
  t->kind = u == 0 ? 1 : ((u >> 52) == 0x7ff ? ((u & ((1ull << 52) - 1)) ? 3 : 2) : 0);
  if (t->kind) {
    if (t->kind == 3) t->neg = false;
    t->len = 3 + (t->neg ? 1 : 0);
    return;
  }
  if (!cs_decimal_fast(u, &t->dec)) {
    int nk;
    t->dec.d = cs_decimal_slow(t->neg ? -v : v, &nk);
    t->dec.n = nk & 255;
    t->dec.k = nk >> 8;
  }
  const int n = t->dec.n, k = t->dec.k;
  int len = t->neg ? 1 : 0;
  if (k > -4 && k <= 16) {
    len += k <= 0 ? 2 - k + n : (n > k ? n + 1 : k + 2);
  } else {
    const int x = k - 1;
    len += n + (n > 1 ? 1 : 0) + 2 + ((x >= 100 || x <= -100) ? 3 : 2);
  }
  t->len = len;
}

// The planned text at out (t.len characters, no terminator).
CS_HD void cs_text_put(const CsText& t, char* out) {
  int p = 0;
  if (t.neg) out[p++] = '-';
  if (t.kind) {
    const char* w = t.kind == 1 ? "0.0" : (t.kind == 2 ? "inf" : "nan");
    for (int i = 0; i < 3; ++i) out[p + i] = w[i];
    return;
  }
  const int n = t.dec.n, k = t.dec.k;
  const bool fixed = k > -4 && k <= 16;
  // digit i goes to p + lead + i, one further from the point on
  const int lead = (fixed && k <= 0) ? 2 - k : 0;
  const int point = fixed ? (k <= 0 ? n : k) : 1;  // digits before the point
  uint32_t part[3];  // 8 digits each, from the last
  part[0] = (uint32_t)(t.dec.d % 100000000ull);
  const uint64_t hi = t.dec.d / 100000000ull;
  part[1] = (uint32_t)(hi % 100000000ull);
  part[2] = (uint32_t)(hi / 100000000ull);
  uint32_t x = part[0];
  for (int i = n - 1; i >= 0; --i) {
    const uint32_t y = x / 10;
    out[p + lead + i + (i >= point ? 1 : 0)] = (char)('0' + (x - 10 * y));
    x = y;
    const int done = n - i;
    if (done == 8) x = part[1];
    if (done == 16) x = part[2];
  }
  if (fixed) {
    if (k <= 0) {
      out[p] = '0';
      out[p + 1] = '.';
      for (int i = 0; i < -k; ++i) out[p + 2 + i] = '0';
    } else {
      for (int i = n; i < k; ++i) out[p + i] = '0';
      out[p + k] = '.';
      if (n <= k) out[p + k + 1] = '0';
    }
    return;
  }
  if (n > 1) out[p + 1] = '.';
  p += n + (n > 1 ? 1 : 0);
  out[p++] = 'e';
  int e = k - 1;
  out[p++] = e < 0 ? '-' : '+';
  if (e < 0) e = -e;
  if (e >= 100) {
    out[p++] = (char)('0' + e / 100);
    e %= 100;
  }
  out[p++] = (char)('0' + e / 10);
  out[p] = (char)('0' + e % 10);
}

// Text of v into out (at most CS_DTOA_MAX characters, no terminator);
// returns the length.
CS_HD int cs_format_double_text(double v, char* out) {
  CsText t;
  cs_text_plan(v, &t);
  cs_text_put(t, out);
  return t.len;
}
