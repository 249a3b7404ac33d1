/*
 * xb_hash.h
 *
 * Hash and numeric helpers shared by host and device code.
 *
 * xb_hash_bytes() is Bob Jenkins' lookup3 "hashlittle" in the form
 * PostgreSQL's hash_any() uses (little-endian word fetch, initial value
 * 0x9e3779b9 + len + 3923095, the final() mix returning c).  PG-Strom's
 * device copy pg_hash_any() (xpu_common.cu:2898-3041) and the host-side
 * inner-relation hash (gpu_join.c:1549-1584 via codegen.c:544-660) must both
 * agree with it, because inner hash tables are built on the host and probed
 * on the device.  The fixed-width variants below are the same function
 * specialised for values already held in registers.
 */
#ifndef XB_HASH_H
#define XB_HASH_H
#include <stdint.h>

#if defined(__CUDACC__)
#define XB_HD __host__ __device__ __forceinline__
#else
#define XB_HD static inline
#endif

#define XB_ROT(x, k)    (((x) << (k)) | ((x) >> (32 - (k))))
#define XB_MIX(a, b, c) do {                        \
        a -= c; a ^= XB_ROT(c, 4);  c += b;          \
        b -= a; b ^= XB_ROT(a, 6);  a += c;          \
        c -= b; c ^= XB_ROT(b, 8);  b += a;          \
        a -= c; a ^= XB_ROT(c, 16); c += b;          \
        b -= a; b ^= XB_ROT(a, 19); a += c;          \
        c -= b; c ^= XB_ROT(b, 4);  b += a;          \
    } while (0)
#define XB_FINAL(a, b, c) do {                      \
        c ^= b; c -= XB_ROT(b, 14);                  \
        a ^= c; a -= XB_ROT(c, 11);                  \
        b ^= a; b -= XB_ROT(a, 25);                  \
        c ^= b; c -= XB_ROT(b, 16);                  \
        a ^= c; a -= XB_ROT(c, 4);                   \
        b ^= a; b -= XB_ROT(a, 14);                  \
        c ^= b; c -= XB_ROT(b, 24);                  \
    } while (0)

/* little-endian gather of up to 4 bytes starting at k[0] */
XB_HD uint32_t xb_le_gather(const uint8_t *k, uint32_t n)
{
    uint32_t v = 0;
    for (uint32_t i = 0; i < n; i++)
        v |= ((uint32_t)k[i]) << (8 * i);
    return v;
}

/* hash_any() over an arbitrary (possibly unaligned) byte string */
XB_HD uint32_t xb_hash_bytes(const uint8_t *k, uint32_t len)
{
    uint32_t a, b, c;
    a = b = c = 0x9e3779b9U + len + 3923095U;
    while (len >= 12) {
        a += xb_le_gather(k, 4);
        b += xb_le_gather(k + 4, 4);
        c += xb_le_gather(k + 8, 4);
        XB_MIX(a, b, c);
        k += 12;
        len -= 12;
    }
    /* the low byte of c is reserved for the length: tail bytes 8..10 go
     * into c shifted up by one byte */
    if (len > 8) {
        c += xb_le_gather(k + 8, len - 8) << 8;
        b += xb_le_gather(k + 4, 4);
        a += xb_le_gather(k, 4);
    } else if (len > 4) {
        b += xb_le_gather(k + 4, len - 4);
        a += xb_le_gather(k, 4);
    } else if (len > 0) {
        a += xb_le_gather(k, len);
    }
    XB_FINAL(a, b, c);
    return c;
}

/*
 * The bytes of a datum at any address as 64-bit words, read by aligned
 * 8-byte loads: every aligned word that overlaps the datum lies in its page
 * or buffer, and no other is read.  next() gives bytes 8i..8i+7 (those past
 * the datum's end are whatever its last word holds).
 */
struct XbWords {
    const uint64_t *w;
    uint64_t        cur;
    uint32_t        i, last, s;
};

XB_HD void xb_words_start(XbWords *r, const uint8_t *p, uint32_t len)
{
    const uint32_t o = (uint32_t)((uintptr_t)p & 7);
    r->w = (const uint64_t *)((uintptr_t)p - o);
    r->s = 8 * o;
    r->i = 0;
    r->last = (o + len - 1) >> 3;
    r->cur = r->w[0];
}

XB_HD uint64_t xb_words_next(XbWords *r)
{
    const uint64_t hi = r->i < r->last ? r->w[r->i + 1] : 0;
    const uint64_t v = r->s ? (r->cur >> r->s) | (hi << (64 - r->s)) : r->cur;
    r->cur = hi;
    r->i++;
    return v;
}

/* the first n (0..8) bytes of a word */
XB_HD uint64_t xb_low_bytes(uint64_t v, uint32_t n)
{
    return n >= 8 ? v : v & ((1ULL << (8 * n)) - 1);
}

/* xb_hash_bytes by words (a query over 1M rows that groups by text of 150
 * bytes and sums numerics of every form, by bytes 2.86 ms, by words and with
 * xb_numeric_sum_value's wider reach 0.93 ms) */
XB_HD uint32_t xb_hash_words(const uint8_t *k, uint32_t len)
{
    uint32_t a, b, c;
    a = b = c = 0x9e3779b9U + len + 3923095U;
    if (len > 0) {
        XbWords r;
        xb_words_start(&r, k, len);
        while (len >= 24) {
            const uint64_t q0 = xb_words_next(&r), q1 = xb_words_next(&r), q2 = xb_words_next(&r);
            a += (uint32_t)q0;
            b += (uint32_t)(q0 >> 32);
            c += (uint32_t)q1;
            XB_MIX(a, b, c);
            a += (uint32_t)(q1 >> 32);
            b += (uint32_t)q2;
            c += (uint32_t)(q2 >> 32);
            XB_MIX(a, b, c);
            len -= 24;
        }
        uint64_t q0 = len > 0 ? xb_words_next(&r) : 0;
        uint64_t q1 = len > 8 ? xb_words_next(&r) : 0;
        if (len >= 12) {
            const uint64_t q2 = len > 16 ? xb_words_next(&r) : 0;
            a += (uint32_t)q0;
            b += (uint32_t)(q0 >> 32);
            c += (uint32_t)q1;
            XB_MIX(a, b, c);
            len -= 12;
            q0 = (q1 >> 32) | (q2 << 32);
            q1 = q2 >> 32;
        }
        q0 = xb_low_bytes(q0, len);
        q1 = len > 8 ? xb_low_bytes(q1, len - 8) : 0;
        a += (uint32_t)q0;
        b += (uint32_t)(q0 >> 32);
        c += (uint32_t)q1 << 8;
    }
    XB_FINAL(a, b, c);
    return c;
}

/* equality of two byte strings of n bytes, by words */
XB_HD int xb_words_eq(const uint8_t *a, const uint8_t *b, uint32_t n)
{
    if (a == b || n == 0)
        return 1;
    XbWords x, y;
    xb_words_start(&x, a, n);
    xb_words_start(&y, b, n);
    for (; n >= 16; n -= 16) {
        const uint64_t x0 = xb_words_next(&x), x1 = xb_words_next(&x);
        const uint64_t y0 = xb_words_next(&y), y1 = xb_words_next(&y);
        if ((x0 ^ y0) | (x1 ^ y1))
            return 0;
    }
    if (n >= 8) {
        if (xb_words_next(&x) != xb_words_next(&y))
            return 0;
        n -= 8;
    }
    return n == 0 || xb_low_bytes(xb_words_next(&x) ^ xb_words_next(&y), n) == 0;
}

/* hash_any() of a 1, 2 or 4 byte little-endian value held in a register */
XB_HD uint32_t xb_hash_u32(uint32_t v, uint32_t len)
{
    uint32_t a, b, c;
    a = b = c = 0x9e3779b9U + len + 3923095U;
    if (len < 4)
        v &= (1U << (8 * len)) - 1U;
    a += v;
    XB_FINAL(a, b, c);
    return c;
}

/* hash_any() of an 8 byte value held in a register */
XB_HD uint32_t xb_hash_u64(uint64_t v)
{
    uint32_t a, b, c;
    a = b = c = 0x9e3779b9U + 8U + 3923095U;
    a += (uint32_t)v;
    b += (uint32_t)(v >> 32);
    XB_FINAL(a, b, c);
    return c;
}

/* hash_any() of a 16 byte little-endian int128 (lo, hi) */
XB_HD uint32_t xb_hash_u128(uint64_t lo, uint64_t hi)
{
    uint32_t a, b, c;
    a = b = c = 0x9e3779b9U + 16U + 3923095U;
    a += (uint32_t)lo;
    b += (uint32_t)(lo >> 32);
    c += (uint32_t)hi;
    XB_MIX(a, b, c);
    a += (uint32_t)(hi >> 32);
    XB_FINAL(a, b, c);
    return c;
}

/* pg_hash_merge (xpu_common.h:3470-3476) */
XB_HD uint32_t xb_hash_merge(uint32_t prev, uint32_t next)
{
    return ((prev >> 3) | (prev << 29)) ^ next;
}

/* ----------------------------------------------------------------
 * PostgreSQL numeric varlena -> (kind, scale, int128)
 *
 * Follows __decimal_from_varlena (xpu_numeric.h:216-277): base-10000
 * digits are accumulated into an int128, the scale ("weight" in PG-Strom's
 * naming) is 4 * (ndigits - (pgweight + 1)), then trailing decimal zeros
 * are stripped while the scale is positive (NUMERIC_NORMALIZE).
 * ---------------------------------------------------------------- */
#define XB_NUM_VALID    0
#define XB_NUM_NAN      1
#define XB_NUM_PINF     2
#define XB_NUM_NINF     3

typedef __int128 xb_i128;

/* returns 0 on success, or a non-zero error (1: corrupted, 2: out of range) */
XB_HD int xb_numeric_decode(const uint8_t *vl, uint8_t *p_kind, int16_t *p_weight,
                            xb_i128 *p_value)
{
    uint32_t len, hdr;
    if ((vl[0] & 0x01) == 0x01) {
        if (vl[0] == 0x01)
            return 1;                       /* external toast pointer */
        len = (vl[0] >> 1) & 0x7f;
        hdr = 1;
    } else {
        if ((vl[0] & 0x03) == 0x02)
            return 1;                       /* compressed */
        len = xb_le_gather(vl, 4) >> 2;
        hdr = 4;
    }
    if (len < hdr + 2)
        return 1;
    const uint8_t *nc = vl + hdr;
    uint32_t nc_len = len - hdr;
    uint16_t n_head = (uint16_t)xb_le_gather(nc, 2);
    if ((n_head & 0xC000) == 0xC000) {
        if (n_head == 0xC000)       *p_kind = XB_NUM_NAN;
        else if (n_head == 0xD000)  *p_kind = XB_NUM_PINF;
        else if (n_head == 0xF000)  *p_kind = XB_NUM_NINF;
        else return 1;
        *p_weight = 0;
        *p_value = 0;
        return 0;
    }
    int is_short = ((n_head & 0xC000) == 0x8000);
    int pgweight;
    const uint8_t *digits;
    uint32_t ndigits;
    int negative;
    if (is_short) {
        pgweight = n_head & 0x003F;
        if (n_head & 0x0040)
            pgweight |= ~0x003F;
        digits = nc + 2;
        ndigits = (nc_len - 2) / 2;
        negative = (n_head & 0x2000) != 0;
    } else {
        if (nc_len < 4)
            return 1;
        pgweight = (int16_t)xb_le_gather(nc + 2, 2);
        digits = nc + 4;
        ndigits = (nc_len - 4) / 2;
        negative = (n_head & 0xC000) == 0x4000;
    }
    xb_i128 value = 0;
    for (uint32_t i = 0; i < ndigits; i++) {
        int16_t dig = (int16_t)xb_le_gather(digits + 2 * i, 2);
        if ((value >> 114) != 0)
            return 2;
        value = value * 10000 + dig;
    }
    if (negative)
        value = -value;
    int weight = 4 * ((int)ndigits - (pgweight + 1));
    /* NUMERIC_NORMALIZE */
    if (value == 0) {
        weight = 0;
    } else {
        while (weight > 0) {
            if (weight >= 5 && (value % 100000) == 0) { value /= 100000; weight -= 5; }
            else if (weight >= 4 && (value % 10000) == 0) { value /= 10000; weight -= 4; }
            else if (weight >= 3 && (value % 1000) == 0) { value /= 1000; weight -= 3; }
            else if (weight >= 2 && (value % 100) == 0) { value /= 100; weight -= 2; }
            else if (weight >= 1 && (value % 10) == 0) { value /= 10; weight -= 1; }
            else break;
        }
    }
    *p_kind = XB_NUM_VALID;
    *p_weight = (int16_t)weight;
    *p_value = value;
    return 0;
}

/* rescale an int128 from scale weight_s to weight_d (__normalize_numeric_int128,
 * xpu_numeric.cu:1076-1126: multiply up, or truncate down) */
XB_HD xb_i128 xb_numeric_rescale(int weight_d, int weight_s, xb_i128 v)
{
    int shift;
    if (weight_d > weight_s) {
        for (shift = weight_d - weight_s; shift > 0; ) {
            int k = shift < 18 ? shift : 18;
            xb_i128 p = 1;
            for (int i = 0; i < k; i++) p *= 10;
            v *= p;
            shift -= k;
        }
    } else if (weight_d < weight_s) {
        for (shift = weight_s - weight_d; shift > 0; ) {
            int k = shift < 18 ? shift : 18;
            xb_i128 p = 1;
            for (int i = 0; i < k; i++) p *= 10;
            v /= p;
            shift -= k;
        }
    }
    return v;
}

/* v * 10^k; 0 when that leaves 64 bits */
XB_HD int xb_scale_up_i64(int64_t v, int k, int64_t *out)
{
    uint64_t p = 1;
    if (k > 18)
        return 0;
    for (; k >= 4; k -= 4) p *= 10000;
    for (; k > 0; k--) p *= 10;
    const uint64_t m = v < 0 ? 0 - (uint64_t)v : (uint64_t)v;
    if (p > 1 && m > (uint64_t)INT64_MAX / p)
        return 0;
    *out = v * (int64_t)p;
    return 1;
}

/*
 * The value of a numeric varlena rescaled to weight_d, for sums: the same
 * number as xb_numeric_rescale(weight_d, w, v) of xb_numeric_decode, which
 * normalises trailing zeros away first; rescaling the digits as stored
 * gives the same result (the removed digits are zeros).  Numerics of up to
 * four base-10000 digits, in the short or the long format and under a
 * varlena header of either size, are read with aligned 8-byte loads (every
 * aligned word that overlaps the datum lies in its page or buffer) and
 * rescaled in 64-bit arithmetic: down by constant divisors (10^k for the
 * remainder of 4 that weight_d decides, then 10^4), which the compiler turns
 * into multiplications.  The others take the general decode, whose 128-bit
 * divisions two thirds of the numerics above went through.
 * Returns 0, or 1 on a corrupt datum.
 */
XB_HD int
xb_numeric_sum_value(const uint8_t *vl, int weight_d, uint8_t *p_kind, xb_i128 *p_out)
{
    const uint32_t o = (uint32_t)((uintptr_t)vl & 7);
    const uint64_t *wp = (const uint64_t *)((uintptr_t)vl - o);
    const uint64_t w0 = wp[0];
    const uint32_t h = (uint32_t)(w0 >> (8 * o)) & 0xff;
    /* the varlena header: 1 byte, or 4 when it lies in this word */
    uint32_t hdr = 0, len = 0;
    if (h & 1) {
        hdr = 1;
        len = h >> 1;
    } else if ((h & 2) == 0 && o <= 4) {
        hdr = 4;
        len = (uint32_t)(w0 >> (8 * o)) >> 2;
    }
    if (hdr && len >= hdr + 2 && len <= hdr + 12 && o + len <= 24) {
        const uint64_t w1 = (o + len > 8) ? wp[1] : 0;
        const uint64_t w2 = (o + len > 16) ? wp[2] : 0;
        /* the 16 bytes from the numeric's header on */
        const uint32_t at = o + hdr, s = 8 * (at & 7);
        const uint64_t a = at < 8 ? w0 : w1, b = at < 8 ? w1 : w2, c = at < 8 ? w2 : 0;
        const uint64_t q0 = s ? (a >> s) | (b << (64 - s)) : a;
        const uint64_t q1 = s ? (b >> s) | (c << (64 - s)) : b;
        const uint32_t n_head = (uint32_t)q0 & 0xffff;
        const int is_short = (n_head & 0xC000) == 0x8000;
        const uint32_t body = len - hdr - (is_short ? 2 : 4);   /* digit bytes */
        if ((n_head & 0xC000) != 0xC000 && (int32_t)body >= 0 && body <= 8 && (body & 1) == 0) {
            int pgweight;
            uint64_t digs;
            int negative;
            if (is_short) {
                pgweight = n_head & 0x003F;
                if (n_head & 0x0040)
                    pgweight |= ~0x003F;
                negative = (n_head & 0x2000) != 0;
                digs = (q0 >> 16) | (q1 << 48);
            } else {
                pgweight = (int16_t)(q0 >> 16);
                negative = (n_head & 0xC000) == 0x4000;
                digs = (q0 >> 32) | (q1 << 32);
            }
            int64_t v = 0;
            for (uint32_t i = 0; i < body; i += 2, digs >>= 16)
                v = v * 10000 + (int16_t)digs;
            if (negative)
                v = -v;
            int shift = weight_d - 4 * ((int)(body / 2) - (pgweight + 1));
            if (shift < 0 && v != 0) {
                switch (-shift & 3) {               /* truncates toward zero */
                case 1: v /= 10; break;
                case 2: v /= 100; break;
                case 3: v /= 1000; break;
                default: break;
                }
                for (shift = -(-shift & ~3); shift < 0 && v != 0; shift += 4)
                    v /= 10000;
                shift = 0;
            }
            if (shift == 0 || v == 0 || xb_scale_up_i64(v, shift, &v)) {
                *p_kind = XB_NUM_VALID;
                *p_out = v;
                return 0;
            }
        }
    }
    int16_t w;
    xb_i128 v;
    if (xb_numeric_decode(vl, p_kind, &w, &v))
        return 1;
    *p_out = (*p_kind == XB_NUM_VALID) ? xb_numeric_rescale(weight_d, w, v) : 0;
    return 0;
}

/* hash of a decoded numeric (xpu_numeric.cu:177-193) */
XB_HD uint32_t xb_hash_numeric(uint8_t kind, int16_t weight, xb_i128 value)
{
    if (kind != XB_NUM_VALID)
        return xb_hash_u32(kind, 1);
    return xb_hash_u32((uint16_t)weight, 2) ^
           xb_hash_u128((uint64_t)value, (uint64_t)(value >> 64));
}

/* order-preserving map of IEEE754 doubles onto int64 (NaN canonicalised as
 * the largest value, as PostgreSQL orders float8) */
XB_HD int64_t xb_f64_ordered(double x)
{
    union { double d; int64_t i; } u;
    u.d = x;
    if (x != x)
        u.i = 0x7ff8000000000000LL;
    return u.i >= 0 ? u.i : (u.i ^ 0x7fffffffffffffffLL);
}
XB_HD double xb_f64_from_ordered(int64_t o)
{
    union { double d; int64_t i; } u;
    u.i = o >= 0 ? o : (o ^ 0x7fffffffffffffffLL);
    return u.d;
}

#endif  /* XB_HASH_H */
