/*
 * make_precise_tables.c -- build-time generator of the constant tables of
 * rocrand_b200/csrc/precise_math.cuh (near-correctly-rounded double log and sincos).
 *
 * Every value is computed in binary128 (libquadmath) and split into double-double pairs:
 *  * log: x = 2^k z with z in [OFF, 2 OFF) split into 256 subintervals by the top 8 bits of
 *    z's offset from OFF (bit patterns, OFF = 0x3FE6A80000000000, just above sqrt(1/2), so
 *    that 1.0 lies inside subinterval 149); per subinterval invc_i = 1/c_i for c_i its
 *    midpoint, rounded to a multiple of 2^-8 (z < 1) or 2^-9 (z >= 1) and moved until
 *    r = z invc_i - 1 stays below 2^-8 over the whole subinterval, which makes r exact in
 *    one fma; the subinterval holding 1.0 takes c = 1.  -log(invc_i) is stored as a head
 *    rounded to a multiple of 2^-42 and a tail, so k ln2_hi + head is exact;
 *    ln 2 as a 42-bit head (exact times any exponent) and a tail;
 *  * sincos: for m = 0..464, sin(m C) and cos(m C), C = 2 pi / 464 as a double, as (hi, lo)
 *    pairs; at the multiples of pi/2 the one that is only C's rounding error is all low word.
 *    (464 C is within 5e-18 of 2 pi, which no power of two of divisions gives: the kernels
 *    leave out that error's product with cos b - 1.)
 *
 * Usage: make_precise_tables <output.inc>
 */
#include <math.h>
#include <quadmath.h>
#include <stdio.h>
#include <string.h>

static double round_bits(__float128 v, int bits)
{
    /* v rounded to `bits` significant bits */
    int        e = 0;
    __float128 m = frexpq(v, &e); /* v = m 2^e, 0.5 <= |m| < 1 */
    m            = rintq(ldexpq(m, bits));
    return (double)ldexpq(m, e - bits);
}

int main(int argc, char** argv)
{
    if(argc != 2)
    {
        fprintf(stderr, "usage: %s <output.inc>\n", argv[0]);
        return 2;
    }
    FILE* f = fopen(argv[1], "w");
    if(!f)
    {
        perror(argv[1]);
        return 1;
    }
    fprintf(f, "/* generated by rocrand_b200/data/make_precise_tables.c */\n");
    /* log table of the offset split: rows (invc, -log(invc) head, tail, 0), i = 0..255 */
    {
        const unsigned long long off = 0x3FE6A80000000000ull;
        fprintf(f, "#define RB_LOG_OFF 0x%016llxull\n#define RB_LOG_ROWS 256\n", off);
        fprintf(f, "#define RB_LOG_INIT { \\\n");
        for(unsigned i = 0; i < 256; i++)
        {
            const unsigned long long blo = off + ((unsigned long long)i << 44);
            const unsigned long long bhi = blo + (1ull << 44) - 1; /* last z of the subinterval */
            double                   zlo, zhi;
            memcpy(&zlo, &blo, 8);
            memcpy(&zhi, &bhi, 8);
            double invc;
            if(zlo <= 1.0 && 1.0 <= zhi)
                invc = 1.0;
            else
            {
                const __float128 c    = ((__float128)zlo + (__float128)zhi) / 2;
                const double     step = zlo < 1.0 ? 0x1p-8 : 0x1p-9;
                invc                  = (double)(rintq((1.0Q / c) / step) * step);
                /* move invc by its step until |r| < 2^-8 at both ends */
                for(int tries = 0; tries < 8; tries++)
                {
                    const __float128 rl = (__float128)zlo * invc - 1, rh = (__float128)zhi * invc - 1;
                    if(fabsq(rl) < 0x1p-8Q && fabsq(rh) < 0x1p-8Q)
                        break;
                    invc += (fabsq(rl) > fabsq(rh) ? (rl < 0 ? step : -step) : (rh > 0 ? -step : step));
                }
            }
            const __float128 rl = (__float128)zlo * invc - 1, rh = (__float128)zhi * invc - 1;
            if(!(fabsq(rl) < 0x1p-8Q && fabsq(rh) < 0x1p-8Q))
            {
                fprintf(stderr, "log table row %u: |r| >= 2^-8\n", i);
                return 1;
            }
            const __float128 l  = -logq((__float128)invc);
            const double     hi = (double)(rintq(ldexpq(l, 42)) / 0x1p42Q);
            const double     lo = (double)(l - (__float128)hi);
            /* the kernels' first sum takes |head| >= |r| (or a zero head) for granted; with
               k ln 2 added it holds by far */
            if(hi != 0.0 && (fabs(hi) < fabsq(rl) || fabs(hi) < fabsq(rh)))
            {
                fprintf(stderr, "log table row %u: |head| < |r|\n", i);
                return 1;
            }
            fprintf(f, "    {%a, %a, %a, 0.0}, \\\n", invc, hi, lo);
        }
        fprintf(f, "}\n");
    }
    const __float128 ln2   = logq(2.0Q);
    const double     l2h   = round_bits(ln2, 42);
    const double     l2l   = (double)(ln2 - (__float128)l2h);
    fprintf(f, "#define RB_LN2_HI %a\n#define RB_LN2_LO %a\n", l2h, l2l);
    /* float log table of the host-logf replay's base (logf_replay.cuh), the same split in
       single precision: t = 2^k z with z in [OFF, 2 OFF), OFF = 0x3f354000 (the 0.708 of
       the double split), 128 subintervals by the top 7 bits of z's offset (1.0 inside
       subinterval 74, which takes c = 1); invc_i rounded to a multiple of 2^-7 (z < 1) or
       2^-8 (z >= 1), at most 8 significant bits, and moved until |r| < 2^-7 over the whole
       subinterval, so that r = z invc_i - 1 is exact in one float fma; -log(invc_i) as a
       head that is a multiple of 2^-19 (k ln2_hi + head is exact in float for |k| <= 31)
       and a float tail; rows (invc, head, tail, 0) */
    {
        const unsigned off = 0x3f354000u;
        fprintf(f, "#define RB_LOGF_OFF 0x%08xu\n#define RB_LOGF_ROWS 128\n", off);
        fprintf(f, "#define RB_LOGF_INIT { \\\n");
        for(unsigned i = 0; i < 128; i++)
        {
            const unsigned blo = off + (i << 16);
            const unsigned bhi = blo + (1u << 16) - 1u;
            float          zlo, zhi;
            memcpy(&zlo, &blo, 4);
            memcpy(&zhi, &bhi, 4);
            double invc;
            if(zlo <= 1.0f && 1.0f <= zhi)
                invc = 1.0;
            else
            {
                const __float128 c    = ((__float128)zlo + (__float128)zhi) / 2;
                const double     step = zlo < 1.0f ? 0x1p-7 : 0x1p-8;
                invc                  = (double)(rintq((1.0Q / c) / step) * step);
                for(int tries = 0; tries < 8; tries++)
                {
                    const __float128 rl = (__float128)zlo * invc - 1, rh = (__float128)zhi * invc - 1;
                    if(fabsq(rl) < 0x1p-7Q && fabsq(rh) < 0x1p-7Q)
                        break;
                    invc += (fabsq(rl) > fabsq(rh) ? (rl < 0 ? step : -step) : (rh > 0 ? -step : step));
                }
            }
            const __float128 rl = (__float128)zlo * invc - 1, rh = (__float128)zhi * invc - 1;
            if(!(fabsq(rl) < 0x1p-7Q && fabsq(rh) < 0x1p-7Q) || (float)invc != invc)
            {
                fprintf(stderr, "float log table row %u: |r| >= 2^-7\n", i);
                return 1;
            }
            const __float128 l  = -logq((__float128)invc);
            const double     hi = (double)(rintq(ldexpq(l, 19)) / 0x1p19Q);
            const float      lo = (float)(l - (__float128)hi);
            fprintf(f, "    %a, %a, %a, 0.0, \\\n", invc, hi, (double)lo);
        }
        fprintf(f, "}\n");
        const double l2fh = (double)(rintq(ldexpq(ln2, 19)) / 0x1p19Q);
        const float  l2fl = (float)(ln2 - (__float128)l2fh);
        fprintf(f, "#define RB_LN2F_HI %af\n#define RB_LN2F_LO %af\n", l2fh, (double)l2fl);
    }
    /* sincos table: rows (sin hi, sin lo, cos hi, cos lo) at m C, m = 0..464 */
    const double step = (double)(2.0Q * M_PIq / 464.0Q);
    fprintf(f, "#define RB_SC_STEP %a\n#define RB_SC_INV_STEP %a\n", step, (double)(1.0Q / (__float128)step));
    fprintf(f, "#define RB_SC_TABLE_ROWS 465\n#define RB_SC_TABLE_INIT { \\\n");
    for(int m = 0; m <= 464; m++)
    {
        const __float128 a  = (__float128)m * (__float128)step; /* exact: 53 + 9 bits */
        const __float128 s  = sinq(a), c = cosq(a);
        const double     sh = m % 232 == 0 ? 0.0 : (double)s, ch = m % 232 == 116 ? 0.0 : (double)c;
        fprintf(f, "    {%a, %a, %a, %a}, \\\n", sh, (double)(s - (__float128)sh), ch,
                (double)(c - (__float128)ch));
    }
    fprintf(f, "}\n");
    if(fclose(f) != 0)
    {
        perror(argv[1]);
        return 1;
    }
    return 0;
}
