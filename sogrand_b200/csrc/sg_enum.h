/* sg_enum.h -- the order in which SOGRAND tests error patterns.
 *
 * sogrand_main_logic (SOGRAND_C/cubic_decoder_final.c:587-746) tests the
 * hard decision first, then loops over logistic weights wt = IC+1 ..
 * 16*IC+136; within a weight over Hamming weights w from the bound of :653
 * upwards; within (wt, w) over the patterns produced by mountain_build
 * (:775-789) and the landslide step (:689-734).  Over the 16 reliability-
 * sorted positions the sequence of patterns depends on IC alone (n = 16,
 * even = 0).  The decoder therefore reads pattern t of a line from a table
 * built once per IC instead of re-running the successor logic per guess.
 *
 * Entry t (t = 0 is the hard decision itself), one field per byte so that
 * the decoder forms each table address with one byte permute:
 *   byte 0  sg_swz(low byte of the pattern over sorted positions): the
 *           decoder's storage index of the low byte's per-line table entries
 *           (sg_swz is its own inverse)
 *   byte 1  the high byte of the pattern (bit r = position 8 + r)
 *   byte 2  8 * (1 + j) for the lowest set position 8 + j of the high byte,
 *           0 if the high byte is empty
 *   byte 3  the same for the second-lowest set high position
 * Bytes 2 and 3 are offsets into a per-line table of path-metric increments
 * whose entry 0 is zero, so the decoder adds the first two high-position
 * increments without a loop.  Two more facts about an order come from
 * counting subsets by logistic weight, not from the table (sg_order_meta):
 * where the first logistic weight whose patterns may hold three high
 * positions starts, and where the reference's Tmax check cuts.
 * For IC >= SG_ENUM_IC_CANON the weight ranges of different Hamming weights
 * no longer interleave and the table is identical for every IC; the decoder
 * uses table SG_ENUM_IC_CANON for all of them (checked by
 * tests/test_enum.py for IC up to 4096 and sampled larger values).
 */
#pragma once
#include <stddef.h>
#include <stdint.h>

#include "sg_math.h" /* SG_HD */

#define SG_ENUM_LEN 65536u
#define SG_ENUM_GS 0x10000u /* exported order: first pattern of a logistic weight */

/* Storage index of the per-line tables' entry for low byte lo: the low
 * nibble XORed with a function of bits 5..7 (their 8 values, 0, 5, 11, 14,
 * 15, 10, 4, 1, are the nibbles of the constant, low first); it leaves bits
 * 4..7 alone, so it is its own inverse.  The 32 patterns of a warp step
 * concentrate on few residues of lo mod 16, an 8-byte table entry's
 * shared-memory bank pair; this permutation, the best of a search over
 * linear maps on the steps of 2 dB decodes, spreads them: 3.3 wavefronts
 * per lookup on average instead of 5.3. */
SG_HD uint32_t sg_swz(uint32_t lo)
{
    return lo ^ ((0x14AFEB50u >> ((lo >> 3) & 28u)) & 15u);
}

/* The pattern (bits 0..15 over sorted positions) of an order-table entry. */
SG_HD uint32_t sg_ent_pattern(uint32_t ent)
{
    return sg_swz(ent & 0xffu) | (ent & 0xff00u);
}
#define SG_ENUM_IC_CANON 56
#define SG_ENUM_NTAB (SG_ENUM_IC_CANON + 1)

/* mountain_build (cubic_decoder_final.c:775-789): set u[k+1..w) to u[k],
 * then pile the weight still missing onto the high end, n1 at a time. */
SG_HD bool sg_enum_fill(int32_t* u, int32_t k, int32_t w, int32_t W1, int32_t n1)
{
    for (int32_t i = k + 1; i < w; i++)
        u[i] = u[k];
    int64_t rest = W1;
    for (int32_t i = 0; i < w; i++)
        rest -= u[i];
    int64_t room = (int64_t)n1 - u[k];
    if (rest < 0 || room <= 0)
        return false;
    int64_t q = rest / room;
    int64_t r = rest - q * room;
    if (q > w)
        return false;
    for (int64_t i = w - q; i < w; i++)
        u[i] = n1;
    if (w > q)
        u[w - q - 1] += (int32_t)r;
    return true;
}

/* Entry of pattern m (bits 0..15). */
SG_HD uint32_t sg_enum_entry(uint32_t m)
{
    uint32_t hi = (m >> 8) & 0xffu, o1 = 0, o2 = 0;
    if (hi) {
        int j = 0;
        while (!((hi >> j) & 1u))
            j++;
        o1 = 8u * (uint32_t)(1 + j);
        hi &= hi - 1u;
    }
    if (hi) {
        int j = 0;
        while (!((hi >> j) & 1u))
            j++;
        o2 = 8u * (uint32_t)(1 + j);
    }
    return sg_swz(m & 0xffu) | (m & 0xff00u) | (o1 << 16) | (o2 << 24);
}

/* Logistic weight of pattern m: IC per set position plus its 1-based rank. */
SG_HD int32_t sg_enum_weight(int32_t ic, uint32_t m)
{
    int32_t wt = 0;
    for (int r = 0; r < 16; r++)
        if ((m >> r) & 1u)
            wt += ic + r + 1;
    return wt;
}

/* Per IC: h3, the first pattern of the first logistic weight that a pattern
 * with three high positions can have (3*IC + 9 + 10 + 11); and lim, the
 * number of patterns tested when Tmax cuts the decode: the reference checks
 * T < Tmax before each new logistic weight (:652), so the cut is at the
 * first weight that starts at or after Tmax (SG_ENUM_LEN without one). */
typedef struct {
    uint32_t h3[SG_ENUM_NTAB];
    uint32_t lim[SG_ENUM_NTAB];
} sg_order_meta;

/* cnt[w][s]: subsets of {1..16} with w elements and sum s. */
static inline void sg_enum_counts(uint32_t cnt[17][137])
{
    for (int w = 0; w <= 16; w++)
        for (int s = 0; s <= 136; s++)
            cnt[w][s] = 0;
    cnt[0][0] = 1;
    for (int r = 1; r <= 16; r++)
        for (int w = r; w >= 1; w--)
            for (int s = 136; s >= r; s--)
                cnt[w][s] += cnt[w - 1][s - r];
}

/* Starts of the logistic weights of IC `ic` in ascending order (at most
 * 16*ic + 136); returns how many. */
static inline int sg_enum_starts(int32_t ic, const uint32_t cnt[17][137], uint32_t* start, uint32_t* h3)
{
    int n = 0;
    uint32_t t = 1; /* after the hard decision */
    *h3 = SG_ENUM_LEN;
    for (int32_t wt = ic + 1; wt <= 16 * ic + 136; wt++) {
        uint32_t c = 0;
        for (int w = 1; w <= 16; w++) {
            const int32_t s = wt - ic * w;
            if (s >= 0 && s <= 136)
                c += cnt[w][s];
        }
        if (wt >= 3 * ic + 30 && *h3 == SG_ENUM_LEN)
            *h3 = t;
        if (c) {
            start[n++] = t;
            t += c;
        }
    }
    return n;
}

/* The builder, usable on host and device (same source, same order): writes
 * the pattern order for `ic` (ic >= 0) to out[0..SG_ENUM_LEN) and returns the
 * number of patterns written: SG_ENUM_LEN on success, 0 if the successor
 * logic left its domain (never for 0 <= ic < 2^20). */
SG_HD size_t sg_enum_build_impl(int32_t ic, uint32_t* out)
{
    const int32_t n = 16;
    size_t t = 0;
    out[t++] = 0; /* the hard decision, tested before the loop (:624-641) */
    const int32_t wt_max = ic * n + n * (n + 1) / 2;
    const double temp = 1 + 2 * ((double)n + (double)ic);
    int32_t u[16];
    for (int32_t wt = ic + 1; wt <= wt_max; wt++) {
        /* smallest Hamming weight that can reach logistic weight wt (:653) */
        int32_t w = (int32_t)ceil((temp - sqrt(temp * temp - 8.0 * wt)) / 2);
        if (w < 1)
            w = 1;
        for (; w <= n; w++) {
            const int32_t W = wt - ic * w;
            if (W < w * (w + 1) / 2)
                break;
            const int32_t W1 = W - w * (w + 1) / 2;
            const int32_t n1 = n - w;
            if (n1 == 0) { /* the all-ones pattern; the reference divides by zero here */
                if (t >= SG_ENUM_LEN)
                    return 0;
                out[t++] = sg_enum_entry(0xffffu);
                continue;
            }
            for (int i = 0; i < 16; i++)
                u[i] = 0;
            if (!sg_enum_fill(u, 0, w, W1, n1))
                return 0;
            for (;;) {
                if (t >= SG_ENUM_LEN)
                    return 0;
                uint32_t m = 0;
                for (int32_t i = 0; i < w; i++)
                    m |= 1u << (i + u[i]);
                out[t++] = sg_enum_entry(m);
                /* landslide (:689-734): move the highest position that is at
                 * least 2 below the top one place up and refill above it */
                if (u[w - 1] - u[0] < 2)
                    break;
                int32_t k = 0;
                for (int32_t i = w - 1; i > 0; i--)
                    if (u[w - 1] - u[i] >= 2) {
                        k = i;
                        break;
                    }
                u[k]++;
                if (!sg_enum_fill(u, k, w, W1, n1))
                    return 0;
            }
        }
    }
    return t;
}
