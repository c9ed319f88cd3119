/* sg_line.cuh -- one SOGRAND component decode per warp.
 *
 * Restates SOGRAND_bitSO + sogrand_main_logic
 * (SOGRAND_C/cubic_decoder_final.c:521-746) for n = 16, k = 8, even = 0,
 * as warp-cooperative code with results bit-identical to the sequential
 * reference (given the same exp/log):
 *
 *  set-up   lanes 0..15 own the 16 positions: hard decision, |LLR|,
 *           JacLog terms, the sort (rank sort, or the reference's exact
 *           quicksort when magnitudes tie), IC, the PM increment and
 *           syndrome column of each sorted position.  From these the warp
 *           builds per-line tables:
 *             A[lo]     PM_HD + the increments of the bits of lo, added in
 *                       ascending order -- exactly the prefix of getPM's
 *                       sequential sum (:765) over the 8 least reliable
 *                       positions;
 *             synlo/hi  syndrome of each byte of a pattern (ParityCheck,
 *                       :748-755, is linear), the hard decision's own
 *                       syndrome folded into synlo.
 *  guesses  32 consecutive patterns of the order table per step, one per
 *           lane: PM = A[lo] + increments of the high bits (ascending),
 *           syndrome = synlo[lo] ^ synhi[hi], e = exp(-PM).
 *  P_notGuess  the reference subtracts e of every guess in order (:626,
 *           :672, :712).  Within one binade every difference rounds to the
 *           binade's grid, so a step without codeword, exact tie or binade
 *           crossing moves P's bit pattern by the warp's exact integer sum of
 *           the rounded terms (SgGrid).  A step with codewords only takes the
 *           sum up to each of them; any other step replays the reference's
 *           sequence from shared memory, every lane performing the 32 IEEE
 *           subtractions in order.  The result equals the sequential loop
 *           bit for bit.
 *  list     codewords are taken in lane order; getLConf (:767-774) uses the
 *           running P_notGuess at each, so T and the list match exactly.
 *  output   soft output of :536-577 on lanes 0..15.
 *
 * What bounds it: issue slots (81 % used) and shared-memory cycles (75 %).
 * Per line decode at 2 dB 3 510 warp instructions and 810 shared-memory
 * cycles; of its 23 steps 15 end in the sum, 2 hold codewords, 6 are
 * replayed.  Why 32 patterns a step and not 64, two per lane: the longer step
 * is summed half as often but has to be looked at again by halves, and half
 * of such steps are replayed (4 740 instructions, 1 280 cycles; 20 000
 * codewords at 2 dB, batched form, 229 against 202 ms).  The shorter set-up
 * and soft output take that to 193, exp constants read from constant memory
 * to 186 ms; with correctly rounded math 60 ms for 4 096.
 * The file is built with -fmad=false: every floating-point operation the
 * reference performs is a separately rounded IEEE operation here.
 */
#pragma once
#include <stddef.h>
#include <stdint.h>
#include "sg_crmath.h"
#include "sg_enum.h"
#include "sg_math.h"

/* The decoder's exp and log, chosen per instantiation by the template
 * parameter CR of sg_decode_line: false (the default decoder) -- the
 * table-driven routines of sg_math.h, within 0.51 ulp; true (the
 * reference-exact mode) -- the correctly rounded routines of sg_crmath.h,
 * with which every result equals the reference's under a correctly rounded
 * libm, at about 2x the cost per exp. */
template <bool CR>
__device__ __forceinline__ double sg_dec_exp(double x, SgTab tab)
{
    return CR ? sg_exp_cr(x, tab) : sg_exp(x, tab);
}
template <bool CR>
__device__ __forceinline__ double sg_dec_exp_neg(double x, SgTab tab)
{
    return CR ? sg_exp_cr_neg(x, tab) : sg_exp_neg(x, tab);
}
template <bool CR>
__device__ __forceinline__ double sg_dec_log(double x, SgTab tab)
{
    return CR ? sg_log_cr(x, tab) : sg_log(x, tab);
}

/* log of a positive normal argument */
template <bool CR>
__device__ __forceinline__ double sg_dec_log_pos(double x, SgTab tab)
{
    return CR ? sg_log_cr(x, tab) : sg_log_core(sg_bits(x), 0, tab);
}

#define SG_FULL 0xffffffffu

/* Shared-memory loads at a 32-bit shared address.  Plain C++ accesses add
 * the kernel's shared base to every index; the guess loop's addresses hold
 * it already. */
__device__ __forceinline__ uint32_t sg_saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
template <int OFF>
__device__ __forceinline__ double sg_lds_f64(uint32_t a)
{
    double v;
    asm volatile("ld.shared.f64 %0, [%1 + %2];" : "=d"(v) : "r"(a), "n"(OFF));
    return v;
}
template <int OFF>
__device__ __forceinline__ uint32_t sg_lds_u8(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1 + %2];" : "=r"(v) : "r"(a), "n"(OFF));
    return v;
}
__device__ __forceinline__ double2 sg_lds_f64x2(uint32_t a)
{
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
    return v;
}

/* The constants of sg_exp_neg, in constant memory. */
struct SgExpK {
    double inv, ln2_hi, ln2_lo, c3, c4, c5, c6, c7;
};
__constant__ __align__(16) SgExpK sg_exp_consts = {SG_EXP_INV_LN2_N, SG_EXP_LN2_N_HI, SG_EXP_LN2_N_LO, SG_EXP_C3,
                                     SG_EXP_C4,        SG_EXP_C5,       SG_EXP_C6,       SG_EXP_C7};
/* Volatile loads: literals, or plain loads, the compiler would put together
 * again in every step of the guess loop. */
__device__ __forceinline__ SgExpK sg_exp_k()
{
    SgExpK k;
    asm volatile("ld.const.v2.f64 {%0, %1}, [sg_exp_consts];" : "=d"(k.inv), "=d"(k.ln2_hi));
    asm volatile("ld.const.v2.f64 {%0, %1}, [sg_exp_consts + 16];" : "=d"(k.ln2_lo), "=d"(k.c3));
    asm volatile("ld.const.v2.f64 {%0, %1}, [sg_exp_consts + 32];" : "=d"(k.c4), "=d"(k.c5));
    asm volatile("ld.const.v2.f64 {%0, %1}, [sg_exp_consts + 48];" : "=d"(k.c6), "=d"(k.c7));
    return k;
}

/* A kernel's exp table in shared memory: T8 -- eight copies, with the
 * adjusted H_j for the table-driven exp (sg_math.h); otherwise one. */
template <bool T8>
struct SgEtab {
    static constexpr int len = T8 ? 8 * SG_EXP_TAB_LEN : SG_EXP_TAB_LEN;
    alignas(16) double d[len];
};
template <bool CR, bool T8>
__device__ __forceinline__ void sg_etab_fill(SgEtab<T8>& dst, const double* src, int tid, int nt)
{
    for (int i = tid; i < SgEtab<T8>::len; i += nt) {
        const int j = T8 ? i >> 4 : i >> 1;
        double v = src[2 * j + (i & 1)];
        if (T8 && !CR && !(i & 1))
            v = sg_from_bits(sg_bits(v) - ((uint64_t)j << 45));
        dst.d[i] = v;
    }
}
template <bool CR, bool T8>
__device__ __forceinline__ SgTab sg_etab_of(const SgEtab<T8>& tab, const double* k)
{
    return {tab.d + (T8 ? 2 * (threadIdx.x & 7) : 0), k, T8 ? 16 : 2, T8 && !CR};
}

/* exp(x) for x in [-707.5, 0]: sg_exp_neg's operations with the constants
 * of k and the lane's copy of the table (its shared address). */
__device__ __forceinline__ double sg_exp_neg_k(double x, uint32_t tab, const SgExpK& k)
{
    const double z = __dmul_rn(x, k.inv);
    double kd = __dadd_rn(z, SG_EXP_SHIFT);
    const int n = __double2loint(kd);
    kd = __dsub_rn(kd, SG_EXP_SHIFT);
    double r = __fma_rn(-kd, k.ln2_hi, x);
    r = __fma_rn(-kd, k.ln2_lo, r);
    const double2 Ht = sg_lds_f64x2(tab + (uint32_t)(n & 127) * 128u);
    const double r2 = __dmul_rn(r, r);
    double p = __fma_rn(r, k.c7, k.c6);
    p = __fma_rn(r, p, k.c5);
    p = __fma_rn(r, p, k.c4);
    p = __fma_rn(r, p, k.c3);
    p = __fma_rn(r, p, SG_EXP_C2);
    p = __dmul_rn(p, r2);
    const double u = __fma_rn(Ht.y, r, Ht.y);
    const double tmp = __dadd_rn(r, __dadd_rn(u, p));
    const double S = __hiloint2double(__double2hiint(Ht.x) + (n << 13), __double2loint(Ht.x));
    return __fma_rn(S, tmp, S);
}

template <bool B>
struct SgBoolTag {
    static constexpr bool value = B;
};

struct SgLineParams {
    int32_t L;
    double thres;
    const sg_order_meta* meta; /* per IC, Tmax included */
};

/* Per-warp shared scratch of one line decode. */
#define SG_LIST_MAX 8 /* SG_MAX_L of the C ABI; the entry points reject larger L */

/* Every record starts at a multiple of 256 bytes: the guess loop puts an
 * entry's byte into the low byte of the record's shared address to address
 * the tables below (A by a scaled index). */
struct alignas(256) SgWarpScratch {
    double A[256];      /* PM prefix over the low byte of a pattern, entry lo
                           stored at sg_swz(lo) */
    uint8_t synlo[256]; /* syndrome of the low byte (and of the hard decision),
                           entry lo stored at sg_swz(lo) */
    uint8_t synhi[256]; /* syndrome of the high byte */
    double dz[9];       /* dz[0] = 0, dz[1 + j] = PM increment of sorted
                           position 8 + j; indexed by the byte offsets of an
                           order-table entry */
    /* the list (touched only at codewords and in the soft output, so it
     * lives here rather than in registers): entry k = exp(-PM) and pattern
     * (bit r = sorted position r) of the k-th codeword found */
    double lst_e[SG_LIST_MAX];
    double ppos;        /* sum of lst_e in order */
    uint32_t lst_m[SG_LIST_MAX];
    double pnl;         /* pNL of the last getLConf */
    int32_t curl;       /* codewords listed */
    uint32_t hdm;       /* hard decision, bit i = position i */
    int32_t itab;       /* order table of the line's IC */
    uint8_t rank[16];   /* position -> sorted rank */
    uint8_t perm[16];   /* sorted rank -> position (tied magnitudes only) */
    alignas(16) uint8_t hcol[16]; /* syndrome columns of sorted positions r and r + 8 at bytes 2r, 2r + 1 */
    alignas(256) double es[32]; /* replay: exp(-PM) of the 32 patterns of a step */
    double qa[16];      /* sorted magnitudes, then the input LLRs */
    double ex[16];      /* exp(input LLR) of each position, for the soft output */
};
static_assert(offsetof(SgWarpScratch, synlo) == 2048 && offsetof(SgWarpScratch, synhi) == 2304 &&
                  offsetof(SgWarpScratch, dz) == 2560 && sizeof(SgWarpScratch) == 3328,
              "tables addressed by a byte in the record's address");

static __constant__ uint8_t c_hcol[16];
static __constant__ uint8_t c_prow[8];
static __constant__ uint8_t c_ptab[256];

/* (int32_t) of a double as x86-64 cvttsd2si computes it: NaN and values
 * outside int32 give INT32_MIN (the reference casts round(...) at :621). */
__device__ __forceinline__ int32_t sg_cvt_i32(double v)
{
    if (!(v > -2147483649.0 && v < 2147483648.0))
        return INT32_MIN;
    return (int32_t)v;
}

/* Exact restatement of the reference's recursive quicksort (:763) on 16
 * values with an explicit stack.  The two partitions are disjoint, so the
 * processing order of the stack does not change the result.  Run by one
 * lane, only when the line has tied reliabilities (a rank sort orders ties
 * differently). */
static __device__ __noinline__ void sg_quicksort16(double* a, uint8_t* perm)
{
    int32_t st_off[32], st_n[32];
    int sp = 0;
    st_off[sp] = 0;
    st_n[sp] = 16;
    sp++;
    while (sp > 0) {
        sp--;
        int32_t off = st_off[sp], n = st_n[sp];
        if (n < 2)
            continue;
        double* x = a + off;
        uint8_t* pm = perm + off;
        double p = x[n / 2];
        int32_t i = 0, j = n - 1;
        while (i <= j) {
            while (x[i] < p)
                i++;
            while (x[j] > p)
                j--;
            if (i <= j) {
                double t = x[i];
                x[i] = x[j];
                x[j] = t;
                uint8_t tt = pm[i];
                pm[i] = pm[j];
                pm[j] = tt;
                i++;
                j--;
            }
        }
        if (j > 0 && sp < 32) {
            st_off[sp] = off;
            st_n[sp] = j + 1;
            sp++;
        }
        if (i < n && sp < 32) {
            st_off[sp] = off + i;
            st_n[sp] = n - i;
            sp++;
        }
    }
}

struct SgLineResult {
    double lapp;      /* lanes 0..15 */
    double le;        /* lanes 0..15 */
    uint32_t hdword;  /* bit i = hard decision of L_APP at position i (all lanes) */
    uint32_t T;       /* guesses (all lanes) */
    int32_t ncw;      /* codewords found (all lanes) */
};

/* The codeword of lane j, whose guess left P_notGuess = P: list insertion
 * and getLConf (:674-686, :767-774), by that lane.  Returns true (all lanes)
 * when the line decode stops.  The confidence ppos / (ppos + pneg) is
 * divided out only within a few units of the threshold, where its rounding
 * could matter; the products decide everywhere else. */
__device__ __forceinline__ bool sg_list_hit(SgWarpScratch* ws, const SgLineParams& lp, uint32_t ent, double P, double e,
                                            int j, int lane)
{
    const int curl = ws->curl;
    bool stop = curl + 1 == lp.L;
    __syncwarp();
    if (lane == j) {
        const double pneg = __dmul_rn(0x1p-8, P); /* 2^-(n-k) * P_notGuess */
        const double ppos = __dadd_rn(ws->ppos, e);
        ws->lst_e[curl] = e;
        ws->lst_m[curl] = sg_ent_pattern(ent);
        ws->ppos = ppos;
        ws->pnl = pneg;
        ws->curl = curl + 1;
        if (!stop) {
            const double den = __dadd_rn(ppos, pneg);
            const double b = __dmul_rn(lp.thres, den), m = __fma_rn(fabs(b), 0x1p-50, 0x1p-900);
            if (!(den > 1e-40))
                stop = 1.0 > lp.thres;
            else if (ppos > __dadd_rn(b, m))
                stop = true;
            else if (!(ppos < __dsub_rn(b, m)))
                stop = __ddiv_rn(ppos, den) > lp.thres;
        }
    }
    __syncwarp();
    return __any_sync(SG_FULL, stop);
}

/* P_notGuess in the guess loop.  P in [2^E, 2^(E+1)) has the grid
 * u = 2^(E-52), and its binary64 bit pattern counts units of u: subtracting
 * k*u subtracts k from the pattern.  Each lane rounds its term to the grid as
 * P - e does by adding it to 2^E (s1) and to 2^E + u (s2).  The two start
 * with different parity, so an exact tie (a term whose units end in 1/2,
 * rounded to even) leaves them something else than one unit apart.
 * SgGrid: the two addends of P's binade.  A P below 2^-970 or not positive
 * has no such grid: NaNs, whose sums never differ by one unit and whose high
 * word no P exceeds, send every step to the replay.  (A NaN P stays one in
 * either.) */
struct SgGrid {
    double b1, b2;
};

__device__ __forceinline__ SgGrid sg_grid(uint64_t Pb)
{
    const int32_t ph = (int32_t)(Pb >> 32);
    const int32_t hi = ph >= 0x03500000 ? (int32_t)(ph & 0xfff00000) : 0x7fffffff;
    SgGrid g;
    g.b1 = __hiloint2double(hi, 0);
    g.b2 = __hiloint2double(hi, ph >= 0x03500000 ? 1 : 0);
    return g;
}

/* The warp's sum of units given as 26-bit halves per lane. */
__device__ __forceinline__ uint64_t sg_units_sum(uint32_t lo, uint32_t hi)
{
    const uint32_t tlo = __reduce_add_sync(SG_FULL, lo);
    const uint32_t thi = __reduce_add_sync(SG_FULL, hi);
    return (uint64_t)thi * (1u << 26) + tlo;
}

/* The reference's own sequence P -= e (:626, :672, :712) over a step's 32
 * patterns, one IEEE subtraction per pattern in order, evaluated by every
 * lane from the terms staged in shared memory: exact whatever the step
 * holds.  With codewords (hits), P at each of them goes to the list.
 * Returns true when one stops the decode, at pattern T of the line. */
__device__ __forceinline__ bool sg_replay(double e, uint32_t ent, uint32_t hits, uint32_t base, uint64_t& Pb,
                                          SgWarpScratch* ws, uint32_t& T, const SgLineParams& lp, int lane)
{
    ws->es[lane] = e;
    __syncwarp();
    double p = sg_from_bits(Pb);
    if (!hits) {
        const double2* e2 = reinterpret_cast<const double2*>(ws->es);
#pragma unroll
        for (int q = 0; q < 16; q++) {
            const double2 v = e2[q];
            p = __dsub_rn(p, v.x);
            p = __dsub_rn(p, v.y);
        }
    } else {
        int k = 0;
        do {
            const int j = hits ? __ffs(hits) - 1 : 31;
#pragma unroll 4
            for (; k <= j; k++)
                p = __dsub_rn(p, ws->es[k]);
            if (hits && sg_list_hit(ws, lp, ent, p, e, j, lane)) {
                T = base + (uint32_t)j + 1u;
                return true;
            }
            hits &= hits - 1u;
        } while (k < 32);
    }
    Pb = sg_bits(p);
    __syncwarp();
    return false;
}

/* A step that holds codewords and neither ties nor crosses: P at each of
 * them is P less the units up to its lane, and nb after the step.  Returns
 * as sg_replay. */
__device__ __forceinline__ bool sg_sum_hits(double e, uint32_t ent, uint32_t hits, uint32_t lo, uint32_t hi, uint32_t base,
                                            uint64_t& Pb, uint64_t nb, SgWarpScratch* ws, uint32_t& T,
                                            const SgLineParams& lp, int lane)
{
    do {
        const int j = __ffs(hits) - 1;
        const bool in = lane <= j;
        const uint64_t pj = Pb - sg_units_sum(in ? lo : 0u, in ? hi : 0u);
        if (sg_list_hit(ws, lp, ent, sg_from_bits(pj), e, j, lane)) {
            T = base + (uint32_t)j + 1u;
            return true;
        }
        hits &= hits - 1u;
    } while (hits);
    Pb = nb;
    return false;
}

/* Extra results of a line decode run for the adjoint (ADJ = true): the
 * sums over the counted guesses that P_notGuess depends on, and the list.
 * Valid for decodes that stop at a list insertion (Tmax >= 65536). */
struct SgAdjOut {
    double etot;    /* uniform: sum of exp(-PM) over the counted guesses */
    double esort;   /* lanes 2 r and 2 r + 1: the same sum over guesses whose pattern holds sorted position r */
    double pnl;     /* uniform: pNL of the last list insertion (before the 1e-40 clamp) */
    double my_e;    /* lane k < curl: exp(-PM) of list entry k */
    uint32_t my_cm; /* lane k < curl: bits of list entry k */
    uint32_t hdm;   /* hard decision, bit i = position i */
    int32_t curl;
    int32_t myrank; /* lanes i and i + 16: sorted rank of position i */
    /* lanes i and i + 16, when curl > 0: 1/(1 + e^{x_i}), p0_i and p1_i of the soft output */
    double q1, p0, p1;
    bool want_app; /* in: L_APP is needed (otherwise left out) */
    double* bins;  /* in: shared, [9][32]; a lane's sums over guesses holding high position j in row 1 + j */
};

/* Decode one line.  llr: the input LLR of position lane & 15 (all lanes).  enum_tabs: SG_ENUM_NTAB tables of SG_ENUM_LEN entries.
 * etab/ltab: shared-memory copies of the exp/log tables.  U: steps whose
 * terms are worked out together; two where few warps share an SM and the
 * line's own chain of operations is the bound (16 lines in one call 45.2 ->
 * 41.0 us, one codeword on 256 warps 435 -> 423 us), one where the SM is
 * full (twice the registers). */
template <bool ADJ = false, bool CR = false, bool T8 = true, int U = 1>
__device__ __forceinline__ SgLineResult sg_decode_line(double llr, const SgLineParams& lp,
                                                        const uint32_t* __restrict__ enum_tabs,
                                                        SgTab etab, SgTab ltab, SgWarpScratch* ws,
                                                        SgAdjOut* adj = nullptr)
{
    const uint32_t ra = sg_saddr(ws); /* low byte zero */
    const int lane = threadIdx.x & 31;
    const bool act = lane < 16;
    const double a = fabs(llr);
    /* HardDec (:758): 1 unless llr > 0 */
    const uint32_t hdm = __ballot_sync(SG_FULL, !(llr > 0.0)) & 0xffffu;
    /* JacLog(xj) = xj if xj > 50, 0 if xj < -50, else log(1 + e^xj) (:762):
     * lanes 0..15 take -|L| (getPM_HD, :617, :764), lanes 16..31 +|L| (the PM
     * increments).  A NaN, which weights that are 0 or large can make of
     * finite LLRs, stays one; sg_dec_log_pos takes positive numbers only. */
    const double xj = act ? -a : a;
    double ex = CR ? sg_exp_cr(xj, etab) : sg_exp_mid(xj, etab);
    if (!CR && !(a < 700.0))
        ex = sg_exp(xj, etab);
    const double jl = !(xj <= 50) ? xj : (xj < -50 ? 0.0 : sg_dec_log_pos<CR>(1.0 + ex, ltab));
    /* the soft output's exp(LLR) is this exp of lane p + 16 when the LLR is
     * positive, of lane p otherwise (a NaN LLR is its own exp) */
    if (act ? !(llr > 0.0) : (llr > 0.0))
        ws->ex[lane & 15] = llr == llr ? ex : llr;
    const double dl = __dsub_rn(__shfl_down_sync(SG_FULL, jl, 16), jl); /* lanes 0..15: PM increment (getPM, :765) */

    /* QuickSort of |L| ascending (:618): rank of each position.  Lane p and
     * lane p + 16 count the smaller magnitudes among positions 0..7 and
     * 8..15, then add.  The magnitudes are non-negative, so their high 32
     * bits order them unless two are equal there, which leaves a rank
     * unoccupied; only then are the full values compared. */
    int lt = 0;
    {
        const int j0 = lane & 16 ? 8 : 0;
        const uint32_t ah = (uint32_t)(sg_bits(a) >> 32);
#pragma unroll
        for (int k = 0; k < 8; k++)
            lt += __shfl_sync(SG_FULL, ah, j0 + k) < ah;
        lt += __shfl_xor_sync(SG_FULL, lt, 16);
        bool sorted = __reduce_or_sync(SG_FULL, a == a ? 1u << lt : 0u) == 0xffffu && __all_sync(SG_FULL, a == a);
        if (!sorted) {
            lt = 0;
#pragma unroll 1
            for (int k = 0; k < 8; k++)
                lt += __shfl_sync(SG_FULL, a, j0 + k) < a;
            lt += __shfl_xor_sync(SG_FULL, lt, 16);
            sorted = __reduce_or_sync(SG_FULL, 1u << lt) == 0xffffu && __all_sync(SG_FULL, a == a);
        }
        /* ties (and NaN, which no comparison orders) take the exact quicksort */
        if (sorted) {
            if (act) {
                ws->rank[lane] = (uint8_t)lt;
                ws->qa[lt] = a;
            }
        } else {
            if (act) {
                ws->qa[lane] = a;
                ws->perm[lane] = (uint8_t)lane;
            }
            __syncwarp();
            if (lane == 0)
                sg_quicksort16(ws->qa, ws->perm);
            __syncwarp();
            if (act)
                ws->rank[ws->perm[lane]] = (uint8_t)lane;
            __syncwarp();
            lt = ws->rank[lane & 15];
        }
    }
    /* by position: the JacLog terms (A[0..15] is free until the tables below
     * are built); by sorted rank: increments and syndrome columns */
    if (act) {
        ws->A[lane] = jl;
        ws->es[lt] = dl;
        ws->hcol[2 * (lt & 7) + (lt >> 3)] = c_hcol[lane];
    }
    __syncwarp();
    /* getPM_HD: summed in position order */
    double pmhd = 0.0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const double2 v = reinterpret_cast<const double2*>(ws->A)[i];
        pmhd = __dadd_rn(pmhd, v.x);
        pmhd = __dadd_rn(pmhd, v.y);
    }

    /* IC (:619-622): beta = (|L|_(7) - |L|_(0)) / 7, IC = max(round(.), 0) of
     * |L|_(0) / beta - 1.  Only the integer matters, and in single precision
     * the quotient below 64 is good to 1e-4: the divisions are done only near
     * a half, or outside single precision's range. */
    int itab;
    {
        const double a0 = ws->qa[0], d70 = __dsub_rn(ws->qa[7], a0);
        const float df = (float)d70, t = __fdividef(7.0f * (float)a0, df) - 1.0f, k = rintf(t);
        if (df > 1e-30f && df < 1e30f && t < 64.0f && fabsf(t - k) < 0.499f) {
            itab = max((int)k, 0);
        } else {
            const double beta = __ddiv_rn(d70, 7.0);
            itab = max(sg_cvt_i32(round(__dsub_rn(__ddiv_rn(a0, beta), 1.0))), 0);
        }
        itab = min(itab, SG_ENUM_IC_CANON);
    }
    /* exp(-PM) needs no range check when no path metric of the line passes
     * 700: JacLog(-|L|) and increment of a position add up to |L| + log 2 */
    bool wide = false;
    if (!(ws->qa[15] < 42.0)) {
        double pmax = act ? dl : 0.0;
        for (int off = 16; off > 0; off >>= 1)
            pmax = __dadd_rn(pmax, __shfl_xor_sync(SG_FULL, pmax, off));
        wide = !(pmax + pmhd < 700.0);
    }

    /* per-line tables; lane j fills A entries j + 32*i, i = 0..7, and
     * syndrome entries 8*j + k, k = 0..7 */
    {
        double d[8];
#pragma unroll
        for (int b = 0; b < 8; b += 2) {
            const double2 v = reinterpret_cast<const double2*>(ws->es)[b / 2];
            d[b] = v.x;
            d[b + 1] = v.y;
        }
        const uint4 h = *reinterpret_cast<const uint4*>(ws->hcol); /* columns of bits b of the low and high byte: 16-bit b */
        __syncwarp(); /* A, qa read before they are overwritten */
        double v0 = pmhd;
        /* low byte: the hard decision's own syndrome, H = [P^T | I]; both:
         * columns of the lane's bits */
        uint32_t s = c_ptab[hdm & 0xffu] ^ (hdm >> 8);
        const uint32_t h5[5] = {h.y >> 16, h.z, h.z >> 16, h.w, h.w >> 16};
#pragma unroll
        for (int b = 0; b < 5; b++)
            if ((lane >> b) & 1) {
                v0 = __dadd_rn(v0, d[b]);
                s ^= h5[b];
            }
        const double v1 = __dadd_rn(v0, d[5]);
        const double v2 = __dadd_rn(v0, d[6]);
        const double v3 = __dadd_rn(v1, d[6]);
        /* entry i is stored at sg_swz(i) */
        ws->A[sg_swz(lane)] = v0;
        ws->A[sg_swz(lane + 32)] = v1;
        ws->A[sg_swz(lane + 64)] = v2;
        ws->A[sg_swz(lane + 96)] = v3;
        ws->A[sg_swz(lane + 128)] = __dadd_rn(v0, d[7]);
        ws->A[sg_swz(lane + 160)] = __dadd_rn(v1, d[7]);
        ws->A[sg_swz(lane + 192)] = __dadd_rn(v2, d[7]);
        ws->A[sg_swz(lane + 224)] = __dadd_rn(v3, d[7]);
        /* byte k of the 8 entries 8*lane + k: the lane's syndrome (bits 3..7)
         * XOR those of bits 0..2 selected by k, built in place in two 32-bit
         * words by byte permutes */
        const uint32_t lo0 = __byte_perm(s, 0u, 0x0000) ^ __byte_perm(h.x, 0u, 0x0404) ^ __byte_perm(h.x, 0u, 0x2244);
        const uint32_t hi0 = __byte_perm(s, 0u, 0x1111) ^ __byte_perm(h.x, 0u, 0x1414) ^ __byte_perm(h.x, 0u, 0x3344);
        {
            /* stored at sg_swz(8*lane + k) = 8*lane' + (k ^ c): group lane' =
             * lane ^ (g >> 3), bytes permuted by c = g & 7, g the XOR value
             * of the group's bits 5..7 */
            const uint32_t g = (0x14AFEB50u >> (4 * (lane >> 2))) & 15u;
            const uint32_t lo1 = lo0 ^ __byte_perm(h.y, 0u, 0x0000);
            const uint32_t sel = 0x3210u ^ ((g & 3u) * 0x1111u);
            const uint32_t w0 = __byte_perm(lo0, 0u, sel), w1 = __byte_perm(lo1, 0u, sel);
            reinterpret_cast<uint2*>(ws->synlo)[lane ^ (g >> 3)] = (g & 4u) ? make_uint2(w1, w0) : make_uint2(w0, w1);
        }
        reinterpret_cast<uint2*>(ws->synhi)[lane] = make_uint2(hi0, hi0 ^ __byte_perm(h.y, 0u, 0x1111));
        if (lane < 9)
            ws->dz[lane] = lane ? ws->es[lane + 7] : 0.0;
    }
    /* the sorted magnitudes are done with: qa keeps the input LLRs for the soft
     * output */
    if (act)
        ws->qa[lane] = llr;
    if (lane == 0) {
        ws->curl = 0;
        ws->pnl = 0.0;
        ws->ppos = 0.0;
        ws->hdm = hdm;
        ws->itab = itab;
    }
    __syncwarp();

    /* Guess loop (:624-744), 32 patterns a step.  From pattern `special` on
     * a step may hold patterns with three or more high positions, end at the
     * Tmax cut, or (special = 0) hold terms below the normal range. */
    uint32_t idx = (uint32_t)itab * SG_ENUM_LEN + (uint32_t)lane; /* low 16 bits: the pattern, low 5: the lane */
    const uint32_t special =
        (uint32_t)itab * SG_ENUM_LEN + (wide ? 0u : min(lp.meta->h3[itab], lp.meta->lim[itab]) & ~31u);
    const uint32_t ea = sg_saddr(etab.t);
    uint64_t Pb = 0x3ff0000000000000ull; /* P_notGuess, as its bit pattern */
    SgGrid g = sg_grid(Pb);
    uint32_t T = 0;
    double adj_tot = 0.0, adj_r[ADJ ? 16 : 1];
#pragma unroll
    for (int r = 0; r < (ADJ ? 8 : 1); r++)
        adj_r[r] = 0.0;
    if (ADJ)
#pragma unroll
        for (int r = 1; r < 9; r++)
            adj->bins[32 * r + lane] = 0.0;
    /* A guess that entered P_notGuess.  The sums of the low positions stay in
     * registers, a pattern holding any of them; of the high ones it holds at
     * most two but for special steps, so theirs are in shared memory, picked
     * by the entry's offsets (row 0: none). */
    auto adj_add = [&](double e, uint32_t ent, bool general) {
        adj_tot += e;
        const uint32_t m = sg_swz(ent & 0xffu);
#pragma unroll
        for (int r = 0; r < (ADJ ? 8 : 1); r++)
            if ((m >> r) & 1u)
                adj_r[r] += e;
        double* bin = adj->bins + lane;
        bin[((ent >> 16) & 0xffu) * 4u] += e;
        bin[(ent >> 24) * 4u] += e;
        if (general) {
            uint32_t rest = (ent >> 8) & 0xffu;
            rest &= rest - 1u;
            rest &= rest - 1u;
            for (; rest; rest &= rest - 1u)
                bin[32 * __ffs(rest)] += e;
        }
    };
    /* path metric (up to two high positions) and syndrome of an entry: the
     * high positions in ascending order, from the entry's offsets (offset 0
     * reads dz[0] = 0, and pm + 0 = pm since pm >= +0) */
    auto metric = [&](uint32_t ent) {
        double pm = sg_lds_f64<offsetof(SgWarpScratch, A)>(ra + (ent & 0xffu) * 8u);
        pm = __dadd_rn(pm, sg_lds_f64<offsetof(SgWarpScratch, dz)>(__byte_perm(ent, ra, 0x7652)));
        return __dadd_rn(pm, sg_lds_f64<offsetof(SgWarpScratch, dz)>(__byte_perm(ent, ra, 0x7653)));
    };
    auto is_codeword = [&](uint32_t ent) {
        return sg_lds_u8<offsetof(SgWarpScratch, synlo)>(__byte_perm(ent, ra, 0x7650)) ==
               sg_lds_u8<offsetof(SgWarpScratch, synhi)>(__byte_perm(ent, ra, 0x7651));
    };
    /* Units of a lane's term on the grid, as 26-bit halves; true when it
     * ties or leaves the binade. */
    auto term_units = [&](double e, uint32_t& lo, uint32_t& hi) {
        const double s1 = __dadd_rn(g.b1, e), s2 = __dadd_rn(g.b2, e);
        const uint32_t l1 = (uint32_t)__double2loint(s1);
        const uint32_t dh = (uint32_t)(__double2hiint(s1) - __double2hiint(g.b1));
        lo = l1 & 0x3ffffffu;
        hi = __funnelshift_r(l1, dh, 26);
        return (uint32_t)__double2loint(s2) - l1 != 1u || dh >= 0x100000u;
    };
    for (;;) {
        uint32_t ent, lo, hi;
        double e;
        uint64_t tot;
        bool out = false, hit, tie;
        const SgExpK ek = sg_exp_k();
        /* P is moved by the step's units.  2^26 in place of the upper half of
         * a lane that cannot be summed, or that holds a codeword, makes them
         * 2^52 or more, which leaves the binade. */
        if constexpr (U == 2) {
            /* two steps at a time: their terms and sums do not depend on each
             * other, only the tests do */
#pragma unroll 1
            while (idx + 32u < special) {
                const uint32_t enta = __ldg(enum_tabs + idx), entb = __ldg(enum_tabs + idx + 32u);
                const double pma = metric(enta), pmb = metric(entb);
                const bool hita = is_codeword(enta), hitb = is_codeword(entb);
                const double ea_ = CR || !T8 ? sg_dec_exp_neg<CR>(-pma, etab) : sg_exp_neg_k(-pma, ea, ek);
                const double eb_ = CR || !T8 ? sg_dec_exp_neg<CR>(-pmb, etab) : sg_exp_neg_k(-pmb, ea, ek);
                uint32_t loa, hia, lob, hib;
                const bool tiea = term_units(ea_, loa, hia), tieb = term_units(eb_, lob, hib);
                const uint64_t tota = sg_units_sum(loa, (tiea || hita) ? 0x4000000u : hia);
                const uint64_t totb = sg_units_sum(lob, (tieb || hitb) ? 0x4000000u : hib);
                const uint64_t pa = Pb - tota, pb = pa - totb;
                if ((int32_t)(pa >> 32) <= __double2hiint(g.b1)) {
                    Pb = pa;
                    tot = tota;
                    ent = enta;
                    e = ea_;
                    hit = hita;
                    tie = tiea;
                    lo = loa;
                    hi = hia;
                    out = true;
                    break;
                }
                if (ADJ)
                    adj_add(ea_, enta, false);
                idx += 32u;
                Pb = pb;
                if ((int32_t)(pb >> 32) <= __double2hiint(g.b1)) {
                    tot = totb;
                    ent = entb;
                    e = eb_;
                    hit = hitb;
                    tie = tieb;
                    lo = lob;
                    hi = hib;
                    out = true;
                    break;
                }
                if (ADJ)
                    adj_add(eb_, entb, false);
                idx += 32u;
            }
        }
#pragma unroll 1
        while ((U == 1 || !out) && idx < special) {
            ent = __ldg(enum_tabs + idx);
            const double pm = metric(ent);
            hit = is_codeword(ent);
            e = CR || !T8 ? sg_dec_exp_neg<CR>(-pm, etab) : sg_exp_neg_k(-pm, ea, ek);
            tie = term_units(e, lo, hi);
            tot = sg_units_sum(lo, (tie || hit) ? 0x4000000u : hi);
            Pb -= tot;
            if ((int32_t)(Pb >> 32) <= __double2hiint(g.b1)) {
                out = true;
                break;
            }
            if (ADJ)
                adj_add(e, ent, false);
            idx += 32u;
        }
        if (!out) {
            const uint32_t end = (uint32_t)ws->itab * SG_ENUM_LEN + lp.meta->lim[ws->itab];
            if (idx - (uint32_t)lane >= end) {
                T = lp.meta->lim[ws->itab];
                break;
            }
            ent = __ldg(enum_tabs + idx);
            double pm = metric(ent);
            uint32_t rest = (ent >> 8) & 0xffu;
            rest &= rest - 1u;
            rest &= rest - 1u;
            while (rest) {
                pm = __dadd_rn(pm, ws->dz[__ffs(rest)]);
                rest &= rest - 1u;
            }
            hit = idx < end && is_codeword(ent);
            e = idx < end ? sg_dec_exp<CR>(-pm, etab) : 0.0;
            tie = term_units(e, lo, hi);
            tot = sg_units_sum(lo, (tie || hit) ? 0x4000000u : hi);
            Pb -= tot;
            if ((int32_t)(Pb >> 32) > __double2hiint(g.b1)) {
                if (ADJ)
                    adj_add(e, ent, true);
                idx += 32u;
                continue;
            }
        }
        Pb += tot;
        const uint32_t hits = __ballot_sync(SG_FULL, hit);
        const uint32_t base = (idx - (uint32_t)lane) & (SG_ENUM_LEN - 1u);
        bool done;
        uint64_t nb = 0;
        /* a step without codewords failed the sum because it ties or crosses */
        bool exact = hits != 0u && !__any_sync(SG_FULL, tie);
        if (exact) {
            nb = Pb - sg_units_sum(lo, hi);
            exact = (int32_t)(nb >> 32) > __double2hiint(g.b1);
        }
        if (exact) {
            done = sg_sum_hits(e, ent, hits, lo, hi, base, Pb, nb, ws, T, lp, lane);
        } else {
            done = sg_replay(e, ent, hits, base, Pb, ws, T, lp, lane);
            g = sg_grid(Pb);
        }
        if (ADJ && (!done || (idx & (SG_ENUM_LEN - 1u)) < T))
            adj_add(e, ent, true);
        if (done)
            break;
        idx += 32u;
    }
    if (ADJ) {
        /* sums over the warp: halving exchanges, which leave lanes 2 r and
         * 2 r + 1 with sorted position r's (15 exchanges and an addition
         * instead of 16 full reductions, in the same order) */
        for (int off = 16; off > 0; off >>= 1)
            adj_tot += __shfl_xor_sync(SG_FULL, adj_tot, off);
#pragma unroll
        for (int r = 8; r < (ADJ ? 16 : 8); r++)
            adj_r[r] = adj->bins[32 * (r - 7) + lane];
#pragma unroll
        for (int h = ADJ ? 8 : 0; h > 0; h >>= 1) {
            const bool up = (lane & (2 * h)) != 0;
#pragma unroll
            for (int r = 0; r < h; r++) {
                const double give = up ? adj_r[r] : adj_r[r + h], keep = up ? adj_r[r + h] : adj_r[r];
                adj_r[r] = keep + __shfl_xor_sync(SG_FULL, give, 2 * h);
            }
        }
        const double mine_r = adj_r[0] + __shfl_xor_sync(SG_FULL, adj_r[0], 1);
        adj->etot = adj_tot;
        adj->esort = mine_r;
        const int curl = ws->curl;
        adj->pnl = ws->pnl;
        adj->my_e = lane < curl ? ws->lst_e[lane] : 0.0;
        /* codeword bits of the list entries (AddTEP, :761): position i flips
         * when its sorted rank is in the pattern */
        adj->my_cm = 0u;
        for (int k = 0; k < curl; k++) {
            const uint32_t cm = hdm ^ (__ballot_sync(SG_FULL, act && ((ws->lst_m[k] >> ws->rank[lane & 15]) & 1u)) & 0xffffu);
            if (lane == k)
                adj->my_cm = cm;
        }
        adj->hdm = hdm;
        adj->curl = curl;
        adj->myrank = ws->rank[lane & 15];
    }

    /* Soft output (:536-577) */
    SgLineResult res;
    res.T = T;
    const int curl = ws->curl;
    res.ncw = curl;
    /* the input LLR of position lane & 15, kept in qa during the loop */
    const double x = ws->qa[lane & 15];
    double lapp = x, le = 0.0;
    if (curl != 0) {
        /* every lane works on position lane & 15; lanes 0..15 then take
         * log(p0), lanes 16..31 log(p1) */
        const int pos = lane & 15;
        const uint32_t rk = ws->rank[pos], hb = ws->hdm >> pos;
        const double pnlc = fmax(ws->pnl, 1e-40);
        /* 1/(1 + e^L) and its complement are at most 1, so only the lower
         * clamps of :541-:548 can act */
        const double q1 = __drcp_rn(__dadd_rn(1.0, ws->ex[pos]));
        const double pp0 = fmax(__dsub_rn(1.0, q1), 1e-40), pp1 = fmax(q1, 1e-40);
        double p1 = 0.0, p0 = 0.0;
        for (int j = 0; j < curl; j++) {
            /* AddTEP (:761): position i flips when its sorted rank is in the
             * pattern.  The reference adds c * p_j and (1 - c) * p_j; the
             * zero one changes nothing. */
            const double pj = ws->lst_e[j];
            if (((ws->lst_m[j] >> rk) ^ hb) & 1u)
                p1 = __dadd_rn(p1, pj);
            else
                p0 = __dadd_rn(p0, pj);
        }
        p0 = __dadd_rn(p0, __dmul_rn(pnlc, pp0));
        p1 = __dadd_rn(p1, __dmul_rn(pnlc, pp1));
        if (ADJ) {
            adj->q1 = q1;
            adj->p0 = p0;
            adj->p1 = p1;
        }
        if (!ADJ || adj->want_app) {
            const double lg = sg_dec_log_pos<CR>(fmax(act ? p0 : p1, 1e-40), ltab);
            lapp = __dsub_rn(lg, __shfl_down_sync(SG_FULL, lg, 16));
            le = __dsub_rn(lapp, x);
        }
    }
    res.lapp = lapp;
    res.le = le;
    res.hdword = __ballot_sync(SG_FULL, act && !(lapp > 0.0)) & 0xffffu;
    __syncwarp();
    return res;
}
