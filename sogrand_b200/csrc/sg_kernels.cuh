/* sg_kernels.cuh -- the decoder kernels, instantiated by sg_api.cu with the
 * table-driven exp/log and by sg_cr.cu with the correctly rounded ones: two
 * translation units, since the correctly rounded routines take their
 * constants as launch arguments and the table-driven ones as literals, and
 * built side by side.
 *
 *   sg_decode_kernel   the whole iterative decode of a codeword per CTA
 *                      (SOGRAND_C/cubic_decoder_final.c:119-289): the
 *                      extrinsic cube stays in shared memory for all
 *                      iterations, the channel cube too (one bulk
 *                      asynchronous copy, cp.async.bulk on an mbarrier) or in
 *                      L2; the warps take the 256 lines of a phase from a
 *                      shared counter and decode one line each
 *                      (sg_line.cuh); after every phase one warp runs the
 *                      early-termination test on the 256 hard-decision words.
 *   sg_persist_kernel  the batched form (sg_persist.cuh)
 *   sg_bitso_kernel    SOGRAND_bitSO on independent lines, one warp per line.
 *
 * Built with -fmad=false: no floating-point contraction anywhere, as in the
 * reference's plain gcc build; the exp/log routines use explicit FMAs.
 */
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include "../../include/sogrand_b200.h"
#include "sg_code.h"
#include "sg_enum.h"
#include "sg_line.cuh"
#include "sg_line16.cuh"
#include "sg_math.h"

#define SG_THREADS 256
/* Bounded device-side waits.  The limit of a wait that can give up (the
 * bulk-copy wait here, the persistent decoder's idle rounds) is a launch
 * argument, SG_WAIT_LIMIT_DEFAULT unless sg_set_wait_limit() changed it.
 * After a bulk-copy wait gave up, the copy may still be writing into the
 * CTA's shared memory: the CTA waits for it again, up to SG_DRAIN_LIMIT
 * polls, before it releases that memory. */
#define SG_WAIT_LIMIT_DEFAULT (1ll << 22)
#define SG_DRAIN_LIMIT (1ll << 26)

static __device__ const double g_etab[SG_EXP_TAB_LEN] = SG_EXP_TAB_INIT;
static __device__ const double g_ltab[SG_LOG_TAB_LEN] = SG_LOG_TAB_INIT;

/* ------------------------------------------------------------ device -- */

struct SgDecodeArgs {
    const double* llr;
    uint8_t* bits;
    double* lapp;
    sg_cw_stats* stats;
    const uint32_t* enum_tabs;
    unsigned int* err;
    double* ckpt; /* nullable: [n_cw][3*imax][4096], L_E entering each phase */
    sg_decode_summary* sum; /* nullable: totals, added to by every codeword */
    const uint8_t* ref;     /* nullable: info bits to compare with, for sum */
    unsigned long long n_cw;
    long long wait_limit; /* polls or idle rounds before a bounded wait gives up */
    int32_t L;
    int32_t imax;
    int32_t use_bulk;
    int32_t pad;
    double thres;
    double alpha[SG_MAX_PHASES];
    SgK k; /* constants of exp and log */
    sg_order_meta meta;
};

/* Poll the mbarrier for phase `parity` at most `limit` times; 1 when it
 * completed. */
__device__ __forceinline__ uint32_t sg_mbar_wait(uint32_t mbar, uint32_t parity, long long limit)
{
    uint32_t ok = 0;
    for (long long it = 0; it < limit && !ok; it++) {
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(ok)
            : "r"(mbar), "r"(parity)
            : "memory");
    }
    return ok;
}

/* Outputs of a codeword, by one warp: bytes `lane` and `lane + 32` of its info
 * bits (b0, b1), its statistics, and its share of the totals.  Iterations are
 * multiples of 0.5, their total below 2^52, so that the atomic double
 * additions are exact and their order does not matter.  Totals kept here
 * need neither the per-codeword statistics in memory nor a kernel that reads
 * them. */
__device__ __forceinline__ void sg_cw_output(const SgDecodeArgs& args, unsigned long long cw, uint32_t b0, uint32_t b1,
                                             const sg_cw_stats& st, int lane)
{
    if (args.bits) {
        args.bits[cw * SG_INFO_BYTES + lane] = (uint8_t)b0;
        args.bits[cw * SG_INFO_BYTES + 32 + lane] = (uint8_t)b1;
    }
    if (lane == 0 && args.stats)
        args.stats[cw] = st;
    if (args.sum) {
        uint32_t e = 0;
        if (args.ref) {
            const uint8_t* r = args.ref + cw * SG_INFO_BYTES + lane;
            e = __popc(b0 ^ r[0]) + __popc(b1 ^ r[32]);
        }
        e = __reduce_add_sync(SG_FULL, e);
        if (lane == 0) {
            typedef unsigned long long u64;
            sg_decode_summary* s = args.sum;
            atomicAdd((u64*)&s->blocks, 1ull);
            uint64_t* what = st.converged == 1 ? &s->converged
                                               : (st.converged == -1 ? &s->nonfinite
                                                                     : (st.converged == -2 ? &s->timeouts : nullptr));
            if (what)
                atomicAdd((u64*)what, 1ull);
            atomicAdd((u64*)&s->total_ng, (u64)st.ng);
            atomicAdd((u64*)&s->total_ng_p, (u64)st.ng_p);
            atomicAdd(&s->total_iterations, st.iterations);
            if (args.ref) {
                atomicAdd((u64*)&s->bits_compared, (u64)SG_INFO_BITS);
                atomicAdd((u64*)&s->bit_errors, (u64)e);
                atomicAdd((u64*)&s->block_errors, e ? 1ull : 0ull);
            }
            const unsigned int err = *(volatile const unsigned int*)args.err;
            if (err)
                atomicOr(&s->device_error, err);
        }
    }
}

/* Outputs of a codeword that is not decoded: zero bits and statistics with
 * the given converged code (-1 non-finite input, -2 a wait gave up).
 * Called by the whole CTA. */
__device__ __forceinline__ void sg_cw_not_decoded(const SgDecodeArgs& args, unsigned long long cw, int code)
{
    if (threadIdx.x < 32) {
        sg_cw_stats st;
        st.iterations = 0;
        st.ng = 0;
        st.ng_p = 0;
        st.converged = code;
        st.phases = 0;
        sg_cw_output(args, cw, 0u, 0u, st, (int)threadIdx.x);
    }
}

/* Shared memory of a decode CTA.  With LCH_SMEM the channel cube is staged
 * here by one bulk copy; otherwise each line reads its 16 channel LLRs from
 * global memory (L2-resident) once per phase. */
template <int NW, bool LCH_SMEM, int LPW = 1> /* LPW: lines decoded per warp at a time */
struct SgCwSmem {
    alignas(16) double lch[LCH_SMEM ? SG_CUBE : 2]; /* bulk-copy destination */
    double le[SG_CUBE];
    /* eight copies where the CTAs per SM that this costs are outweighed:
     * w10-l2-g2 falls from two CTAs to one, and 12 000 codewords at 2 dB from
     * 507 to 406 ms */
    static constexpr bool T8 = NW * LPW >= 16 && !LCH_SMEM;
    SgEtab<T8> etab;
    alignas(16) double ltab[SG_LOG_TAB_LEN];
    SgWarpScratch ws[NW * LPW];
    uint16_t hdw[256];
    unsigned long long mbar;
    unsigned long long ng;
    unsigned int ngmax;
    int line_next;
    int conv;
    int bad;
};

/* Cube index of bit `i` of line `l` in phase `axis` (lines of the reference's
 * column phase run along the stride-1 index, rows along stride 16, slices
 * along stride 256; cubic_decoder_final.c:157-247). */
__device__ __forceinline__ int sg_pos(int axis, int l, int i)
{
    const int a = l >> 4, b = l & 15;
    if (axis == 0)
        return a * 256 + b * 16 + i;
    if (axis == 1)
        return a * 256 + i * 16 + b;
    return i * 256 + a * 16 + b;
}

/* Early termination (cubic_decoder_final.c:317-391) on the 256 line words
 * of the phase just run: the hard decisions form a product codeword iff
 * every word is a component codeword and the words satisfy the component
 * parity equations along both other axes (bitwise).  Warp-wide. */
__device__ __forceinline__ bool sg_is_codeword(const uint16_t* hdw, int lane)
{
    bool bad = false;
    for (int q = lane; q < 256; q += 32) {
        const uint32_t x = hdw[q];
        bad |= ((x >> 8) & 0xffu) != c_ptab[x & 0xffu];
    }
    for (int q = lane; q < 128; q += 32) {
        const int a = q >> 3, j = q & 7;
        uint32_t acc = 0;
#pragma unroll
        for (int b = 0; b < 8; b++)
            if ((c_prow[b] >> j) & 1u)
                acc ^= hdw[a * 16 + b];
        bad |= acc != hdw[a * 16 + 8 + j];
    }
    for (int q = lane; q < 128; q += 32) {
        const int b = q >> 3, j = q & 7;
        uint32_t acc = 0;
#pragma unroll
        for (int a = 0; a < 8; a++)
            if ((c_prow[a] >> j) & 1u)
                acc ^= hdw[a * 16 + b];
        bad |= acc != hdw[(8 + j) * 16 + b];
    }
    return !__any_sync(SG_FULL, bad);
}

__device__ __forceinline__ uint32_t sg_smem_u32(const void* p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

extern __shared__ __align__(1024) unsigned char sg_smem_raw[];

template <int NW, bool LCH_SMEM, int MINB, int G, bool CR, int LPW = 1>
__global__ void __launch_bounds__(NW * 32, MINB) sg_decode_kernel(const __grid_constant__ SgDecodeArgs args)
{
    constexpr int NT = NW * 32;
    SgCwSmem<NW, LCH_SMEM, LPW>& S = *reinterpret_cast<SgCwSmem<NW, LCH_SMEM, LPW>*>(sg_smem_raw);
    constexpr bool T8 = SgCwSmem<NW, LCH_SMEM, LPW>::T8;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool use_bulk = LCH_SMEM && args.use_bulk;
    sg_etab_fill<CR, T8>(S.etab, g_etab, tid, NT);
    for (int i = tid; i < SG_LOG_TAB_LEN; i += NT)
        S.ltab[i] = g_ltab[i];
    const uint32_t mbar = sg_smem_u32(&S.mbar);
    if (tid == 0 && use_bulk) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    uint32_t phase_bit = 0;
    const SgTab etab = sg_etab_of<CR, T8>(S.etab, args.k.v), ltab{S.ltab, args.k.v};
    SgLineParams lp;
    lp.L = args.L;
    lp.meta = &args.meta;
    lp.thres = args.thres;

    for (unsigned long long cw = blockIdx.x; cw < args.n_cw; cw += gridDim.x) {
        const double* g = args.llr + cw * SG_CUBE;
        if (use_bulk) {
            if (tid == 0) {
                /* order earlier generic-proxy reads of lch before the async write */
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar),
                             "r"((uint32_t)(SG_CUBE * 8))
                             : "memory");
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        sg_smem_u32(S.lch)),
                    "l"(g), "r"((uint32_t)(SG_CUBE * 8)), "r"(mbar)
                    : "memory");
            }
        } else if (LCH_SMEM) {
            for (int i = tid; i < SG_CUBE; i += NT)
                S.lch[i] = g[i];
        }
        for (int i = tid; i < SG_CUBE; i += NT)
            S.le[i] = 0.0;
        if (tid == 0) {
            S.ng = 0;
            S.conv = 0;
            S.bad = 0;
        }
        if (use_bulk && tid == 0) {
            if (!sg_mbar_wait(mbar, phase_bit, args.wait_limit)) {
                /* gave up: report it, then let the copy land before this
                 * CTA's shared memory is reused or released */
                atomicOr(args.err, 1u);
                if (!sg_mbar_wait(mbar, phase_bit, SG_DRAIN_LIMIT))
                    atomicOr(args.err, 2u);
                S.bad = 2;
            }
        }
        phase_bit ^= 1u;
        __syncthreads();
        if (S.bad == 2) {
            /* this codeword and the CTA's later ones are reported as not
             * decoded (converged = -2) */
            for (unsigned long long c = cw; c < args.n_cw; c += gridDim.x)
                sg_cw_not_decoded(args, c, -2);
            return;
        }
        bool nonfinite = false;
        for (int i = tid; i < SG_CUBE; i += NT)
            nonfinite |= !isfinite(LCH_SMEM ? S.lch[i] : __ldg(g + i));
        if (__syncthreads_or(nonfinite)) {
            sg_cw_not_decoded(args, cw, -1);
            __syncthreads();
            continue;
        }

        int phases = 0;
        unsigned long long ng_p = 0;
        int axis_last = 0;
        bool conv = false;
        for (int iter = 1; iter <= args.imax && !conv; iter++) {
            for (int axis = 0; axis < 3 && !conv; axis++) {
                const double alpha = args.alpha[3 * (iter - 1) + axis];
                if (tid == 0) {
                    S.line_next = 0;
                    S.ngmax = 0;
                }
                __syncthreads();
                if constexpr (LPW == 2) {
                    /* the warp takes two lines at a time, one per half, and
                     * decodes them in lockstep (sg_line16.cuh) */
                    const int hb = lane & 16, sl = lane & 15;
                    SgWarpScratch* wsl = &S.ws[2 * warp + (hb >> 4)];
                    for (;;) {
                        int l = 0;
                        if (lane == 0)
                            l = atomicAdd(&S.line_next, 2);
                        l = __shfl_sync(SG_FULL, l, 0) + (hb >> 4);
                        if (l >= 256) /* 256 lines: both halves leave together */
                            break;
                        const int pos = sg_pos(axis, l, sl);
                        const double le0 = S.le[pos];
                        const double v = __dadd_rn(LCH_SMEM ? S.lch[pos] : __ldg(g + pos), __dmul_rn(alpha, le0));
                        if (args.ckpt)
                            args.ckpt[(cw * (3ull * args.imax) + 3 * (iter - 1) + axis) * SG_CUBE + pos] = le0;
                        const SgLineResult r = sg_decode_line16<G, CR>(v, lp, args.enum_tabs, etab, ltab, wsl);
                        S.le[pos] = r.le;
                        if (args.lapp)
                            args.lapp[cw * SG_CUBE + pos] = r.lapp;
                        if (sl == 0) {
                            S.hdw[l] = (uint16_t)r.hdword;
                            atomicAdd(&S.ng, (unsigned long long)r.T);
                            atomicMax(&S.ngmax, r.T);
                        }
                    }
                } else {
                    for (;;) {
                        int l = 0;
                        if (lane == 0)
                            l = atomicAdd(&S.line_next, 1);
                        l = __shfl_sync(SG_FULL, l, 0);
                        if (l >= 256)
                            break;
                        const int pos = sg_pos(axis, l, lane & 15);
                        /* L_ch + (alpha*L_E), lanes p and p + 16 alike */
                        const double le0 = S.le[pos];
                        const double v = __dadd_rn(LCH_SMEM ? S.lch[pos] : __ldg(g + pos), __dmul_rn(alpha, le0));
                        if (args.ckpt && lane < 16)
                            args.ckpt[(cw * (3ull * args.imax) + 3 * (iter - 1) + axis) * SG_CUBE + pos] = le0;
                        const SgLineResult r =
                            sg_decode_line<false, CR, T8>(v, lp, args.enum_tabs, etab, ltab, &S.ws[warp]);
                        if (lane < 16) {
                            S.le[pos] = r.le;
                            if (args.lapp)
                                args.lapp[cw * SG_CUBE + pos] = r.lapp;
                        }
                        if (lane == 0) {
                            S.hdw[l] = (uint16_t)r.hdword;
                            atomicAdd(&S.ng, (unsigned long long)r.T);
                            atomicMax(&S.ngmax, r.T);
                        }
                    }
                }
                __syncthreads();
                phases++;
                axis_last = axis;
                ng_p += S.ngmax;
                if (warp == 0) {
                    const bool c = sg_is_codeword(S.hdw, lane);
                    if (lane == 0)
                        S.conv = c;
                }
                __syncthreads();
                conv = S.conv != 0;
            }
        }

        /* hard_decision (:393-415): info bit b = s*64 + r*8 + c is the sign of
         * L_APP at cube index s*256 + r*16 + c; packed MSB first (:272-280) */
        if (warp == 0) {
            uint32_t byte[2];
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
                uint32_t v = 0;
                for (int q = 0; q < 8; q++) {
                    const int b = (lane + 32 * h) * 8 + q;
                    const int p = (b >> 6) * 256 + ((b >> 3) & 7) * 16 + (b & 7);
                    int l, bit;
                    if (axis_last == 0) {
                        l = (p >> 8) * 16 + ((p >> 4) & 15);
                        bit = p & 15;
                    } else if (axis_last == 1) {
                        l = (p >> 8) * 16 + (p & 15);
                        bit = (p >> 4) & 15;
                    } else {
                        l = ((p >> 4) & 15) * 16 + (p & 15);
                        bit = p >> 8;
                    }
                    v = (v << 1) | ((S.hdw[l] >> bit) & 1u);
                }
                (h ? byte[1] : byte[0]) = v;
            }
            sg_cw_stats st;
            st.iterations = 0.5 * phases;
            st.ng = S.ng;
            st.ng_p = ng_p;
            st.converged = conv ? 1 : 0;
            st.phases = phases;
            sg_cw_output(args, cw, byte[0], byte[1], st, lane);
        }
        __syncthreads();
    }
}

#include "sg_persist.cuh"
#include "sg_cluster.cuh"

template <int NW, bool T8>
struct SgLineSmem {
    SgEtab<T8> etab;
    alignas(16) double ltab[SG_LOG_TAB_LEN];
    int next; /* of the CTA's lines, the next to hand out */
    SgWarpScratch ws[NW];
};

/* SOGRAND_bitSO on independent lines, one per warp.  CTA b takes the lines
 * [b * per, (b + 1) * per), its warps from a shared counter: the searches'
 * lengths differ by an order of magnitude, and fixed shares would leave warps
 * idle. */
template <int NW, bool T8, bool CR>
__global__ void __launch_bounds__(NW * 32, NW == 16 ? 2 : 1)
    sg_bitso_kernel(const double* __restrict__ llr, unsigned long long n_lines, unsigned long long per, int32_t L,
                    double thres, double* lapp, double* le, int32_t* nguess, int32_t* ncw, const uint32_t* enum_tabs,
                    const __grid_constant__ SgK k, const __grid_constant__ sg_order_meta meta)
{
    SgLineSmem<NW, T8>& S = *reinterpret_cast<SgLineSmem<NW, T8>*>(sg_smem_raw);
    const SgTab etab = sg_etab_of<CR, T8>(S.etab, k.v), ltab{S.ltab, k.v};
    const SgLineParams lp{L, thres, &meta};
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    sg_etab_fill<CR, T8>(S.etab, g_etab, tid, NW * 32);
    for (int i = tid; i < SG_LOG_TAB_LEN; i += NW * 32)
        S.ltab[i] = g_ltab[i];
    if (tid == 0) {
        S.next = 0;
    }
    __syncthreads();
    const unsigned long long l0 = blockIdx.x * per, l1 = l0 + per < n_lines ? l0 + per : n_lines;
    for (;;) {
        int q = 0;
        if (lane == 0)
            q = atomicAdd(&S.next, 1);
        const unsigned long long l = l0 + (unsigned)__shfl_sync(SG_FULL, q, 0);
        if (l >= l1)
            break;
        const double v = llr[l * 16 + (lane & 15)];
        if (__any_sync(SG_FULL, !isfinite(v))) { /* not decoded: NaN out, N_guess -1 */
            if (lane < 16) {
                lapp[l * 16 + lane] = __longlong_as_double(0x7ff8000000000000ll);
                le[l * 16 + lane] = __longlong_as_double(0x7ff8000000000000ll);
            }
            if (lane == 0) {
                nguess[l] = -1;
                if (ncw)
                    ncw[l] = 0;
            }
            continue;
        }
        const SgLineResult r = sg_decode_line<false, CR, T8, NW <= 4 ? 2 : 1>(v, lp, enum_tabs, etab, ltab, &S.ws[warp]);
        if (lane < 16) {
            lapp[l * 16 + lane] = r.lapp;
            le[l * 16 + lane] = r.le;
        }
        if (lane == 0) {
            nguess[l] = (int32_t)r.T;
            if (ncw)
                ncw[l] = r.ncw;
        }
    }
}

/* SG_TU_CR: the math of this translation unit's instantiations. */
#ifndef SG_TU_CR
#define SG_TU_CR false
#endif

/* Decoder kernel configurations: warps per codeword CTA, channel cube in
 * shared memory (bulk copy) or read from global memory, minimum resident
 * CTAs per SM for the register budget, and lines per warp (1: 32 lanes per
 * line, sg_line.cuh; 2: 16 lanes per line and G patterns per lane,
 * sg_line16.cuh).  A one-line kernel has two names: X decodes every batch
 * with it, X-g2 hands small batches to the cluster configurations below. */
struct SgVariant {
    const char* name;
    int nw;
    bool lch_smem;
    bool clusters; /* small batches go to clusters */
    size_t smem;
    const void* fn;
};

#define SG_VARIANT(NW, L, M, CL, NAME) \
    { NAME, NW, L, CL, sizeof(SgCwSmem<NW, L>), (const void*)sg_decode_kernel<NW, L, M, 1, SG_TU_CR> }
#define SG_VARIANT_L2(NW, M, G, NAME) \
    { NAME, NW, false, false, sizeof(SgCwSmem<NW, false, 2>), \
      (const void*)sg_decode_kernel<NW, false, M, G, SG_TU_CR, 2> }
static const SgVariant k_variants[] = {
    SG_VARIANT(8, false, 3, false, "w8-gmem"),
    SG_VARIANT(8, true, 2, false, "w8-smem"),
    SG_VARIANT(12, true, 2, false, "w12-smem"),
    SG_VARIANT(16, false, 2, false, "w16-gmem"),
    SG_VARIANT(16, false, 2, true, "w16-gmem-g2"),
    SG_VARIANT(8, false, 3, true, "w8-gmem-g2"),
    SG_VARIANT(12, true, 2, true, "w12-smem-g2"),
    SG_VARIANT_L2(8, 2, 2, "w8-l2-g2"),
    SG_VARIANT_L2(8, 2, 4, "w8-l2-g4"),
    SG_VARIANT_L2(10, 1, 2, "w10-l2-g2"),
    SG_VARIANT_L2(16, 1, 2, "w16-l2-g2"),
    SG_VARIANT(8, true, 2, true, "w8-smem-g2"),
};
#define SG_NVARIANTS ((int)(sizeof(k_variants) / sizeof(k_variants[0])))

#define SG_VARIANT_DEFAULT 4 /* w16-gmem-g2 */

/* Batched persistent decoder configurations: warps per CTA (one CTA per
 * SM), codeword slots per CTA; names as above. */
struct SgPVariant {
    const char* name;
    int nw;
    int slots;
    bool clusters;
    size_t smem;
    const void* fn;
};
#define SG_PVARIANT(NW, C, CL, NAME) \
    { NAME, NW, C, CL, sizeof(SgPersistSmem<NW, C>), (const void*)sg_persist_kernel<NW, C, SG_TU_CR> }
static const SgPVariant k_pvariants[] = {
    SG_PVARIANT(24, 3, false, "p24x3"),
    SG_PVARIANT(28, 3, false, "p28x3"),
    SG_PVARIANT(16, 3, false, "p16x3"),
    SG_PVARIANT(20, 4, false, "p20x4"),
    SG_PVARIANT(32, 3, false, "p32x3"),
    SG_PVARIANT(32, 3, true, "p32x3-g2"),
    SG_PVARIANT(24, 3, true, "p24x3-g2"),
    SG_PVARIANT(28, 3, true, "p28x3-g2"),
    SG_PVARIANT(16, 3, true, "p16x3-g2"),
    SG_PVARIANT(20, 4, true, "p20x4-g2"),
};
#define SG_NPVARIANTS ((int)(sizeof(k_pvariants) / sizeof(k_pvariants[0])))
#define SG_PVARIANT_DEFAULT 5 /* p32x3-g2 */

/* Cluster configurations (sg_cluster.cuh): warps per CTA and CTAs per
 * codeword, the latter descending. */
struct SgCVariant {
    int nw;
    int cs;
    size_t smem;
    const void* fn;
};
#define SG_CVARIANT(NW, CS) {NW, CS, sizeof(SgClusterSmem<NW>), (const void*)sg_cluster_kernel<NW, CS, SG_TU_CR>}
static const SgCVariant k_cvariants[] = {SG_CVARIANT(16, 16), SG_CVARIANT(32, 8), SG_CVARIANT(32, 4), SG_CVARIANT(32, 2)};
#define SG_NCVARIANTS ((int)(sizeof(k_cvariants) / sizeof(k_cvariants[0])))

/* Line kernels: few lines (one per warp), and many (a full SM per two CTAs). */
struct SgBVariant {
    int nw;
    size_t smem;
    const void* fn;
};
#define SG_BVARIANT(NW, T8) {NW, sizeof(SgLineSmem<NW, T8>), (const void*)sg_bitso_kernel<NW, T8, SG_TU_CR>}
static const SgBVariant k_bvariants[] = {SG_BVARIANT(4, false), SG_BVARIANT(16, true)};

/* The code tables, for this translation unit's kernels. */
static cudaError_t sg_load_code(const sg_code_tables& code)
{
    cudaError_t e = cudaMemcpyToSymbol(c_hcol, code.hcol, sizeof code.hcol);
    if (e == cudaSuccess)
        e = cudaMemcpyToSymbol(c_prow, code.prow, sizeof code.prow);
    if (e == cudaSuccess)
        e = cudaMemcpyToSymbol(c_ptab, code.ptab, sizeof code.ptab);
    return e;
}
