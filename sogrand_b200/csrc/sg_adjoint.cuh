/* sg_adjoint.cuh -- FP64 adjoint of the SOGRAND soft-output decoder.
 *
 * The decoder is piecewise smooth in its inputs: the sort, IC, the tested
 * patterns, the codeword list, the stopping guess, the early-termination
 * decisions and the number of phases are piecewise constant, and are held
 * fixed as the branch of the forward pass.  On that branch the soft output
 * of one line (SOGRAND_bitSO, SOGRAND_C/cubic_decoder_final.c:536-577) is
 *   p_j   = exp(-PM_j),  PM_j = sum_k JacLog(-|x_k|) + sum_{k in S_j} delta(|x_k|)
 *   pNL   = 2^-8 (1 - sum_{t <= T} exp(-PM_t))          (all counted guesses t)
 *   pp1_i = 1/(1 + e^{x_i}),  pp0_i = 1 - pp1_i           (clamped to [1e-40, 1])
 *   p0_i  = sum_{j: c_ji = 0} p_j + max(pNL,1e-40) pp0_i,  p1_i likewise
 *   L_APP_i = log max(p0_i,1e-40) - log max(p1_i,1e-40),   L_E_i = L_APP_i - x_i
 * with S_j the positions where pattern j differs from the hard decision and
 *   dPM/dx_i = sign(x_i) (-sigma(-|x_i|) [|x_i| <= 50] + [i in S]),
 * so dpNL/dx_i = 2^-8 sign(x_i) (-sigma(-|x_i|)[|x_i| <= 50] E + E_i) with
 * E = sum_t exp(-PM_t) and E_i the same sum over guesses holding position i.
 * sg_line_vjp applies the transpose of that Jacobian to an upstream vector.
 *
 * The backward kernel re-runs, phase by phase in reverse, every line decode
 * from the checkpointed extrinsic cube entering the phase (the forward
 * writes one 32 KB checkpoint per phase), accumulating E and E_i on the way,
 * and propagates the gradient of the loss
 *   loss = sum_i softplus(s_i L_APP_i),  s_i = +1 for code bit 1, -1 for 0,
 * (the BCE of the final APP against the transmitted bits; loss_mode 1: the
 * sum of that over every phase's APP) to the per-phase extrinsic weights
 * alpha_p, the channel LLRs and the previous phase.
 */
#pragma once

/* sum over positions, lanes p and p + 16 holding position p's term alike */
__device__ __forceinline__ double sg_sum16(double v)
{
    for (int off = 8; off > 0; off >>= 1)
        v += __shfl_xor_sync(SG_FULL, v, off);
    return v;
}

/* Gradient with respect to the line input x of g . L_APP, g the upstream
 * gradient of L_APP; lanes p and p + 16 hold position p alike.  The soft
 * output's exp, reciprocal and sums come from the decode. */
__device__ __forceinline__ double sg_line_vjp(double x, double g, const SgAdjOut& a, SgTab etab, int lane)
{
    if (a.curl == 0)
        return g; /* L_APP = x */
    const bool low = lane < 16;
    const int pos = lane & 15;
    const double eps = 1e-40;
    const bool pnl_live = a.pnl > eps;
    const double p_nl = fmax(a.pnl, eps);
    const double pp1r = a.q1, pp0r = 1.0 - pp1r;
    const double pp1 = fmax(pp1r, eps), pp0 = fmax(pp0r, eps); /* at most 1 */
    /* g / p0 on the low lanes, -g / p1 on the high ones */
    const double pm = low ? a.p0 : a.p1;
    const double mine = pm > eps ? (low ? g : -g) / pm : 0.0, other = __shfl_xor_sync(SG_FULL, mine, 16);
    const double a0 = low ? mine : other, a1 = low ? other : mine;
    const double dsig = pp0r * pp1r; /* d pp0/dx = -d pp1/dx */
    double gx = 0.0;
    if (pp0r > eps)
        gx += a0 * p_nl * dsig;
    if (pp1r > eps)
        gx -= a1 * p_nl * dsig;
    const double sgn = x > 0.0 ? 1.0 : (x < 0.0 ? -1.0 : 0.0);
    const double ax = fabs(x);
    const double sm = ax <= 50.0 ? (x > 0.0 ? pp1r : 1.0 / (1.0 + sg_exp(ax, etab))) : 0.0; /* sigma(-|x|) */
    for (int j = 0; j < a.curl; j++) {
        const double pj = __shfl_sync(SG_FULL, a.my_e, j);
        const uint32_t cm = __shfl_sync(SG_FULL, a.my_cm, j);
        const uint32_t cj = (cm >> pos) & 1u;
        const double gpj = sg_sum16(cj ? a1 : a0);
        const double gpm = -pj * gpj;
        const double inS = (((cm ^ a.hdm) >> pos) & 1u) ? 1.0 : 0.0;
        gx += gpm * sgn * (inS - sm);
    }
    if (pnl_live) {
        const double gpnl = sg_sum16(a0 * pp0 + a1 * pp1);
        const double ei = __shfl_sync(SG_FULL, a.esort, 2 * a.myrank);
        gx += gpnl * 0x1p-8 * sgn * (ei - sm * a.etot);
    }
    return gx;
}

struct SgBackwardArgs {
    const double* llr;
    const double* ckpt;          /* [n_cw][nph][4096]: L_E entering each phase */
    const sg_cw_stats* stats;    /* phases run per codeword (forward output) */
    const uint8_t* code_bits;    /* [n_cw][4096] transmitted bits, 0/1 */
    const uint32_t* enum_tabs;
    double* loss;                /* [n_cw] */
    double* grad_alpha;          /* [n_cw][nph] */
    double* grad_llr;            /* [n_cw][4096] or NULL */
    unsigned long long n_cw;
    int32_t L;
    int32_t nph;                 /* 3 * Imax */
    int32_t loss_mode;           /* 0: BCE of the final APP; 1: summed over all phases' APPs */
    double thres;
    double alpha[SG_MAX_PHASES];
    SgK k; /* constants of exp and log */
    sg_order_meta meta;
};

#define SG_BACK_WINDOW 2048   /* codewords of a launch that are ordered by length */
#define SG_BACK_WARPS 24      /* of the backward kernel's CTAs, one per SM */

struct SgBackSmem {
    union {
        double gle[SG_CUBE]; /* d loss / d L_E of the phase being processed */
        struct { /* before it: the choice of the codeword */
            uint8_t pick[SG_BACK_WINDOW];
            int hist[SG_MAX_PHASES + 1];
        };
    };
    SgEtab<true> etab;
    alignas(16) double ltab[SG_LOG_TAB_LEN];
    SgWarpScratch ws[SG_BACK_WARPS];
    double bins[SG_BACK_WARPS][9 * 32]; /* high positions' guess sums, per lane */
    double ga;   /* d loss / d alpha of the phase */
    double lsum; /* loss of the codeword */
    int line_next;
};

/* The codeword of block b: the last SG_BACK_WINDOW ones are taken in the
 * order of falling phase counts, equal ones in index order.  Codewords differ
 * in length by up to the number of phases, and a long one that starts last
 * runs alone on its SM.  A block counts the window's phases for itself (a few
 * microseconds of the millisecond a codeword takes), so nothing is shared
 * between blocks.  1.5 dB, Imax 10: 1 024 codewords 32.8 -> 26.8 ms, 600 22.4
 * -> 17.4. */
__device__ __forceinline__ unsigned long long sg_back_pick(const SgBackwardArgs& args, unsigned long long b, uint8_t* ph,
                                                           int* hist, int tid)
{
    constexpr int NT = SG_BACK_WARPS * 32;
    const unsigned long long n = args.n_cw, base = n > SG_BACK_WINDOW ? n - SG_BACK_WINDOW : 0;
    if (b < base)
        return b;
    const int m = (int)(n - base);
    int k = (int)(b - base); /* the k-th of m */
    for (int i = tid; i <= SG_MAX_PHASES; i += NT)
        hist[i] = 0;
    __syncthreads();
    for (int i = tid; i < m; i += NT) {
        const int p = min(max(args.stats[base + i].phases, 0), SG_MAX_PHASES);
        ph[i] = (uint8_t)p;
        atomicAdd(&hist[p], 1);
    }
    __syncthreads();
    if (tid < 32) {
        int v = SG_MAX_PHASES;
        for (; k >= hist[v]; v--)
            k -= hist[v];
        int i = tid;
        for (;; i += 32) {
            const uint32_t same = __ballot_sync(SG_FULL, i < m && ph[i] == v);
            const int c = __popc(same);
            if (k < c) {
                if (i < m && ph[i] == v && __popc(same & ((1u << tid) - 1u)) == k)
                    hist[0] = i;
                break;
            }
            k -= c;
        }
    }
    __syncthreads();
    const int i = hist[0];
    __syncthreads();
    return base + (unsigned long long)i;
}

/* One codeword at a time on an SM's 24 warps of 80 registers; 28 warps take
 * as long, 30 spill and take 2 % more.  Two CTAs of 12 warps, each with a
 * codeword of its own, hide the end of each other's phases but take twice as
 * long over the longest codeword: 4 % more for 1 024 codewords at 1.5 dB, Imax
 * 10, and 11.5 against 7.3 ms for 160.
 * Bound by issue slots (71 % used) and latency; 25.9 ms for those 1 024.  A
 * guess costs nine predicated additions and two shared-memory sums besides the
 * forward's work: with all 16 positions' sums in registers there are spills
 * and 7 % more, since the forward's work leaves half of the shared-memory
 * cycles idle.  Per line, whatever the decode has worked out is used again,
 * sums over a phase are kept per lane, and no logarithm is taken where the
 * loss does not need L_APP (a fifth less in all); the exp table in eight
 * copies, as in the decoders, takes 6 %. */
__global__ void __launch_bounds__(SG_BACK_WARPS * 32, 1) sg_backward_kernel(const __grid_constant__ SgBackwardArgs args)
{
    constexpr int NT = SG_BACK_WARPS * 32;
    SgBackSmem& S = *reinterpret_cast<SgBackSmem*>(sg_smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    sg_etab_fill<false, true>(S.etab, g_etab, tid, NT);
    for (int i = tid; i < SG_LOG_TAB_LEN; i += NT)
        S.ltab[i] = g_ltab[i];
    SgLineParams lp;
    lp.L = args.L;
    lp.meta = &args.meta;
    lp.thres = args.thres;
    const SgTab etab = sg_etab_of<false, true>(S.etab, args.k.v), ltab{S.ltab, args.k.v};
    __syncthreads();
    for (unsigned long long b = blockIdx.x; b < args.n_cw; b += gridDim.x) {
        const unsigned long long cw = sg_back_pick(args, b, S.pick, S.hist, tid);
        const int P = args.stats[cw].phases;
        const double* g = args.llr + cw * SG_CUBE;
        for (int i = tid; i < SG_CUBE; i += NT) {
            S.gle[i] = 0.0;
            if (args.grad_llr)
                args.grad_llr[cw * SG_CUBE + i] = 0.0;
        }
        for (int p = tid; p < args.nph; p += NT)
            args.grad_alpha[cw * args.nph + p] = 0.0;
        if (tid == 0)
            S.lsum = 0.0;
        __syncthreads();
        for (int p = P - 1; p >= 0; p--) {
            const int axis = p % 3;
            const double alpha = args.alpha[p];
            const double* ck = args.ckpt + (cw * args.nph + p) * SG_CUBE;
            if (tid == 0) {
                S.line_next = 0;
                S.ga = 0.0;
            }
            __syncthreads();
            const bool scored = p == P - 1 || args.loss_mode == 1;
            double ga = 0.0, ls = 0.0; /* the lane's shares of the phase's sums */
            for (;;) {
                int l = 0;
                if (lane == 0)
                    l = atomicAdd(&S.line_next, 1);
                l = __shfl_sync(SG_FULL, l, 0);
                if (l >= 256)
                    break;
                const int pos = sg_pos(axis, l, lane & 15);
                const double lep = ck[pos];
                const double x = __dadd_rn(g[pos], __dmul_rn(alpha, lep));
                SgAdjOut a;
                a.want_app = scored;
                a.bins = S.bins[warp];
                const SgLineResult r = sg_decode_line<true, false, true>(x, lp, args.enum_tabs, etab, ltab, &S.ws[warp], &a);
                const double gE = S.gle[pos];
                double gL = 0.0;
                if (scored) {
                    const double lapp = __shfl_sync(SG_FULL, r.lapp, lane & 15);
                    const double s = args.code_bits[cw * SG_CUBE + pos] ? 1.0 : -1.0;
                    const double z = s * lapp;
                    ls += (z > 0.0 ? z : 0.0) + log1p(exp(-fabs(z))); /* softplus */
                    gL = s / (1.0 + exp(-z));                          /* s * sigmoid(z) */
                }
                const double gx = sg_line_vjp(x, gL + gE, a, etab, lane) - gE;
                __syncwarp(); /* gle read by both halves */
                if (lane < 16) {
                    S.gle[pos] = alpha * gx;
                    if (args.grad_llr) /* one addition per phase: no result to wait for */
                        atomicAdd(&args.grad_llr[cw * SG_CUBE + pos], gx);
                }
                ga += gx * lep;
            }
            ga = sg_sum16(ga);
            ls = sg_sum16(ls);
            if (lane == 0) {
                atomicAdd(&S.ga, ga);
                if (scored)
                    atomicAdd(&S.lsum, ls);
            }
            __syncthreads();
            if (tid == 0)
                args.grad_alpha[cw * args.nph + p] = S.ga;
            __syncthreads();
        }
        if (tid == 0)
            args.loss[cw] = S.lsum;
        __syncthreads();
    }
}
