/* sg_cluster.cuh -- a codeword decoded by a cluster of CTAs, for batches that
 * leave SMs idle.
 *
 * With one CTA per codeword a small batch is bound by latency: an SM works
 * through the 256 lines of a phase on its own, however many others are idle,
 * and each phase ends with its longest line.  Here the CS CTAs of a cluster
 * take 256 / CS lines of every phase each.  The extrinsic cube is spread over
 * them: an entry is kept by the CTA whose line of the next phase will read
 * it, so each line's results are stored straight into the shared memory of
 * those CTAs (distributed shared memory), its hard-decision word into all of
 * them.  One cluster barrier ends a phase; every warp then runs the
 * early-termination test on its CTA's own copy of the 256 words.
 *
 * No store races with a load: the copy of an entry that a phase reads is the
 * one of the CTA whose line holds it, and only that line's warp replaces it.
 * Words and maxima of a phase alternate between two buffers, since a CTA may
 * be one phase ahead.  Per codeword, the line decodes and their order of
 * phases are those of sg_decode_kernel, and so are the outputs, bit for bit.
 *
 * Bound by the latency of a line decode and of the phase ends (issue slots
 * 64 % used with 70 codewords on pairs).  2 dB, one CTA per codeword against
 * clusters: one codeword 2.4 and 0.31 to 0.45 ms (16 CTAs, by its noise), 100
 * codewords 3.2 and 2.0 ms (2 CTAs each).
 */
#pragma once

template <int NW>
struct SgClusterSmem {
    double le[SG_CUBE];
    SgEtab<true> etab;
    alignas(16) double ltab[SG_LOG_TAB_LEN];
    SgWarpScratch ws[NW];
    uint16_t hdw[2][256];
    unsigned long long ng;   /* rank 0: guesses of the codeword */
    unsigned int ngmax[2];   /* rank 0: largest of the phase */
    int line_next[2];        /* next of the CTA's lines to hand out */
};

/* Shared address of a CTA of the cluster for this CTA's shared address a. */
__device__ __forceinline__ uint32_t sg_mapa(uint32_t a, int rank)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void sg_cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

/* Line of phase `axis` that holds cube position p (the inverse of sg_pos). */
__device__ __forceinline__ int sg_line_of(int axis, int p)
{
    const int s = p >> 8, c = (p >> 4) & 15, r = p & 15;
    return axis == 0 ? s * 16 + c : (axis == 1 ? s * 16 + r : c * 16 + r);
}

template <int NW, int CS, bool CR>
__global__ void __launch_bounds__(NW * 32, 1) sg_cluster_kernel(const __grid_constant__ SgDecodeArgs args)
{
    constexpr int NT = NW * 32, LPC = 256 / CS; /* lines per CTA and phase */
    SgClusterSmem<NW>& S = *reinterpret_cast<SgClusterSmem<NW>*>(sg_smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned long long cw = blockIdx.x / CS;
    const int rank = (int)(blockIdx.x % CS);
    sg_etab_fill<CR, true>(S.etab, g_etab, tid, NT);
    for (int i = tid; i < SG_LOG_TAB_LEN; i += NT)
        S.ltab[i] = g_ltab[i];
    for (int i = tid; i < SG_CUBE; i += NT)
        S.le[i] = 0.0;
    const double* g = args.llr + cw * SG_CUBE;
    bool nonfinite = false;
    for (int i = tid; i < SG_CUBE; i += NT)
        nonfinite |= !isfinite(__ldg(g + i));
    if (tid == 0) {
        S.ng = 0;
        S.ngmax[0] = S.ngmax[1] = 0;
        S.line_next[0] = S.line_next[1] = 0;
    }
    /* every CTA of the cluster looks at the whole cube and decides alike */
    if (__syncthreads_or(nonfinite)) {
        if (rank == 0)
            sg_cw_not_decoded(args, cw, -1);
        return;
    }
    const SgTab etab = sg_etab_of<CR, true>(S.etab, args.k.v), ltab{S.ltab, args.k.v};
    const SgLineParams lp{args.L, args.thres, &args.meta};
    const uint32_t le_a = sg_saddr(S.le);
    const uint32_t ng_a = sg_mapa(sg_saddr(&S.ng), 0), ngmax_a = sg_mapa(sg_saddr(S.ngmax), 0);
    const uint32_t hdw_a = sg_mapa(sg_saddr(S.hdw), lane % CS);
    const int nphase = 3 * args.imax;
    unsigned long long ng_p = 0; /* rank 0, thread 0 */
    int phase = 0, axis = 0;
    bool conv = false;
    sg_cluster_barrier(); /* the shared memory of all CTAs is set up */
    for (;;) {
        const int buf = phase & 1, axis_next = axis == 2 ? 0 : axis + 1;
        const double alpha = args.alpha[phase];
        for (;;) {
            int q = 0;
            if (lane == 0)
                q = atomicAdd(&S.line_next[buf], 1);
            q = __shfl_sync(SG_FULL, q, 0);
            if (q >= LPC)
                break;
            const int l = rank * LPC + q, pos = sg_pos(axis, l, lane & 15);
            /* L_ch + (alpha*L_E), lanes p and p + 16 alike */
            const double le0 = S.le[pos];
            const double v = __dadd_rn(__ldg(g + pos), __dmul_rn(alpha, le0));
            if (args.ckpt && lane < 16)
                args.ckpt[(cw * (unsigned long long)nphase + phase) * SG_CUBE + pos] = le0;
            const SgLineResult r = sg_decode_line<false, CR, true, NW <= 16 ? 2 : 1>(v, lp, args.enum_tabs, etab, ltab, &S.ws[warp]);
            if (lane < 16) {
                const uint32_t a = sg_mapa(le_a + 8u * (uint32_t)pos, sg_line_of(axis_next, pos) / LPC);
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(r.le) : "memory");
                if (args.lapp)
                    args.lapp[cw * SG_CUBE + pos] = r.lapp;
            }
            if (lane < CS) {
                const uint32_t a = hdw_a + 2u * (uint32_t)(buf * 256 + l);
                asm volatile("st.shared::cluster.u16 [%0], %1;" ::"r"(a), "h"((uint16_t)r.hdword) : "memory");
            }
            if (lane == 0) {
                asm volatile("red.relaxed.cluster.shared::cluster.add.u64 [%0], %1;" ::"r"(ng_a),
                             "l"((unsigned long long)r.T)
                             : "memory");
                asm volatile("red.relaxed.cluster.shared::cluster.max.u32 [%0], %1;" ::"r"(ngmax_a + 4u * buf), "r"(r.T)
                             : "memory");
            }
        }
        __syncwarp();
        sg_cluster_barrier(); /* the phase's results are everywhere */
        conv = sg_is_codeword(S.hdw[buf], lane);
        if (tid == 0) { /* the next phase uses the other buffers, the one after it these */
            ng_p += S.ngmax[buf];
            S.ngmax[buf] = 0;
            S.line_next[buf] = 0;
        }
        phase++;
        if (conv || phase == nphase)
            break;
        axis = axis_next;
    }
    if (rank != 0)
        return;
    ng_p = __shfl_sync(SG_FULL, ng_p, 0); /* of warp 0; the others leave */
    if (warp != 0)
        return;
    /* hard_decision (:393-415) and packing (:272-280) as in sg_decode_kernel */
    const uint16_t* hdw = S.hdw[(phase - 1) & 1];
    uint32_t byte[2];
#pragma unroll 1
    for (int h = 0; h < 2; h++) {
        uint32_t v = 0;
        for (int q = 0; q < 8; q++) {
            const int b = (lane + 32 * h) * 8 + q;
            const int p = (b >> 6) * 256 + ((b >> 3) & 7) * 16 + (b & 7);
            const int l = sg_line_of(axis, p), bit = axis == 0 ? p & 15 : (axis == 1 ? (p >> 4) & 15 : p >> 8);
            v = (v << 1) | ((hdw[l] >> bit) & 1u);
        }
        (h ? byte[1] : byte[0]) = v;
    }
    sg_cw_stats st;
    st.iterations = 0.5 * phase;
    st.ng = S.ng;
    st.ng_p = ng_p;
    st.converged = conv ? 1 : 0;
    st.phases = phase;
    sg_cw_output(args, cw, byte[0], byte[1], st, lane);
}
