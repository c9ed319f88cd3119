/* sg_api.cu -- B200 SOGRAND cubic decoder: C ABI, and the kernels of the
 * table-driven math (sg_kernels.cuh; sg_cr.cu holds the correctly rounded
 * ones), the generator (sg_gen_kernel: seeded source, encoder, AWGN channel)
 * and the adjoint.
 *
 * Built with -fmad=false: no floating-point contraction anywhere, as in the
 * reference's plain gcc build; the exp/log routines use explicit FMAs.
 */
#include <cuda_runtime.h>

#include <errno.h>
#include <stddef.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "../../include/sogrand_b200.h"
#include "sg_cr.h"
#include "sg_gen.h"
#include "sg_kernels.cuh"
#include "sg_adjoint.cuh"

struct SgGenSmem {
    alignas(16) double etab[SG_EXP_TAB_LEN];
    alignas(16) double ltab[SG_LOG_TAB_LEN];
    alignas(16) ulonglong2 key[SG_POLAR_TRIES]; /* of the two noise streams of each attempt */
    double u[SG_CUBE];                          /* accepted pairs: u, and u^2 + v^2 */
    double ss[SG_CUBE];
    uint16_t W[256];
    uint8_t ib[SG_INFO_BYTES];
    uint8_t prow[8];
    uint8_t ptab[256];
};

/* a / b correctly rounded, y = 1 / b correctly rounded, for quotients and
 * remainders in the normal range: two corrections of a * y by the exact
 * remainder (P. Markstein, "Computation of elementary functions on the IBM RISC
 * System/6000 processor", IBM J. Res. Dev. 34(1), 1990). */
__device__ __forceinline__ double sg_div_by(double a, double b, double y)
{
    double q = __dmul_rn(a, y);
    q = __fma_rn(__fma_rn(-q, b, a), y, q);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
}

/* sg_sym_unit from bits 11..63: 1 + (bits 11..62) 2^-52, less 1 or 2 by bit
 * 63; exact. */
__device__ __forceinline__ double sg_sym_unit_bits(uint64_t r)
{
    const uint32_t hi = (uint32_t)(r >> 32);
    const double d = __hiloint2double((int)(0x3ff00000u | ((hi >> 11) & 0xfffffu)), (int)__funnelshift_r((uint32_t)r, hi, 11));
    return __dsub_rn(d, (int32_t)hi < 0 ? 1.0 : 2.0);
}

/* Seeded codewords and their channel LLRs.  Two passes over a thread's 16
 * positions p = tid + 256 q: the polar attempts, as one stream (a lane moves
 * to its next position when a pair is accepted, so a warp does not wait,
 * position by position, for its unluckiest lane), then log, square root and
 * divisions of the accepted pairs with every lane busy.  Each position keeps
 * its first accepted attempt (after SG_POLAR_TRIES rejections, 0), as
 * sg_normal does.  Bound by issue slots: one attempt is two 64-bit hashes;
 * keyed per attempt once per CTA, not per sample, and with unit and quotient
 * from bits and remainders, 20 000 codewords take 0.86 ms (1.36 ms with one
 * pass, four hashes per attempt and three library divisions per sample). */
__global__ void __launch_bounds__(SG_THREADS, 3) sg_gen_kernel(uint64_t seed, uint64_t cw0, unsigned long long n_cw,
                                                               double sigma, double lo, double hi, uint8_t* info,
                                                               double* llr, const __grid_constant__ SgK k)
{
    SgGenSmem& S = *reinterpret_cast<SgGenSmem*>(sg_smem_raw);
    const SgTab etab{S.etab, k.v}, ltab{S.ltab, k.v};
    const int tid = threadIdx.x;
    for (int i = tid; i < SG_EXP_TAB_LEN; i += SG_THREADS)
        S.etab[i] = g_etab[i];
    for (int i = tid; i < SG_LOG_TAB_LEN; i += SG_THREADS)
        S.ltab[i] = g_ltab[i];
    if (tid < SG_POLAR_TRIES)
        S.key[tid] = make_ulonglong2(sg_rand_key(seed, 1 + 2 * tid), sg_rand_key(seed, 2 + 2 * tid));
    if (tid < 8)
        S.prow[tid] = c_prow[tid];
    S.ptab[tid] = c_ptab[tid];
    __syncthreads();
    for (unsigned long long c = blockIdx.x; c < n_cw; c += gridDim.x) {
        const uint64_t gc = cw0 + c;
        if (tid < 8) {
            const uint64_t r = sg_rand(seed, 0, gc * 8 + tid);
            for (int q = 0; q < 8; q++)
                S.ib[tid * 8 + q] = (uint8_t)(r >> (8 * q));
        }
        __syncthreads();
        /* sg_encode_words, each of its four stages spread over the block:
         * info words, parity columns of the first 8 slices, parity rows,
         * parity slices (the same words, every one written once) */
        if (tid < 64)
            S.W[(tid >> 3) * 16 + (tid & 7)] = (uint16_t)sg_brev8(S.ib[tid]);
        __syncthreads();
        if (tid < 64) {
            const int l = tid >> 3, jj = tid & 7;
            uint16_t acc = 0;
            for (int j = 0; j < 8; j++)
                if ((S.prow[j] >> jj) & 1)
                    acc ^= S.W[l * 16 + j];
            S.W[l * 16 + 8 + jj] = acc;
        }
        __syncthreads();
        if (tid < 128) {
            const uint16_t x = S.W[tid];
            S.W[tid] = (uint16_t)((x & 0xff) | (S.ptab[x & 0xff] << 8));
        }
        __syncthreads();
        if (tid < 128) {
            const int jj = tid >> 4, j = tid & 15;
            uint16_t acc = 0;
            for (int l = 0; l < 8; l++)
                if ((S.prow[l] >> jj) & 1)
                    acc ^= S.W[l * 16 + j];
            S.W[(8 + jj) * 16 + j] = acc;
        }
        if (info && tid < SG_INFO_BYTES)
            info[c * SG_INFO_BYTES + tid] = S.ib[tid];
        __syncthreads();
        const double s = sigma > 0.0 ? sigma : sg_sigma_draw(seed, gc, lo, hi, etab);
        uint64_t base = sg_rand_ctr(gc * 4096u + tid);
        for (int p = tid, att = 0; p < SG_CUBE;) {
            const ulonglong2 key = S.key[att];
            const double u = sg_sym_unit_bits(sg_mix64(key.x ^ base));
            const double v = sg_sym_unit_bits(sg_mix64(key.y ^ base));
            const double ss = __dadd_rn(__dmul_rn(u, u), __dmul_rn(v, v));
            const bool ok = ss > 0.0 && ss < 1.0;
            if (ok || att + 1 == SG_POLAR_TRIES) {
                S.u[p] = u;
                S.ss[p] = ok ? ss : 2.0;
                p += SG_THREADS;
                base += (uint64_t)SG_THREADS * SG_RAND_CTR_MUL;
                att = 0;
            } else {
                att++;
            }
        }
        const double var = __dmul_rn(s, s), rvar = __drcp_rn(var);
        const bool mid = var > 0x1p-400 && var < 0x1p400; /* noise and quotient stay normal */
        double* out = llr + c * SG_CUBE;
#pragma unroll 2
        for (int q = 0; q < SG_CUBE / SG_THREADS; q++) {
            const int p = tid + SG_THREADS * q;
            const double ss = S.ss[p];
            double z = 0.0;
            if (ss < 1.0) {
                const double m = __dmul_rn(-2.0, sg_log_core(sg_bits(ss), 0, ltab));
                z = __dmul_rn(S.u[p], __dsqrt_rn(sg_div_by(m, ss, __drcp_rn(ss))));
            }
            /* sg_llr_of */
            const double y2 = __dmul_rn(2.0, __dadd_rn((S.W[p >> 4] >> (p & 15)) & 1 ? -1.0 : 1.0, __dmul_rn(s, z)));
            out[p] = mid ? sg_div_by(y2, var, rvar) : __ddiv_rn(y2, var);
        }
        __syncthreads();
    }
}

/* A configuration's shared memory: tables on 16-byte boundaries (double2
 * loads), warp records on 256-byte ones (the guess loop puts table bytes into
 * the low byte of a record's address), and room for the CTAs per SM that it
 * is built for (228 KB per SM, 1 KB of it reserved per CTA; 227 KB per CTA). */
template <class T, int CTAS>
constexpr bool sg_smem_ok()
{
    return offsetof(T, etab) % 16 == 0 && offsetof(T, ltab) % 16 == 0 && offsetof(T, ws) % 256 == 0 &&
           alignof(T) <= 1024 && sizeof(T) <= 227 * 1024 && CTAS * (sizeof(T) + 1024) <= 228 * 1024;
}
static_assert(sg_smem_ok<SgPersistSmem<16, 3>, 1>() && sg_smem_ok<SgPersistSmem<20, 4>, 1>() &&
                  sg_smem_ok<SgPersistSmem<24, 3>, 1>() && sg_smem_ok<SgPersistSmem<28, 3>, 1>() &&
                  sg_smem_ok<SgPersistSmem<32, 3>, 1>(),
              "batched configurations");
static_assert(sg_smem_ok<SgCwSmem<8, false>, 3>() && sg_smem_ok<SgCwSmem<8, true>, 2>() &&
                  sg_smem_ok<SgCwSmem<12, true>, 2>() && sg_smem_ok<SgCwSmem<16, false>, 2>() &&
                  sg_smem_ok<SgCwSmem<8, false, 2>, 2>() && sg_smem_ok<SgCwSmem<10, false, 2>, 1>() &&
                  sg_smem_ok<SgCwSmem<16, false, 2>, 1>(),
              "plain configurations");
static_assert(sg_smem_ok<SgClusterSmem<16>, 1>() && sg_smem_ok<SgClusterSmem<32>, 1>(), "cluster configurations");
static_assert(sg_smem_ok<SgLineSmem<4, false>, 1>() && sg_smem_ok<SgLineSmem<16, true>, 2>(), "line kernels");
static_assert(sg_smem_ok<SgBackSmem, 1>(), "backward kernel");
template <class T>
constexpr bool sg_bulk_aligned()
{
    return offsetof(T, lch) == 0 && offsetof(T, mbar) % 8 == 0;
}
static_assert(sg_bulk_aligned<SgCwSmem<8, true>>() && sg_bulk_aligned<SgCwSmem<12, true>>(), "bulk copy");

/* Static device memory of the allocation-free entry point: the error flag
 * (word 0; while the tables are built, each one's completion flag) and a
 * private copy of the pattern-order tables.  Host code must not use these
 * names as addresses: the set-up below resolves them with
 * cudaGetSymbolAddress on each device. */
static __device__ unsigned int g_noalloc_err[SG_ENUM_NTAB];
static __device__ __align__(256) uint32_t g_noalloc_enum[SG_ENUM_NTAB * SG_ENUM_LEN];

/* One thread per IC builds that IC's pattern order (same source as the host
 * builder); ok[ic] = 1 when complete. */
__global__ void sg_enum_build_kernel(uint32_t* out, unsigned int* ok)
{
    const int ic = blockIdx.x * blockDim.x + threadIdx.x;
    if (ic < SG_ENUM_NTAB)
        ok[ic] = sg_enum_build_impl(ic, out + (size_t)ic * SG_ENUM_LEN) == SG_ENUM_LEN ? 1u : 0u;
}

/* Ceiling of the per-guess floating-point work: each thread evaluates, per
 * iteration, one path-metric addition, exp(-PM) and one P_notGuess
 * subtraction, with no memory traffic beyond the shared exp table.
 * guesses/s of this kernel over all SMs bounds what any decoder with the
 * reference's per-guess arithmetic can reach.  CR: the correctly rounded
 * exp; otherwise the table-driven sg_exp_neg. */
template <bool CR>
__global__ void __launch_bounds__(256) sg_guess_ceiling_kernel(unsigned long long iters, double* sink,
                                                               const __grid_constant__ SgK k)
{
    __shared__ alignas(16) double etab_s[SG_EXP_TAB_LEN];
    const SgTab etab{etab_s, k.v};
    for (int i = threadIdx.x; i < SG_EXP_TAB_LEN; i += 256)
        etab_s[i] = g_etab[i];
    __syncthreads();
    double pm0 = 1e-3 * (threadIdx.x + 1), pm1 = pm0 + 0.37, acc0 = 1.0, acc1 = 1.0;
    for (unsigned long long it = 0; it < iters; it++) {
        pm0 = __dadd_rn(pm0, 1.1e-5);
        pm1 = __dadd_rn(pm1, 1.3e-5);
        acc0 = __dsub_rn(acc0, CR ? sg_exp_cr_neg(-pm0, etab) : sg_exp_neg(-pm0, etab));
        acc1 = __dsub_rn(acc1, CR ? sg_exp_cr_neg(-pm1, etab) : sg_exp_neg(-pm1, etab));
    }
    if (acc0 + acc1 == 12345.0)
        sink[blockIdx.x] = acc0;
}

/* -------------------------------------------------------------- host -- */

namespace {

thread_local std::string t_err;

sg_status fail(sg_status s, const std::string& msg)
{
    t_err = msg;
    return s;
}

sg_status cuda_fail(cudaError_t e, const char* what)
{
    return fail(SG_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

#define SG_CUDA(call)                         \
    do {                                      \
        cudaError_t e_ = (call);              \
        if (e_ != cudaSuccess)                \
            return cuda_fail(e_, #call);      \
    } while (0)


std::mutex g_mu;
std::atomic<long long> g_wait_limit{SG_WAIT_LIMIT_DEFAULT};
std::atomic<int> g_math_mode{0}; /* 0: table-driven exp/log, 1: correctly rounded */
/* Selected kernel variants, one per math mode (sogrand_b200.autotune
 * measures them).  B200, 12 000 codewords at 2 dB, table math: p32x3 112.6
 * ms, p28x3 117.3, p24x3 121.6; w16-gmem 115.3, w8-gmem 134.0, w12-smem
 * 137.0, w8-smem 162.7; correctly rounded, 6 000: p32x3 86.5, p28x3 89.2,
 * p24x3 93.2; w16-gmem 87.7, w8-gmem 93.5. */
int g_pvariant_by_mode[2] = {SG_PVARIANT_DEFAULT, SG_PVARIANT_DEFAULT};
int g_variant_by_mode[2] = {SG_VARIANT_DEFAULT, SG_VARIANT_DEFAULT};
#define g_pvariant (g_pvariant_by_mode[g_math_mode.load()])
#define g_variant (g_variant_by_mode[g_math_mode.load()])
std::vector<uint32_t> g_enum_host;
sg_code_tables g_code;
bool g_host_ready = false;

const double k_etab_host[SG_EXP_TAB_LEN] = SG_EXP_TAB_INIT;
const double k_ltab_host[SG_LOG_TAB_LEN] = SG_LOG_TAB_INIT;
const SgK k_consts = SG_K_INIT;
const SgTab k_etab_tab{k_etab_host, k_consts.v}, k_ltab_tab{k_ltab_host, k_consts.v};

/* Kernel of a configuration, by math mode. */
const void* decode_fn(int v, bool cr) { return cr ? sg_cr_decode_fn(v) : k_variants[v].fn; }
const void* persist_fn(int v, bool cr) { return cr ? sg_cr_persist_fn(v) : k_pvariants[v].fn; }

const void* bitso_fn(int v, bool cr) { return cr ? sg_cr_bitso_fn(v) : k_bvariants[v].fn; }
const void* cluster_fn(int v, bool cr) { return cr ? sg_cr_cluster_fn(v) : k_cvariants[v].fn; }

sg_status host_init_locked()
{
    if (g_host_ready)
        return SG_OK;
    sg_code_build(&g_code);
    g_enum_host.assign((size_t)SG_ENUM_NTAB * SG_ENUM_LEN, 0);
    for (int ic = 0; ic < SG_ENUM_NTAB; ic++)
        if (sg_enum_build_impl(ic, g_enum_host.data() + (size_t)ic * SG_ENUM_LEN) != SG_ENUM_LEN)
            return fail(SG_ERR_ARG, "error-pattern order table incomplete");
    g_host_ready = true;
    return SG_OK;
}

/* What the choice of a cluster configuration needs to know of a device. */
struct ClusterInfo {
    int sms = 0;
    int fit[SG_NCVARIANTS] = {}; /* clusters that run at the same time */
};

/* Decodes in flight on a device, for cluster_for(): a cluster decodes one
 * codeword sooner than a CTA but takes more SM time over it, so callers that
 * decode small batches on streams of their own at the same time must share
 * the SMs, not each take them as if alone.  One event per stream, recorded
 * after its latest decode; earlier ones on that stream run before it, not
 * beside it.  At most MAX events, kept for later calls; streams beyond them
 * are not counted.  A wrong count costs time, never results.  2 dB, 4
 * codewords per call: 64 streams 13.0 -> 3.7 ms, one CTA per codeword 5.8; 16
 * streams 3.2 -> 1.3; 20 per call, 64 streams 23.1 -> 15.9; one stream pays
 * 1 us of host time. */
class Flights {
    static constexpr int MAX = 128, LOOK = 8;
    struct Call {
        unsigned long long stream, n;
        cudaEvent_t done;
        bool live;
    };
    std::mutex mu;
    Call call[MAX];
    int used = 0, first = 0;

public:
    /* Codewords in flight on other streams; calls that have ended are
     * dropped.  After LOOK running ones the rest are not asked and count as
     * running, so that a call's cost stays bounded; the next call starts
     * behind them. */
    unsigned long long others(unsigned long long stream)
    {
        std::lock_guard<std::mutex> lk(mu);
        const bool clean = cudaPeekAtLastError() == cudaSuccess;
        unsigned long long n = 0;
        int running = 0;
        for (int k = 0, from = first; k < used; k++) {
            const int i = (from + k) % used;
            Call& c = call[i];
            if (!c.live || c.stream == stream)
                continue;
            if (running < LOOK) {
                c.live = cudaEventQuery(c.done) == cudaErrorNotReady;
                running += c.live;
                first = i + 1;
            }
            if (c.live)
                n += c.n;
        }
        if (clean && running) /* "not ready" is no error of the caller's */
            cudaGetLastError();
        return n;
    }
    void launched(unsigned long long stream, cudaStream_t st, unsigned long long n)
    {
        std::lock_guard<std::mutex> lk(mu);
        Call* c = nullptr;
        for (int i = 0; i < used; i++) {
            if (call[i].stream == stream) {
                c = &call[i];
                break;
            }
            if (!call[i].live && !c)
                c = &call[i];
        }
        if (!c) {
            if (used == MAX)
                return;
            c = &call[used];
            if (cudaEventCreateWithFlags(&c->done, cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                return;
            }
            used++;
        }
        c->stream = stream;
        c->n = n;
        c->live = cudaEventRecord(c->done, st) == cudaSuccess;
    }
};

struct DevCtx {
    bool ready = false;
    uint32_t* enum_tabs = nullptr;
    unsigned int* err = nullptr;
    double* err_sink = nullptr; /* never-read output of the ceiling kernel */
    int sms = 0;
    ClusterInfo clusters;
    Flights flights;
};
DevCtx g_ctx[64];

cudaLaunchConfig_t cluster_config(int v, unsigned long long clusters, cudaStream_t st, cudaLaunchAttribute* at)
{
    const SgCVariant& c = k_cvariants[v];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * c.cs));
    cfg.blockDim = dim3(c.nw * 32);
    cfg.dynamicSmemBytes = c.smem;
    cfg.stream = st;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = c.cs;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

cudaError_t cluster_setup(int dev, ClusterInfo* info)
{
    cudaError_t e = cudaDeviceGetAttribute(&info->sms, cudaDevAttrMultiProcessorCount, dev);
    for (int v = 0; v < SG_NCVARIANTS && e == cudaSuccess; v++) {
        for (bool cr : {false, true}) {
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(cluster_fn(v, cr), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)k_cvariants[v].smem);
            if (e == cudaSuccess && k_cvariants[v].cs > 8)
                e = cudaFuncSetAttribute(cluster_fn(v, cr), cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        }
        if (e == cudaSuccess) {
            cudaLaunchAttribute at;
            const cudaLaunchConfig_t cfg = cluster_config(v, 1, nullptr, &at);
            e = cudaOccupancyMaxActiveClusters(&info->fit[v], cluster_fn(v, false), &cfg);
        }
    }
    return e;
}

/* The cluster configuration for a batch of n codewords, -1 when it is large
 * enough for one CTA per codeword: the most CTAs per codeword with which all
 * clusters run at the same time; with two, also up to 7/4 codewords per SM.
 * B200, one call at 2 dB, when the rule was set: n = 1 plain 2.29 ms, 16 CTAs
 * 0.43, 8 CTAs 0.52; n = 9: 8 CTAs 0.58, 16 (the ninth cluster waits) 0.66;
 * n = 18: 4 CTAs 1.02, 8 1.18; n = 33: 4 CTAs 1.02, 2 1.57; n = 37 (one too
 * many): 4 CTAs 1.66, 2 1.74; n = 100: 2 CTAs 2.00, plain 3.81; n = 220: 3.92,
 * 4.46; n = 296: 4.35, 4.63 but 4.51 in the batched form; n = 600: 8.7, 8.5.
 * With `others` in flight on other streams, at most three times the clusters
 * that run at the same time: their codewords end at different times and let
 * waiting clusters in, until the SM time that large clusters cost decides.
 * 2 dB, several streams of n codewords, ms a round, as if alone / at most
 * once / twice / three times: 16 of 1 0.83 / 0.69 / 0.67 / 0.84; 64 of 4 13.0
 * / 3.5 / 3.7 / 3.8; 1 dB, 4 of 3 2.7 / 3.5 / 2.7 / 2.7; 6 of 3 3.2 / - / 3.5
 * / 3.2: only with three is nothing slower than as if alone.  Two CTAs per
 * codeword cost a tenth more SM time than one, so these take any number. */
int cluster_for(unsigned long long n, unsigned long long others, const ClusterInfo& info)
{
    constexpr int last = SG_NCVARIANTS - 1;
    for (int v = 0; v < SG_NCVARIANTS; v++) {
        const unsigned long long fit = (unsigned long long)info.fit[v];
        if (n <= fit && (v == last || n + others <= 3 * fit))
            return v;
    }
    return info.fit[last] > 0 && 4 * n <= 7ull * info.sms ? last : -1;
}

cudaError_t launch_cluster(const SgDecodeArgs& a, int v, int mode, cudaStream_t st)
{
    void* kargs[] = {(void*)&a};
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t cfg = cluster_config(v, a.n_cw, st, &at);
    return cudaLaunchKernelExC(&cfg, cluster_fn(v, mode == 1), kargs);
}

/* The choice and launch of one decode on `st` beside those of `fl` (NULL: as
 * if alone): launch(v) starts cluster configuration v, -1 the form for more
 * codewords.  A stream under capture is taken as alone: its launches run
 * when the graph does. */
template <class F>
cudaError_t launch_small_or(unsigned long long n, const ClusterInfo& info, Flights* fl, cudaStream_t st, F launch)
{
    unsigned long long id = 0;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (!fl || cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone ||
        cudaStreamGetId(st, &id) != cudaSuccess)
        return launch(cluster_for(n, 0, info));
    /* event calls are legal here whatever other streams are capturing */
    cudaStreamCaptureMode was = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&was);
    const int v = cluster_for(n, 0, info) >= 0 ? cluster_for(n, fl->others(id), info) : -1;
    cudaThreadExchangeStreamCaptureMode(&was);
    const cudaError_t e = launch(v);
    if (e == cudaSuccess) {
        was = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&was);
        fl->launched(id, st, n);
        cudaThreadExchangeStreamCaptureMode(&was);
    }
    return e;
}

/* Launch of the plain form. */
cudaError_t launch_decode(const SgDecodeArgs& a, const ClusterInfo& info, Flights* fl, int mode, cudaStream_t st)
{
    const int vi = g_variant_by_mode[mode];
    auto launch = [&](int cv) {
        if (cv >= 0)
            return launch_cluster(a, cv, mode, st);
        const SgVariant& v = k_variants[vi];
        void* kargs[] = {(void*)&a};
        return cudaLaunchKernel(decode_fn(vi, mode == 1), dim3((unsigned)std::min<unsigned long long>(a.n_cw, 1 << 30)),
                                dim3(v.nw * 32), kargs, v.smem, st);
    };
    /* as in the batched form, a lowered wait limit keeps a kernel that waits */
    const bool cl = k_variants[vi].clusters && (!k_variants[vi].lch_smem || a.wait_limit == SG_WAIT_LIMIT_DEFAULT);
    return cl ? launch_small_or(a.n_cw, info, fl, st, launch) : launch(-1);
}

sg_status get_ctx(DevCtx** out)
{
    int dev = 0;
    SG_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64)
        return fail(SG_ERR_ARG, "device index out of range");
    std::lock_guard<std::mutex> lk(g_mu);
    DevCtx& c = g_ctx[dev];
    if (!c.ready) {
        sg_status s = host_init_locked();
        if (s != SG_OK)
            return s;
        const size_t bytes = g_enum_host.size() * sizeof(uint32_t);
        SG_CUDA(cudaMalloc(&c.enum_tabs, bytes));
        SG_CUDA(cudaMemcpy(c.enum_tabs, g_enum_host.data(), bytes, cudaMemcpyHostToDevice));
        SG_CUDA(cudaMalloc(&c.err, sizeof(unsigned int)));
        SG_CUDA(cudaMalloc(&c.err_sink, 148 * 64 * sizeof(double)));
        SG_CUDA(cudaMemset(c.err, 0, sizeof(unsigned int)));
        SG_CUDA(sg_load_code(g_code));
        SG_CUDA(sg_cr_load_code(g_code));
        for (int v = 0; v < SG_NVARIANTS; v++) {
            SG_CUDA(cudaFuncSetAttribute(decode_fn(v, false), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)k_variants[v].smem));
            SG_CUDA(cudaFuncSetAttribute(decode_fn(v, true), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)k_variants[v].smem));
        }
        for (int v = 0; v < SG_NPVARIANTS; v++) {
            SG_CUDA(cudaFuncSetAttribute(persist_fn(v, false), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)k_pvariants[v].smem));
            SG_CUDA(cudaFuncSetAttribute(persist_fn(v, true), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)k_pvariants[v].smem));
        }
        SG_CUDA(cluster_setup(dev, &c.clusters));
        for (int v = 0; v < 2; v++)
            for (bool cr : {false, true})
                SG_CUDA(cudaFuncSetAttribute(bitso_fn(v, cr), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)k_bvariants[v].smem));
        SG_CUDA(cudaFuncSetAttribute(sg_gen_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SgGenSmem)));
        SG_CUDA(cudaFuncSetAttribute(sg_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(SgBackSmem)));
        SG_CUDA(cudaDeviceGetAttribute(&c.sms, cudaDevAttrMultiProcessorCount, dev));
        c.ready = true;
    }
    *out = &c;
    return SG_OK;
}

sg_status check_params(const sg_params* p)
{
    if (!p)
        return fail(SG_ERR_ARG, "params is NULL");
    if (p->L < 1 || p->L > SG_MAX_L)
        return fail(SG_ERR_ARG, "L must be in [1, 8]");
    if (p->Imax < 1 || p->Imax > SG_MAX_IMAX)
        return fail(SG_ERR_ARG, "Imax must be in [1, 50]");
    if (!(p->thres == p->thres))
        return fail(SG_ERR_ARG, "thres is NaN");
    for (int i = 0; i < 3 * p->Imax; i++)
        if (!isfinite(p->alpha[i]))
            return fail(SG_ERR_ARG, "alpha must be finite");
    return SG_OK;
}

uint32_t tmax_eff(uint64_t tmax)
{
    if (tmax == 0)
        return 0x7fffffffu; /* if (Tmax==0) Tmax=Inf, :607 */
    return tmax > 0xffffffffull ? 0xffffffffu : (uint32_t)tmax;
}

/* Starts of the logistic weights of every IC's pattern order, counted once. */
struct OrderStarts {
    std::vector<uint32_t> start[SG_ENUM_NTAB];
    uint32_t h3[SG_ENUM_NTAB];
    OrderStarts()
    {
        uint32_t cnt[17][137];
        sg_enum_counts(cnt);
        for (int ic = 0; ic < SG_ENUM_NTAB; ic++) {
            start[ic].resize(16 * ic + 136);
            start[ic].resize(sg_enum_starts(ic, cnt, start[ic].data(), &h3[ic]));
        }
    }
};

/* sg_order_meta for a Tmax as tmax_eff() gives it: the first weight that
 * starts at or after Tmax ends the decode. */
void order_meta(uint32_t tmax, sg_order_meta* m)
{
    static const OrderStarts o;
    for (int ic = 0; ic < SG_ENUM_NTAB; ic++) {
        m->h3[ic] = o.h3[ic];
        m->lim[ic] = SG_ENUM_LEN;
        if (tmax < SG_ENUM_LEN) {
            const auto it = std::lower_bound(o.start[ic].begin(), o.start[ic].end(), tmax);
            if (it != o.start[ic].end())
                m->lim[ic] = *it;
        }
    }
}

int grid_for(unsigned long long n, int cap)
{
    return (int)(n < (unsigned long long)cap ? n : (unsigned long long)cap);
}

/* Host-buffer decode through the batched persistent decoder, defined with
 * the batch handles below. */
sg_status decode_host_pipelined(const double* llr, size_t n_cw, const sg_params* p, uint8_t* bits, double* lapp,
                                sg_cw_stats* stats);
/* The file decoder's pipeline, defined with them. */
sg_status decode_file_pipelined(FILE* fi, FILE* fo, const sg_params* p, size_t chunk_cw, sg_run_summary* sum,
                                bool* any_nonfinite);

} // namespace

extern "C" {

void sg_params_default(sg_params* p)
{
    if (!p)
        return;
    memset(p, 0, sizeof *p);
    p->L = 3;
    p->Imax = 30;
    p->Tmax = UINT64_MAX;
    p->thres = 1.0 - 1e-5;
    for (int i = 0; i < SG_MAX_PHASES; i++)
        p->alpha[i] = 0.7;
}

namespace {
/* The decode with checked arguments; d_bits, d_lapp, d_stats and d_summary
 * may each be NULL, d_ref is for the summary. */
sg_status decode_device(const double* d_llr, size_t n_cw, const sg_params* p, uint8_t* d_bits, double* d_lapp,
                        sg_cw_stats* d_stats, sg_decode_summary* d_summary, const uint8_t* d_ref, void* stream)
{
    sg_status s;
    DevCtx* c = nullptr;
    if ((s = get_ctx(&c)) != SG_OK)
        return s;
    SgDecodeArgs a;
    memset(&a, 0, sizeof a);
    a.llr = d_llr;
    a.bits = d_bits;
    a.lapp = d_lapp;
    a.stats = d_stats;
    a.sum = d_summary;
    a.ref = d_ref;
    a.enum_tabs = c->enum_tabs;
    a.err = c->err;
    a.n_cw = n_cw;
    a.wait_limit = g_wait_limit.load();
    a.L = p->L;
    a.imax = p->Imax;
    order_meta(tmax_eff(p->Tmax), &a.meta);
    a.use_bulk = ((uintptr_t)d_llr & 15u) == 0;
    a.thres = p->thres;
    memcpy(a.alpha, p->alpha, sizeof a.alpha);
    a.k = k_consts;
    SG_CUDA(launch_decode(a, c->clusters, &c->flights, g_math_mode.load(), (cudaStream_t)stream));
    return SG_OK;
}

} // namespace

sg_status sg_decode_device(const double* d_llr, size_t n_cw, const sg_params* p, uint8_t* d_bits,
                           double* d_lapp, sg_cw_stats* d_stats, void* stream)
{
    sg_status s = check_params(p);
    if (s != SG_OK)
        return s;
    if (n_cw == 0)
        return SG_OK;
    if (!d_llr || !d_bits)
        return fail(SG_ERR_ARG, "llr and bits must not be NULL");
    if ((uintptr_t)d_llr & 7u)
        return fail(SG_ERR_ARG, "llr must be 8-byte aligned");
    return decode_device(d_llr, n_cw, p, d_bits, d_lapp, d_stats, nullptr, nullptr, stream);
}

sg_status sg_bitso_device(const double* d_llr, size_t n_lines, int32_t L, uint64_t Tmax, double thres,
                          double* d_lapp, double* d_le, int32_t* d_nguess, int32_t* d_ncw, void* stream)
{
    if (L < 1 || L > SG_MAX_L)
        return fail(SG_ERR_ARG, "L must be in [1, 8]");
    if (n_lines == 0)
        return SG_OK;
    if (!d_llr || !d_lapp || !d_le || !d_nguess)
        return fail(SG_ERR_ARG, "NULL buffer");
    DevCtx* c = nullptr;
    sg_status s = get_ctx(&c);
    if (s != SG_OK)
        return s;
    sg_order_meta meta;
    order_meta(tmax_eff(Tmax), &meta);
    /* up to 16 lines per SM: one per warp, in CTAs spread over the SMs; more:
     * two CTAs of 16 warps on every SM, each with an equal share, which fill
     * their tables once.  The line is where the two meet.  148 SMs, 1 / 2 / 3
     * dB, us, one per warp against resident: 2 000 lines 33 / 35 / 39 and 35 /
     * 35 / 39, 2 368 equal, 4 000 38 / 45 / 51 and 37 / 38 / 42, 4 736 51 / 54
     * / 59 and 41 / 44 / 48, 65 537 327 / 338 / 354 and 232 / 236 / 242;
     * correctly rounded, 2 dB: 1 000 39 and 43, 2 368 41 and 43, 3 552 57 and
     * 46. */
    const unsigned long long full = 2ull * c->sms;
    const int bv = n_lines > 8 * full ? 1 : 0;
    const SgBVariant& v = k_bvariants[bv];
    unsigned long long n = n_lines, per = bv ? (n + full - 1) / full : (n < full ? 1 : v.nw);
    const uint32_t* tabs = c->enum_tabs;
    SgK k = k_consts;
    void* kargs[] = {&d_llr, &n, &per, &L, &thres, &d_lapp, &d_le, &d_nguess, &d_ncw, &tabs, &k, &meta};
    SG_CUDA(cudaLaunchKernel(bitso_fn(bv, g_math_mode.load() == 1), dim3((unsigned)((n + per - 1) / per)),
                             dim3(v.nw * 32), kargs, v.smem, (cudaStream_t)stream));
    return SG_OK;
}

namespace {

/* Pinned staging of a thread's small line calls, mapped into the devices'
 * address spaces; freed when the thread ends. */
struct LineStage {
    static constexpr size_t MAX = 256; /* lines: 100 KB per thread */
    unsigned char* p = nullptr;
    ~LineStage()
    {
        if (p)
            cudaFreeHost(p);
    }
};

/* sg_bitso_host for few lines: the kernel reads the LLRs from pinned host
 * memory and writes its results there, so a call is one launch and one wait,
 * on the thread's own stream.  16 lines: 41 us, with five allocations, six
 * copies and five frees per call 116; 256 lines: 60 us, 158.  The line at 256
 * bounds what a thread keeps pinned.  *done = false: not possible here (no
 * pinned memory), nothing happened. */
sg_status bitso_host_small(const double* llr, size_t n, int32_t L, uint64_t Tmax, double thres, double* lapp, double* le,
                           int32_t* nguess, int32_t* ncw, bool* done)
{
    static thread_local LineStage st;
    *done = false;
    if (!st.p) {
        const size_t bytes = LineStage::MAX * (3 * 16 * sizeof(double) + 2 * sizeof(int32_t));
        if (cudaHostAlloc((void**)&st.p, bytes, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
            cudaGetLastError();
            st.p = nullptr;
            return SG_OK;
        }
    }
    double* h = reinterpret_cast<double*>(st.p); /* LLRs, L_APP, L_E, guesses, codewords */
    double *ha = h + 16 * LineStage::MAX, *he = ha + 16 * LineStage::MAX;
    int32_t *hn = reinterpret_cast<int32_t*>(he + 16 * LineStage::MAX), *hc = hn + LineStage::MAX;
    memcpy(h, llr, n * 16 * sizeof(double));
    *done = true;
    /* unified addressing: the host pointers are valid on the device */
    const sg_status s = sg_bitso_device(h, n, L, Tmax, thres, ha, he, hn, hc, (void*)cudaStreamPerThread);
    if (s != SG_OK)
        return s;
    SG_CUDA(cudaStreamSynchronize(cudaStreamPerThread));
    memcpy(lapp, ha, n * 16 * sizeof(double));
    memcpy(le, he, n * 16 * sizeof(double));
    memcpy(nguess, hn, n * sizeof(int32_t));
    if (ncw)
        memcpy(ncw, hc, n * sizeof(int32_t));
    return SG_OK;
}

} // namespace

sg_status sg_bitso_host(const double* llr, size_t n_lines, int32_t L, uint64_t Tmax, double thres,
                        double* lapp, double* le, int32_t* nguess, int32_t* ncw)
{
    if (n_lines == 0)
        return SG_OK;
    if (!llr || !lapp || !le || !nguess)
        return fail(SG_ERR_ARG, "NULL buffer");
    if (n_lines <= LineStage::MAX) {
        bool done;
        const sg_status s = bitso_host_small(llr, n_lines, L, Tmax, thres, lapp, le, nguess, ncw, &done);
        if (done)
            return s;
    }
    double *dl = nullptr, *da = nullptr, *de = nullptr;
    int32_t *dn = nullptr, *dc = nullptr;
    const size_t vb = n_lines * 16 * sizeof(double), ib = n_lines * sizeof(int32_t);
    sg_status s = SG_OK;
    cudaError_t e;
    if ((e = cudaMalloc(&dl, vb)) != cudaSuccess || (e = cudaMalloc(&da, vb)) != cudaSuccess ||
        (e = cudaMalloc(&de, vb)) != cudaSuccess || (e = cudaMalloc(&dn, ib)) != cudaSuccess ||
        (e = cudaMalloc(&dc, ib)) != cudaSuccess) {
        s = cuda_fail(e, "cudaMalloc");
    } else if ((e = cudaMemcpy(dl, llr, vb, cudaMemcpyHostToDevice)) != cudaSuccess) {
        s = cuda_fail(e, "cudaMemcpy H2D");
    } else if ((s = sg_bitso_device(dl, n_lines, L, Tmax, thres, da, de, dn, dc, nullptr)) == SG_OK) {
        if ((e = cudaDeviceSynchronize()) != cudaSuccess ||
            (e = cudaMemcpy(lapp, da, vb, cudaMemcpyDeviceToHost)) != cudaSuccess ||
            (e = cudaMemcpy(le, de, vb, cudaMemcpyDeviceToHost)) != cudaSuccess ||
            (e = cudaMemcpy(nguess, dn, ib, cudaMemcpyDeviceToHost)) != cudaSuccess ||
            (ncw && (e = cudaMemcpy(ncw, dc, ib, cudaMemcpyDeviceToHost)) != cudaSuccess))
            s = cuda_fail(e, "bitso copy-out");
    }
    cudaFree(dl);
    cudaFree(da);
    cudaFree(de);
    cudaFree(dn);
    cudaFree(dc);
    return s;
}

sg_status sg_decode_host(const double* llr, size_t n_cw, const sg_params* p, uint8_t* bits, double* lapp,
                         sg_cw_stats* stats)
{
    sg_status s = check_params(p);
    if (s != SG_OK)
        return s;
    if (n_cw == 0)
        return SG_OK;
    if (!llr || !bits)
        return fail(SG_ERR_ARG, "llr and bits must not be NULL");
    return decode_host_pipelined(llr, n_cw, p, bits, lapp, stats);
}

sg_status sg_decode_file(const char* in_path, const char* out_path, const sg_params* p, size_t chunk_cw,
                         sg_run_summary* summary)
{
    sg_status s = check_params(p);
    if (s != SG_OK)
        return s;
    if (!in_path || !out_path)
        return fail(SG_ERR_ARG, "NULL path");
    const auto t0 = std::chrono::steady_clock::now();
    FILE* fi = fopen(in_path, "rb");
    if (!fi)
        return fail(SG_ERR_IO, std::string("Error opening input file: ") + strerror(errno));
    FILE* fo = fopen(out_path, "wb");
    if (!fo) {
        fclose(fi);
        return fail(SG_ERR_IO, std::string("Error opening output file: ") + strerror(errno));
    }
    sg_run_summary sum;
    memset(&sum, 0, sizeof sum);
    bool nonfinite = false;
    s = decode_file_pipelined(fi, fo, p, chunk_cw, &sum, &nonfinite);
    fclose(fi);
    if (fclose(fo) != 0 && s == SG_OK)
        s = fail(SG_ERR_IO, "error closing output file");
    if (s == SG_OK && nonfinite)
        s = fail(SG_ERR_NONFINITE, "input contains non-finite LLRs; those codewords were not decoded");
    sum.seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (summary)
        *summary = sum;
    return s;
}

double sg_channel_sigma(double ebn0_db)
{
    const int n = 16, k = 8;
    const double R = pow((double)k / n, 3);
    const double es = ebn0_db + 10 * log10(2 * R);
    return 1.0 / sqrt(pow(10, es / 10.0));
}

sg_status sg_gen_info_host(uint64_t seed, uint64_t cw0, size_t n_cw, uint8_t* info)
{
    if (!info && n_cw)
        return fail(SG_ERR_ARG, "info is NULL");
    for (size_t c = 0; c < n_cw; c++)
        for (int w = 0; w < 8; w++) {
            const uint64_t r = sg_rand(seed, 0, (cw0 + c) * 8 + w);
            for (int q = 0; q < 8; q++)
                info[c * SG_INFO_BYTES + w * 8 + q] = (uint8_t)(r >> (8 * q));
        }
    return SG_OK;
}

sg_status sg_encode_host(const uint8_t* info, size_t n_cw, uint8_t* code_bits)
{
    if ((!info || !code_bits) && n_cw)
        return fail(SG_ERR_ARG, "NULL buffer");
    {
        std::lock_guard<std::mutex> lk(g_mu);
        sg_status s = host_init_locked();
        if (s != SG_OK)
            return s;
    }
    uint16_t W[256];
    for (size_t c = 0; c < n_cw; c++) {
        sg_encode_words(info + c * SG_INFO_BYTES, g_code.prow, g_code.ptab, W);
        for (int p = 0; p < SG_CUBE; p++)
            code_bits[c * SG_CUBE + p] = (uint8_t)((W[p >> 4] >> (p & 15)) & 1);
    }
    return SG_OK;
}

sg_status sg_gen_llr_host(uint64_t seed, uint64_t cw0, size_t n_cw, double sigma, double ebn0_lo_db,
                          double ebn0_hi_db, uint8_t* info, double* llr)
{
    if (!llr && n_cw)
        return fail(SG_ERR_ARG, "llr is NULL");
    {
        std::lock_guard<std::mutex> lk(g_mu);
        sg_status s = host_init_locked();
        if (s != SG_OK)
            return s;
    }
    uint8_t ib[SG_INFO_BYTES];
    uint16_t W[256];
    for (size_t c = 0; c < n_cw; c++) {
        const uint64_t gc = cw0 + c;
        sg_gen_info_host(seed, gc, 1, ib);
        if (info)
            memcpy(info + c * SG_INFO_BYTES, ib, SG_INFO_BYTES);
        sg_encode_words(ib, g_code.prow, g_code.ptab, W);
        const double s = sigma > 0.0 ? sigma : sg_sigma_draw(seed, gc, ebn0_lo_db, ebn0_hi_db, k_etab_tab);
        for (int p = 0; p < SG_CUBE; p++) {
            const int bit = (W[p >> 4] >> (p & 15)) & 1;
            llr[c * SG_CUBE + p] = sg_llr_of(bit, s, sg_normal(seed, gc, (uint32_t)p, k_ltab_tab));
        }
    }
    return SG_OK;
}

sg_status sg_gen_llr_device(uint64_t seed, uint64_t cw0, size_t n_cw, double sigma, double ebn0_lo_db,
                            double ebn0_hi_db, uint8_t* d_info, double* d_llr, void* stream)
{
    if (n_cw == 0)
        return SG_OK;
    if (!d_llr)
        return fail(SG_ERR_ARG, "llr is NULL");
    if ((uintptr_t)d_llr & 7u)
        return fail(SG_ERR_ARG, "llr must be 8-byte aligned");
    DevCtx* c = nullptr;
    sg_status s = get_ctx(&c);
    if (s != SG_OK)
        return s;
    sg_gen_kernel<<<grid_for(n_cw, 148 * 16), SG_THREADS, sizeof(SgGenSmem), (cudaStream_t)stream>>>(
        seed, cw0, n_cw, sigma, ebn0_lo_db, ebn0_hi_db, d_info, d_llr, k_consts);
    SG_CUDA(cudaGetLastError());
    return SG_OK;
}

size_t sg_pattern_order(int32_t ic, uint32_t* out, size_t cap)
{
    if (ic < 0 || !out)
        return 0;
    std::vector<uint32_t> t(SG_ENUM_LEN);
    const size_t n = sg_enum_build_impl(ic, t.data());
    const size_t m = n < cap ? n : cap;
    int32_t prev = 0;
    for (size_t i = 0; i < m; i++) {
        const uint32_t pat = sg_ent_pattern(t[i]);
        const int32_t wt = sg_enum_weight(ic, pat);
        out[i] = pat | (i && wt != prev ? SG_ENUM_GS : 0u);
        prev = wt;
    }
    return m;
}

sg_status sg_decode_summary_device(const double* d_llr, size_t n_cw, const sg_params* p,
                                   const uint8_t* d_ref_info, uint8_t* d_bits, sg_decode_summary* d_summary,
                                   void* stream)
{
    if (!d_summary)
        return fail(SG_ERR_ARG, "summary must not be NULL");
    if (d_ref_info && ((uintptr_t)d_ref_info & 15u))
        return fail(SG_ERR_ARG, "ref_info must be 16-byte aligned");
    if (d_bits && ((uintptr_t)d_bits & 15u))
        return fail(SG_ERR_ARG, "bits must be 16-byte aligned");
    sg_status s = check_params(p);
    if (s != SG_OK)
        return s;
    cudaStream_t st = (cudaStream_t)stream;
    SG_CUDA(cudaMemsetAsync(d_summary, 0, sizeof(sg_decode_summary), st));
    if (n_cw == 0)
        return SG_OK;
    if (!d_llr)
        return fail(SG_ERR_ARG, "llr must not be NULL");
    if ((uintptr_t)d_llr & 7u)
        return fail(SG_ERR_ARG, "llr must be 8-byte aligned");
    /* the decode kernels add each codeword to the totals: with its statistics
     * in memory allocated per call and a second kernel, 2 000 codewords at
     * 1 dB took 95.9 ms, 47 at 2.3 dB 1.2 to 4.7 ms */
    return decode_device(d_llr, n_cw, p, d_bits, nullptr, nullptr, d_summary, d_ref_info, stream);
}

sg_status sg_wilson_interval(uint64_t k, uint64_t n, double z, double* lo, double* hi)
{
    if (!lo || !hi || n == 0 || k > n || !(z > 0))
        return fail(SG_ERR_ARG, "wilson interval needs 0 <= k <= n, n > 0, z > 0");
    const double nn = (double)n, ph = (double)k / nn, z2 = z * z;
    const double den = 1.0 + z2 / nn;
    const double c = (ph + z2 / (2 * nn)) / den;
    const double h = z * sqrt(ph * (1 - ph) / nn + z2 / (4 * nn * nn)) / den;
    *lo = (k == 0 || c - h < 0) ? 0.0 : c - h;
    *hi = (k == n || c + h > 1) ? 1.0 : c + h;
    return SG_OK;
}

namespace {

struct NoAllocCtx {
    bool ready = false;
    unsigned int* err = nullptr;      /* device address of g_noalloc_err */
    uint32_t* enum_tabs = nullptr;    /* device address of g_noalloc_enum */
    ClusterInfo clusters;
};
NoAllocCtx g_noalloc[64];

/* Once per device, with that device current: resolve the static arrays'
 * device addresses, load the code tables, build the pattern orders on the
 * device, allow the decode kernels their shared memory.  No allocation. */
sg_status noalloc_setup(NoAllocCtx** out)
{
    int dev = 0;
    SG_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64)
        return fail(SG_ERR_ARG, "device index out of range");
    std::lock_guard<std::mutex> lk(g_mu);
    NoAllocCtx& c = g_noalloc[dev];
    if (!c.ready) {
        sg_code_tables code;
        sg_code_build(&code);
        SG_CUDA(cudaGetSymbolAddress((void**)&c.err, g_noalloc_err));
        SG_CUDA(cudaGetSymbolAddress((void**)&c.enum_tabs, g_noalloc_enum));
        SG_CUDA(sg_load_code(code));
        SG_CUDA(sg_cr_load_code(code));
        for (int v = 0; v < SG_NVARIANTS; v++) {
            SG_CUDA(cudaFuncSetAttribute(decode_fn(v, false), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)k_variants[v].smem));
            SG_CUDA(cudaFuncSetAttribute(decode_fn(v, true), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)k_variants[v].smem));
        }
        SG_CUDA(cluster_setup(dev, &c.clusters));
        unsigned int* ok = c.err; /* SG_ENUM_NTAB words */
        SG_CUDA(cudaMemset(ok, 0, SG_ENUM_NTAB * sizeof(unsigned int)));
        sg_enum_build_kernel<<<1, 64>>>(c.enum_tabs, ok);
        SG_CUDA(cudaGetLastError());
        unsigned int hok[SG_ENUM_NTAB];
        SG_CUDA(cudaMemcpy(hok, ok, sizeof hok, cudaMemcpyDeviceToHost));
        for (int i = 0; i < SG_ENUM_NTAB; i++)
            if (hok[i] != 1u)
                return fail(SG_ERR_ARG, "device pattern-order build incomplete");
        c.ready = true;
    }
    *out = &c;
    return SG_OK;
}

} // namespace

sg_status sg_decode_summary_device_noalloc(const double* d_llr, size_t n_cw, const sg_params* p,
                                           const uint8_t* d_ref_info, uint8_t* d_bits,
                                           sg_decode_summary* d_summary, void* stream)
{
    if (!d_summary)
        return fail(SG_ERR_ARG, "summary must not be NULL");
    if (n_cw > SG_NOALLOC_MAX_CW)
        return fail(SG_ERR_ARG, "n_cw exceeds SG_NOALLOC_MAX_CW (16384) for the allocation-free entry point");
    if (d_ref_info && ((uintptr_t)d_ref_info & 15u))
        return fail(SG_ERR_ARG, "ref_info must be 16-byte aligned");
    if (d_bits && ((uintptr_t)d_bits & 15u))
        return fail(SG_ERR_ARG, "bits must be 16-byte aligned");
    if (n_cw && !d_llr)
        return fail(SG_ERR_ARG, "llr must not be NULL");
    if ((uintptr_t)d_llr & 7u)
        return fail(SG_ERR_ARG, "llr must be 8-byte aligned");
    sg_status s = check_params(p);
    if (s != SG_OK)
        return s;
    NoAllocCtx* c = nullptr;
    if ((s = noalloc_setup(&c)) != SG_OK)
        return s;
    cudaStream_t st = (cudaStream_t)stream;
    SG_CUDA(cudaMemsetAsync(d_summary, 0, sizeof(sg_decode_summary), st));
    if (n_cw == 0)
        return SG_OK;
    /* the flag keeps the previous call's contents */
    unsigned int* err = c->err;
    SG_CUDA(cudaMemsetAsync(err, 0, sizeof(unsigned int), st));
    SgDecodeArgs a;
    memset(&a, 0, sizeof a);
    a.llr = d_llr;
    a.bits = d_bits;
    a.lapp = nullptr;
    a.sum = d_summary;
    a.ref = d_ref_info;
    a.enum_tabs = c->enum_tabs;
    a.err = err;
    a.n_cw = n_cw;
    a.wait_limit = g_wait_limit.load();
    a.L = p->L;
    a.imax = p->Imax;
    order_meta(tmax_eff(p->Tmax), &a.meta);
    a.use_bulk = ((uintptr_t)d_llr & 15u) == 0;
    a.thres = p->thres;
    memcpy(a.alpha, p->alpha, sizeof a.alpha);
    a.k = k_consts;
    /* no events here: they may take memory, and calls do not overlap */
    SG_CUDA(launch_decode(a, c->clusters, nullptr, g_math_mode.load(), st));
    return SG_OK;
}

} // extern "C"

struct sg_batch_s {
    int device = -1;
    SgQueue* q = nullptr;
    cudaGraphExec_t exec = nullptr;
};

namespace {

sg_status batch_enqueue(sg_batch b, const double* d_llr, size_t n_cw, const sg_params* p, uint8_t* d_bits,
                        double* d_lapp, sg_cw_stats* d_stats, cudaStream_t st)
{
    sg_status s = check_params(p);
    if (s != SG_OK)
        return s;
    if (!b || !b->q)
        return fail(SG_ERR_ARG, "invalid batch handle");
    if (n_cw && (!d_llr || !d_bits))
        return fail(SG_ERR_ARG, "llr and bits must not be NULL");
    if ((uintptr_t)d_llr & 7u)
        return fail(SG_ERR_ARG, "llr must be 8-byte aligned");
    int dev = 0;
    SG_CUDA(cudaGetDevice(&dev));
    if (dev != b->device)
        return fail(SG_ERR_ARG, "batch handle belongs to another device");
    DevCtx* c = nullptr;
    if ((s = get_ctx(&c)) != SG_OK)
        return s;
    SG_CUDA(cudaMemsetAsync(b->q, 0, sizeof(SgQueue), st));
    if (n_cw == 0)
        return SG_OK;
    SgDecodeArgs a;
    memset(&a, 0, sizeof a);
    a.llr = d_llr;
    a.bits = d_bits;
    a.lapp = d_lapp;
    a.stats = d_stats;
    a.enum_tabs = c->enum_tabs;
    a.err = c->err;
    a.n_cw = n_cw;
    a.wait_limit = g_wait_limit.load();
    a.L = p->L;
    a.imax = p->Imax;
    order_meta(tmax_eff(p->Tmax), &a.meta);
    a.use_bulk = 0;
    a.thres = p->thres;
    memcpy(a.alpha, p->alpha, sizeof a.alpha);
    a.k = k_consts;
    const int mode = g_math_mode.load(), vi = g_pvariant_by_mode[mode];
    auto launch = [&](int cv) {
        if (cv >= 0)
            return launch_cluster(a, cv, mode, st);
        const SgPVariant& v = k_pvariants[vi];
        SgQueue* q = b->q;
        void* kargs[] = {(void*)&a, (void*)&q};
        const int grid = (int)(n_cw < (size_t)c->sms ? n_cw : (size_t)c->sms);
        return cudaLaunchKernel(persist_fn(vi, mode == 1), dim3(grid), dim3(v.nw * 32), kargs, v.smem, st);
    };
    /* a small batch goes to clusters; under a lowered wait limit it keeps the
     * kernel whose waits that limit bounds (clusters only meet at hardware
     * barriers) */
    if (k_pvariants[vi].clusters && a.wait_limit == SG_WAIT_LIMIT_DEFAULT)
        SG_CUDA(launch_small_or(n_cw, c->clusters, &c->flights, st, launch));
    else
        SG_CUDA(launch(-1));
    return SG_OK;
}

/* One half of the host-buffer pipeline: device buffers for one chunk, its
 * stream and its work queue. */
struct HostLane {
    double* dl = nullptr;
    double* da = nullptr;
    uint8_t* db = nullptr;
    sg_cw_stats* dst = nullptr;
    cudaStream_t st = nullptr;
    sg_batch_s b;
    size_t off = 0, n = 0;
};

/* Device resources of the host-buffer pipeline, kept per device across
 * calls so that a call allocates nothing after the first: two lanes of
 * chunk buffers, their streams and work queues.  Calls on one device are
 * serialised by the mutex. */
constexpr int SG_HOST_LANES = 2;
constexpr size_t SG_HOST_CHUNK = 16384;
/* Pinned host staging of the file decoder: SG_FILE_BUFS chunks of LLR cubes
 * (a reader thread fills one while the lanes decode the others) and the
 * bits and statistics of each lane's chunk. */
constexpr size_t SG_FILE_CHUNK = 8192;
constexpr int SG_FILE_BUFS = 3;
struct FileStage {
    double* llr[SG_FILE_BUFS] = {};
    uint8_t* bits[SG_HOST_LANES] = {};
    sg_cw_stats* st[SG_HOST_LANES] = {};
    bool ready = false;
};
struct HostPipe {
    std::mutex mu;
    HostLane ln[SG_HOST_LANES];
    bool ready = false;     /* buffers (without L_APP), streams and queues */
    bool has_lapp = false;  /* L_APP buffers too */
    FileStage fs;           /* pinned staging, allocated by the first file decode */
};
constexpr int SG_HOST_MAX_DEV = 64;
HostPipe g_host_pipe[SG_HOST_MAX_DEV];

sg_status host_pipe_setup(HostPipe& hp, int dev, bool want_lapp)
{
    cudaError_t e = cudaSuccess;
    if (!hp.ready) {
        for (HostLane& L : hp.ln) {
            L.b.device = dev;
            if ((e = cudaMalloc(&L.dl, SG_HOST_CHUNK * SG_CUBE * sizeof(double))) != cudaSuccess ||
                (e = cudaMalloc(&L.db, SG_HOST_CHUNK * SG_INFO_BYTES)) != cudaSuccess ||
                (e = cudaMalloc(&L.dst, SG_HOST_CHUNK * sizeof(sg_cw_stats))) != cudaSuccess ||
                (e = cudaMalloc(&L.b.q, sizeof(SgQueue))) != cudaSuccess ||
                (e = cudaStreamCreateWithFlags(&L.st, cudaStreamNonBlocking)) != cudaSuccess)
                break;
        }
        if (e != cudaSuccess) { /* undo a partial set-up; the next call retries */
            for (HostLane& L : hp.ln) {
                cudaFree(L.dl);
                cudaFree(L.db);
                cudaFree(L.dst);
                cudaFree(L.b.q);
                if (L.st)
                    cudaStreamDestroy(L.st);
                L = HostLane();
            }
            return cuda_fail(e, "host pipeline buffers");
        }
        hp.ready = true;
    }
    if (want_lapp && !hp.has_lapp) {
        for (HostLane& L : hp.ln)
            if ((e = cudaMalloc(&L.da, SG_HOST_CHUNK * SG_CUBE * sizeof(double))) != cudaSuccess)
                break;
        if (e != cudaSuccess) {
            for (HostLane& L : hp.ln) {
                cudaFree(L.da);
                L.da = nullptr;
            }
            return cuda_fail(e, "host pipeline L_APP buffers");
        }
        hp.has_lapp = true;
    }
    return SG_OK;
}

/* Chunks of at most 16384 codewords (512 MiB of LLRs) alternate between the
 * two lanes: while chunk k decodes, chunk k + 1 is copied in and queued
 * behind it, so copies overlap decoding and the next chunk's CTAs take each
 * SM as soon as the current chunk's CTA there runs out of work.  Results
 * are read back chunk by chunk in order; a lane is refilled only after its
 * chunk has been read back. */
sg_status decode_host_pipelined(const double* llr, size_t n_cw, const sg_params* p, uint8_t* bits, double* lapp,
                                sg_cw_stats* stats)
{
    const size_t chunk = n_cw < SG_HOST_CHUNK ? n_cw : SG_HOST_CHUNK;
    const size_t nk = (n_cw + chunk - 1) / chunk;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return cuda_fail(e, "cudaGetDevice");
    if (dev < 0 || dev >= SG_HOST_MAX_DEV)
        return fail(SG_ERR_ARG, "device index beyond the host pipeline's table");
    HostPipe& hp = g_host_pipe[dev];
    std::lock_guard<std::mutex> lk(hp.mu);
    sg_status s = host_pipe_setup(hp, dev, lapp != nullptr);
    if (s != SG_OK)
        return s;
    HostLane* ln = hp.ln;
    std::vector<sg_cw_stats> hst(chunk);
    bool any_nonfinite = false;
    auto enqueue = [&](size_t k) -> sg_status {
        HostLane& L = ln[k % SG_HOST_LANES];
        L.off = k * chunk;
        L.n = (n_cw - L.off) < chunk ? (n_cw - L.off) : chunk;
        SG_CUDA(cudaMemcpyAsync(L.dl, llr + L.off * SG_CUBE, L.n * SG_CUBE * sizeof(double), cudaMemcpyHostToDevice,
                                L.st));
        return batch_enqueue(&L.b, L.dl, L.n, p, L.db, lapp ? L.da : nullptr, L.dst, L.st);
    };
    auto drain = [&](size_t k) -> sg_status {
        HostLane& L = ln[k % SG_HOST_LANES];
        SgQueue hq;
        SG_CUDA(cudaMemcpyAsync(bits + L.off * SG_INFO_BYTES, L.db, L.n * SG_INFO_BYTES, cudaMemcpyDeviceToHost,
                                L.st));
        SG_CUDA(cudaMemcpyAsync(hst.data(), L.dst, L.n * sizeof(sg_cw_stats), cudaMemcpyDeviceToHost, L.st));
        if (lapp)
            SG_CUDA(cudaMemcpyAsync(lapp + L.off * SG_CUBE, L.da, L.n * SG_CUBE * sizeof(double),
                                    cudaMemcpyDeviceToHost, L.st));
        SG_CUDA(cudaMemcpyAsync(&hq, L.b.q, sizeof hq, cudaMemcpyDeviceToHost, L.st));
        SG_CUDA(cudaStreamSynchronize(L.st));
        if (hq.err)
            return fail(SG_ERR_TIMEOUT, "a persistent-decoder warp gave up waiting for work");
        for (size_t i = 0; i < L.n; i++)
            any_nonfinite |= hst[i].converged < 0;
        if (stats)
            memcpy(stats + L.off, hst.data(), L.n * sizeof(sg_cw_stats));
        return SG_OK;
    };
    for (size_t k = 0; k < (size_t)SG_HOST_LANES && k < nk && s == SG_OK; k++)
        s = enqueue(k);
    for (size_t k = 0; k < nk && s == SG_OK; k++) {
        if ((s = drain(k)) != SG_OK)
            break;
        if (k + SG_HOST_LANES < nk)
            s = enqueue(k + SG_HOST_LANES);
    }
    /* leave no work of this call running on the lanes' streams */
    for (HostLane& L : hp.ln)
        cudaStreamSynchronize(L.st);
    if (s == SG_OK && any_nonfinite)
        return fail(SG_ERR_NONFINITE, "input contains non-finite LLRs; those codewords were not decoded");
    return s;
}

sg_status file_stage_setup(FileStage& fs)
{
    if (fs.ready)
        return SG_OK;
    cudaError_t e = cudaSuccess;
    for (int b = 0; b < SG_FILE_BUFS && e == cudaSuccess; b++)
        e = cudaHostAlloc((void**)&fs.llr[b], SG_FILE_CHUNK * SG_CUBE * sizeof(double), cudaHostAllocDefault);
    for (int l = 0; l < SG_HOST_LANES && e == cudaSuccess; l++) {
        e = cudaHostAlloc((void**)&fs.bits[l], SG_FILE_CHUNK * SG_INFO_BYTES, cudaHostAllocDefault);
        if (e == cudaSuccess)
            e = cudaHostAlloc((void**)&fs.st[l], SG_FILE_CHUNK * sizeof(sg_cw_stats), cudaHostAllocDefault);
    }
    if (e != cudaSuccess) {
        for (int b = 0; b < SG_FILE_BUFS; b++)
            cudaFreeHost(fs.llr[b]);
        for (int l = 0; l < SG_HOST_LANES; l++) {
            cudaFreeHost(fs.bits[l]);
            cudaFreeHost(fs.st[l]);
        }
        fs = FileStage();
        return cuda_fail(e, "pinned staging buffers of the file decoder");
    }
    fs.ready = true;
    return SG_OK;
}

/* The file decoder's pipeline.  A reader thread fills pinned staging
 * buffers with chunks of whole cubes (fread, as the reference's loop reads
 * them; a trailing partial cube is ignored); the calling thread copies each
 * chunk to a lane of the host pipeline, decodes it with the batched decoder
 * and copies bits and statistics back, alternating between the two lanes,
 * and writes a chunk's bits when its lane is taken again (chunks are
 * written in order).  File reading, both copy directions and decoding
 * overlap.  chunk_cw: codewords per chunk, 0 or above SG_FILE_CHUNK for
 * SG_FILE_CHUNK. */
sg_status decode_file_pipelined(FILE* fi, FILE* fo, const sg_params* p, size_t chunk_cw, sg_run_summary* sum,
                                bool* any_nonfinite)
{
    const size_t chunk = (chunk_cw == 0 || chunk_cw > SG_FILE_CHUNK) ? SG_FILE_CHUNK : chunk_cw;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return cuda_fail(e, "cudaGetDevice");
    if (dev < 0 || dev >= SG_HOST_MAX_DEV)
        return fail(SG_ERR_ARG, "device index beyond the host pipeline's table");
    HostPipe& hp = g_host_pipe[dev];
    std::lock_guard<std::mutex> lk(hp.mu);
    sg_status s = host_pipe_setup(hp, dev, false);
    if (s == SG_OK)
        s = file_stage_setup(hp.fs);
    if (s != SG_OK)
        return s;
    FileStage& fs = hp.fs;

    /* reader: chunk k goes to buffer k % SG_FILE_BUFS once the chunk that
     * used it before has been decoded and read back */
    std::mutex m;
    std::condition_variable cv;
    size_t count[SG_FILE_BUFS] = {};
    bool full[SG_FILE_BUFS] = {};
    bool stop = false, read_err = false;
    std::thread reader([&] {
        for (size_t k = 0;; k++) {
            const int b = (int)(k % SG_FILE_BUFS);
            {
                std::unique_lock<std::mutex> ul(m);
                cv.wait(ul, [&] { return !full[b] || stop; });
                if (stop)
                    return;
            }
            const size_t got = fread(fs.llr[b], sizeof(double) * SG_CUBE, chunk, fi);
            const bool err = got < chunk && ferror(fi);
            {
                std::lock_guard<std::mutex> g(m);
                count[b] = got;
                full[b] = true;
                read_err = read_err || err;
            }
            cv.notify_all();
            if (got < chunk)
                return; /* end of file, or a read error */
        }
    });

    HostLane* ln = hp.ln;
    long pending[SG_HOST_LANES] = {-1, -1}; /* chunk held by each lane */
    size_t pend_n[SG_HOST_LANES] = {0, 0};
    auto drain = [&](int l) -> sg_status {
        if (pending[l] < 0)
            return SG_OK;
        HostLane& L = ln[l];
        SgQueue hq;
        SG_CUDA(cudaMemcpyAsync(&hq, L.b.q, sizeof hq, cudaMemcpyDeviceToHost, L.st));
        SG_CUDA(cudaStreamSynchronize(L.st));
        const size_t n = pend_n[l];
        {
            std::lock_guard<std::mutex> g(m);
            full[pending[l] % SG_FILE_BUFS] = false; /* its input buffer is free again */
        }
        cv.notify_all();
        pending[l] = -1;
        if (hq.err)
            return fail(SG_ERR_TIMEOUT, "a persistent-decoder warp gave up waiting for work");
        if (fwrite(fs.bits[l], SG_INFO_BYTES, n, fo) != n)
            return fail(SG_ERR_IO, "short write to output file");
        for (size_t i = 0; i < n; i++) {
            const sg_cw_stats& c = fs.st[l][i];
            *any_nonfinite |= c.converged < 0;
            sum->total_iterations += c.iterations;
            sum->total_ng += c.ng;
            sum->total_ng_p += c.ng_p;
        }
        sum->blocks += n;
        return SG_OK;
    };
    for (size_t k = 0; s == SG_OK; k++) {
        const int b = (int)(k % SG_FILE_BUFS), l = (int)(k % SG_HOST_LANES);
        size_t n;
        {
            std::unique_lock<std::mutex> ul(m);
            cv.wait(ul, [&] { return full[b]; });
            n = count[b];
        }
        if ((s = drain(l)) != SG_OK)
            break;
        if (n == 0)
            break;
        HostLane& L = ln[l];
        cudaError_t ce = cudaMemcpyAsync(L.dl, fs.llr[b], n * SG_CUBE * sizeof(double), cudaMemcpyHostToDevice,
                                         L.st);
        if (ce != cudaSuccess) {
            s = cuda_fail(ce, "cudaMemcpyAsync H2D");
            break;
        }
        if ((s = batch_enqueue(&L.b, L.dl, n, p, L.db, nullptr, L.dst, L.st)) != SG_OK)
            break;
        if ((ce = cudaMemcpyAsync(fs.bits[l], L.db, n * SG_INFO_BYTES, cudaMemcpyDeviceToHost, L.st)) !=
                cudaSuccess ||
            (ce = cudaMemcpyAsync(fs.st[l], L.dst, n * sizeof(sg_cw_stats), cudaMemcpyDeviceToHost, L.st)) !=
                cudaSuccess) {
            s = cuda_fail(ce, "cudaMemcpyAsync D2H");
            break;
        }
        pending[l] = (long)k;
        pend_n[l] = n;
        if (n < chunk)
            break; /* the last chunk */
    }
    /* the lanes' remaining chunks, in order */
    const int first = (pending[0] >= 0 && (pending[1] < 0 || pending[0] < pending[1])) ? 0 : 1;
    for (int i = 0; i < SG_HOST_LANES; i++) {
        const sg_status d = drain((first + i) % SG_HOST_LANES);
        if (s == SG_OK)
            s = d;
    }
    {
        std::lock_guard<std::mutex> g(m);
        stop = true;
    }
    cv.notify_all();
    reader.join();
    for (HostLane& L : hp.ln)
        cudaStreamSynchronize(L.st);
    if (s == SG_OK && read_err)
        s = fail(SG_ERR_IO, "read error on input file");
    return s;
}

} // namespace

extern "C" {

sg_status sg_batch_create(sg_batch* out)
{
    if (!out)
        return fail(SG_ERR_ARG, "NULL handle pointer");
    *out = nullptr;
    DevCtx* c = nullptr;
    sg_status s = get_ctx(&c);
    if (s != SG_OK)
        return s;
    sg_batch b = new (std::nothrow) sg_batch_s;
    if (!b)
        return fail(SG_ERR_NOMEM, "host allocation failed");
    cudaGetDevice(&b->device);
    cudaError_t e = cudaMalloc(&b->q, sizeof(SgQueue));
    if (e != cudaSuccess) {
        delete b;
        return cuda_fail(e, "cudaMalloc");
    }
    *out = b;
    return SG_OK;
}

sg_status sg_batch_destroy(sg_batch b)
{
    if (!b)
        return SG_OK;
    if (b->exec)
        cudaGraphExecDestroy(b->exec);
    cudaFree(b->q);
    delete b;
    return SG_OK;
}

sg_status sg_batch_decode(sg_batch b, const double* d_llr, size_t n_cw, const sg_params* p, uint8_t* d_bits,
                          double* d_lapp, sg_cw_stats* d_stats, void* stream)
{
    return batch_enqueue(b, d_llr, n_cw, p, d_bits, d_lapp, d_stats, (cudaStream_t)stream);
}

sg_status sg_batch_capture(sg_batch b, const double* d_llr, size_t n_cw, const sg_params* p, uint8_t* d_bits,
                           double* d_lapp, sg_cw_stats* d_stats, void* stream)
{
    if (!b)
        return fail(SG_ERR_ARG, "invalid batch handle");
    cudaStream_t st = (cudaStream_t)stream;
    cudaStream_t own = nullptr;
    if (!st) {
        SG_CUDA(cudaStreamCreateWithFlags(&own, cudaStreamNonBlocking));
        st = own;
    }
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    sg_status s = SG_OK;
    if (e != cudaSuccess) {
        s = cuda_fail(e, "cudaStreamBeginCapture");
    } else {
        s = batch_enqueue(b, d_llr, n_cw, p, d_bits, d_lapp, d_stats, st);
        e = cudaStreamEndCapture(st, &g);
        if (s == SG_OK && e != cudaSuccess)
            s = cuda_fail(e, "cudaStreamEndCapture");
    }
    if (s == SG_OK) {
        if (b->exec) {
            cudaGraphExecDestroy(b->exec);
            b->exec = nullptr;
        }
        e = cudaGraphInstantiate(&b->exec, g, 0);
        if (e != cudaSuccess)
            s = cuda_fail(e, "cudaGraphInstantiate");
    }
    if (g)
        cudaGraphDestroy(g);
    if (own)
        cudaStreamDestroy(own);
    return s;
}

sg_status sg_batch_replay(sg_batch b, void* stream)
{
    if (!b || !b->exec)
        return fail(SG_ERR_ARG, "no captured decode in this batch handle");
    SG_CUDA(cudaGraphLaunch(b->exec, (cudaStream_t)stream));
    return SG_OK;
}

sg_status sg_batch_check(sg_batch b)
{
    if (!b)
        return fail(SG_ERR_ARG, "invalid batch handle");
    SgQueue hq;
    SG_CUDA(cudaMemcpy(&hq, b->q, sizeof hq, cudaMemcpyDeviceToHost));
    if (hq.err)
        return fail(SG_ERR_TIMEOUT, "a persistent-decoder warp gave up waiting for work");
    return SG_OK;
}

int sg_batch_variant_count(void) { return SG_NPVARIANTS; }

const char* sg_batch_variant_name(int v) { return (v >= 0 && v < SG_NPVARIANTS) ? k_pvariants[v].name : ""; }

sg_status sg_batch_set_variant(int v)
{
    if (v < 0 || v >= SG_NPVARIANTS)
        return fail(SG_ERR_ARG, "no such batch variant");
    g_pvariant = v;
    return SG_OK;
}

int sg_batch_get_variant(void) { return g_pvariant; }

sg_status sg_guess_ceiling(unsigned long long iters, int32_t mode, double* guesses_per_second)
{
    if (!guesses_per_second || iters == 0 || (mode != 0 && mode != 1))
        return fail(SG_ERR_ARG, "need iters > 0, mode 0 or 1 and an output pointer");
    void (*kern)(unsigned long long, double*, SgK) =
        mode == 1 ? sg_guess_ceiling_kernel<true> : sg_guess_ceiling_kernel<false>;
    DevCtx* c = nullptr;
    sg_status s = get_ctx(&c);
    if (s != SG_OK)
        return s;
    const int blocks = c->sms * 8; /* 8 CTAs x 8 warps per SM */
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    SG_CUDA(cudaEventCreate(&e0));
    SG_CUDA(cudaEventCreate(&e1));
    kern<<<blocks, 256>>>(iters / 8 + 1, c->err_sink, k_consts); /* warm-up */
    SG_CUDA(cudaEventRecord(e0));
    kern<<<blocks, 256>>>(iters, c->err_sink, k_consts);
    SG_CUDA(cudaEventRecord(e1));
    SG_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    SG_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    SG_CUDA(cudaGetLastError());
    *guesses_per_second = 2.0 * (double)iters * blocks * 256 / (ms / 1000.0);
    return SG_OK;
}

sg_status sg_forward_device(const double* d_llr, size_t n_cw, const sg_params* p, uint8_t* d_bits, double* d_lapp,
                            sg_cw_stats* d_stats, double* d_ckpt, void* stream)
{
    sg_status s = check_params(p);
    if (s != SG_OK)
        return s;
    if (n_cw == 0)
        return SG_OK;
    if (!d_llr || !d_bits || !d_stats || !d_ckpt)
        return fail(SG_ERR_ARG, "llr, bits, stats and ckpt must not be NULL");
    if ((uintptr_t)d_llr & 7u)
        return fail(SG_ERR_ARG, "llr must be 8-byte aligned");
    DevCtx* c = nullptr;
    if ((s = get_ctx(&c)) != SG_OK)
        return s;
    SgDecodeArgs a;
    memset(&a, 0, sizeof a);
    a.llr = d_llr;
    a.bits = d_bits;
    a.lapp = d_lapp;
    a.stats = d_stats;
    a.enum_tabs = c->enum_tabs;
    a.err = c->err;
    a.ckpt = d_ckpt;
    a.n_cw = n_cw;
    a.wait_limit = g_wait_limit.load();
    a.L = p->L;
    a.imax = p->Imax;
    order_meta(tmax_eff(p->Tmax), &a.meta);
    a.use_bulk = ((uintptr_t)d_llr & 15u) == 0;
    a.thres = p->thres;
    memcpy(a.alpha, p->alpha, sizeof a.alpha);
    a.k = k_consts;
    SG_CUDA(launch_decode(a, c->clusters, &c->flights, 0, (cudaStream_t)stream));
    return SG_OK;
}

sg_status sg_backward_device(const double* d_llr, size_t n_cw, const sg_params* p, const sg_cw_stats* d_stats,
                             const double* d_ckpt, const uint8_t* d_code_bits, int32_t loss_mode, double* d_loss,
                             double* d_grad_alpha, double* d_grad_llr, void* stream)
{
    sg_status s = check_params(p);
    if (s != SG_OK)
        return s;
    if (loss_mode != 0 && loss_mode != 1)
        return fail(SG_ERR_ARG, "loss_mode must be 0 (final APP) or 1 (every phase's APP)");
    if (p->Tmax < SG_ENUM_LEN && p->Tmax != 0)
        return fail(SG_ERR_ARG, "the adjoint needs Tmax >= 65536 (every line stops at a list insertion)");
    if (n_cw == 0)
        return SG_OK;
    if (!d_llr || !d_stats || !d_ckpt || !d_code_bits || !d_loss || !d_grad_alpha)
        return fail(SG_ERR_ARG, "NULL buffer");
    DevCtx* c = nullptr;
    if ((s = get_ctx(&c)) != SG_OK)
        return s;
    SgBackwardArgs a;
    memset(&a, 0, sizeof a);
    a.llr = d_llr;
    a.ckpt = d_ckpt;
    a.stats = d_stats;
    a.code_bits = d_code_bits;
    a.enum_tabs = c->enum_tabs;
    a.loss = d_loss;
    a.grad_alpha = d_grad_alpha;
    a.grad_llr = d_grad_llr;
    a.n_cw = n_cw;
    a.L = p->L;
    a.nph = 3 * p->Imax;
    order_meta(0xffffffffu, &a.meta);
    a.loss_mode = loss_mode;
    a.thres = p->thres;
    memcpy(a.alpha, p->alpha, sizeof a.alpha);
    a.k = k_consts;
    void* kargs[] = {(void*)&a};
    SG_CUDA(cudaLaunchKernel((const void*)sg_backward_kernel, dim3(grid_for(n_cw, 1 << 30)),
                             dim3(SG_BACK_WARPS * 32), kargs, sizeof(SgBackSmem), (cudaStream_t)stream));
    return SG_OK;
}

sg_status sg_set_math_mode(int32_t mode)
{
    if (mode != 0 && mode != 1)
        return fail(SG_ERR_ARG, "math mode must be 0 (table-driven) or 1 (correctly rounded)");
    g_math_mode.store(mode);
    return SG_OK;
}

int32_t sg_get_math_mode(void) { return g_math_mode.load(); }

sg_status sg_set_wait_limit(uint64_t limit)
{
    g_wait_limit.store(limit > (uint64_t)SG_WAIT_LIMIT_DEFAULT ? SG_WAIT_LIMIT_DEFAULT : (long long)limit);
    return SG_OK;
}

uint64_t sg_get_wait_limit(void) { return (uint64_t)g_wait_limit.load(); }

sg_status sg_check_device(void* stream)
{
    DevCtx* c = nullptr;
    sg_status s = get_ctx(&c);
    if (s != SG_OK)
        return s;
    SG_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    unsigned int flags = 0;
    SG_CUDA(cudaMemcpy(&flags, c->err, sizeof flags, cudaMemcpyDeviceToHost));
    if (flags) {
        SG_CUDA(cudaMemset(c->err, 0, sizeof flags));
        return fail(SG_ERR_TIMEOUT, (flags & 2u) ? "a bulk-copy wait gave up and the copy did not complete"
                                                 : "a bulk-copy wait gave up; the affected codewords report "
                                                   "converged = -2");
    }
    return SG_OK;
}

int sg_decoder_variant_count(void) { return SG_NVARIANTS; }

const char* sg_decoder_variant_name(int v)
{
    return (v >= 0 && v < SG_NVARIANTS) ? k_variants[v].name : "";
}

sg_status sg_decoder_set_variant(int v)
{
    if (v < 0 || v >= SG_NVARIANTS)
        return fail(SG_ERR_ARG, "no such decoder variant");
    g_variant = v;
    return SG_OK;
}

int sg_decoder_get_variant(void) { return g_variant; }

const char* sg_status_string(sg_status s)
{
    switch (s) {
    case SG_OK: return "ok";
    case SG_ERR_ARG: return "invalid argument";
    case SG_ERR_CUDA: return "CUDA error";
    case SG_ERR_NONFINITE: return "non-finite input";
    case SG_ERR_IO: return "I/O error";
    case SG_ERR_NOMEM: return "out of memory";
    case SG_ERR_TIMEOUT: return "device wait timed out";
    }
    return "unknown status";
}

const char* sg_last_error(void) { return t_err.c_str(); }

const char* sg_version(void) { return "sogrand_b200 0.1.0 (sm_100a)"; }

} // extern "C"
