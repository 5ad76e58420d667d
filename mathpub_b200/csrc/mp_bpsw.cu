// mp_bpsw.cu -- 64-bit BPSW primality test for B200 (sm_100a): batches of candidate lists.
//
// Reference (paths inside the Mathpub project): bpsw A350826/a350826.c:965 (the base-2 strong
// test sprp2_64 :618 and the strong Lucas test slprp64 :766 with Selfridge's D :739), after
// the trivial small-factor handling of is_prime_ref :529; the breadth-first batching of
// test_batch64 :1392.  The arithmetic and the two tests are in mp_mont64.cuh.  Trial division
// by the odd primes up to 127 uses the multiplicative-inverse test (q | r iff r q^-1 mod 2^32
// <= (2^32 - 1) / q, for odd q) on 32-bit residues of n / 2^32 modulo six products of them, all 30
// primes for every candidate, with no early exit.  The
// verdict is primality for every n < 2^64 (BPSW has no pseudoprime below 2^64).
//
// Two launch structures:
//   plain    one launch per candidate list, one thread per candidate, all phases inline;
//   batched  four launches over every list at once.  The first trial-divides the candidates, writes
//            the verdict words of the ones that settles, and files the survivors in two size
//            classes (below 2^63 and above; mp_mont64.cuh runs a different squaring for each).
//            The second runs the base-2 test over the survivors, one per thread, every warp full
//            and of one class; the third Selfridge's search over the passers, which files them by
//            D (D = 5 apart); the fourth the Lucas ladders, which set the bits of the primes, those
//            with D = 5 in a two-product step.  (The base-2 test as z = 2^((n-1)/2), with the whole
//            strong test only where z = 1 leaves it open, saves the squarings after 2^d for most
//            composites, but 6% of this workload's candidates are built to have z = 1: 0.96 ms
//            instead of 0.89 at 2^24 candidates.)
//            One launch of persistent warps that took chunks of 1024 candidates through trial
//            division and the base-2 test left batches partly filled (25 of 32 lanes active) and,
//            at 2^24 candidates, 2.3 chunks a warp: 1.13 ms for the two
//            phases that take 1.01 ms now (1.38 ms before the windowed ladder).
//   few      up to BPSW_FEW candidates: one launch whose warps take the phases of a candidate at the
//            same time, since latency is all that counts there
#include "mp_mont64.cuh"
#include <algorithm>

// Up to BPSW_FEW candidates a batch runs in one launch (a whole call with host copies, batched form
// against this: 100 candidates 83 and 51 us, 4000 89 and 66, 16000 118 and 86, 24000 122 and 102; the
// former needs no Lucas tests of composites, so that it is taken well before they meet), of 8
// candidates a CTA up to BPSW_VERY_FEW (8 against 32 a CTA: 1000 candidates 53 and 59 us, 2000 57 and
// 65, 4000 67 and 66).  The few form does several times the work; with four serving workers busy, 256 requests
// of up to 4000 or 16000 candidates take what the batched form took (2.1 and 2.9 ms).
#define BPSW_FEW 16384
#define BPSW_VERY_FEW 2048

#define TD_N 30            // odd primes 3..127
#define TD_NG 6            // in six groups whose products are below 2^32

__constant__ u32 c_tdg_prod[TD_NG];      // the groups' products
__constant__ u32 c_tdg_inv[TD_NG];       // product^-1 mod 2^32
__constant__ u32 c_td_inv32[TD_N];       // p^-1 mod 2^32
__constant__ u32 c_td_lim32[TD_N];       // floor((2^32 - 1) / p)
__constant__ u64 c_small_prime_mask[2];   // bit n set iff n < 128 is prime

// ---- trial division ----
// 1 = prime, 0 = composite, -1 = undecided (odd, no factor <= 127, n >= 131^2).  Per group one
// word of Montgomery reduction by the product P of the group: n / 2^32 = n1 - hi(m P) (mod P) with
// m = n0 P^-1 mod 2^32, plus P on a borrow, a 32-bit residue that the primes of P divide exactly
// when they divide n.  Then p | r iff r p^-1 mod 2^32 <= (2^32 - 1) / p: one 32-bit multiply and
// one compare a prime.  (A 64-bit Barrett remainder per group took four times as long.)
__device__ __forceinline__ int td_verdict(u64 n)
{
    if (n < 128) return (int)((c_small_prime_mask[n >> 6] >> (n & 63)) & 1);
    bool f = !(n & 1);
    const int gsize[TD_NG] = {8, 5, 5, 5, 4, 3};   // 3..23, 29..43, 47..67, 71..89, 97..107, 109..127
    int k = 0;
#pragma unroll
    for (int g = 0; g < TD_NG; g++) {
        const u32 P = c_tdg_prod[g], hp = __umulhi((u32)n * c_tdg_inv[g], P), n1 = (u32)(n >> 32);
        const u32 r = n1 - hp + (n1 < hp ? P : 0u);
#pragma unroll
        for (int j = 0; j < gsize[g]; j++, k++) f |= r * c_td_inv32[k] <= c_td_lim32[k];
    }
    if (f) return 0;
    return n < 131ull * 131ull ? 1 : -1;
}

__device__ __forceinline__ bool bpsw_full(u64 n)
{
    const int v = td_verdict(n);
    if (v >= 0) return v != 0;
    return bpsw_odd(n);
}

// ---- plain form: one thread per candidate of one list ----
__global__ void __launch_bounds__(256) bpsw_plain_kernel(const u64 *__restrict__ n, u32 len, u32 *__restrict__ bits)
{
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    bool v = false;
    if (i < len) v = bpsw_full(__ldg(n + i));
    const u32 b = __ballot_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0 && i < len) bits[i >> 5] = b;
}

// ---- few candidates ----
// G candidates of one list per CTA, whose four warps take the phases at the same time: the base-2 test
// below 2^63 and above, and the Lucas test for D = 5 and for any other D, each after its own search for
// D (W = 32 / G lanes a candidate try W values of D at once).  Latency is all that counts, so the Lucas
// ladders of composites, which the phases in turn would save, cost nothing (100 candidates: 21 us of
// kernel, 28 with a thread per candidate and the phases in turn).
template <int G>
__global__ void __launch_bounds__(128) bpsw_few_kernel(const u64 *__restrict__ n, u32 total, u32 *__restrict__ bits)
{
    constexpr u32 W = 32 / G;
    __shared__ u32 s_pass[4];
    const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % W, i = blockIdx.x * G + lane / W;
    const u64 x = i < total ? __ldg(n + i) : 0;
    const int td = td_verdict(x);
    const bool open = td < 0 && x != ~0ull;                              // 3 | 2^64 - 1
    bool v = false;
    if (warp < 2) {
        if (open && sub == 0 && x >> 63 == warp) v = warp ? spsp2<SP_WIDE>(x) : spsp2<SP_MID>(x);
    } else {
        // selfridge_d, W tries a round: the first D with (D/n) <= 0 decides
        i32 D = 0;
        bool more = open;
        for (int k0 = 0; k0 < 2048 && __any_sync(0xffffffffu, more); k0 += W) {
            const int k = k0 + (int)sub;
            const i32 a = 5 + 2 * k, d = (k & 1) ? -a : a;
            const int j = more ? jacobi_dn(d, x) : 1;
            const u32 neg = __ballot_sync(0xffffffffu, more && j < 0), zero = __ballot_sync(0xffffffffu, more && j == 0);
            const u32 own = (W == 32 ? 0xffffffffu : (1u << (W & 31)) - 1) << (lane - sub), ev = (neg | zero) & own;
            const u32 first = ev ? __ffs((int)ev) - 1 : lane;
            const i32 df = __shfl_sync(0xffffffffu, d, (int)first);
            if (more && ev) {
                more = false;
                D = neg >> first & 1 ? df : 0;
            } else if (more && k0 <= 23 && k0 + (int)W > 23 && is_square64(x)) {
                more = false;
            }
        }
        if (D && sub == 0 && (D == 5) == (warp == 2)) {
            const Mod64 M = mm_setup(x);
            v = warp == 2 ? lucas_strong_d5(M) : lucas_strong(M, D);
        }
    }
    __syncwarp();
    const u32 m = __ballot_sync(0xffffffffu, v);
    if (lane == 0) s_pass[warp] = m;
    __syncthreads();
    if (warp == 0) {
        const u32 pass = (s_pass[0] | s_pass[1]) & (s_pass[2] | s_pass[3]), at = lane * W & 31;
        const int tj = __shfl_sync(0xffffffffu, td, (int)at);
        const u32 b = __ballot_sync(0xffffffffu, lane < G && (tj == 1 || (pass >> at & 1)));
        if (lane == 0) {
            if (G == 32) bits[blockIdx.x] = b;
            else ((u8 *)bits)[blockIdx.x] = (u8)b;
        }
    }
}

// ---- batched form ----
// a list of two kinds of entries shares one array of cap entries: the first kind from the front,
// the second from the back.  ctr[0] and ctr[1] count them.

// warp-aggregated append of v to the front of a list (every lane takes part)
__device__ __forceinline__ void list_append(bool keep, u32 v, u32 *list, u32 *ctr)
{
    const u32 lane = threadIdx.x & 31, m = __ballot_sync(0xffffffffu, keep);
    if (!m) return;
    u32 g = 0;
    if (lane == 0) g = atomicAdd(ctr, (u32)__popc(m));
    g = __shfl_sync(0xffffffffu, g, 0) + __popc(m & ((1u << lane) - 1));
    if (keep) list[g] = v;
}

// 1. trial division: verdict words of all candidates (bits of the primes it settles), survivors
//    to `surv` (below 2^63 in front, the others at the back).  cap = total.  A warp collects the
//    survivors of TRIAL_RUN candidates in shared memory, so that one atomic on the two counters
//    (one 64-bit word) covers them: an atomic per 32 candidates and kind made the launch wait on
//    one address of L2 (0.69 ms at 2^24 candidates, 0.12 now)
#define TRIAL_RUN 512u
__global__ void __launch_bounds__(256) bpsw_trial_kernel(const u64 *__restrict__ n, u32 total, u32 *__restrict__ bits,
                                                         u32 *__restrict__ surv, unsigned long long *ctr)
{
    __shared__ u16 s_idx[8][TRIAL_RUN];                  // one kind from the front, the other from the back
    const u32 lane = threadIdx.x & 31, lt = (1u << lane) - 1;
    u16 *idx = s_idx[threadIdx.x >> 5];
    const u64 step = (u64)gridDim.x * 8 * TRIAL_RUN;
    for (u64 b0 = ((u64)blockIdx.x * 8 + (threadIdx.x >> 5)) * TRIAL_RUN; b0 < total; b0 += step) {
        const u32 len = (u32)min((u64)TRIAL_RUN, total - b0);
        u32 nm = 0, nw = 0;
        for (u32 r = 0; r < len; r += 32) {
            const u32 i = r + lane;
            const u64 x = i < len ? __ldcs(n + b0 + i) : 0;
            const int v = i < len ? td_verdict(x) : 0;
            const bool cm = v < 0 && x >> 63 == 0, cw = v < 0 && x >> 63;
            const u32 pm = __ballot_sync(0xffffffffu, v == 1), mm = __ballot_sync(0xffffffffu, cm);
            const u32 mw = __ballot_sync(0xffffffffu, cw);
            if (lane == 0) bits[(b0 + r) >> 5] = pm;
            if (cm) idx[nm + __popc(mm & lt)] = (u16)i;
            if (cw) idx[TRIAL_RUN - 1 - nw - __popc(mw & lt)] = (u16)i;
            nm += __popc(mm);
            nw += __popc(mw);
        }
        __syncwarp();
        unsigned long long g = 0;
        if (lane == 0 && nm + nw) g = atomicAdd(ctr, (unsigned long long)nw << 32 | nm);
        g = __shfl_sync(0xffffffffu, g, 0);
        const u32 gm = (u32)g, gw = (u32)(g >> 32);
        for (u32 k = lane; k < nm; k += 32) surv[gm + k] = (u32)b0 + idx[k];
        for (u32 k = lane; k < nw; k += 32) surv[total - 1 - gw - k] = (u32)b0 + idx[TRIAL_RUN - 1 - k];
        __syncwarp();
    }
}

// 2. base-2 test of the survivors; passers to `pass`.  64 to 512 threads a CTA (mp_tune_set)
__global__ void __launch_bounds__(512) bpsw_base2_kernel(const u64 *__restrict__ n, u32 total,
                                                         const u32 *__restrict__ surv, const u32 *sctr,
                                                         u32 *__restrict__ pass, u32 *ctr)
{
    // the warps of the wider class first (they take longer), each class rounded up to whole warps
    const u32 nm = sctr[0], nw = sctr[1], lane = threadIdx.x & 31, ww = (nw + 31) / 32, wall = ww + (nm + 31) / 32;
    const u32 step = gridDim.x * (blockDim.x >> 5);
    for (u32 w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < wall; w += step) {
        u32 idx = 0;
        bool p = false;
        if (w < ww) {
            const u32 k = w * 32 + lane;
            if (k < nw) {
                idx = surv[total - 1 - k];
                p = spsp2<SP_WIDE>(__ldg(n + idx));
            }
        } else {
            const u32 k = (w - ww) * 32 + lane;
            if (k < nm) {
                idx = surv[k];
                p = spsp2<SP_MID>(__ldg(n + idx));
            }
        }
        __syncwarp();
        list_append(p, idx, pass, ctr);
    }
}

// 3. Selfridge's search for D over the passers, whose length differs from candidate to candidate (a
//    few Jacobi symbols, each after a 64-bit remainder): D = 5 (about half of them: n = 2 or 3 mod 5)
//    to the front of `luc`, any other D to the back with its value in dl; D = 0 (shown composite
//    by the search) to neither
__global__ void __launch_bounds__(256) bpsw_selfridge_kernel(const u64 *__restrict__ n, u32 total,
                                                             const u32 *__restrict__ pass, const u32 *pctr,
                                                             u32 *__restrict__ luc, i32 *__restrict__ dl, u32 *ctr)
{
    const u32 cnt = *pctr, lane = threadIdx.x & 31;
    // warp-uniform trip count, so that every lane takes part in the ballots
    for (u32 b0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); b0 < cnt; b0 += gridDim.x * blockDim.x) {
        const u32 i = b0 + lane;
        u32 idx = 0;
        i32 D = 0;
        if (i < cnt) {
            idx = pass[i];
            const u64 x = __ldg(n + idx);
            D = x == ~0ull ? 0 : selfridge_d(x);                         // 3 | 2^64 - 1
        }
        __syncwarp();
        list_append(D == 5, idx, luc, ctr);
        const u32 m = __ballot_sync(0xffffffffu, D != 0 && D != 5);
        if (m) {
            u32 g = 0;
            if (lane == 0) g = atomicAdd(ctr + 1, (u32)__popc(m));
            g = __shfl_sync(0xffffffffu, g, 0) + __popc(m & ((1u << lane) - 1));
            if (D != 0 && D != 5) {
                luc[total - 1 - g] = idx;
                dl[g] = D;
            }
        }
    }
}

// 4. the Lucas ladders, the D = 5 list first with its two-product step (Q = -1); a prime's verdict
//    bit is set in its word
__global__ void __launch_bounds__(256) bpsw_lucas_kernel(const u64 *__restrict__ n, u32 total,
                                                         const u32 *__restrict__ luc, const i32 *__restrict__ dl,
                                                         const u32 *ctr, u32 *bits)
{
    const u32 c5 = ctr[0], cnt = c5 + ctr[1];
    for (u32 i = blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += gridDim.x * blockDim.x) {
        const bool f = i < c5;
        const u32 idx = f ? luc[i] : luc[total - 1 - (i - c5)];
        const Mod64 M = mm_setup(__ldg(n + idx));
        if (f ? lucas_strong_d5(M) : lucas_strong(M, dl[i - c5])) atomicOr(bits + (idx >> 5), 1u << (idx & 31));
    }
}

// ---- host side ----

static bool g_bpsw_consts[16] = {false};

static int bpsw_consts(mp_handle *h)
{
    if (h->device >= 0 && h->device < 16 && g_bpsw_consts[h->device]) return MP_OK;
    static const u32 tdp[TD_N] = {3,  5,  7,  11, 13, 17, 19, 23, 29, 31, 37, 41,  43,  47,  53,
                                  59, 61, 67, 71, 73, 79, 83, 89, 97, 101, 103, 107, 109, 113, 127};
    static const int gsize[TD_NG] = {8, 5, 5, 5, 4, 3};
    u32 inv[TD_N], lim[TD_N], prod[TD_NG], ginv[TD_NG];
    u64 mask[2] = {0, 0};
    for (int k = 0; k < TD_N; k++) {
        const u32 q = tdp[k];
        inv[k] = (u32)inv64(q);              // q^-1 mod 2^64, so also mod 2^32
        lim[k] = 0xffffffffu / q;
    }
    for (int g = 0, k = 0; g < TD_NG; g++) {
        u64 pr = 1;
        for (int j = 0; j < gsize[g]; j++, k++) pr *= tdp[k];
        if (pr >> 32) return mp_set_error(h, MP_EINVAL, "trial-division group product above 2^32");
        prod[g] = (u32)pr;
        ginv[g] = (u32)inv64(pr);
    }
    for (u32 v = 2; v < 128; v++) {
        bool p = true;
        for (u32 d = 2; d * d <= v; d++) if (v % d == 0) { p = false; break; }
        if (p) mask[v >> 6] |= 1ull << (v & 63);
    }
    MP_CUDA(h, cudaMemcpyToSymbol(c_td_inv32, inv, sizeof inv));
    MP_CUDA(h, cudaMemcpyToSymbol(c_td_lim32, lim, sizeof lim));
    MP_CUDA(h, cudaMemcpyToSymbol(c_tdg_prod, prod, sizeof prod));
    MP_CUDA(h, cudaMemcpyToSymbol(c_tdg_inv, ginv, sizeof ginv));
    MP_CUDA(h, cudaMemcpyToSymbol(c_small_prime_mask, mask, sizeof mask));
    if (h->device >= 0 && h->device < 16) g_bpsw_consts[h->device] = true;
    return MP_OK;
}

// a grid of as many CTAs as fit on the device at once, no more than `need`
template <class F>
static cudaError_t resident_grid(mp_handle *h, F kernel, u32 threads, u64 need, unsigned *grid)
{
    int per_sm = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, (int)threads, 0);
    if (e != cudaSuccess) return e;
    const u64 g = (u64)h->sm_count * (u32)std::max(per_sm, 1);
    *grid = (unsigned)std::max<u64>(1, std::min(g, need));
    return cudaSuccess;
}

// the four launches over `total` candidates; list: 4 total words
static int bpsw_batched_launch(mp_handle *h, const u64 *d_n, u32 total, u32 *d_bits, u32 *list, cudaStream_t st)
{
    // threads per CTA of the base-2 launch: the tuned choice
    static const u32 kThreads[4] = {256, 128, 512, 64};
    const u32 nth = kThreads[h->tune.bpsw_variant & 3];
    u32 *ctr = h->queue.as<u32>(), *surv = list, *pass = list + total, *luc = list + 2 * (size_t)total;
    i32 *dl = (i32 *)(list + 3 * (size_t)total);
    unsigned g = 1;
    MP_CUDA(h, cudaMemsetAsync(ctr, 0, 24, st));
    const u64 need = ((u64)total + 255) / 256;
    MP_CUDA(h, resident_grid(h, bpsw_trial_kernel, 256, ((u64)total + 8 * TRIAL_RUN - 1) / (8 * TRIAL_RUN), &g));
    bpsw_trial_kernel<<<g, 256, 0, st>>>(d_n, total, d_bits, surv, (unsigned long long *)ctr);
    MP_CUDA(h, resident_grid(h, bpsw_base2_kernel, nth, ((u64)total + nth - 1) / nth, &g));
    bpsw_base2_kernel<<<g, nth, 0, st>>>(d_n, total, surv, ctr, pass, ctr + 2);
    MP_CUDA(h, resident_grid(h, bpsw_selfridge_kernel, 256, need, &g));
    bpsw_selfridge_kernel<<<g, 256, 0, st>>>(d_n, total, pass, ctr + 2, luc, dl, ctr + 4);
    MP_CUDA(h, resident_grid(h, bpsw_lucas_kernel, 256, need, &g));
    bpsw_lucas_kernel<<<g, 256, 0, st>>>(d_n, total, luc, dl, ctr + 4, d_bits);
    MP_CUDA(h, cudaGetLastError());
    return MP_OK;
}

// lists at d_n + offs[i] (offs multiples of 32, host array of nlists + 1 entries), verdict
// words at d_bits + offs[i] / 32
int mp_bpsw_run(mp_handle *h, const u64 *d_n, const u64 *offs, const u32 *lens, u32 nlists, u32 *d_bits,
                u32 mode, cudaStream_t st)
{
    MP_TRY(bpsw_consts(h));
    if (mode == MP_MODE_PLAIN) {
        for (u32 i = 0; i < nlists; i++) {
            if (!lens[i]) continue;
            if (offs[i] & 31) return mp_set_error(h, MP_EINVAL, "list offsets must be multiples of 32");
            ProfScope ps(h, PROF_BPSW_PLAIN, st);
            bpsw_plain_kernel<<<(lens[i] + 255) / 256, 256, 0, st>>>(d_n + offs[i], lens[i], d_bits + offs[i] / 32);
            MP_CUDA(h, cudaGetLastError());
        }
        return MP_OK;
    }
    const u64 total = offs[nlists];
    if (!total) return MP_OK;
    if (total <= BPSW_FEW) {
        ProfScope ps(h, PROF_BPSW_BATCHED, st);
        const unsigned words = (unsigned)((total + 31) / 32);
        if (total <= BPSW_VERY_FEW) bpsw_few_kernel<8><<<4 * words, 128, 0, st>>>(d_n, (u32)total, d_bits);
        else bpsw_few_kernel<32><<<words, 128, 0, st>>>(d_n, (u32)total, d_bits);
        MP_CUDA(h, cudaGetLastError());
        return MP_OK;
    }
    // slices of at most 2^31 candidates, so that the lists hold 32-bit indices
    const u64 slice = 1ull << 31;
    MP_CUDA(h, h->queue.ensure(64));
    MP_CUDA(h, h->bpsw_list.ensure((size_t)std::min(total, slice) * 16));   // survivors; passers; by D; their D
    ProfScope ps(h, PROF_BPSW_BATCHED, st);
    for (u64 b = 0; b < total; b += slice)
        MP_TRY(bpsw_batched_launch(h, d_n + b, (u32)std::min(slice, total - b), d_bits + b / 32,
                                   h->bpsw_list.as<u32>(), st));
    return MP_OK;
}

const char *mp_bpsw_variant_name(int v)
{
    static const char *names[4] = {"256 threads per CTA", "128 threads per CTA", "512 threads per CTA",
                                   "64 threads per CTA"};
    return names[v & 3];
}
