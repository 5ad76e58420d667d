// mp_gap.cu -- statistics of the prime-gap stream (include/mathpub_gpu.h, gap statistics):
// the histogram of the gaps that follow the primes of a range, from which A252768's power
// sums come, and the run lengths of A158939 (L(p) = the number of strictly increasing gaps
// that follow p, A158939/a158939.c:17-30) with the smallest prime of each length.
//
// The range is sieved a chunk at a time (2^34 integers) into the odd-only bitmap, with a
// look-ahead of 2^16 integers past the chunk, and gap_kernel reads the bitmap: a CTA takes a window of
// it at a time, compacts the prime positions into shared memory in order, and every thread takes
// primes of the window's segment, reads the gap to the next prime and walks on while the gaps
// increase (L(p) depends only on the gaps after p, the fact (F1) of A158939/a158939.c:32-35, so
// segments need nothing from each other; a walk that leaves the window goes on in the bitmap).  The
// same walk gives the chains of gapchain_ps (gapchain/gapchain_ps.c:336-366): from a head p the gaps
// 2, 4, 6, ..., that is 1, 2, 3, ... bits of the odd-only map.  Counts go to shared histograms and at
// the end to the device accumulator with one atomic per bin; chain heads of at least the requested
// length go to a device list.
#include "mp_common.cuh"
#include <algorithm>

#define GAP_THREADS 256
#define GAP_WPT 5u                          // words of the map a thread compacts
#define GAP_WORDS (GAP_THREADS * GAP_WPT)   // words of a window
#define GAP_LOOK_WORDS 64u                  // of which look-ahead: 4096 integers (walks that leave it go on
                                            // in global memory)
#define GAP_SEG_BITS ((GAP_WORDS - GAP_LOOK_WORDS) * 32u)
#define GAP_MAXP 8064u                      // primes per window; the densest, the odd numbers below 81920,
                                            // holds 8,016
#define GAP_CHUNK ((u64)1 << 34)            // integers sieved per pass
#define GAP_LOOK ((u64)1 << 16)

struct ChainOut {
    u32 min_len;                            // list heads with at least this many primes (0: none)
    u64 cap;
    u64 *heads;
    u32 *lens;
    unsigned long long *n;
};

// the first prime bit after bit `pos`, or ~0 when none is sieved
__device__ __noinline__ u64 gap_next(const u32 *__restrict__ bm, u64 pos, u64 nbits_all)
{
    u64 b = pos + 1;
    if (b >= nbits_all) return ~0ull;
    u32 v = __ldg(bm + (b >> 5)) & (~0u << (b & 31));
    for (b &= ~31ull;;) {
        if (v) {
            b += __ffs(v) - 1;
            return b < nbits_all ? b : ~0ull;
        }
        b += 32;
        if (b >= nbits_all) return ~0ull;
        v = __ldg(bm + (b >> 5));
    }
}

// Persistent CTAs, each over every gridDim-th segment: the histograms stay in shared memory until the
// end.  Per segment the window's prime positions are compacted in order (16 bits each: a window of
// 40960 bits), then each thread takes primes of the segment.  (Segments of 2^16 bits with 2^15 of
// look-ahead, 32-bit positions and a flush of the histograms per segment: 1.50 ms for 2^32 integers
// at 1e13, two CTAs an SM; 1.0 now.)
__global__ void __launch_bounds__(GAP_THREADS) gap_kernel(const u32 *__restrict__ bm, u64 nbits_in, u64 nbits_all,
                                                          u64 base, u32 nseg, mp_gap_stats *acc, u32 *err, ChainOut co)
{
    __shared__ u32 w[GAP_WORDS];            // the map's words of the window
    __shared__ u16 P[GAP_MAXP];             // prime positions (bits from the segment's start)
    __shared__ u64 rf[MP_RUN_MAX];
    __shared__ u32 hist[MP_GAP_BINS], rh[MP_RUN_MAX], ch[MP_CHAIN_MAX], s_wsum[GAP_THREADS / 32];
    __shared__ u32 s_uns;
    const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (u32 i = tid; i < MP_GAP_BINS; i += GAP_THREADS) hist[i] = 0;
    if (tid < MP_RUN_MAX) { rh[tid] = 0; rf[tid] = ~0ull; }
    if (tid < MP_CHAIN_MAX) ch[tid] = 0;
    if (tid == 0) s_uns = 0;
    // nearly every chain has one prime, and nearly every run at most four gaps: those are counted in
    // registers (same-address atomics of a warp wait for one another).  seen: the run lengths the thread
    // has met (its primes ascend, so a later one of the same length is never the first)
    // (16 bits a count: a launch of 2^34 integers gives a thread some 4000 primes)
    u32 c1 = 0, c2 = 0, r12 = 0, r34 = 0, seen = 0;
    for (u32 seg = blockIdx.x; seg < nseg; seg += gridDim.x) {
        const u64 seg0 = (u64)seg * GAP_SEG_BITS;
        __syncthreads();
        for (u32 i = tid; i < GAP_WORDS; i += GAP_THREADS) {   // zero at and past the sieved bits
            const u64 b = seg0 + 32ull * i;
            u32 v = 0;
            if (b < nbits_all) {
                v = __ldg(bm + (b >> 5));
                if (b + 32 > nbits_all) v &= (1u << (u32)(nbits_all - b)) - 1u;
            }
            w[i] = v;
        }
        __syncthreads();
        // compaction in order: thread t owns words [t GAP_WPT, (t + 1) GAP_WPT)
        u32 c = 0;
#pragma unroll
        for (u32 k = 0; k < GAP_WPT; k++) c += __popc(w[tid * GAP_WPT + k]);
        u32 incl = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const u32 v = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (u32)d) incl += v;
        }
        if (lane == 31) s_wsum[warp] = incl;
        __syncthreads();
        u32 pos = incl - c, total = 0;
#pragma unroll
        for (u32 i = 0; i < GAP_THREADS / 32; i++) {
            const u32 v = s_wsum[i];
            if (i < warp) pos += v;
            total += v;
        }
#pragma unroll
        for (u32 k = 0; k < GAP_WPT; k++)
            for (u32 y = w[tid * GAP_WPT + k]; y; y &= y - 1) {
                if (pos < GAP_MAXP) P[pos] = (u16)((tid * GAP_WPT + k) * 32 + __ffs(y) - 1);
                pos++;
            }
        if (tid == 0 && total > GAP_MAXP) atomicOr(err, 8u);
        __syncthreads();
        const u32 n = total < GAP_MAXP ? total : GAP_MAXP;
        const u64 in = nbits_in - seg0;                        // bits of the segment in [lo, hi)
        const u32 lim = (u32)min((u64)GAP_SEG_BITS, in);
        // the position after place j at position x (relative to the segment), ~0 when none is sieved
        const auto after = [&](u32 j, u32 x) -> u32 {
            if (j + 1 < n) return P[j + 1];
            const u64 b = gap_next(bm, seg0 + x, nbits_all);
            return b == ~0ull ? ~0u : (u32)(b - seg0);
        };
        // The primes of this segment in [lo, hi), 32 consecutive ones a step, each warp a contiguous run
        // of steps.  A place is a descent when the gap after it is no wider: L(p) is the distance to the
        // first descent from p on, read off the ballots of the step and the next one.
        const u32 steps = (n + 31) / 32, per = (steps + GAP_THREADS / 32 - 1) / (GAP_THREADS / 32);
        const u32 g0 = warp * per, ge = min(g0 + per, steps);
        u32 np = 0, np1 = 0, np2 = 0, ndown = 0;
        const auto load = [&](u32 g) {
            const u32 i = g * 32 + lane;
            if (g * 32 + 34 <= n) {
                np = P[i];
                np1 = P[i + 1];
                np2 = P[i + 2];
            } else {
                np = i < n ? P[i] : ~0u;
                np1 = i + 1 < n ? P[i + 1] : ~0u;
                np2 = i + 2 < n ? P[i + 2] : ~0u;
            }
            ndown = __ballot_sync(0xffffffffu, np2 != ~0u && np2 - np1 <= np1 - np);
        };
        if (g0 < ge) load(g0);
        for (u32 g = g0; g < ge; g++) {
            const u32 p = np, p2 = np2, down = ndown, i = g * 32 + lane;
            u32 p1 = np1;
            load(g + 1);
            const auto take = [&] {
                if (p1 == ~0u) {                                        // the window's last prime
                    p1 = after(i, p);
                    if (p1 == ~0u) { atomicAdd(&s_uns, 1u); return; }
                }
                const u32 g1 = p1 - p;                                  // the gap / 2 (every gap < 2048)
                atomicAdd(&hist[g1 < MP_GAP_BINS ? g1 : MP_GAP_BINS - 1], 1u);
                c1 += g1 != 1;
                if (g1 == 1) {
                    // chain: the m-th gap after p is 2m integers = m bits
                    if (p2 != ~0u && p2 - p1 != 2 && co.min_len != 2) c2++;
                    else {
                        u32 cl = 2, jc = i + 1, x = p1, y = after(jc, x);
                        while (y != ~0u && y - x == cl) { cl++; jc++; x = y; y = after(jc, x); }
                        if (y == ~0u) atomicAdd(&s_uns, 1u);            // still a chain at the end of the sieved bits
                        else {
                            const u32 cc = cl < MP_CHAIN_MAX ? cl : MP_CHAIN_MAX - 1;
                            atomicAdd(&ch[cc], 1u);
                            if (co.min_len && cl >= co.min_len) {
                                const unsigned long long k = atomicAdd(co.n, 1ull);
                                if (k < co.cap) {
                                    co.heads[k] = base + 2 * (seg0 + p) + 1;
                                    co.lens[k] = cc;
                                }
                            }
                        }
                    }
                }
                u32 L = __ffs(__funnelshift_r(down, ndown, lane));
                if (!L) {
                    // no descent in sight: walk on past the window
                    u32 j = i + 1, gp = g1, x = p1, k = 1;
                    for (;;) {
                        const u32 y = after(j, x);
                        if (y == ~0u) break;
                        if (y - x <= gp) { L = k; break; }
                        k++;
                        gp = y - x;
                        j++;
                        x = y;
                    }
                    if (!L) { atomicAdd(&s_uns, 1u); return; }
                }
                if (L > 4) atomicAdd(&rh[L < MP_RUN_MAX ? L : MP_RUN_MAX - 1], 1u);
                else if (L > 2) r34 += 1u << (16 * (L - 3));
                else r12 += 1u << (16 * (L - 1));
                if (L >= 32 || !((seen >> L) & 1)) {
                    seen |= L < 32 ? 1u << L : 0u;
                    atomicMin((unsigned long long *)&rf[L < MP_RUN_MAX ? L : MP_RUN_MAX - 1],
                              (unsigned long long)(base + 2 * (seg0 + p) + 1));
                }
            };
            if (p < lim) take();
            __syncwarp();                                           // the next step's ballot takes every lane
        }
    }
    __syncwarp();
    c1 = __reduce_add_sync(0xffffffffu, c1);
    c2 = __reduce_add_sync(0xffffffffu, c2);
    const u32 r1 = __reduce_add_sync(0xffffffffu, r12 & 0xffffu), r2 = __reduce_add_sync(0xffffffffu, r12 >> 16);
    const u32 r3 = __reduce_add_sync(0xffffffffu, r34 & 0xffffu), r4 = __reduce_add_sync(0xffffffffu, r34 >> 16);
    if (lane == 0) {
        atomicAdd(&ch[1], c1);
        atomicAdd(&ch[2], c2);
        atomicAdd(&rh[1], r1);
        atomicAdd(&rh[2], r2);
        atomicAdd(&rh[3], r3);
        atomicAdd(&rh[4], r4);
    }
    __syncthreads();
    for (u32 i = tid; i < MP_GAP_BINS; i += GAP_THREADS)
        if (hist[i]) atomicAdd((unsigned long long *)&acc->gap_hist[i], (unsigned long long)hist[i]);
    if (tid < MP_RUN_MAX && rh[tid]) {
        atomicAdd((unsigned long long *)&acc->run_hist[tid], (unsigned long long)rh[tid]);
        atomicMin((unsigned long long *)&acc->run_first[tid], (unsigned long long)rf[tid]);
    }
    if (tid < MP_CHAIN_MAX && ch[tid]) atomicAdd((unsigned long long *)&acc->chain_hist[tid], (unsigned long long)ch[tid]);
    if (tid == 0 && s_uns) atomicAdd((unsigned long long *)&acc->unsettled, (unsigned long long)s_uns);
}

// sieve [lo, hi) a chunk at a time and run gap_kernel over it; the accumulator and the chain
// list stay on the device (the caller copies them)
static int gap_run(mp_handle *h, u64 lo, u64 hi, mp_gap_stats *acc, ChainOut co, cudaStream_t st)
{
    int per_sm = 0;
    MP_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gap_kernel, GAP_THREADS, 0));
    const u64 resident = (u64)h->sm_count * (u32)std::max(per_sm, 1);
    MP_CUDA(h, cudaMemsetAsync(acc, 0, sizeof(mp_gap_stats), st));
    MP_CUDA(h, cudaMemsetAsync(acc->run_first, 0xff, sizeof acc->run_first, st));
    MP_CUDA(h, h->small_out.ensure(256));
    mp_sieve_opts o;
    memset(&o, 0, sizeof o);
    o.mode = MP_MODE_BATCHED;
    for (u64 c = lo; c < hi;) {
        const u64 c1 = hi - c > GAP_CHUNK ? c + GAP_CHUNK : hi;
        const u64 ext = c1 + GAP_LOOK;
        const u64 base = c & ~1ull;
        const u64 nbits_all = (ext - base) >> 1, nbits_in = (c1 - base) >> 1;
        MP_CUDA(h, h->scratch_bitmap.ensure((size_t)((nbits_all + 63) >> 6) * 8 + 64));
        MP_TRY(mp_sieve_run(h, c, ext, &o, h->small_out.as<mp_range_stats>(), nullptr, nullptr,
                            h->scratch_bitmap.as<u64>(), st));
        const u64 nseg = (nbits_in + GAP_SEG_BITS - 1) / GAP_SEG_BITS;
        if (nseg) {
            gap_kernel<<<(unsigned)std::min(nseg, resident), GAP_THREADS, 0, st>>>(
                h->scratch_bitmap.as<u32>(), nbits_in, nbits_all, base, (u32)nseg, acc, h->errflag.as<u32>(), co);
            MP_CUDA(h, cudaGetLastError());
        }
        c = c1;
    }
    return MP_OK;
}

// the prime 2 is outside the odd-only map: its gap is 1; 1 < 2 (3 -> 5) >= 2 (5 -> 7) gives
// L(2) = 2; and no chain starts with the gap 1
static void add_two(mp_gap_stats *out, u64 lo, u64 hi)
{
    if (lo <= 2 && 2 < hi) {
        out->gap_hist[0]++;
        out->run_hist[2]++;
        if (out->run_first[2] > 2) out->run_first[2] = 2;
        out->chain_hist[1]++;
    }
    for (int l = 0; l < MP_RUN_MAX; l++)
        if (out->run_first[l] == ~0ull) out->run_first[l] = 0;
}

extern "C" int mp_gap_stats_range(mp_handle *h, uint64_t lo, uint64_t hi, mp_gap_stats *out)
{
    if (!h || !out) return MP_EINVAL;
    memset(out, 0, sizeof *out);
    if (hi <= lo) return MP_OK;
    std::lock_guard<std::recursive_mutex> lk(h->mu);
    if (hi > MP_HI_MAX - 2 * GAP_LOOK) return mp_set_error(h, MP_ERANGE, "hi must be <= 2^64 - 2^18 - 2^17");
    MP_CUDA(h, cudaSetDevice(h->device));
    cudaStream_t st = h->stream;
    MP_CUDA(h, h->gap_acc.ensure(sizeof(mp_gap_stats) + 64));
    mp_gap_stats *acc = h->gap_acc.as<mp_gap_stats>();
    ChainOut co;
    memset(&co, 0, sizeof co);
    MP_TRY(gap_run(h, lo, hi, acc, co, st));
    MP_CUDA(h, cudaMemcpyAsync(out, acc, sizeof *out, cudaMemcpyDeviceToHost, st));
    MP_TRY(mp_sieve_errors(h, st));                      // synchronises
    add_two(out, lo, hi);
    return MP_OK;
}

extern "C" int mp_gap_chains(mp_handle *h, uint64_t lo, uint64_t hi, uint32_t min_len, uint64_t *heads, uint32_t *lens,
                             size_t cap, size_t *count)
{
    if (!h || !count || (cap && (!heads || !lens))) return MP_EINVAL;
    *count = 0;
    if (min_len < 2) return mp_set_error(h, MP_EINVAL, "min_len must be at least 2");
    if (hi <= lo) return MP_OK;
    std::lock_guard<std::recursive_mutex> lk(h->mu);
    if (hi > MP_HI_MAX - 2 * GAP_LOOK) return mp_set_error(h, MP_ERANGE, "hi must be <= 2^64 - 2^18 - 2^17");
    MP_CUDA(h, cudaSetDevice(h->device));
    cudaStream_t st = h->stream;
    MP_CUDA(h, h->gap_acc.ensure(sizeof(mp_gap_stats) + 64));
    mp_gap_stats *acc = h->gap_acc.as<mp_gap_stats>();
    // the list: cap entries (at least one, so that the device pointers are valid)
    const u64 dcap = cap ? cap : 1;
    MP_CUDA(h, h->ferm_p.ensure((size_t)dcap * 12 + 64));
    ChainOut co;
    co.min_len = min_len;
    co.cap = cap;
    co.heads = h->ferm_p.as<u64>();
    co.lens = (u32 *)(co.heads + dcap);
    co.n = (unsigned long long *)((char *)h->gap_acc.p + sizeof(mp_gap_stats));
    MP_CUDA(h, cudaMemsetAsync(co.n, 0, 8, st));
    MP_TRY(gap_run(h, lo, hi, acc, co, st));
    u64 n = 0;
    MP_CUDA(h, cudaMemcpyAsync(&n, co.n, 8, cudaMemcpyDeviceToHost, st));
    MP_TRY(mp_sieve_errors(h, st));                      // synchronises
    const u64 m = n < cap ? n : cap;
    std::vector<u64> hd(m);
    std::vector<u32> ln(m);
    if (m) {
        MP_CUDA(h, cudaMemcpyAsync(hd.data(), co.heads, m * 8, cudaMemcpyDeviceToHost, st));
        MP_CUDA(h, cudaMemcpyAsync(ln.data(), co.lens, m * 4, cudaMemcpyDeviceToHost, st));
        MP_CUDA(h, cudaStreamSynchronize(st));
    }
    // the device appends in arbitrary order: sort by head (only when the list is complete is
    // the order of a partial list meaningful, so a partial list is sorted as found)
    std::vector<u64> ord(m);
    for (u64 i = 0; i < m; i++) ord[i] = i;
    std::sort(ord.begin(), ord.end(), [&](u64 x, u64 y) { return hd[x] < hd[y]; });
    for (u64 i = 0; i < m; i++) { heads[i] = hd[ord[i]]; lens[i] = ln[ord[i]]; }
    *count = (size_t)n;
    return MP_OK;
}
