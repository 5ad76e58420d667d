// mp_planes.cu -- the batched sieve in residue planes mod 30 for B200 (sm_100a).
//
// Of every 30 integers only the eight 30 i + r, r = 1, 7, 11, 13, 17, 19, 23, 29, can be primes
// above 5.  Plane r is the bitmap over i of the numbers 30 i + r.  In a plane the multiples of a
// sieving prime q lie exactly q bits apart, so marking needs no wheel: one progression of stride
// q per prime, of which 32 lanes take every 32nd term (a stride of q whole words with one bit
// mask per lane).  A bit of a plane stands for 3.75 integers instead of the odd-only map's 2, so
// a shared-memory tile spans twice the integers and the sparse primes are visited half as often.
//
// A range is processed in waves of whole scan stretches (2^tlog bits of the odd-only map, the unit
// of the summaries).  Per wave:
//   scatter   the bucket primes (above the tile): their hits in the eight planes, filed by tile
//   tile      one (plane, block of pt bits) per CTA step: patterns for 7 .. 89, marks, records;
//             the prime bits go to the wave's plane buffer
//   scan      the planes of each stretch side by side: pi, twins, 6-tuples with their checksum,
//             first / last prime, widest gap; where asked for the odd-only bitmap words
//   emit      (prime lists only) the in-range primes in order
// The summaries and the outputs are those of the odd-only form (mp_sieve.cu), bit for bit.
//
// Reference behaviour (paths inside the Mathpub project): see mp_sieve.cu; the mod-30 layout is
// the one of A158939/cuda/a158939_cuda.cu:26-41 with a plane instead of a bit per residue.
#include "mp_sieve.cuh"
#include "mp_planes_cap.h"
#include <algorithm>
#include <atomic>
#include <math.h>

// c_res(k): the residues in order
__host__ __device__ __forceinline__ u32 pl_res(u32 k) { return (u32)(0x1d1713110d0b0701ull >> (8 * k)) & 0xffu; }

// For plane residue r and c = q mod 30 (q a unit): the multiples of q in the plane are the q k with
// k = u (mod 30), u = r q^-1 mod 30, and q u = 30 (a u + v) + r with a = q / 30, v = (c u - r) / 30.
// So i = a u + v (mod q) is the class of their indices.
struct PlaneUV {
    u8 u, v;
};
__host__ __device__ __forceinline__ PlaneUV pl_uv(u32 r, u32 c)
{
    const u32 inv = c * c % 30u * c % 30u;               // every unit mod 30 has an order dividing 4
    const u32 u = r * inv % 30u;
    return PlaneUV{(u8)u, (u8)((c * u - r) / 30u)};
}

#define PL_PTMAX 1769472u             // bits of a tile at most (216 KB of shared memory)
#define PL_NPAT MP_NPAT
#define PL_IMOD_MIN 4096u            // primes from which on a launch for their remainders pays

struct PlaneTileArgs {
    u64 i0;                           // index of the wave's first plane bit
    u32 nb, pt, ntile;                // blocks per plane, bits per block, tiles = 8 nb
    const u32 *q;
    const u64 *magic;
    u32 iw0, iw1, it1;                // warp tier [iw0, iw1), thread tier [iw1, it1)
    const u32 *pat[PL_NPAT];
    u32 period[PL_NPAT], zoff[PL_NPAT][8];
    const u32 *rec, *cnt;             // bucket records by tile (nullable)
    u32 cap;
    u32 *planes;                      // [8][nb pt / 32] words, set bits are primes
    u32 *tstate;                      // per CTA: next multiple of each thread-tier prime
    const u32 *imod;                  // i0 mod q for the primes from iw0 on (nullable)
};

// index (relative to is) of the first multiple of q at or after `is` in the CTA's plane, the prime
// itself excepted, from m = is mod q; uv: the plane's table by q mod 30
__device__ __forceinline__ u32 plane_first(u64 is, u32 q, u32 m, const u16 *uv)
{
    const u32 a = q / 30u, t = uv[q - 30u * a], u = t & 0xffu;
    const u32 s = a * u + (t >> 8);                      // < q
    u32 j = s - m;
    j = min(j, j + q);                                   // s < m: below zero, so the sum is the smaller
    if (is <= a && u == 1 && is + j == a) j += q;
    return j;
}

// (i0 + off) mod q from r = i0 mod q, which a launch of its own took once for the wave, and M = floor(2^32
// / q): a 32-bit remainder instead of a 64-bit one.  The quotient is at most 2 short, so 3 q and r + off have to
// be below 2^32, which plan_planes sees to: off < 2^31, and q is a prime below the buckets (up to 1.5 tiles,
// 2654208, and a few primes more)
__device__ __forceinline__ u32 plane_mod(u32 r, u32 off, u32 q, u32 M)
{
    const u32 x = r + off;
    u32 m = x - __umulhi(x, M) * q;                      // < 3 q
    m = min(m, m - q);
    return min(m, m - q);
}

__global__ void __launch_bounds__(256) plane_imod_kernel(const u32 *__restrict__ q, const u64 *__restrict__ magic, u32 n,
                                                         u64 i0, u32 *__restrict__ out)
{
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = mp_mod_barrett(i0, q[i], magic[i]);
}

__device__ __forceinline__ void plane_presieve(u32 *sm, u32 nw, const PlaneTileArgs &a, const u32 *s_off)
{
    const u32 tid = threadIdx.x, nth = blockDim.x;
    for (u32 w4 = tid * 4; w4 < nw; w4 += nth * 4) {
        u32 o0 = 0, o1 = 0, o2 = 0, o3 = 0;
        uint4 LO[PL_NPAT], HI[PL_NPAT];
#pragma unroll
        for (int p = 0; p < PL_NPAT; p++) {              // all loads first: ten in flight per thread
            const u32 a4 = ((s_off[p] >> 5) + w4) & ~3u;
            LO[p] = __ldg((const uint4 *)(a.pat[p] + a4));
            HI[p] = __ldg((const uint4 *)(a.pat[p] + a4 + 4));
        }
#pragma unroll
        for (int p = 0; p < PL_NPAT; p++) {
            const u32 bit = s_off[p] + w4 * 32;
            const u32 s = bit >> 5, sh = bit & 31;
            const uint4 lo = LO[p], hi = HI[p];
            u32 v0, v1, v2, v3, v4;
            switch (s & 3) {                             // the same in the whole CTA
            case 0: v0 = lo.x; v1 = lo.y; v2 = lo.z; v3 = lo.w; v4 = hi.x; break;
            case 1: v0 = lo.y; v1 = lo.z; v2 = lo.w; v3 = hi.x; v4 = hi.y; break;
            case 2: v0 = lo.z; v1 = lo.w; v2 = hi.x; v3 = hi.y; v4 = hi.z; break;
            default: v0 = lo.w; v1 = hi.x; v2 = hi.y; v3 = hi.z; v4 = hi.w; break;
            }
            o0 |= __funnelshift_r(v0, v1, sh);
            o1 |= __funnelshift_r(v1, v2, sh);
            o2 |= __funnelshift_r(v2, v3, sh);
            o3 |= __funnelshift_r(v3, v4, sh);
        }
        *(uint4 *)&sm[w4] = make_uint4(o0, o1, o2, o3);
    }
}

// CTA b sieves the tiles [b per, (b + 1) per) of the wave in order; tile t is block t mod nb of
// plane t / nb, so that the thread-tier primes carry their next multiple along a plane.  Bound by
// shared-memory atomics: [1e15, +2^34) 3.45 ms, 1.75e12 marks and records a second or 0.88 of the rate of
// atomics on random words (the odd-only tiles: 5.85 ms with their scans of 1.2, 0.51 of that rate)
template <int NTH>
__global__ void __launch_bounds__(NTH) plane_tile_kernel(PlaneTileArgs a)
{
    extern __shared__ __align__(16) u32 sm[];            // pt / 32 words
    __shared__ u32 s_off[PL_NPAT];
    __shared__ u16 s_uv[30];
    const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr u32 nth = NTH, nwarps = NTH / 32;
    const u32 pt = a.pt, nw = pt >> 5;
    const u32 per = (a.ntile + gridDim.x - 1) / gridDim.x;
    const u32 tb = blockIdx.x * per, te = min(tb + per, a.ntile);
    u32 *const tst = a.tstate + (u64)blockIdx.x * (a.it1 - a.iw1);
    for (u32 t = tb; t < te; t++) {
        const u32 pl = t / a.nb, blk = t - pl * a.nb;
        const bool fresh = t == tb || blk == 0;          // no carried state yet
        const bool keep = t + 1 < te && blk + 1 < a.nb;  // the plane's next block follows here
        const u64 is = a.i0 + (u64)blk * pt;
        if (tid < PL_NPAT) {
            const u32 o = (u32)(is % a.period[tid]) + a.zoff[tid][pl];
            s_off[tid] = o >= a.period[tid] ? o - a.period[tid] : o;
        }
        if (tid < 30) {
            const PlaneUV x = pl_uv(pl_res(pl), tid);
            s_uv[tid] = (u16)(x.u | x.v << 8);           // (used at the units only)
        }
        __syncthreads();
        plane_presieve(sm, nw, a, s_off);
        __syncthreads();
        if (is <= 2 && tid == 0) {
            // the pattern primes themselves are prime; 1 is not
            const u32 pp[22] = {7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61, 67, 71, 73, 79, 83, 89, 0};
            for (int k = 0; pp[k]; k++)
                if (pp[k] % 30 == pl_res(pl) && pp[k] / 30 >= is) {
                    const u32 j = pp[k] / 30 - (u32)is;
                    atomicAnd(&sm[j >> 5], ~(1u << (j & 31)));
                }
            if (is == 0 && pl == 0) atomicOr(&sm[0], 1u);
        }
        // The marks, in any order: the warp tier is bound by shared memory, the thread tier and the
        // records by L2, so a third of the warps starts with each ([1e15, +2^34): 3.44 ms of tile kernel
        // against 3.79 with every warp in the same order; by warp & 1 3.53)
        for (u32 step = 0; step < 3; step++) {
            const u32 part = (step + warp) % 3u;
            if (part == 0) {
                // warp tier.  Warp w takes the primes w, w + nwarps, ... of the tier, 32 at a time: lane i
                // sets up prime i of the batch, then the warp marks the batch one prime after the other,
                // lane l the multiples l, l + 32, ...: 32 q bits apart, so a lane's mask stays and its word
                // advances by q
                for (u32 kb = a.iw0 + warp; kb < a.iw1; kb += 32 * nwarps) {
                    const u32 k = kb + nwarps * lane;
                    u32 q = 0, j = 0;
                    if (k < a.iw1) {
                        q = __ldg(a.q + k);
                        const u64 M = __ldg(a.magic + k);
                        const u32 m = a.imod ? plane_mod(__ldg(a.imod + (k - a.iw0)), blk * pt, q, (u32)(M >> 32))
                                             : mp_mod_barrett(is, q, M);
                        j = plane_first(is, q, m, s_uv);
                    }
                    const u32 n = min(32u, (a.iw1 - kb + nwarps - 1) / nwarps);
                    for (u32 i = 0; i < n; i++) {
                        const u32 qi = __shfl_sync(0xffffffffu, q, i), ji = __shfl_sync(0xffffffffu, j, i) + lane * qi;
                        const u32 m = __funnelshift_l(0u, 1u, ji);
                        u32 w = ji >> 5;
                        if (33 * qi <= nw) {
                            // at least 32 steps a lane: the lanes start at different steps, lane l at the one
                            // whose word is in bank l (q is odd), go to the end and on from the first word, so
                            // that a step meets each bank once, twice while some lanes have wrapped
                            u32 inv = qi;
                            inv *= 2 - qi * inv;                  // 1 / q mod 64
                            const u32 first = w, start = w + qi * (((lane - w) * inv) & 31u);
                            w = start;
                            do {
                                atomicOr(&sm[w], m);
                                w += qi;
                                if (w >= nw) w = first;
                            } while (w != start);
                            continue;
                        }
                        for (; w + 3 * qi < nw; w += 4 * qi) {
                            atomicOr(&sm[w], m);
                            atomicOr(&sm[w + qi], m);
                            atomicOr(&sm[w + 2 * qi], m);
                            atomicOr(&sm[w + 3 * qi], m);
                        }
                        for (; w < nw; w += qi) atomicOr(&sm[w], m);
                    }
                }
            } else if (part == 1) {
                // thread tier, one thread per prime, its next multiple carried to the plane's next block.  Half
                // of a visit was address arithmetic and bounds, so the thread count is a constant (the eight
                // primes a thread loads ahead are immediate offsets) and whole batches run without checks
                {
                    const u32 n = a.it1 - a.iw1;
                    const u32 *pq = a.q + a.iw1 + tid;
                    u32 *ps = tst + tid;
                    u32 i = tid;
                    if (!fresh) {
                        for (; i + 7 * NTH < n; i += 8 * NTH, pq += 8 * NTH, ps += 8 * NTH) {
                            u32 qv[8], jv[8];
#pragma unroll
                            for (int u = 0; u < 8; u++) {
                                qv[u] = __ldg(pq + u * NTH);
                                jv[u] = ps[u * NTH];
                            }
#pragma unroll
                            for (int u = 0; u < 8; u++) {
                                u32 j = jv[u];
                                for (; j < pt; j += qv[u]) atomicOr(&sm[j >> 5], __funnelshift_l(0u, 1u, j));
                                if (keep) ps[u * NTH] = j - pt;
                            }
                        }
                    } else if (a.imod) {
                        const u32 *pr = a.imod + (a.iw1 - a.iw0) + i, *pm = (const u32 *)(a.magic + a.iw1 + i) + 1;
                        for (; i + 3 * NTH < n; i += 4 * NTH, pq += 4 * NTH, ps += 4 * NTH, pr += 4 * NTH, pm += 8 * NTH) {
                            u32 qv[4], jv[4], mv[4];
#pragma unroll
                            for (int u = 0; u < 4; u++) {
                                qv[u] = __ldg(pq + u * NTH);
                                jv[u] = __ldg(pr + u * NTH);
                                mv[u] = __ldg(pm + 2 * u * NTH);
                            }
#pragma unroll
                            for (int u = 0; u < 4; u++) {
                                u32 j = plane_first(is, qv[u], plane_mod(jv[u], blk * pt, qv[u], mv[u]), s_uv);
                                for (; j < pt; j += qv[u]) atomicOr(&sm[j >> 5], __funnelshift_l(0u, 1u, j));
                                if (keep) ps[u * NTH] = j - pt;
                            }
                        }
                    }
                    for (; i < n; i += NTH, pq += NTH, ps += NTH) {
                        const u32 q = __ldg(pq);
                        u32 j;
                        if (!fresh) j = *ps;
                        else j = plane_first(is, q, mp_mod_barrett(is, q, __ldg(a.magic + a.iw1 + i)), s_uv);
                        for (; j < pt; j += q) atomicOr(&sm[j >> 5], __funnelshift_l(0u, 1u, j));
                        if (keep) *ps = j - pt;
                    }
                }
            } else if (a.rec) {
                // bucket records of this tile: read once, with streaming hints
                {
                    const u32 n = min(__ldg(a.cnt + t), a.cap);
                    const u32 *R = a.rec + (u64)t * a.cap;       // cap is a multiple of 4
                    const uint4 *R4 = (const uint4 *)R;
                    const u32 n4 = n >> 2;
                    u32 i = tid;
                    for (; i + 3 * nth < n4; i += 4 * nth) {     // 16 records in flight per thread
                        const uint4 r0 = __ldcs(R4 + i), r1 = __ldcs(R4 + i + nth);
                        const uint4 r2 = __ldcs(R4 + i + 2 * nth), r3 = __ldcs(R4 + i + 3 * nth);
                        const u32 js[16] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w,
                                            r2.x, r2.y, r2.z, r2.w, r3.x, r3.y, r3.z, r3.w};
#pragma unroll
                        for (int k = 0; k < 16; k++) atomicOr(&sm[js[k] >> 5], __funnelshift_l(0u, 1u, js[k]));
                    }
                    for (; i < n4; i += nth) {
                        const uint4 r0 = __ldcs(R4 + i);
                        atomicOr(&sm[r0.x >> 5], __funnelshift_l(0u, 1u, r0.x));
                        atomicOr(&sm[r0.y >> 5], __funnelshift_l(0u, 1u, r0.y));
                        atomicOr(&sm[r0.z >> 5], __funnelshift_l(0u, 1u, r0.z));
                        atomicOr(&sm[r0.w >> 5], __funnelshift_l(0u, 1u, r0.w));
                    }
                    for (u32 k = (n4 << 2) + tid; k < n; k += nth) {
                        const u32 j = __ldcs(R + k);
                        atomicOr(&sm[j >> 5], __funnelshift_l(0u, 1u, j));
                    }
                }
            }
        }
        __syncthreads();
        u32 *out = a.planes + (u64)pl * a.nb * nw + (u64)blk * nw;
        for (u32 w4 = tid * 4; w4 < nw; w4 += nth * 4) {
            const uint4 v = *(const uint4 *)&sm[w4];
            *(uint4 *)(out + w4) = make_uint4(~v.x, ~v.y, ~v.z, ~v.w);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------
// bucket scatter
// ---------------------------------------------------------------------------------------

struct PlaneScatterArgs {
    u64 i0;
    u32 ni;                           // plane bits of the wave that matter (< 2^31)
    u32 nb, pt, blk_magic;            // block of bit j: ((j >> 10) blk_magic) >> 32 (pt a multiple of 1024)
    const u32 *q;
    const u64 *magic;
    u32 k0, k1;                       // the bucket primes
    u32 kc, run;                      // primes a warp takes from the queue at once: 32 below kc, then run
    u32 parts, part;                  // below kc a unit is 32 primes over one of `parts` parts of `part` bits
    u32 *rec, *cnt;                   // [8 nb][cap], [8 nb] zeroed before the launch
    u32 cap;
    u32 *queue;                       // zeroed before the launch
    u32 *err;
};

#define PS_THREADS 512
#define PS_STAGE 8192                 // staged records per CTA (two buffers of them)
#define PS_CTAS_PER_SM 3
#define PS_OFF_BITS 21                // staged record: tile << 21 | offset
#define PS_NONE 0xffffffffu           // an empty place of the stage

// sort the staged records by tile and write them to their buckets (all threads)
__device__ __forceinline__ void plane_flush(const PlaneScatterArgs &a, u32 nt, u32 *stage, u32 *sorted, u32 *hist,
                                            u32 *gb, u32 *s_fill, u32 *s_wsum)
{
    const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __syncthreads();
    const u32 n = *s_fill;
    // exclusive scan of the tile counts; thread t owns tiles [t per, (t + 1) per)
    const u32 per = (nt + PS_THREADS - 1) / PS_THREADS;
    const u32 t0 = tid * per;
    u32 sum = 0;
    for (u32 t = t0; t < t0 + per && t < nt; t++) sum += hist[t];
    u32 incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const u32 v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= (u32)d) incl += v;
    }
    if (lane == 31) s_wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const u32 v = lane < PS_THREADS / 32 ? s_wsum[lane] : 0u;
        u32 iv = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const u32 u = __shfl_up_sync(0xffffffffu, iv, d);
            if (lane >= (u32)d) iv += u;
        }
        if (lane < PS_THREADS / 32) s_wsum[lane] = iv - v;
        if (lane == PS_THREADS / 32 - 1) s_wsum[PS_THREADS / 32] = iv;    // all records
    }
    __syncthreads();
    // reserve each tile's run in its bucket; hist becomes the placement cursor and gb the
    // bucket slot of sorted index 0 of that run (mod 2^32)
    u32 start = s_wsum[warp] + incl - sum;
    for (u32 t = t0; t < t0 + per && t < nt; t++) {
        const u32 c = hist[t];
        if (c) {
            const u32 g = atomicAdd(a.cnt + t, c);
            if (g + c > a.cap) atomicOr(a.err, 2u);
            gb[t] = g - start;
        }
        hist[t] = start;
        start += c;
    }
    __syncthreads();
    for (u32 i = tid; i < n; i += PS_THREADS) {
        const u32 r = stage[i];
        if (r != PS_NONE) sorted[atomicAdd(&hist[r >> PS_OFF_BITS], 1u)] = r;
    }
    const u32 nrec = s_wsum[PS_THREADS / 32];
    __syncthreads();
    // the runs of one tile are consecutive in sorted order and in the bucket
    for (u32 i = tid; i < nrec; i += PS_THREADS) {
        const u32 r = sorted[i], tl = r >> PS_OFF_BITS, slot = gb[tl] + i;
        if (slot < a.cap) __stcs(a.rec + (u64)tl * a.cap + slot, r & ((1u << PS_OFF_BITS) - 1u));
    }
    __syncthreads();
    for (u32 t = tid; t < nt; t += PS_THREADS) hist[t] = 0;
    if (tid == 0) *s_fill = 0;
    __syncthreads();
}

// The hits of a bucket prime q in the wave: in each plane one progression of stride q from the class
// of its multiples.  A thread holds one prime and the next hit of each plane, and files one hit per
// plane and round; in plane order the eight starts follow from one remainder i0 mod q.  Warps take
// runs of primes from a queue and hand them to the lanes that have none, so no lane waits for a
// neighbour with more hits; the queue replaces bounds computed on the host for each range.  Bound by the
// stage's shared memory traffic and issue: 3.2e11 records a second at 1e15 (2.24 ms for 2^34 integers; the
// odd-only wheel of 210, with 1/7 fewer records by half as many turns, 4.19 ms), 1.7e11 at 9e17, where a
// prime has 7.5 hits for its set-up (2.2 ms for 2^32, 5.5 before).  SMALL, for
// waves with few units of work or few hits (2^16 integers at 9e17: 754 -> 260 us of scatter; 2^28 at
// 1e12: 88 -> 42 us): units cover parts of the wave, a round looks for primes with hits up to eight
// times, and primes far apart are first asked for any multiple at all.
template <bool SMALL>
__global__ void __launch_bounds__(PS_THREADS, PS_CTAS_PER_SM) plane_scatter_kernel(PlaneScatterArgs a)
{
    extern __shared__ __align__(16) u32 ssm[];
    const u32 nt = 8 * a.nb;
    u32 *stage = ssm, *sorted = ssm + PS_STAGE, *hist = ssm + 2 * PS_STAGE, *gb = hist + nt;
    __shared__ u32 s_fill;
    __shared__ u32 s_wsum[PS_THREADS / 32 + 1];
    __shared__ __align__(8) u64 s_u[30], s_v[30];        // u and v of the eight planes, a byte each, by q mod 30
    const u32 tid = threadIdx.x, lane = tid & 31, lt = (1u << lane) - 1;
    for (u32 i = tid; i < nt; i += PS_THREADS) hist[i] = 0;
    if (tid == 0) s_fill = 0;
    if (tid < 30) {
        u64 U = 0, V = 0;
        for (u32 k = 0; k < 8; k++) {
            const PlaneUV x = pl_uv(pl_res(k), tid);
            U |= (u64)x.u << (8 * k);
            V |= (u64)x.v << (8 * k);
        }
        s_u[tid] = U;
        s_v[tid] = V;
    }
    const u32 ni = a.ni, pt = a.pt, nb = a.nb, dense_q = (SMALL ? a.part : ni) / 2;
    u32 jj[8], q = 0;
    bool have = false;
    u32 wk = 0, wend = 0, wlo = 0, whi = ni;             // the warp's run of primes and part of the wave
    u32 lim = 0;                                         // SMALL: the end of the lane's prime's part
    bool dry = false;                                    // the queue is empty
    __syncthreads();
    for (;;) {
        // hand out primes to the lanes that have none; a prime without a hit is dropped on the spot and
        // its lane tries again, at most eight times a round
        for (int tries = 0; tries < (SMALL ? 8 : 1); tries++) {
            const u32 need = __ballot_sync(0xffffffffu, !have);
            if (SMALL && tries && __popc(need) <= 16) break;
            if (need && wk >= wend && !dry) {
                u32 c = 0;
                if (lane == 0) c = atomicAdd(a.queue, 1u);
                c = __shfl_sync(0xffffffffu, c, 0);
                const u32 parts = SMALL ? a.parts : 1u, fine = ((a.kc - a.k0) >> 5) * parts;   // kc - k0: whole 32s
                const u32 pc = c / parts;
                const u64 k = c < fine ? a.k0 + 32ull * pc : a.kc + (u64)a.run * (c - fine);
                wk = (u32)min(k, (u64)a.k1);
                wend = min(wk + (c < fine ? 32u : a.run), a.k1);
                if (SMALL) {
                    wlo = c < fine ? (c - pc * parts) * a.part : 0u;
                    whi = c < fine ? min(wlo + a.part, ni) : ni;
                }
                dry = wk >= a.k1;
            }
            if (!need || wk >= wend) break;
            const u32 k = wk + __popc(need & lt);
            if (!have && k < wend) {
                q = __ldg(a.q + k);
                const u64 magic = __ldg(a.magic + k), is = a.i0 + wlo;
                bool hit = true;
                if (SMALL && q / 32 > whi - wlo) {
                    // far apart: most have no multiple, in a plane or not, in the part's integers
                    const u32 r = mp_mod_barrett(30 * is, q, magic);
                    hit = r == 0 || q - r < 30 * (whi - wlo);
                }
                if (hit) {
                    const u32 m = mp_mod_barrett(is, q, magic);
                    const u32 qa = q / 30u, c = q - 30u * qa;
                    const u64 U = s_u[c], V = s_v[c];
                    u32 jmin = 0xffffffffu;
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const u32 u = (u32)(U >> (8 * i)) & 0xffu, v = (u32)(V >> (8 * i)) & 0xffu;
                        const u32 s = qa * u + v;
                        u32 j = s - m + (s < m ? q : 0u);
                        if (is <= qa && u == 1 && is + j == qa) j = q < ni ? j + q : ni;    // not q itself
                        if (SMALL) j = j < ni ? j + wlo : 0xffffffffu;   // from the wave's start
                        jj[i] = j;
                        jmin = min(jmin, j);
                    }
                    if (SMALL) lim = whi;
                    have = jmin < (SMALL ? lim : ni);
                }
            }
            wk = min(wk + (u32)__popc(need), wend);
        }
        if (!__syncthreads_or(have || wk < wend || !dry)) break;   // the last round's appends are done
        // every thread takes the fill before any thread appends again, so the flush decision
        // (and the barriers inside the flush) is the same in every thread
        const u32 fill = s_fill;
        __syncthreads();
        if (fill > PS_STAGE - 8 * PS_THREADS) plane_flush(a, nt, stage, sorted, hist, gb, &s_fill, s_wsum);
        // one hit per plane: rec = tile << 21 | bit in the tile, as blk (2^21 - pt) + j + (plane nb << 21)
        u32 rec[8], jmin = 0xffffffffu;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const u32 j = jj[i];
            const bool v = have && j < (SMALL ? lim : ni);
            rec[i] = v ? __umulhi(j >> 10, a.blk_magic) * ((1u << PS_OFF_BITS) - pt) + (j + i * (nb << PS_OFF_BITS))
                       : PS_NONE;
            const u32 jn = v ? j + q : PS_NONE;
            jj[i] = jn < j ? PS_NONE : jn;               // no wrap: q may be close to 2^32
            jmin = min(jmin, jj[i]);
        }
        if (__all_sync(0xffffffffu, have && q <= dense_q)) {
            // nearly every place is taken: the lane's eight go down as they are, empty ones marked
            u32 base = 0;
            if (lane == 0) base = atomicAdd(&s_fill, 256u);
            base = __shfl_sync(0xffffffffu, base, 0);
            uint4 *const at = (uint4 *)(stage + base + 8 * lane);
            at[0] = make_uint4(rec[0], rec[1], rec[2], rec[3]);
            at[1] = make_uint4(rec[4], rec[5], rec[6], rec[7]);
#pragma unroll
            for (int i = 0; i < 8; i++)
                if (rec[i] != PS_NONE) atomicAdd(&hist[rec[i] >> PS_OFF_BITS], 1u);
        } else {
            u32 nmine = 0;
#pragma unroll
            for (int i = 0; i < 8; i++) nmine += rec[i] != PS_NONE;
            u32 incl = nmine;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const u32 u = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= (u32)d) incl += u;
            }
            const u32 tot = __shfl_sync(0xffffffffu, incl, 31), res = (tot + 3) & ~3u;   // 16-byte steps
            u32 base = 0;
            if (lane == 0 && tot) base = atomicAdd(&s_fill, res);
            base = __shfl_sync(0xffffffffu, base, 0);
            u32 pos = base + incl - nmine;
            if (lane < res - tot) stage[base + tot + lane] = PS_NONE;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                if (rec[i] != PS_NONE) {
                    stage[pos++] = rec[i];
                    atomicAdd(&hist[rec[i] >> PS_OFF_BITS], 1u);
                }
            }
        }
        have = have && jmin < (SMALL ? lim : ni);
    }
    plane_flush(a, nt, stage, sorted, hist, gb, &s_fill, s_wsum);
}

// ---------------------------------------------------------------------------------------
// scan
// ---------------------------------------------------------------------------------------

struct PlaneScanArgs {
    SieveGeom g;
    u32 t0, nt;                       // stretches [t0, t0 + nt)
    u64 i0;
    const u32 *planes;
    u32 pstride;                      // words per plane
    TileSum *sums;                    // by stretch
    u32 *bitmap32;                    // nullable
    const u64 *emit_off;              // emit: number of primes before each stretch
    u64 *emit;
    u64 emit_cap;
};

#define SCAN_WARPS 8                  // warps per CTA at most

// the stretch's numbers x, A < x < E (x < base + 2 nbx), as index ranges of the planes relative to i0,
// and the part of them below the range's end
struct Stretch {
    u64 A, E, LIM;                    // LIM = base + 2 limit
    u32 lo[8], hi[8], lim[8];
    u32 lomax, limmin, w0, w1;        // words [w0, w1)
};

// the first i with 30 i + r >= x, relative to i0
__device__ __forceinline__ u32 first_index(u64 x, u32 r, u64 i0) { return (u32)((x > r ? (x - r + 29) / 30 : 0) - i0); }

__device__ __forceinline__ void stretch_setup(Stretch &S, const PlaneScanArgs &a, u32 t)
{
    const u64 G = (u64)t << a.g.tlog, T = 1ull << a.g.tlog;
    const u64 A = a.g.base + 2 * G, E = a.g.base + 2 * min(G + T, a.g.nbx), LIM = a.g.base + 2 * a.g.limit;
    if (threadIdx.x < 8) {
        const u32 k = threadIdx.x, r = pl_res(k);
        S.lo[k] = first_index(A + 1, r, a.i0);
        S.hi[k] = first_index(E, r, a.i0);
        S.lim[k] = first_index(min(max(LIM, A + 1), E), r, a.i0);          // LIM may lie below the stretch
    }
    if (threadIdx.x == 0) {
        S.A = A;
        S.E = E;
        S.LIM = LIM;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        u32 lomax = 0, limmin = ~0u, lomin = ~0u, himax = 0;
        for (int k = 0; k < 8; k++) {
            lomax = max(lomax, S.lo[k]);
            lomin = min(lomin, S.lo[k]);
            limmin = min(limmin, S.lim[k]);
            himax = max(himax, S.hi[k]);
        }
        S.lomax = lomax;
        S.limmin = limmin;
        S.w0 = lomin >> 5;
        S.w1 = (himax + 31) >> 5;
    }
    __syncthreads();
}

// bits b0 .. b0 + 31 that lie in [lo, hi)
__device__ __forceinline__ u32 range_mask(u32 lo, u32 hi, u32 b0)
{
    if (hi <= b0 || lo >= b0 + 32) return 0;
    u32 m = ~0u;
    if (lo > b0) m = ~0u << (lo - b0);
    if (hi < b0 + 32) m &= ~0u >> (b0 + 32 - hi);
    return m;
}

// the planes' words w of the stretch, masked to it (to the range's end with in)
__device__ __forceinline__ void load_masked(u32 (&p)[8], const Stretch &S, const u32 *planes, u32 pstride, u32 w,
                                            bool in)
{
#pragma unroll
    for (int k = 0; k < 8; k++)
        p[k] = planes[(u64)k * pstride + w] & range_mask(S.lo[k], in ? S.lim[k] : S.hi[k], w * 32);
}

// first / last prime of block b of the words (which holds one)
__device__ __forceinline__ u64 block_first(const u32 (&p)[8], u64 i, u32 b)
{
    u64 x = 0;
#pragma unroll
    for (int k = 7; k >= 0; k--)
        if ((p[k] >> b) & 1u) x = 30 * i + pl_res(k);
    return x;
}
__device__ __forceinline__ u64 block_last(const u32 (&p)[8], u64 i, u32 b)
{
    u64 x = 0;
#pragma unroll
    for (int k = 0; k < 8; k++)
        if ((p[k] >> b) & 1u) x = 30 * i + pl_res(k);
    return x;
}

// 8 words, bit b of word k -> 32 bytes, bit k of byte b: byte b of the result is byte b & 3 of v[b / 4]
__device__ __forceinline__ void transpose_planes(u32 (&v)[8], const u32 (&p)[8])
{
    u32 x[4], y[4];
    {
        const u32 a = __byte_perm(p[0], p[1], 0x5140), b = __byte_perm(p[0], p[1], 0x7362);
        const u32 c = __byte_perm(p[2], p[3], 0x5140), d = __byte_perm(p[2], p[3], 0x7362);
        x[0] = __byte_perm(a, c, 0x5410); x[1] = __byte_perm(a, c, 0x7632);
        x[2] = __byte_perm(b, d, 0x5410); x[3] = __byte_perm(b, d, 0x7632);
    }
    {
        const u32 a = __byte_perm(p[4], p[5], 0x5140), b = __byte_perm(p[4], p[5], 0x7362);
        const u32 c = __byte_perm(p[6], p[7], 0x5140), d = __byte_perm(p[6], p[7], 0x7362);
        y[0] = __byte_perm(a, c, 0x5410); y[1] = __byte_perm(a, c, 0x7632);
        y[2] = __byte_perm(b, d, 0x5410); y[3] = __byte_perm(b, d, 0x7632);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        u32 t = (x[i] ^ (x[i] >> 7)) & 0x00AA00AAu;
        x[i] ^= t ^ (t << 7);
        t = (x[i] ^ (x[i] >> 14)) & 0x0000CCCCu;
        x[i] ^= t ^ (t << 14);
        t = (y[i] ^ (y[i] >> 7)) & 0x00AA00AAu;
        y[i] ^= t ^ (t << 7);
        t = (y[i] ^ (y[i] >> 14)) & 0x0000CCCCu;
        y[i] ^= t ^ (t << 14);
        t = (x[i] ^ (y[i] << 4)) & 0xF0F0F0F0u;
        v[2 * i] = x[i] ^ t;
        v[2 * i + 1] = y[i] ^ (t >> 4);
    }
}

// a block's byte -> its 15 bits of the odd-only map (bit (r - 1) / 2 for residue r)
__device__ __forceinline__ u32 block_odds(u32 byte)
{
    u32 o = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) o |= ((byte >> k) & 1u) << ((pl_res(k) - 1) / 2);
    return o;
}

// widest gap found so far by a lane: the wider, then the earlier one
__device__ __forceinline__ void gap_take(u32 &bg, u64 &bs, u64 p, u64 next, u64 LIM)
{
    if (p >= LIM) return;
    const u32 g = (u32)(next - p);
    if (g > bg || (g == bg && p < bs)) { bg = g; bs = p; }
}

// starts of runs of at least Z (1 .. 32) empty blocks among the 32 of a word: any = non-empty blocks,
// next = those of the next word, prev = whether the block before the word is non-empty
__device__ __forceinline__ u32 run_starts(u32 any, u32 next, bool prev, u32 Z)
{
    u64 v = ~((u64)next << 32 | any);
    u32 have = 1;
    while (2 * have <= Z) { v &= v >> have; have *= 2; }
    if (Z > have) v &= v >> (Z - have);
    return (u32)v & ((any << 1) | (prev ? 1u : 0u));
}

// one CTA per stretch; warp w takes a contiguous run of its words, 32 a row, lane l word l of the row:
// 32 blocks of 30 integers, eight words, one per plane.  Counts are popcounts; twins and 6-tuples are
// ANDs of planes.  The widest gap is found from the empty blocks: a run of z of them lies in a gap
// between 30 z + 2 and 30 z + 58, so once a gap of g is known only runs of at least (g - 28) / 30
// empty blocks can hold a wider one, and of at least (g - 30) / 30 one as wide, which are rare.  A gap as
// wide counts where it may come first: against another warp's, and in the row whose own search for long
// runs first gave g, since the earliest of equal gaps can have a block fewer than the one found.  Until
// (g - 30) / 30 is at least 1 the row's primes are walked.
// 0.43 ms for 2^33 integers without the bitmap (4.6 GB of planes a ms: issue and the latency of a row),
// 0.6 in the odd-only tiles; a short range waits some 20 us for one stretch's rows
template <bool BITMAP>
__global__ void __launch_bounds__(32 * SCAN_WARPS, 2) plane_scan_kernel(PlaneScanArgs a)
{
    __shared__ Stretch S;
    __shared__ Part s_part[SCAN_WARPS];
    __shared__ u16 s_odds[BITMAP ? 256 : 1];
    __shared__ u32 s_row[BITMAP ? SCAN_WARPS : 1][BITMAP ? 481 : 1];
    __shared__ u32 s_best;              // the CTA's widest gap
    const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const u32 t = a.t0 + blockIdx.x;
    const u64 base = a.g.base, i0 = a.i0;
    if (tid == 0) s_best = 0;
    if (BITMAP)
        for (u32 i = tid; i < 256; i += blockDim.x) s_odds[i] = (u16)block_odds(i);
    stretch_setup(S, a, t);
    const u64 LIM = S.LIM;
    const u32 nrow = (S.w1 - S.w0 + 31) / 32, wrow = (nrow + nwarps - 1) / nwarps;
    const u32 c0 = min(S.w0 + warp * wrow * 32, S.w1), c1 = min(c0 + wrow * 32, S.w1);
    const u32 *const P0 = a.planes;
    u32 cnt = 0, tw = 0, tu = 0, bg = 0, fw = ~0u, lw = 0, liw = 0;     // lw, liw: word + 1
    u64 cks = 0, bs = ~0ull;
    u32 best = 0;                       // the warp's widest gap
    u64 carry = 0;                      // last prime of the rows walked so far (0: none)
    bool walked = false, prevtop = false;
    // bitmap: bit j of the odd-only map is string position j - D of the planes' 15-bit blocks
    const i64 D = (i64)(15 * i0 - base / 2);
    const u32 ds = (u32)(D & 31);
    const i64 dq = D >> 5;
    if (BITMAP && lane == 0) {
        u32 v = 0;
        if (c0 > 0 && c0 < c1) {                         // the last 32 string bits before word c0
            u32 b31 = 0, b30 = 0, b29 = 0;
            for (int k = 0; k < 8; k++) {
                const u32 w = P0[(u64)k * a.pstride + c0 - 1];
                b31 |= ((w >> 31) & 1u) << k;
                b30 |= ((w >> 30) & 1u) << k;
                b29 |= ((w >> 29) & 1u) << k;
            }
            v = block_odds(b31) << 17 | block_odds(b30) << 2 | block_odds(b29) >> 13;
        }
        s_row[warp][0] = v;
    }
    u32 nx[8];
#pragma unroll
    for (int k = 0; k < 8; k++) nx[k] = c0 + lane < c1 ? P0[(u64)k * a.pstride + c0 + lane] : 0u;
    for (u32 wr = c0; wr < c1; wr += 32) {
        const u32 w = wr + lane, b0 = w * 32;
        u32 p[8], raw[8], any = 0, anyin = 0, nany = 0;
        const bool inside = b0 >= S.lomax && (u64)b0 + 32 <= S.limmin;
#pragma unroll
        for (int k = 0; k < 8; k++) raw[k] = nx[k];
#pragma unroll
        for (int k = 0; k < 8; k++) nx[k] = w + 32 < c1 ? P0[(u64)k * a.pstride + w + 32] : 0u;
        const u32 q1 = w < c1 ? P0[w + 1] : 0u;          // plane 1 of the next word (padded buffer)
        if (__all_sync(0xffffffffu, inside || w >= c1)) {
#pragma unroll
            for (int k = 0; k < 8; k++) { p[k] = raw[k]; any |= raw[k]; }
            anyin = any;
        } else {
#pragma unroll
            for (int k = 0; k < 8; k++) {
                any |= raw[k] & range_mask(S.lo[k], S.hi[k], b0);
                p[k] = raw[k] & range_mask(S.lo[k], S.lim[k], b0);
                anyin |= p[k];
            }
        }
        if (wr + 32 < c1) {                              // lane 0's blocks of the next row, for lane 31
            const u32 nw = w + 32;
#pragma unroll
            for (int k = 0; k < 8; k++) nany |= nx[k];
            if (!(nw * 32 >= S.lomax && (u64)nw * 32 + 32 <= S.limmin)) {
                nany = 0;
#pragma unroll
                for (int k = 0; k < 8; k++) nany |= nx[k] & range_mask(S.lo[k], S.hi[k], nw * 32);
            }
        }
        // counts: p are the in-range primes, raw also the members past the end
#pragma unroll
        for (int k = 0; k < 8; k++) cnt += __popc(p[k]);
        tw += __popc(p[2] & raw[3]) + __popc(p[4] & raw[5]) + __popc(p[7] & __funnelshift_r(raw[0], q1, 1));
        u32 six = p[1] & raw[2] & raw[3] & raw[4] & raw[5] & raw[6];
        if (six) {
            tu += __popc(six);
            while (six) {
                const u32 b = __ffs(six) - 1;
                six &= six - 1;
                cks += mp_mix64(30 * (i0 + b0 + b) + 7);
            }
        }
        if (any) {
            if (fw == ~0u) fw = w;
            lw = w + 1;
        }
        if (anyin) liw = w + 1;
        // gaps
        u32 nxt = __shfl_down_sync(0xffffffffu, any, 1);
        const u32 n0 = __shfl_sync(0xffffffffu, nany, 0);
        if (lane == 31) nxt = n0;
        const u32 up = __shfl_up_sync(0xffffffffu, any, 1);
        const bool prev = lane ? (up >> 31) != 0 : prevtop;
        prevtop = (__shfl_sync(0xffffffffu, any, 31) >> 31) != 0;
        // the gaps after the runs that start at the blocks st of this lane's word
        const auto close_runs = [&](u32 st) {
            while (st) {
                const u32 b = __ffs(st) - 1;
                st &= st - 1;
                u32 pm[8];
                const u32 pw = b ? w : w - 1, pb = b ? b - 1 : 31;       // the non-empty block before
                load_masked(pm, S, P0, a.pstride, pw, false);
                const u64 x = block_last(pm, i0 + (u64)pw * 32 + pb, pb);
                u32 nw = w, f = any & (~0u << b);
                while (!f && ++nw < c1) {
                    load_masked(pm, S, P0, a.pstride, nw, false);
                    f = pm[0] | pm[1] | pm[2] | pm[3] | pm[4] | pm[5] | pm[6] | pm[7];
                }
                if (!f) break;                            // past the warp's words: joined by the summaries
                load_masked(pm, S, P0, a.pstride, nw, false);
                gap_take(bg, bs, x, block_first(pm, i0 + (u64)nw * 32 + (__ffs(f) - 1), __ffs(f) - 1), LIM);
            }
        };
        const auto reduce_best = [&] {
            const u32 r = __reduce_max_sync(0xffffffffu, bg);
            if (r > best) {
                best = r;
                if (lane == 0) atomicMax(&s_best, r);
            }
        };
        const bool first = best < 60;                    // no threshold from the rows before
        if (first) {
            // the longest runs of the row first, which settles the threshold at once at most heights
            for (u32 Z = 16; Z; Z >>= 1) {
                const u32 st = run_starts(any, nxt, prev, Z);
                if (__any_sync(0xffffffffu, st != 0)) {
                    close_runs(st);
                    __syncwarp();
                    reduce_best();
                    break;
                }
            }
        }
        const bool walk = best < 60;
        if (walk || walked) {
            // exact primes of the row's words: the lane's first and last, and the last before the lane
            u32 pm[8];
            u64 lf = 0, ll = 0;
            if (w < c1 && any) {
                load_masked(pm, S, P0, a.pstride, w, false);
                const u32 fb = __ffs(any) - 1, lb = 31 - __clz(any);
                lf = block_first(pm, i0 + b0 + fb, fb);
                ll = block_last(pm, i0 + b0 + lb, lb);
                if (walk) {
                    u64 x = 0;
                    for (u32 y = any; y; y &= y - 1) {
                        const u32 b = __ffs(y) - 1;
#pragma unroll
                        for (int k = 0; k < 8; k++)
                            if ((pm[k] >> b) & 1u) {
                                const u64 z = 30 * (i0 + b0 + b) + pl_res(k);
                                if (x) gap_take(bg, bs, x, z, LIM);
                                x = z;
                            }
                    }
                }
            }
            __syncwarp();
            u64 sc = ll;                                  // inclusive max-scan of the last primes
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const u64 u = __shfl_up_sync(0xffffffffu, sc, d);
                if (lane >= (u32)d && u > sc) sc = u;
            }
            u64 ex = __shfl_up_sync(0xffffffffu, sc, 1);
            if (lane == 0) ex = 0;
            if (!ex) ex = carry;
            if (lf && ex) gap_take(bg, bs, ex, lf, LIM);
            const u64 rl = __shfl_sync(0xffffffffu, sc, 31);
            if (rl) carry = rl;
            reduce_best();
            // the gap that leaves the rows walked is settled by the first prime of a later row
            walked = walk || !rl;
        }
        if (!walk) {
            // a gap found by another warp counts too, but one that ties it may come first here, as one that ties
            // this row's own first find may
            const u32 other = *(volatile u32 *)&s_best;
            const u32 Z = max(best - (first ? 30 : 28), other > 30 ? other - 30 : 0u) / 30;
            const u32 st = run_starts(any, nxt, prev, min(32u, Z));
            if (__any_sync(0xffffffffu, st != 0)) {
                close_runs(st);
                __syncwarp();
                reduce_best();
            }
        }
        if (BITMAP) {
            u32 v[8], o[16];
            transpose_planes(v, raw);
#pragma unroll
            for (int k = 0; k < 16; k++) o[k] = 0;
#pragma unroll
            for (int b = 0; b < 32; b++) {
                const u32 x = s_odds[(v[b >> 2] >> (8 * (b & 3))) & 0xffu];
                o[(15 * b) >> 5] |= x << ((15 * b) & 31);
                if (((15 * b) & 31) > 17) o[((15 * b) >> 5) + 1] |= x >> (32 - ((15 * b) & 31));
            }
            u32 *const row = s_row[warp];
#pragma unroll
            for (int k = 0; k < 15; k++) row[1 + 15 * lane + k] = o[k];
            __syncwarp();
            // string word K of the row goes, with the top of word K - 1, to map word K + dq
            const u64 G = (u64)t << a.g.tlog;
            const i64 m0 = (i64)(G >> 5), m1 = (i64)((min(G + (1ull << a.g.tlog), (a.g.limit + 63) & ~63ull) + 31) >> 5);
            const u32 nk = 15 * min(32u, c1 - wr);
            const i64 mr = (i64)15 * wr + dq;             // the row's first map word
            if (nk == 480 && mr > 0 && mr >= m0 && mr + 480 <= m1 && (u64)(mr + 480) * 32 <= a.g.limit) {
                u32 *const out = a.bitmap32 + mr + lane;
#pragma unroll
                for (u32 k = 0; k < 15; k++)
                    out[32 * k] = __funnelshift_l(row[32 * k + lane], row[32 * k + lane + 1], ds);
            } else
            for (u32 k = lane; k < nk; k += 32) {
                const i64 m = (i64)15 * wr + k + dq;
                if (m < m0 || m >= m1) continue;
                u32 x = ds ? (row[k] >> (32 - ds)) | (row[k + 1] << ds) : row[k + 1];
                if (m == 0) {                             // 3 and 5 are in no plane
                    if (base < 3) x |= 1u << ((3 - (u32)base) / 2);
                    if (base < 5) x |= 1u << ((5 - (u32)base) / 2);
                }
                a.bitmap32[m] = x & bits_mask((u64)m * 32, a.g.limit);
            }
            __syncwarp();
            if (lane == 0) row[0] = row[480];
            __syncwarp();
        }
    }
    // the warp's summary in bits of the odd-only map
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
        cnt += __shfl_xor_sync(0xffffffffu, cnt, d);
        tw += __shfl_xor_sync(0xffffffffu, tw, d);
        tu += __shfl_xor_sync(0xffffffffu, tu, d);
        cks += __shfl_xor_sync(0xffffffffu, cks, d);
        fw = min(fw, __shfl_xor_sync(0xffffffffu, fw, d));
        lw = max(lw, __shfl_xor_sync(0xffffffffu, lw, d));
        liw = max(liw, __shfl_xor_sync(0xffffffffu, liw, d));
        const u32 og = __shfl_xor_sync(0xffffffffu, bg, d);
        const u64 os = __shfl_xor_sync(0xffffffffu, bs, d);
        if (og > bg || (og == bg && os < bs)) { bg = og; bs = os; }
    }
    if (lane == 0) {
        const auto bit = [&](u64 x) { return (x - base - 1) / 2; };
        Part P;
        part_init(P);
        P.count = cnt; P.twins = tw; P.tuples = tu; P.cks = cks;
        u32 pm[8];
        if (fw != ~0u) {
            load_masked(pm, S, P0, a.pstride, fw, false);
            u32 y = pm[0] | pm[1] | pm[2] | pm[3] | pm[4] | pm[5] | pm[6] | pm[7];
            P.first = bit(block_first(pm, i0 + (u64)fw * 32 + (__ffs(y) - 1), __ffs(y) - 1));
            load_masked(pm, S, P0, a.pstride, lw - 1, false);
            y = pm[0] | pm[1] | pm[2] | pm[3] | pm[4] | pm[5] | pm[6] | pm[7];
            P.last = bit(block_last(pm, i0 + (u64)(lw - 1) * 32 + (31 - __clz(y)), 31 - __clz(y)));
        }
        if (liw) {
            load_masked(pm, S, P0, a.pstride, liw - 1, true);
            const u32 y = pm[0] | pm[1] | pm[2] | pm[3] | pm[4] | pm[5] | pm[6] | pm[7];
            P.lastin = bit(block_last(pm, i0 + (u64)(liw - 1) * 32 + (31 - __clz(y)), 31 - __clz(y)));
        }
        if (bg) { P.mg = bg / 2; P.mgs = bit(bs); }
        s_part[warp] = P;
    }
    __syncthreads();
    if (warp == 0) {
        Part Q;
        if (lane < nwarps) Q = s_part[lane];
        else part_init(Q);
        Q = part_warp_reduce(Q, a.g.limit);
        if (lane == 0) {
            if (S.A < 5) {
                // 3 and 5, which are in no plane, come before everything else
                Part L;
                part_init(L);
                for (u32 x = 3; x <= 5; x += 2) {
                    if (x <= S.A || x >= S.E) continue;
                    Part X;
                    part_init(X);
                    X.first = X.last = (x - base - 1) / 2;
                    if (x < LIM) {
                        X.lastin = X.first;
                        X.count = 1;
                        X.twins = 1;                      // (3, 5) and (5, 7)
                    }
                    L = part_join(L, X, a.g.limit);
                }
                Q = part_join(L, Q, a.g.limit);
            }
            TileSum R;
            R.first = Q.first; R.last = Q.last; R.lastin = Q.lastin; R.mgs = Q.mgs; R.cks = Q.cks;
            R.mg = Q.mg; R.count = Q.count; R.twins = Q.twins; R.tuples = Q.tuples;
            a.sums[t] = R;
        }
    }
}

// the in-range primes of each stretch, in order, from place emit_off on.  A warp takes 32 words (1024
// blocks of 30) at a time: the lanes put their primes as 16-bit offsets into the warp's part of shared
// memory, and the warp writes them out in whole rows (36 M primes near 1e12: 0.13 ms, 0.44 with every
// lane writing its own run).  Its part holds as many as any window of 30720 integers is known to have
// (pi(30720) = 3314); that no window has more is not proved, so a row of more is written lane by lane
#define EMIT_WARPS 8
#ifndef EMIT_ROW
#define EMIT_ROW 3328u
#endif
__global__ void __launch_bounds__(32 * EMIT_WARPS) plane_emit_kernel(PlaneScanArgs a)
{
    extern __shared__ __align__(16) u16 s_offs[];         // [EMIT_WARPS][EMIT_ROW]
    __shared__ Stretch S;
    __shared__ u32 s_cnt[EMIT_WARPS];
    const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const u32 t = a.t0 + blockIdx.x;
    u16 *const out = s_offs + warp * EMIT_ROW;
    stretch_setup(S, a, t);
    u64 at = a.emit_off[t];
    if (S.A < 5)
        for (u32 x = 3; x <= 5; x += 2)
            if (x > S.A && x < S.E && x < S.LIM) {
                if (tid == 0 && at < a.emit_cap) a.emit[at] = x;
                at++;
            }
    for (u32 wr = S.w0; wr < S.w1; wr += 32 * EMIT_WARPS) {
        const u32 w = wr + tid;
        u32 p[8], c = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) p[k] = 0;
        if (w < S.w1) load_masked(p, S, a.planes, a.pstride, w, true);
#pragma unroll
        for (int k = 0; k < 8; k++) c += __popc(p[k]);
        u32 incl = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const u32 v = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (u32)d) incl += v;
        }
        const u32 n = __shfl_sync(0xffffffffu, incl, 31);
        if (lane == 0) s_cnt[warp] = n;
        __syncthreads();
        u32 before = 0, total = 0;
#pragma unroll
        for (int i = 0; i < EMIT_WARPS; i++) {
            const u32 v = s_cnt[i];
            if (i < (int)warp) before += v;
            total += v;
        }
        u32 v[8], pos = incl - c;
        transpose_planes(v, p);
        const u64 first = 30 * (a.i0 + (u64)(wr + 32 * warp) * 32), to = at + before;
        const bool staged = n <= EMIT_ROW;                // the same in the whole warp
#pragma unroll
        for (int m = 0; m < 8; m++) {
            const u32 x0 = 30 * (32 * lane + 4 * m);
            for (u32 y = v[m]; y; y &= y - 1) {           // four blocks, a byte each
                const u32 k = __ffs(y) - 1, x = x0 + 30 * (k >> 3) + (__byte_perm(0x0d0b0701u, 0x1d171311u, k & 7) & 0xffu);
                if (staged) out[pos] = (u16)x;
                else if (to + pos < a.emit_cap) a.emit[to + pos] = first + x;
                pos++;
            }
        }
        __syncwarp();
        if (staged)
            for (u32 i = lane; i < n; i += 32)
                if (to + i < a.emit_cap) __stcs(a.emit + to + i, first + out[i]);
        at += total;
        __syncthreads();
    }
}

// emit_off of the stretches [t0, t0 + nt) from their counts, *total the primes before and after them
// (one CTA)
__global__ void __launch_bounds__(1024) plane_offsets_kernel(const TileSum *sums, u32 t0, u32 nt, u64 *off, u64 *total)
{
    __shared__ u64 s_w[32];
    const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const u32 per = (nt + 1023) / 1024, b = min(tid * per, nt), e = min(b + per, nt);
    const u64 start = *total;
    u64 c = 0;
    for (u32 t = b; t < e; t++) c += sums[t0 + t].count;
    u64 incl = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const u64 v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= (u32)d) incl += v;
    }
    if (lane == 31) s_w[warp] = incl;
    __syncthreads();
    u64 before = start;
    for (u32 i = 0; i < warp; i++) before += s_w[i];
    u64 at = before + incl - c;
    for (u32 t = b; t < e; t++) {
        if (off) off[t0 + t] = at;
        at += sums[t0 + t].count;
    }
    if (tid == 1023) *total = at;                         // every thread has read *total before the barrier
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------

// raise a kernel's limit on dynamic shared memory to the device's, once per device
template <class F>
static cudaError_t raise_smem(F kernel, std::atomic<bool> (&done)[16], int device, int bytes)
{
    if (device < 0 || device >= 16) return cudaErrorInvalidDevice;
    if (done[device]) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) done[device] = true;
    return e;
}

struct PlanePlan {
    u32 nb, pt, threads, waves, tw;   // blocks per plane, bits per block; waves of tw stretches
    u32 iw0, iw1, it1, iend;
    u32 cap;
    u64 ni;                           // plane bits of a full wave
    u32 grid, nmod;                   // CTAs of the tile launch; primes of the remainders' launch
    size_t psize, tsize, rsize;       // bytes of the planes, the threads' state and the records
};

static void (*const kTile[3])(PlaneTileArgs) = {plane_tile_kernel<256>, plane_tile_kernel<512>, plane_tile_kernel<1024>};
static int tile_form(u32 threads) { return threads == 1024 ? 2 : threads == 512 ? 1 : 0; }

// the buffers' bytes of a plan, without what they may have to spare
static int plan_sizes(mp_handle *h, PlanePlan &P)
{
    static std::atomic<bool> done[3][16];
    const int tk = tile_form(P.threads);
    MP_CUDA(h, raise_smem(kTile[tk], done[tk], h->device, (int)(PL_PTMAX / 8)));
    int occ = 0;
    MP_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kTile[tk], (int)P.threads, P.pt / 8));
    const u32 ntile = 8 * P.nb;
    P.grid = (u32)std::min<u64>(ntile, (u64)h->sm_count * (u32)std::max(occ, 1));
    P.nmod = P.it1 - P.iw0 >= PL_IMOD_MIN ? P.it1 - P.iw0 : 0;
    P.psize = ((size_t)ntile * (P.pt / 32) + 64) * 4;
    P.tsize = ((size_t)P.grid * (P.it1 - P.iw1) + P.nmod) * 4 + 64;
    P.rsize = P.cap ? (size_t)ntile * P.cap * 4 : 0;
    return MP_OK;
}

// most: the bytes that a wave's buffers may take (one stretch at the least)
static int plan_planes(mp_handle *h, const PrimeTable &tb, const SieveGeom &g, u64 most, PlanePlan &P)
{
    const u64 S = 2ull << g.tlog, top = g.base + 2 * g.nbx;
    const u64 sq = mp_isqrt64(top - 1) + 1;
    const u64 total = 2 * g.nbx / 30 + 4;
    const u32 group = (u32)std::max(1, h->sm_count / 4);                  // 8 planes x 37 blocks = 2 x 148 tiles
    u64 blocks = (total + PL_PTMAX - 1) / PL_PTMAX;
    u64 waves = (blocks + 4 * group - 1) / (4 * group);
    for (;; waves++) {
        P.tw = (u32)((g.ntiles + waves - 1) / waves);
        P.waves = (g.ntiles + P.tw - 1) / P.tw;
        P.ni = std::min<u64>(P.tw * S, 2 * g.nbx) / 30 + 4;
        if (P.ni >= (1ull << 31)) continue;
        // tiles in whole rounds over the SMs, of at least PL_PTMIN bits
        const u64 ptmin = 4096;
        u64 nb = (P.ni + PL_PTMAX - 1) / PL_PTMAX;
        if (P.ni >= ptmin * group) nb = (nb + group - 1) / group * group;
        else nb = std::max<u64>(nb, P.ni / ptmin);
        P.pt = (u32)(((P.ni + nb - 1) / nb + 1023) & ~1023ull);
        if (P.pt < 2048) P.pt = 2048;
        if (nb > 4 * group && P.tw > 1) continue;
        P.nb = (u32)((P.ni + P.pt - 1) / P.pt);
        P.threads = P.pt >= (1u << 19) ? 1024 : P.pt >= (1u << 17) ? 512 : 256;
        // tiers: a prime has pt / q multiples in a tile.  The buckets start at 1.5 pt: a visit of a prime
        // that often misses costs a thread less than its hits cost the scatter ([1e15, +2^34): 1.0 pt 7.60,
        // 1.25 pt 7.57, 1.5 pt 7.52, 1.75 pt 7.61, 2 pt 7.66 ms a call)
        P.iend = (u32)tb.count_le(sq);
        P.iw0 = (u32)std::min<u64>(tb.count_le(89), P.iend);
        P.iw1 = std::max(P.iw0, (u32)std::min<u64>(tb.count_le(std::min<u32>(8192, P.pt / 64)), P.iend));
        P.it1 = std::max(P.iw1, (u32)std::min<u64>(tb.count_le((u64)P.pt * 3 / 2), P.iend));
        // a few primes more a thread than a launch of their own
        if (P.iend - P.it1 <= 16 * P.threads) P.it1 = P.iend;
        P.cap = 0;
        if (P.iend > P.it1) {
            P.cap = plane_bucket_cap(P.pt, tb.inv_prefix[P.iend] - tb.inv_prefix[P.it1], g.base / 30, tb.host[P.iend - 1]);
            // records of a wave within 3 GB
            if ((u64)P.cap * 8 * P.nb * 4 > (3072ull << 20) && P.tw > 1) continue;
        }
        if (P.it1 && ((u64)tb.host[P.it1 - 1] + (u64)P.nb * P.pt >> 32 || 3ull * tb.host[P.it1 - 1] >> 32)) {
            if (P.tw > 1) continue;
            return mp_set_error(h, MP_ERANGE, "a plane's wave is too long for 32-bit remainders");
        }
        MP_TRY(plan_sizes(h, P));
        if (P.psize + P.tsize + P.rsize > most && P.tw > 1) continue;
        return MP_OK;
    }
}

int mp_planes_shape(mp_handle *h, const PrimeTable &tb, const SieveGeom &g, u32 *tile_bits, u32 *bucket_above)
{
    PlanePlan P;
    MP_TRY(plan_planes(h, tb, g, h->planes_max, P));
    *tile_bits = P.pt;
    *bucket_above = P.it1 ? tb.host[P.it1 - 1] : 0;
    return MP_OK;
}

int mp_planes_bytes(mp_handle *h, const PrimeTable &tb, const SieveGeom &g, u64 *bytes)
{
    PlanePlan P;
    MP_TRY(plan_planes(h, tb, g, ~0ull, P));
    *bytes = P.psize + P.tsize + P.rsize;
    return MP_OK;
}

int mp_planes_run(mp_handle *h, const PrimeTable &tb, const SieveGeom &g, TileSum *sums, u32 *bitmap32, u64 *emit,
                  u64 emit_cap, u64 *emit_total, cudaStream_t st)
{
    static std::atomic<bool> scat_done[2][16];
    PlanePlan P;
    int smem_max = 0;
    MP_CUDA(h, cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device));
    // The buffers follow the range's length and, a little, its height; a growth frees the old one, which
    // waits for the device ([1e12 + x, +2^30) for growing x: 1.1 ms instead of 0.27).  So they grow with
    // something to spare; a third for the threads' state, which is largest below the longest waves
    // (tiles of less than half an SM's shared memory run two to an SM).  Where the device has no room, they do
    // without, and then with shorter waves (2^32 integers at 9e17 take 1.9 GB in one wave)
    for (bool lean = false;;) {
        MP_TRY(plan_planes(h, tb, g, h->planes_max, P));
        const size_t spare = lean ? 0 : 32u << 20;
        cudaError_t e = h->planes.ensure(P.psize, lean ? 0 : P.psize / 16 + spare);
        if (e == cudaSuccess) e = h->tstate.ensure(P.tsize, lean ? 0 : P.tsize / 3 + spare / 4);
        if (e == cudaSuccess && P.cap) e = h->rec.ensure(P.rsize, lean ? 0 : P.rsize / 16 + spare);
        if (e == cudaSuccess && P.cap) e = h->reccnt.ensure(((size_t)8 * P.nb + 1) * 4, 16384);
        if (e == cudaSuccess) break;
        if (e != cudaErrorMemoryAllocation || (lean && P.tw == 1)) MP_CUDA(h, e);
        if (lean) h->planes_max = (P.psize + P.tsize + P.rsize) / 2;
        lean = true;
        h->planes.release();
        h->tstate.release();
        h->rec.release();
    }
    const int tk = tile_form(P.threads);
    const u32 ntile = 8 * P.nb, nw = P.pt / 32, grid = P.grid, nmod = P.nmod;
    const size_t tsm = P.pt / 8;
    const bool large = P.iend > P.it1;
    PlaneTileArgs a;
    memset(&a, 0, sizeof a);
    a.nb = P.nb; a.pt = P.pt; a.ntile = ntile;
    a.q = tb.q.as<u32>(); a.magic = tb.magic.as<u64>();
    a.iw0 = P.iw0; a.iw1 = P.iw1; a.it1 = P.it1;
    for (int p = 0; p < PL_NPAT; p++) {
        // pattern bit j: 2 j + 1 has a factor of the group (product M).  30 i + r has one exactly when
        // 2 j + 1 has, for j = i + r / 30 + (M - 1) / 2 (mod M)
        const u64 M = p ? h->pat.period[p] : h->pat.period7;
        u64 y = 0;
        while ((1 + M * y) % 30) y++;
        const u64 z = (1 + M * y) / 30;                                    // 1 / 30 mod M
        a.pat[p] = p ? h->pat.d_words[p] : h->pat.d_words7;
        a.period[p] = (u32)M;
        for (u32 k = 0; k < 8; k++) a.zoff[p][k] = (u32)((pl_res(k) * z + (M - 1) / 2) % M);
    }
    a.cap = P.cap;
    a.planes = h->planes.as<u32>();
    a.tstate = h->tstate.as<u32>() + nmod;
    a.imod = nmod ? h->tstate.as<u32>() : nullptr;
    PlaneScanArgs c;
    memset(&c, 0, sizeof c);
    c.g = g;
    c.planes = a.planes;
    c.pstride = P.nb * nw;
    c.sums = sums;
    c.bitmap32 = bitmap32;
    c.emit = emit;
    c.emit_cap = emit_cap;
    u64 *off = nullptr;
    if (emit_total) {
        MP_CUDA(h, h->emit_off.ensure((size_t)g.ntiles * 8 + 64, 65536));
        off = h->emit_off.as<u64>();
        c.emit_off = off;
        MP_CUDA(h, cudaMemsetAsync(emit_total, 0, 8, st));
    }
    const u64 S = 2ull << g.tlog;
    for (u32 w = 0; w < P.waves; w++) {
        const u32 t0 = w * P.tw, nt = std::min(P.tw, g.ntiles - t0);
        const u64 lo = g.base + t0 * S, hi = std::min(lo + nt * S, g.base + 2 * g.nbx);
        a.i0 = c.i0 = lo / 30;
        if (large) {
            PlaneScatterArgs s;
            s.i0 = a.i0;
            s.ni = (u32)std::min<u64>((hi - 1) / 30 - a.i0 + 3, (u64)P.nb * P.pt);
            s.nb = P.nb; s.pt = P.pt;
            s.blk_magic = (u32)((1ull << 32) / (P.pt >> 10)) + 1;
            s.q = a.q; s.magic = a.magic;
            s.k0 = P.it1; s.k1 = P.iend;
            const u32 nblk = (u32)h->sm_count * PS_CTAS_PER_SM;
            // runs of 32 primes where they take several rounds, then up to 512, so that the queue is no
            // bottleneck and no warp is left with a long run (measured: runs of 512 throughout, 6.4 ms
            // instead of 2.2 at 9e17, where a few warps held the smallest primes)
            const bool far = tb.host[s.k1 - 1] / 32 > s.ni;                  // most primes have no hit
            const u64 many = far ? 4ull * s.ni : s.ni / 4;                   // several rounds to here
            s.kc = s.k0 + (std::min(s.k1, std::max(s.k0, (u32)tb.count_le(many))) - s.k0 & ~31u);
            const u32 each = (s.k1 - s.kc) / (nblk * (PS_THREADS / 32));      // primes a warp
            s.run = std::max(32u, std::min(512u, (far ? each / 2 : each / 8) & ~31u));
            // with fewer of the former than eight per warp, each covers a part of the wave only, of four
            // rounds or more: a wave of a small range waited for one warp's rounds
            const u32 fine = (s.kc - s.k0) >> 5, rounds = s.ni / (P.pt + P.pt / 2) + 1;
            s.parts = fine ? std::max(1u, std::min(8 * nblk * (PS_THREADS / 32) / fine, rounds / 4)) : 1u;
            s.part = (s.ni + s.parts - 1) / s.parts;
            s.rec = h->rec.as<u32>(); s.cnt = h->reccnt.as<u32>(); s.cap = P.cap;
            s.queue = s.cnt + ntile;
            s.err = h->errflag.as<u32>();
            a.rec = s.rec;
            a.cnt = s.cnt;
            MP_CUDA(h, cudaMemsetAsync(s.cnt, 0, ((size_t)ntile + 1) * 4, st));
            const size_t ssm = ((size_t)2 * PS_STAGE + 2 * ntile) * 4;
            // the form for small waves: parts, or primes so far apart that most have no multiple in the wave
            const int sk = s.parts > 1 || far;
            static void (*const scat[2])(PlaneScatterArgs) = {plane_scatter_kernel<false>, plane_scatter_kernel<true>};
            MP_CUDA(h, raise_smem(scat[sk], scat_done[sk], h->device, smem_max - 4096));
            ProfScope ps(h, PROF_SCATTER, st);
            // a unit per CTA before a second one in any: a round's barriers are what a small wave waits for
            const u32 units = fine * s.parts + (s.k1 - s.kc + s.run - 1) / s.run;
            scat[sk]<<<std::min(nblk, units), PS_THREADS, ssm, st>>>(s);
            MP_CUDA(h, cudaGetLastError());
        }
        if (nmod) {
            plane_imod_kernel<<<(nmod + 255) / 256, 256, 0, st>>>(a.q + P.iw0, a.magic + P.iw0, nmod, a.i0,
                                                                  h->tstate.as<u32>());
            MP_CUDA(h, cudaGetLastError());
        }
        {
            ProfScope ps(h, PROF_TILE, st);
            kTile[tk]<<<grid, P.threads, tsm, st>>>(a);
        }
        MP_CUDA(h, cudaGetLastError());
        c.t0 = t0;
        c.nt = nt;
        ProfScope ps(h, PROF_FOLD, st);
        // two warps a stretch of 2^19 bits and more: a warp's first row and its summary cost several rows
        // (at 2^20 bits 0.86 ms of scans a 2^34 integers, eight warps 0.96)
        const u32 sth = g.tlog >= 19 ? 64 : 32 * SCAN_WARPS;
        if (bitmap32) plane_scan_kernel<true><<<nt, sth, 0, st>>>(c);
        else plane_scan_kernel<false><<<nt, sth, 0, st>>>(c);
        MP_CUDA(h, cudaGetLastError());
        if (emit_total) {
            plane_offsets_kernel<<<1, 1024, 0, st>>>(sums, t0, nt, off, emit_total);
            if (emit) {
                static std::atomic<bool> emit_done[16];
                MP_CUDA(h, raise_smem(plane_emit_kernel, emit_done, h->device, EMIT_WARPS * EMIT_ROW * 2));
                plane_emit_kernel<<<nt, 32 * EMIT_WARPS, EMIT_WARPS * EMIT_ROW * 2, st>>>(c);
            }
            MP_CUDA(h, cudaGetLastError());
        }
    }
    return MP_OK;
}
