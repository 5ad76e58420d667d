// mp_sieve.cuh -- what the two tile forms of the sieve share: the geometry of a range in the
// odd-only map, the summary of a stretch of it, and the in-order join of summaries.
//   mp_sieve.cu   odd-only tiles (the plain per-segment form, pinned geometries, the prime table)
//   mp_planes.cu  residue planes mod 30 (the batched default)
#pragma once
#include "mp_common.cuh"

struct TileSum {
    u64 first, last;   // first / last prime bit in the tile (bits < nbx); MP_NONE if none
    u64 lastin;        // last prime bit below limit; MP_NONE if none
    u64 mgs;           // bit of the prime starting the widest internal gap; MP_NONE if none
    u64 cks;           // sum of mix64(p) over the 6-tuple starts p (bits < limit)
    u32 mg;            // widest internal gap in bits (pairs whose first prime is in range)
    u32 count;         // primes with bit < limit
    u32 twins, tuples;
};

struct SieveGeom {
    u64 base, limit, nbx;   // base even; bits [0, limit) in range; bits [0, nbx) sieved
    u32 tlog, ntiles;
};

// ---------------------------------------------------------------------------------------
// ordered combine of tile / thread summaries
// ---------------------------------------------------------------------------------------

struct Part {
    u64 first, last, lastin, mgs, cks;
    u32 mg, count, twins, tuples;
};

__device__ __forceinline__ void part_init(Part &p)
{
    p.first = p.last = p.lastin = p.mgs = MP_NONE;
    p.cks = 0;
    p.mg = p.count = p.twins = p.tuples = 0;
}

// L followed by R (R's bits all above L's); gaps compare strictly so the earliest start wins
__device__ __forceinline__ Part part_join(const Part &L, const Part &R, u64 limit)
{
    Part o;
    o.count = L.count + R.count;
    o.twins = L.twins + R.twins;
    o.tuples = L.tuples + R.tuples;
    o.cks = L.cks + R.cks;
    o.mg = L.mg;
    o.mgs = L.mgs;
    if (L.first == MP_NONE) {
        o.first = R.first; o.last = R.last; o.lastin = R.lastin; o.mg = R.mg; o.mgs = R.mgs;
        return o;
    }
    o.first = L.first;
    if (R.first == MP_NONE) { o.last = L.last; o.lastin = L.lastin; return o; }
    o.last = R.last;
    o.lastin = R.lastin != MP_NONE ? R.lastin : L.lastin;
    if (L.last < limit) {
        const u32 g = (u32)(R.first - L.last);
        if (g > o.mg) { o.mg = g; o.mgs = L.last; }
    }
    if (R.mg > o.mg) { o.mg = R.mg; o.mgs = R.mgs; }
    return o;
}

__device__ __forceinline__ Part part_shfl_down(const Part &p, int d)
{
    Part o;
    o.first = __shfl_down_sync(0xffffffffu, p.first, d);
    o.last = __shfl_down_sync(0xffffffffu, p.last, d);
    o.lastin = __shfl_down_sync(0xffffffffu, p.lastin, d);
    o.mgs = __shfl_down_sync(0xffffffffu, p.mgs, d);
    o.cks = __shfl_down_sync(0xffffffffu, p.cks, d);
    o.mg = __shfl_down_sync(0xffffffffu, p.mg, d);
    o.count = __shfl_down_sync(0xffffffffu, p.count, d);
    o.twins = __shfl_down_sync(0xffffffffu, p.twins, d);
    o.tuples = __shfl_down_sync(0xffffffffu, p.tuples, d);
    return o;
}

// in-order reduction over the lanes of a warp; lane 0 holds the result
__device__ __forceinline__ Part part_warp_reduce(Part p, u64 limit)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        Part r = part_shfl_down(p, d);
        if ((lane & (2 * d - 1)) == 0) p = part_join(p, r, limit);
    }
    return p;
}

__device__ __forceinline__ u32 bits_mask(u64 start, u64 bound)
{
    // bits start .. start+31 below bound
    if (start >= bound) return 0;
    const u64 n = bound - start;
    return n >= 32 ? 0xffffffffu : ((1u << n) - 1);
}

// the sieve of [g.base, g.base + 2 g.nbx) in residue planes mod 30 (mp_planes.cu): summaries of
// the stretches of 2^g.tlog bits to `sums`, and, where asked for, the in-range bits of the odd-only
// map to `bitmap32`, or the in-range primes in order to `emit` (at most emit_cap of them; their
// number goes to *emit_total, a device word, as always)
int mp_planes_run(mp_handle *h, const PrimeTable &tb, const SieveGeom &g, TileSum *sums, u32 *bitmap32, u64 *emit,
                  u64 emit_cap, u64 *emit_total, cudaStream_t st);

// the stretches of a range in that form; and the tile of a plane in bits, with the bound above which
// its primes go through the bucket scatter
int mp_planes_geom(mp_handle *h, u64 lo, u64 hi, u32 block_log2, SieveGeom &g);
int mp_planes_shape(mp_handle *h, const PrimeTable &tb, const SieveGeom &g, u32 *tile_bits, u32 *bucket_above);
// bytes of the buffers of a wave of that form, without what they may have to spare
int mp_planes_bytes(mp_handle *h, const PrimeTable &tb, const SieveGeom &g, u64 *bytes);
