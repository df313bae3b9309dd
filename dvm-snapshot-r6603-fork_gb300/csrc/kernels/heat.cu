// Explicit 2-D heat step with SUM and MINLOC reductions, FP64, for sm_103a:
// the loop of dvm-snapshot-r6603-fork_gb300/workloads/heat.c
//   dst[i][j] = src[i][j] + c * (src[i-1][j] + src[i+1][j] + src[i][j-1] + src[i][j+1] - 4.0 * src[i][j])
//   sum += dst[i][j];  if (dst[i][j] < mn) { mn = dst[i][j]; loc = {i, j}; }
//
// A warp walks a strip: up to DVMHGB_HEAT_ROWS(variant) consecutive rows of one
// 64-wide chunk of j aligned to a multiple of 64 of the array index (lane l
// holds j = base+2l, base+2l+1 as one 128-bit access).  Rows i-1, i, i+1 roll
// through registers with row i+2 in flight, so every source row is read once
// per chunk; lanes 0 and 31 also fetch the chunk's edge columns.
//
// The sum of the four neighbours runs on the FP32 pipe (fixlimb.cuh): a row is
// split into limbs once, when it arrives, its left and right neighbours come by
// shuffles of the limbs.  S - 4 src, exact in the limbs' unit, is rounded once
// from a 63-bit integer, as the source's two operations round it (4 src is exact).
// The product with c and the last addition are two operations on the FP64 unit.
// The limbs' range of nine binades follows the values of the warp's rows; a row
// that does not fit it is computed on the FP64 unit from memory.
//
// Per row the warp writes one SUM item -- the pairwise tree over the chunk's 64
// positions (pair sum, then the lanes by 1, 2, 4, 8, 16), the canonical order
// the reduction engine folds -- and one MINLOC item: the smallest value, ties to
// the smallest j, i.e. the first in loop order, as the strict '<' of the source
// gives.  The pair sums of 8 rows wait in shared memory; then four lanes take a
// row each and walk its tree in registers: 9 FP64 instructions per 8 rows,
// where a butterfly per row takes 40.  Items are in row-major (row, chunk) order.
//
// What bounds it: about 320 instructions per row of a strip at half the issue
// rate (16 warps an SM, for 128 registers a thread), and beside them 6.1
// operations on the FP64 unit, 76 cycles each for a warp.  The kernel that took
// the sums and the tree's pair on the FP64 unit (13 operations a row) and the
// rest of the trees as butterflies on the integer pipe: 3171 us for 256 plates of
// 64..2048 (159 M cells, 380 us of HBM traffic at the copy rate), 124 us for 24
// of 64..512.  Now 1240 and 25.  On the way: limbs for the four neighbours 1620;
// S - 4 src on the integer pipe too 1577; the next row's loads no longer waited
// for in the step that issues them 1240.
//
// The same strip code serves one array (plain per-loop launches) and a table
// of arrays of uneven sizes (batched mode): there the strips of all arrays
// form one index space that a persistent grid strides over (strip bases
// cached in shared memory), so small and large arrays share the GPU in a
// single launch.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../../include/dvmh_gb.h"
#include "../../../include/dvmh_gb_kernels.h"
#include "devinfo.cuh"
#include "rowlimb.cuh"

namespace {

constexpr int HT = 256;  // threads per CTA (8 warps)

__device__ __forceinline__ uint64_t minKey(double v) {
    // IEEE order as unsigned order; -0 keyed as +0 (they compare equal); NaN last
    uint64_t b = (uint64_t)__double_as_longlong(v);
    if ((b & 0x7FFFFFFFFFFFFFFFull) == 0) b = 0;
    if ((b & 0x7FFFFFFFFFFFFFFFull) > 0x7FF0000000000000ull) return ~0ull;
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}

constexpr int MAX_CACHED = 2048;  // strip bases cached in shared memory

constexpr int RB = 8;               // rows whose pair sums wait for their trees, 4 lanes a row
constexpr int RS = 36;              // stride of such a row: lane l at l + l / 8, read without bank conflicts
using fx::f32x2;

// strip `local` of loop d: chunk local / nrb, rows (local % nrb) * sr ...; sums: RB * RS doubles of the warp's own
__device__ __forceinline__ void heatStrip(const dvmhgb_heat_desc &d, long local, double *sums) {
    const int lane = threadIdx.x & 31;
    const long nrows = d.hi0 - d.lo0 + 1;
    const long sr = d.sr;
    const unsigned nrb = (unsigned)((nrows + sr - 1) / sr);
    const unsigned ch = (unsigned)local / nrb, rb = (unsigned)local - ch * nrb;
    const long r0 = (long)rb * sr;
    int left = (int)((r0 + sr < nrows ? r0 + sr : nrows) - r0);  // rows to do
    const long base = (d.c0 + ch) * 64;
    const long j = base + 2 * lane;
    const long last = d.hi1 + 1;  // the last column a cell of the loop reads
    const bool in0 = j >= d.lo1 && j <= d.hi1, in1 = j + 1 >= d.lo1 && j + 1 <= d.hi1;
    // edge columns: lane 0 the left neighbour of j = base, lane 31 the right one of base + 63.  Elements that no cell of
    // the loop needs are replaced by others of the row, so that they do not leave the limbs' range.
    const int jo = j <= last ? 0 : (int)((last & ~1L) - j);                 // the pair's offset from j
    const bool needY = j + jo + 1 <= last;                                  // its second element (else the row's padding)
    const int eo = lane == 0 ? (j >= 1 ? -1 : 0) : (lane == 31 && j + 2 <= last ? 2 : jo);
    const double c = __ldg(d.coef);
    const long s0 = d.s0;
    const int nck = (int)d.nck;
    const double *p = d.src + (d.lo0 + r0 - 1) * s0 + j;  // the pair of row i-1 (+ jo)
    const long toOut = d.dst - d.src + s0;                // from there to row i of dst
    int item = (int)(r0 * nck + ch);                      // (a loop's items are fewer than 2^31)
    int row = (int)(d.lo0 + r0);  // i
    double *const sumItems = d.sumItems, *const minItems = d.minItems;
    int *const locItems = d.locItems;
    int E = fx::E_DEFAULT;
    auto load = [&](const double *q, rows::Row &r) {
        r.d = rows::ldGlobal2(q + jo);
        r.e = rows::ldGlobal(q + eo);
    };
    auto split = [&](rows::Row &r) {
        if (!needY) r.d.y = r.d.x;  // (not at the load: it would be waited for there)
        rows::split(r, E);
    };
    rows::Row ra, rc, rd;
    load(p, ra);
    load(p + s0, rc);
    load(p + 2 * s0, rd);
    split(ra);
    split(rc);
    split(rd);
    int rr = 0;  // rows in the batch

    // row i from up, mid, dn; up then takes row i + 2's place
    auto step = [&](rows::Row &up, rows::Row &mid, rows::Row &dn) -> bool {
        rows::Row nx;
        const bool more = left > 1;
        if (more) load(p + 3 * s0, nx);
        if (__builtin_expect(!(up.ok && mid.ok && dn.ok), 0)) {
            const int e = rows::rangeOf(up, mid, dn, E);
            if (e != E) {  // move the range
                E = e;
                load(p, up);
                load(p + s0, mid);
                load(p + 2 * s0, dn);
                split(up);
                split(mid);
                split(dn);
            }
        }
        double v0, v1;
        if (__builtin_expect(up.ok && mid.ok && dn.ok, 1)) {
            fx::Limbs<f32x2> lt, rt;
            rows::sides(mid.v.h, mid.eh, lane, lt.h, rt.h);
            rows::sides(mid.v.m, mid.em, lane, lt.m, rt.m);
            rows::sides(mid.v.l, mid.el, lane, lt.l, rt.l);
            // ((src[i-1] + src[i+1]) + src[j-1]) + src[j+1]
            const fx::Limbs<f32x2> s = fx::add(fx::add(fx::add(up.v, dn.v), lt), rt);
            // S - 4 src as an integer of the limbs' unit, rounded once
            const f32x2 m4 = fx::pack(-4.0f, -4.0f), sc = fx::pack(0x1p-11f, 0x1p-11f);
            const f32x2 th = fx::vmul(fx::vfma(mid.v.h, m4, s.h), sc), tm = fx::vfma(mid.v.m, m4, s.m);
            const f32x2 tl = fx::vfma(mid.v.l, m4, s.l);
            const int64_t tx = ((int64_t)__float2int_rz(fx::lo(th)) << 40) + ((int64_t)__float2int_rz(fx::lo(tm)) << 20) +
                               (int64_t)__float2int_rz(fx::lo(tl));
            const int64_t ty = ((int64_t)__float2int_rz(fx::hi(th)) << 40) + ((int64_t)__float2int_rz(fx::hi(tm)) << 20) +
                               (int64_t)__float2int_rz(fx::hi(tl));
            v0 = mid.d.x + c * fx::round63(tx, E);
            v1 = mid.d.y + c * fx::round63(ty, E);
        } else {
            const double *q = p;  // row i-1
            v0 = v1 = 0.0;
            if (in0) v0 = q[s0] + c * ((((q[0] + q[2 * s0]) + q[s0 - 1]) + q[s0 + 1]) - 4.0 * q[s0]);
            if (in1) v1 = q[s0 + 1] + c * ((((q[1] + q[2 * s0 + 1]) + q[s0]) + q[s0 + 2]) - 4.0 * q[s0 + 1]);
        }
        double *out = const_cast<double *>(p) + toOut;
        if (in0 && in1) rows::stGlobal(out, make_double2(v0, v1));
        else if (in0) rows::stGlobal(out, v0);
        else if (in1) rows::stGlobal(out + 1, v1);
        // SUM: -0.0 outside the loop
        sums[rr * RS + lane + (lane >> 3)] = (in0 ? v0 : -0.0) + (in1 ? v1 : -0.0);
        // MINLOC: the smallest value's first cell.  Non-negative values below infinity are ordered as their bits are;
        // other rows go by minKey.  The lane that holds the minimum writes the item.
        {
            uint32_t h0 = in0 ? sf::hi32(sf::bits(v0)) : 0x7FF00000u, h1 = in1 ? sf::hi32(sf::bits(v1)) : 0x7FF00000u;
            uint32_t l0 = (uint32_t)sf::bits(v0), l1 = (uint32_t)sf::bits(v1);
            bool none = false;  // no cell below infinity
            if (__builtin_expect(__any_sync(0xffffffffu, max(h0, h1) > 0x7FF00000u || (in0 && h0 == 0x7FF00000u) ||
                                                             (in1 && h1 == 0x7FF00000u)), 0)) {
                const uint64_t k0 = in0 ? minKey(v0) : ~0ull, k1 = in1 ? minKey(v1) : ~0ull;
                h0 = sf::hi32(k0), l0 = (uint32_t)k0, h1 = sf::hi32(k1), l1 = (uint32_t)k1;
                none = __all_sync(0xffffffffu, (k0 & k1) == ~0ull);
            }
            const bool second = h1 < h0 || (h1 == h0 && l1 < l0);
            const uint32_t h = second ? h1 : h0, l = second ? l1 : l0, mh = __reduce_min_sync(0xffffffffu, h);
            unsigned who = __ballot_sync(0xffffffffu, h == mh);
            if (who & (who - 1)) {  // equal high words
                const uint32_t ml = __reduce_min_sync(0xffffffffu, h == mh ? l : ~0u);
                who = __ballot_sync(0xffffffffu, h == mh && l == ml);
            }
            if (lane == __ffs(who) - 1) {
                rows::stGlobal(minItems + item, none ? __builtin_huge_val() : second ? v1 : v0);
                rows::stGlobal(locItems + 2 * (long)item, row);
                rows::stGlobal(locItems + 2 * (long)item + 1, (int)j + (second ? 1 : 0));
            }
        }
        if (++rr == RB || !more) {
            __syncwarp();
            double x[RB];
            const double *q = sums + (lane >> 2) * RS + (lane & 3) * 9;
#pragma unroll
            for (int i = 0; i < 8; i++) x[i] = q[i];
#pragma unroll
            for (int w = 1; w < 8; w <<= 1)
#pragma unroll
                for (int i = 0; i < 8; i += 2 * w) x[i] = x[i] + x[i + w];
            double total = x[0] + __shfl_xor_sync(0xffffffffu, x[0], 1);
            total = total + __shfl_xor_sync(0xffffffffu, total, 2);
            if ((lane & 3) == 0 && (lane >> 2) < rr) rows::stGlobal(sumItems + item + ((lane >> 2) + 1 - rr) * nck, total);
            __syncwarp();
            rr = 0;
        }
        if (!more) return false;
        up = nx;
        split(up);
        p += s0;
        item += nck;
        row++;
        left--;
        return true;
    };
    // three rows a trip, so that the limbs stay where they are
    while (step(ra, rc, rd) && step(rc, rd, ra) && step(rd, ra, rc)) {
    }
}

constexpr int HB = 2;  // CTAs per SM

__global__ void __launch_bounds__(HT, HB) kHeatOne(dvmhgb_heat_desc d) {
    __shared__ double sums[HT / 32][RB * RS];
    for (long s = (blockIdx.x * (long)HT + threadIdx.x) >> 5; s < d.strips; s += (long)gridDim.x * (HT / 32))
        heatStrip(d, s, sums[threadIdx.x >> 5]);
}

// strips of array k are [d[k].stripBase, d[k].stripBase + d[k].strips)
__global__ void __launch_bounds__(HT, HB) kHeatMany(const dvmhgb_heat_desc *__restrict__ ds, int n, long total) {
    __shared__ int sb[MAX_CACHED];
    __shared__ double sums[HT / 32][RB * RS];
    const bool cached = n <= MAX_CACHED && total < (1L << 31);
    if (cached)
        for (int q = threadIdx.x; q < n; q += HT) sb[q] = (int)ds[q].stripBase;
    __syncthreads();
    for (long s = (blockIdx.x * (long)HT + threadIdx.x) >> 5; s < total; s += (long)gridDim.x * (HT / 32)) {
        int lo = 0, hi = n - 1;  // last array whose stripBase <= s
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if ((cached ? sb[mid] : ds[mid].stripBase) <= s) lo = mid;
            else hi = mid - 1;
        }
        heatStrip(ds[lo], s - (cached ? sb[lo] : ds[lo].stripBase), sums[threadIdx.x >> 5]);
    }
}

long residentWarps() { return (long)gbdev::smCount() * HB * (HT / 32); }

// strips of sr rows over a loop
long stripsOf(const dvmhgb_heat_desc &d, long sr) { return d.nck * ((d.hi0 - d.lo0 + sr) / sr); }

// What `strips` strips of sr rows cost, in rows of one warp: each begins with three rows loaded and split before its
// first result, and the warps the GPU holds take them in rounds.  Measured, us: 256 plates of 64..2048 (159 M cells)
// 1283 / 1241 / 1240 / 1282 at 16 / 32 / 64 / 128 rows; 24 of 64..512 27.7 / 24.8 / 34.9 / 61.7 at 8 / 16 / 32 / 64;
// 60 of 16..256 14.6 / 20.1 / 33.5 at 8 / 16 / 32.
long stripCost(long strips, long sr) { return (strips + residentWarps() - 1) / residentWarps() * (2 * sr + 5); }

}  // namespace

extern "C" {

int dvmhgb_heat_desc_fill(dvmhgb_heat_desc *d, const double *src, double *dst, long rowStride, const long lo[2],
                          const long hi[2], const double *coefDev) {
    // 128-bit accesses: even row stride and 16-byte aligned bases
    if (!d || hi[0] < lo[0] || hi[1] < lo[1] || lo[0] < 1 || lo[1] < 1 || (rowStride & 1) ||
        ((uintptr_t)src & 15) || ((uintptr_t)dst & 15))
        return -1;
    d->src = src;
    d->dst = dst;
    d->s0 = rowStride;
    d->lo0 = lo[0];
    d->hi0 = hi[0];
    d->lo1 = lo[1];
    d->hi1 = hi[1];
    d->coef = coefDev;
    d->c0 = lo[1] / 64;
    d->nck = hi[1] / 64 - d->c0 + 1;
    d->units = (hi[0] - lo[0] + 1) * d->nck;
    d->unitBase = 0;
    d->sr = DVMHGB_HEAT_STRIP;
    d->strips = d->nck * ((hi[0] - lo[0] + d->sr) / d->sr);
    d->stripBase = 0;
    if (d->units >= (1L << 31) || d->strips >= (1L << 31)) return -1;
    d->sumItems = d->minItems = nullptr;
    d->locItems = nullptr;
    return 0;
}

int dvmhgb_heat(const dvmhgb_heat_desc *d, void *stream) {
    if (!d || !d->sumItems || !d->minItems || !d->locItems) return -1;
    dvmhgb_heat_desc e = *d;
    for (long sr = e.sr = 1; sr <= DVMHGB_HEAT_STRIP; sr *= 2)
        if (stripCost(stripsOf(*d, sr), sr) <= stripCost(stripsOf(*d, e.sr), e.sr)) e.sr = sr;
    e.strips = stripsOf(e, e.sr);
    long blocks = (e.strips + HT / 32 - 1) / (HT / 32);
    if (blocks > (long)gbdev::smCount() * HB) blocks = (long)gbdev::smCount() * HB;
    kHeatOne<<<(unsigned)blocks, HT, 0, (cudaStream_t)stream>>>(e);
    dvmhgb_count_launches(1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int dvmhgb_heat_desc_rows(dvmhgb_heat_desc *d, long sr) {
    if (!d || sr < 1) return -1;
    d->sr = sr;
    d->strips = stripsOf(*d, sr);
    return d->strips < (1L << 31) ? 0 : -1;
}

int dvmhgb_heat_default_variant(const dvmhgb_heat_desc *d, int n) {
    if (!d || n < 1) return -1;
    int best = -1;
    long bestCost = 0;
    for (int v = 0; v < DVMHGB_HEAT_VARIANTS; v++) {
        if (DVMHGB_HEAT_CTAS(v) != HB) continue;
        const long sr = DVMHGB_HEAT_ROWS(v);
        long strips = 0;
        for (int q = 0; q < n; q++) strips += stripsOf(d[q], sr);
        const long cost = stripCost(strips, sr);
        if (best < 0 || cost < bestCost) best = v, bestCost = cost;
    }
    return best;
}

int dvmhgb_heat_many_grid(const dvmhgb_heat_desc *dDev, int n, long totalStrips, int ctasPerSm, void *stream) {
    if (!dDev || n < 1 || totalStrips < 1 || ctasPerSm < 1 || ctasPerSm > 8) return -1;
    long blocks = (totalStrips + HT / 32 - 1) / (HT / 32);
    if (ctasPerSm > HB) ctasPerSm = HB;  // more would wait for the resident ones' whole walk
    if (blocks > (long)gbdev::smCount() * ctasPerSm) blocks = (long)gbdev::smCount() * ctasPerSm;
    kHeatMany<<<(unsigned)blocks, HT, 0, (cudaStream_t)stream>>>(dDev, n, totalStrips);
    dvmhgb_count_launches(1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int dvmhgb_heat_many(const dvmhgb_heat_desc *dDev, int n, long totalStrips, void *stream) {
    return dvmhgb_heat_many_grid(dDev, n, totalStrips, 8, stream);
}

}  // extern "C"
