// The 2-D Jacobi loops with the sums on FP32 limbs (fixlimb.cuh).  FUSED = false:
// Out = (4 neighbours of A) / 4 over the box.  FUSED = true: the update loop
// eps = Max(|B - A|, eps); A = B and then Out = (4 neighbours of A_new) / 4, A_new
// = B inside the box and A outside it; Out also gets B's values beside the box in
// the box's rows and, with `rowsToo`, in the rows above and below it.  Included by
// jacobi.cu inside its anonymous namespace (Box2, ctaMax come from there).
//
// A warp walks a strip: `sr` consecutive rows of one 64-wide chunk of columns, as
// the heat kernel does (rowlimb.cuh).  Rows i-1, i, i+1 are in registers as limbs,
// the next seven on their way to shared memory; the left and right neighbours come
// by shuffles.  The range of the limbs follows the values of the warp's rows; a row
// that does not fit it is computed on the FP64 unit; after a move in vain the next
// 32 such rows are not tried (values of 24 decades at 4097^2, a move in every row:
// stencil 172 us, fused 341; with every sum on the FP64 unit 169 and 259; now 138 and
// 245).
// |B - A| is taken on the FP64 unit, which is otherwise idle: one operation a cell,
// used a row later.
//
// What bounds it: instruction issue, about 200 (FUSED 330) a row of a chunk, at 16
// warps an SM.  With one row in flight in registers in place of the ring the
// stencil took 128 us at 4097^2 (8 KB in flight per SM), with it 67; all additions
// on the FP64 unit, 76 cycles each for a warp, 166 (the older variants).  Fused,
// with the copy of B's outside that the older kernels leave to another launch:
// 280 -> 198 us at 4097^2, 26.9 -> 14.1 at 1024^2, 12.0 -> 5.0 at 130^2.
template <bool FUSED>
__global__ void __launch_bounds__(256, 2)
    kStencil2L(double *A, const double *B, double *Out, Box2 b, int c0, int nchunks, int sr, long strips, double *items,
               int nitems, int rowsToo) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ double shr[8];
    if (FUSED) gbdev::nextMayLaunch();
    const int lane = threadIdx.x & 31;
    const long strip = blockIdx.x * 8L + (threadIdx.x >> 5);
    uint64_t mb = 0;
    bool seen = false;
    if (strip < strips) {
        const int rb = (int)(strip / nchunks), ch = (int)(strip - (long)rb * nchunks);
        const long base = (c0 + ch) * 64L, j = base + 2 * lane;
        const bool in0 = j >= b.lo1 && j <= b.hi1, in1 = j + 1 >= b.lo1 && j + 1 <= b.hi1;
        // the columns that the loop's cells read (0 outside the array); other elements are replaced by neighbours of
        // theirs, so that they do not leave the limbs' range
        const long first = b.lo1 - 1 > 0 ? b.lo1 - 1 : 0, last = b.hi1 + 1 < b.e1 ? b.hi1 + 1 : b.e1 - 1;
        long jj = j;  // the pair that this lane loads
        if (j > last) jj = last & ~1L;
        if (j + 1 < first) jj = first & ~1L;
        const bool dupY = jj + 1 > last, whole = jj + 1 < b.e1;  // (the last column of an odd row has no pair)
        const bool zeroX = j == b.e1 && b.hi1 + 1 == b.e1, zeroY = j + 1 == b.e1 && b.hi1 + 1 == b.e1;
        // edge columns: lane 0 the left neighbour of j = base, lane 31 the right one of base + 63
        long ej = lane == 0 ? base - 1 : (lane == 31 ? base + 64 : jj);
        const bool zeroE = (ej < 0 && b.lo1 == 0) || (ej == b.e1 && b.hi1 + 1 == b.e1);
        if (ej < first || ej > last) ej = jj;
        // FUSED: the elements that come from B in the box's rows
        const bool xB = jj >= b.lo1 && jj <= b.hi1, yB = jj + 1 >= b.lo1 && jj + 1 <= b.hi1, eB = ej >= b.lo1 && ej <= b.hi1;
        const bool mixed = xB != yB && !dupY;
        const long i0 = b.lo0 + (long)rb * sr;
        const int count = (int)(i0 + sr - 1 < b.hi0 ? sr : b.hi0 - i0 + 1);  // rows of this strip
        const long s0 = b.s0;
        int E = fx::E_DEFAULT;
        // the lane's part in a row, as bits that are tested (not comparisons made again in every row)
        enum { IN0 = 1, IN1 = 2, PLAIN = 4, EDGE = 8, DUPY = 16, ZEROX = 32, ZEROY = 64, ZEROE = 128, FIX = 16 + 32 + 64 + 128,
               OLD2 = 256, OLD1 = 512, OUT0 = 1024, OUT1 = 2048 };
        const bool edgeLane = lane == 0 || lane == 31;
        int f = (in0 ? IN0 : 0) | (in1 ? IN1 : 0) | (whole && !(FUSED && mixed) ? PLAIN : 0) | (edgeLane ? EDGE : 0) |
                (dupY ? DUPY : 0) | (zeroX ? ZEROX : 0) | (zeroY ? ZEROY : 0) | (zeroE ? ZEROE : 0) |
                (j + 1 < b.e1 ? OLD2 : (j < b.e1 ? OLD1 : 0)) | (!in0 && j < b.e1 ? OUT0 : 0) |
                (!in1 && j + 1 < b.e1 ? OUT1 : 0);
        asm volatile("" : "+r"(f));
        // rows are numbered from i0 - 1; numbers boxLo .. boxLo + boxN are rows of the box
        const int boxLo = i0 > b.lo0 ? 0 : 1;
        const unsigned boxN = (unsigned)((b.hi0 - i0 + 1 < count + 1 ? b.hi0 - i0 + 1 : count + 1) - boxLo);
        // FUSED: A's own pair of the row beside it
        rows::Ring &ring = reinterpret_cast<rows::Ring *>(dyn)[(FUSED ? 2 : 1) * (threadIdx.x >> 5)];
        rows::Ring &oldRing = reinterpret_cast<rows::Ring *>(dyn)[(FUSED ? 2 : 1) * (threadIdx.x >> 5) + (FUSED ? 1 : 0)];
        // this lane's source of row i: B in the box (FUSED), else A
        auto from = [&](long i, bool fromB) { return (FUSED && fromB && i >= b.lo0 && i <= b.hi0 ? B : A) + i * s0; };
        // copies of the strip's rows, number 0 being row i0 - 1: the next number, its place in the ring, its sources
        int asked = 0;
        double2 *dst = &ring.pair[0][lane], *dstOld = &oldRing.pair[0][lane];
        double *dstEdge = &ring.edge[0][lane & 1];
        const double *px = (FUSED && (xB || yB) ? B : A) + (i0 - 1) * s0 + jj, *pe = (FUSED && eB ? B : A) + (i0 - 1) * s0 + ej;
        const double *po = A + (i0 - 1) * s0 + j;
        auto ask = [&]() {
            if (asked < count + 2) {
                const bool box = (unsigned)(asked - boxLo) <= boxN;
                if (__builtin_expect(box && (f & PLAIN), 1)) {
                    rows::copy16(dst, px);
                    if (f & EDGE) rows::copy8(dstEdge, pe);
                } else {  // a row beside the box, a pair that is not one of a single array
                    const long i = i0 - 1 + asked;
                    const bool in = i >= 0 && i < b.e0;
                    rows::copy8(&dst->x, in ? from(i, xB) + jj : A, in);
                    if (whole) rows::copy8(&dst->y, in ? from(i, yB) + jj + 1 : A, in);
                    if (f & EDGE) rows::copy8(dstEdge, in ? from(i, eB) + ej : A, in);
                }
                if (FUSED && box) {
                    if (f & OLD2) rows::copy16(dstOld, po);
                    else if (f & OLD1) rows::copy8(&dstOld->x, po);
                }
                px += s0;
                pe += s0;
                po += s0;
            }
            asked++;
            const bool wrap = asked % rows::DEPTH == 0;
            dst += wrap ? 32 - 32 * rows::DEPTH : 32;
            dstOld += wrap ? 32 - 32 * rows::DEPTH : 32;
            dstEdge += wrap ? 2 - 2 * rows::DEPTH : 2;
            rows::commit();
        };
        auto fix = [&](rows::Row &r) {
            if (!(f & EDGE)) r.e = r.d.x;
            if (__builtin_expect(f & FIX, 0)) {
                if (f & DUPY) r.d.y = r.d.x;
                if (f & ZEROX) r.d.x = 0.0;
                if (f & ZEROY) r.d.y = 0.0;
                if (f & ZEROE) r.e = 0.0;
            }
            rows::split(r, E);
        };
        int taken = 0;
        // the strip's next row, and the copy of the row DEPTH - 1 after it
        auto take = [&](rows::Row &r) {
            rows::landed();
            r.d = ring.pair[taken % rows::DEPTH][lane];
            r.e = ring.edge[taken % rows::DEPTH][lane & 1];
            taken++;
            ask();
            fix(r);
        };
        auto again = [&](long i, rows::Row &r) {  // from memory
            r.d = make_double2(0.0, 0.0);
            r.e = 0.0;
            if (i >= 0 && i < b.e0) {
                r.d.x = from(i, xB)[jj];
                if (whole) r.d.y = from(i, yB)[jj + 1];
                r.e = from(i, eB)[ej];
            }
            fix(r);
        };
        rows::Row ra, rc, rd;
        for (int q = 0; q < rows::DEPTH - 1; q++) ask();
        take(ra);
        take(rc);
        double2 old = FUSED ? oldRing.pair[1][lane] : make_double2(0.0, 0.0);  // A's own pair of row i
        take(rd);
        double2 dif = make_double2(0.0, 0.0);
        uint32_t mh = 0, ml = 0;  // the largest |B - A| so far, as bits
        auto absmax = [&](double d) {  // a NaN leaves it, as Max(t, eps) does
            const uint32_t h = sf::hi32(sf::bits(d)) & 0x7FFFFFFFu, l = (uint32_t)sf::bits(d);
            const bool more = (((uint64_t)h << 32) | l) > (((uint64_t)mh << 32) | ml) && h < 0x7FF00000u + (l == 0 ? 1u : 0u);
            mh = more ? h : mh;
            ml = more ? l : ml;
        };
        double *out = Out + i0 * s0 + j, *a = FUSED ? A + i0 * s0 + j : nullptr;
        long i = i0;
        int left = count;
        int hold = 0;  // rows that are not tried in another range, the last move having been in vain
        constexpr int HOLD = 32;

        // row i from up, mid, dn; up then takes row i + 2's place
        auto step = [&](rows::Row &up, rows::Row &mid, rows::Row &dn) -> bool {
            const bool more = left > 1;
            if (__builtin_expect(!(up.ok && mid.ok && dn.ok), 0)) {
                if (hold > 0) {
                    hold--;
                } else {
                    const int e = rows::rangeOf(up, mid, dn, E);
                    if (e != E) {  // move the range
                        E = e;
                        again(i - 1, up);
                        again(i, mid);
                        again(i + 1, dn);
                        if (!(up.ok && mid.ok && dn.ok)) hold = HOLD;
                    }
                }
            }
            double v0, v1;
            if (__builtin_expect(up.ok && mid.ok && dn.ok, 1)) {
                fx::Limbs<rows::f32x2> lt, rt;
                rows::sides(mid.v.h, mid.eh, lane, lt.h, rt.h);
                rows::sides(mid.v.m, mid.em, lane, lt.m, rt.m);
                rows::sides(mid.v.l, mid.el, lane, lt.l, rt.l);
                // (((A[i-1][j] + A[i][j-1]) + A[i][j+1]) + A[i+1][j]) / 4.0
                const fx::Quotient<rows::f32x2> z = fx::whole(fx::add(fx::add(fx::add(up.v, lt), rt), dn.v));
                v0 = fx::assemble(fx::lo(z.hm), fx::lo(z.mm), fx::lo(z.l), fx::lo(z.b), E, 2);
                v1 = fx::assemble(fx::hi(z.hm), fx::hi(z.mm), fx::hi(z.l), fx::hi(z.b), E, 2);
                if (__builtin_expect(fminf(fx::lo(z.b), fx::hi(z.b)) == 0.0f, 0)) {  // four zeros
                    if (fx::lo(z.b) == 0.0f) v0 = 0.0;
                    if (fx::hi(z.b) == 0.0f) v1 = 0.0;
                }
            } else {
                const double lx = __shfl_up_sync(0xffffffffu, mid.d.y, 1), ry = __shfl_down_sync(0xffffffffu, mid.d.x, 1);
                const double l = lane == 0 ? mid.e : lx, r = lane == 31 ? mid.e : ry;
                // a loop: as straight code the compiler issues these FP64 instructions, predicated off, in every row,
                // and each still takes the unit (FUSED, 4096^2: 187 us an iteration, so 183)
                v0 = v1 = 0.0;
#pragma unroll 1
                for (int e = 0; e < 2; e++) {
                    v0 = v1;
                    v1 = sf::scale_down(sf::nadd(sf::nadd(sf::nadd(e ? up.d.y : up.d.x, e ? mid.d.x : l),
                                                          e ? r : mid.d.y), e ? dn.d.y : dn.d.x), 2);
                }
            }
            if (__builtin_expect((f & (IN0 | IN1)) == (IN0 | IN1), 1)) {
                rows::stGlobal(out, make_double2(v0, v1));
                if (FUSED) rows::stGlobal(a, mid.d);
            } else {
                if (f & IN0) {
                    rows::stGlobal(out, v0);
                    if (FUSED) rows::stGlobal(a, mid.d.x);
                } else if (FUSED && (f & OUT0)) {
                    rows::stGlobal(out, __ldg(B + (out - Out)));
                }
                if (f & IN1) {
                    rows::stGlobal(out + 1, v1);
                    if (FUSED) rows::stGlobal(a + 1, mid.d.y);
                } else if (FUSED && (f & OUT1)) {
                    rows::stGlobal(out + 1, __ldg(B + (out - Out) + 1));
                }
            }
            if (FUSED) {
                // the last row's differences enter the MAX now: nothing waits for the FP64 unit
                absmax(dif.x);
                absmax(dif.y);
                dif.x = sf::nadd(mid.d.x, f & IN0 ? -old.x : -mid.d.x);
                dif.y = sf::nadd(mid.d.y, f & IN1 ? -old.y : -mid.d.y);
            }
            if (!more) return false;
            if (FUSED) old = oldRing.pair[(taken - 1) % rows::DEPTH][lane];
            take(up);
            i++;
            out += s0;
            if (FUSED) a += s0;
            left--;
            return true;
        };
        // three rows a trip, so that the limbs stay where they are
        while (step(ra, rc, rd) && step(rc, rd, ra) && step(rd, ra, rc)) {
        }
        seen = in0 || in1;
        if (FUSED) {
            absmax(dif.x);
            absmax(dif.y);
            mb = ((uint64_t)mh << 32) | ml;
        }
        if (FUSED && rowsToo) {  // the rows above and below the box, in this chunk's columns
            auto copyRow = [&](long r) {
                for (int e = 0; e < 2; e++)
                    if (j + e < b.e1) Out[r * s0 + j + e] = B[r * s0 + j + e];
            };
            if (rb == 0)
                for (long r = 0; r < b.lo0; r++) copyRow(r);
            if (i0 + count > b.hi0)
                for (long r = b.hi0 + 1; r < b.e0; r++) copyRow(r);
        }
    }
    if (FUSED) {
        const double m = ctaMax(seen ? sf::from(mb) : -__builtin_huge_val(), shr);
        if (threadIdx.x == 0) items[blockIdx.x] = m;
        if (blockIdx.x == 0)  // the items that this launch has no CTA for
            for (int q = gridDim.x + threadIdx.x; q < nitems; q += 256) items[q] = -__builtin_huge_val();
    }
}

struct St2LGeom {
    int c0, nchunks, sr;
    long strips, blocks;
    bool ok;
};

// The strip length that costs least: the GPU's 2 x 8 warps per SM take the strips in rounds, and a strip of sr rows
// costs about 2 sr + 5 half-rows (three rows are loaded and split before its first result).
St2LGeom st2LGeom(const long lo[2], const long hi[2]) {
    St2LGeom g{};
    const long ni = hi[0] - lo[0] + 1;
    g.ok = ni > 0 && hi[1] >= lo[1] && lo[1] >= 0 && lo[0] >= 0 && hi[1] / 64 < (1L << 31);
    if (!g.ok) return g;
    g.c0 = (int)(lo[1] / 64);
    const long nchunks = hi[1] / 64 - g.c0 + 1, warps = (long)smCount() * 16;
    long best = -1, bestSr = 1;
    for (long sr = 1; sr <= 128 && (sr == 1 || sr <= ni); sr++) {
        const long cost = ((ni + sr - 1) / sr * nchunks + warps - 1) / warps * (2 * sr + 5);
        if (best < 0 || cost < best) best = cost, bestSr = sr;
    }
    g.nchunks = (int)nchunks;
    g.sr = (int)bestSr;
    g.strips = (ni + bestSr - 1) / bestSr * nchunks;
    g.blocks = (g.strips + 7) / 8;
    g.ok = g.blocks < (1L << 31);
    return g;
}
