// The 3-D Jacobi stencil loop, Out = (6 neighbours of A) / 6, with A's planes
// staged in shared memory by the Tensor Memory Accelerator and the sums on the
// FP32 pipe (fixlimb.cuh).  M = 0: the loop alone; M = 3: a time step's stencil
// loop followed by the next step's update loop, eps = Max(|B - A|, eps); A = B.
// Included by jacobi.cu inside its anonymous namespace, after stencil_tma.cuh.
//
// A CTA covers 64 columns of k (lane l owns the pair 2l, 2l + 1) and TY rows of
// j, one warp each, and streams the planes i of its chunk.  One thread issues
// one TMA box copy per plane -- the CTA's columns with both edge columns and its
// rows with both halo rows, a (TY + 2) x 68 box starting at k = kb - 2 so that
// the copy's x coordinate stays 16-byte aligned, 0 outside the array -- into a
// ring of NS plane slots, NS - 2 planes ahead.  Step t (plane ib + t, sequence
// number t + 1 of the copies) waits for plane t + 2, splits it into limbs --
// every element once, by the CTA; a thread keeps its own pair's limbs in
// registers, so the neighbours in i come from there -- and writes them to the
// limb ring; then it computes plane t + 1 from the registers and the limb slot
// that was written a step before.  One barrier per step separates the writes of
// a limb slot (two slots) from its readers, and a plane slot's readers from the
// next copy into it.
//
// Range.  The limbs hold +0 and nine binades of positive values, [2^-9, 1) at
// first.  When a plane has another value, the CTA looks up the largest exponent
// of that plane and the one before, moves the range so that it ends there, and
// splits the two again: a field in degrees or an initial spike costs a few such
// steps, not the whole loop.  A cell whose neighbours still do not fit
// (negative, tiny beside its neighbours, infinite) is computed on the FP64 unit
// from the doubles of the plane slots, bit for bit the same; so is one whose
// quotient is too small for the assembly, by the integer division.
//
// Plain planes.  A plane that no range holds is done by a loop of its own, with
// no split before it and the limbs of the next two planes made anew after it; the
// third in a row (the first of a chunk) is followed by eight such planes, then
// sixteen, up to sixty-four at a time.  With every plane split and looked through
// first, and rows outside the box computed too, values in [-1, 1) took 254 us for
// the stencil and 342 for the cross-step pass at 255^3, 1500 and 2220 at 512^3,
// 1186 and 2790 for a box of 2000 x 2 x 2000; now 178 and 270, 1350 and 1940, 150
// and 425 (the kernels before the limbs: 205 and 285, 1535 and 2046, 226 and 336).
// A loop of its own also because as a branch of the step, in its three copies, it
// took the FP64 path 2790 us at 512^3: instruction fetches.
//
// M = 3: the new B of a cell meets A's limbs (the plane's own) in registers, so
// |B - A| is a difference of limbs, exact as an integer.  Only its FP32 value
// (off by less than 2^-21 relatively) is formed for every cell; the exact
// difference enters the thread's MAX where that value comes within 2^-20 of the
// largest one the CTA has seen.  RN(max |b - a|) = max |RN(b - a)|: RN is
// monotone and odd.  B is stored twice, into B and into A's second buffer, which
// becomes A when the pair ends; the cells of the box's rows beside it (k outside
// [lo2, hi2], inside the CTAs' columns) get A's value there.  24 bytes a cell.
//
// What bounds it: instruction issue.  A cell takes about 130 instructions (two
// cells per FP32 instruction in the sums) against 178 of the q61 form, whose
// 64-bit integer additions kept the ALU pipe busy; at 512^3 the stencil alone
// takes 0.61 ms (q61 0.82) and the cross-step pass 0.68 ms (q61, with a quarter
// of the warps on the FP64 unit, 1.05) of the 0.48 ms its 24 bytes a cell take at
// the copy rate.  FP64-unit warps made both slower here (0.76 and 0.99 ms with
// one in eight): the others wait for them at the barrier.  mbarriers in its
// place, so that warps may run a step ahead, cost more in polling and in
// instruction-cache misses than the barrier (0.82 ms).
//
// Every wait is bounded (tma::mbarWait): after 2 s the kernel writes
// DVMHGB_ERR_TMA_TIMEOUT to the status word (when one is given), the CTA leaves
// its loop, and thread 0 waits (bounded again) for the copies in flight.
namespace limb {

constexpr int BX = tma::BX;
constexpr int rowsOf(int jt) { return TY * jt; }                      // rows of j a CTA computes
constexpr int cellsOf(int jt) { return BX * (rowsOf(jt) + 2); }       // of a plane's box
constexpr int slotOf(int jt) { return (cellsOf(jt) * 8 + 127) / 128 * 128; }
constexpr int ringOf(int jt) { return 2 * 3 * cellsOf(jt) * 4; }      // two planes' limbs
constexpr int smemBytes(int jt, int ns) { return ns * slotOf(jt) + ringOf(jt) + ns * 8 + 128; }
static_assert(BX % 2 == 0, "pairs of limbs are 8-byte aligned");

__device__ __forceinline__ fx::f32x2 ld2f(const float *p) {
    return {*reinterpret_cast<const unsigned long long *>(p)};
}
__device__ __forceinline__ void st2f(float *p, fx::f32x2 v) { *reinterpret_cast<unsigned long long *>(p) = v.v; }

// a row's limbs of one plane
__device__ __forceinline__ fx::Limbs<fx::f32x2> ldLimbs(const float *p, int cells) {
    return {ld2f(p), ld2f(p + cells), ld2f(p + 2 * cells)};
}
__device__ __forceinline__ void stLimbs(float *p, int cells, const fx::Limbs<fx::f32x2> &v) {
    st2f(p, v.h);
    st2f(p + cells, v.m);
    st2f(p + 2 * cells, v.l);
}

}  // namespace limb

template <int M, int JT, int NS, int MINB>
__global__ void __launch_bounds__(TX *TY, MINB)
    kStencil3L(const __grid_constant__ CUtensorMap map, double *Out, Box3 b, long p0, int ichunk, double *items,
               int *status, double *Out2) {
    static_assert(NS >= 4, "the ring holds planes i - 1, i, i + 1 and the slot being refilled");
    static_assert(M == 0 || M == 3, "the loop alone, or with the next update");
    constexpr bool U = M == 3;
    constexpr int BX = limb::BX, CELLS = limb::cellsOf(JT), SLOT = limb::slotOf(JT), TJ = limb::rowsOf(JT);
    using fx::f32x2;
    using Limbs = fx::Limbs<f32x2>;
    extern __shared__ unsigned char dyn[];
    if (U) gbdev::nextMayLaunch();
    unsigned char *base = dyn + ((128u - (tma::smemAddr(dyn) & 127u)) & 127u);
    float *ring = reinterpret_cast<float *>(base + NS * SLOT);
    uint64_t *bars = reinterpret_cast<uint64_t *>(base + NS * SLOT + limb::ringOf(JT));
    // the timeout flag, one per parity of the step: set before the step's barrier, read after it
    __shared__ int stopAt[2];
    __shared__ unsigned topExp;
    // planes that no range held: the last one's step, how many in a row (the chunk's first counts as the third), how many
    // plain planes follow the next that is one too many
    __shared__ int missAt, missed, nextPlain;
    __shared__ float seenMax;  // U: |B - A| (u units) some thread has entered exactly, times (1 - 2^-20)
    __shared__ double shr[TY];

    const int lane = threadIdx.x, ty = threadIdx.y, tid = ty * TX + lane;
    const long kb = 2 * (p0 + (long)blockIdx.x * TX);
    const long jb = b.lo1 + (long)blockIdx.y * TJ;
    const long ib = b.lo0 + (long)blockIdx.z * ichunk;
    const long ie = ib + ichunk - 1 < b.hi0 ? ib + ichunk - 1 : b.hi0;
    const int nplanes = (int)(ie - ib + 1), nseq = nplanes + 2;  // planes ib - 1 .. ie + 1
    const long k = kb + 2 * lane, j = jb + JT * ty;
    const bool k0 = k >= b.lo2 && k <= b.hi2, k1 = k + 1 >= b.lo2 && k + 1 <= b.hi2;
    // the cells of the loop box: bits 0, 1 the first row's pair, bits 2, 3 the second's; U: from bit 4, the others of a
    // row of the box, whose A carries over; MINE: the warp has a row of the box
    constexpr int MINE = 256;
    int cells = j <= b.hi1 ? MINE : 0;
    float tiny[JT][2];
    f32x2 mask[JT];
#pragma unroll
    for (int r = 0; r < JT; r++) {
        const bool in0 = j + r <= b.hi1 && k0, in1 = j + r <= b.hi1 && k1;
        cells |= (in0 ? 1 << 2 * r : 0) | (in1 ? 2 << 2 * r : 0);
        if (U && j + r <= b.hi1)
            cells |= (!in0 && k < b.e2 ? 16 << 2 * r : 0) | (!in1 && k + 1 < b.e2 ? 32 << 2 * r : 0);
        // a quotient below the assembly's range counts in the box only; |B - A| outside it is 0
        tiny[r][0] = in0 ? fx::SMALL6 : -__builtin_huge_valf();
        tiny[r][1] = in1 ? fx::SMALL6 : -__builtin_huge_valf();
        mask[r] = fx::pack(in0 ? 1.0f : 0.0f, in1 ? 1.0f : 0.0f);
    }
    asm volatile("" : "+r"(cells));  // kept, not computed again every step

    auto slotOf = [&](int q) { return reinterpret_cast<const double *>(base + (size_t)(q % NS) * SLOT); };
    auto limbsOf = [&](int q) { return ring + (q & 1) * 3 * CELLS; };
    auto barOf = [&](int q) { return tma::smemAddr(bars + q % NS); };
    auto parityOf = [](int q) { return (uint32_t)((q / NS) & 1); };
    int issued = 0;  // thread 0: planes issued (q = 0 .. issued - 1)
    auto issue = [&](int q) {
        const uint32_t bar = barOf(q);
        tma::mbarExpect(bar, CELLS * 8);
        tma::copyBox(&map, tma::smemAddr(slotOf(q)), bar, (int)(kb - 2), (int)(jb - 1), (int)(ib - 1 + q));
        issued = q + 1;
    };

    // the pairs this thread splits: its own (rows JT ty + 1 .. of the box, pair lane + 1) and, HALO threads, one of
    // the halo (the first and last row, then the first and last pair of the others); which warps have those differs
    // from CTA to CTA, so that the SM's four schedulers get the same work
    constexpr int RP = BX / 2;  // pairs of a row
    constexpr int HALO = 2 * RP + 2 * TJ;
    static_assert(HALO == CELLS / 2 - TX * TJ && HALO <= TX * TY, "own pairs, then halo pairs");
    // (a thread whose pairs no cell of the box reads takes the CTA's first one, so that theirs do not count)
    const int place = (JT * ty + 1) * BX + 2 + 2 * lane;
    const int own = j <= b.hi1 + 1 && k <= b.hi2 + 1 ? place : BX + 2;
    int halo = -1;
    {
        const int h = (tid + 32 * (int)((blockIdx.x + blockIdx.y + blockIdx.z) & 7)) & (TX * TY - 1);
        if (h < RP) halo = 2 * h;
        else if (h < 2 * RP) halo = (TJ + 1) * BX + 2 * (h - RP);
        else if (h < HALO) halo = (1 + (h - 2 * RP) / 2) * BX + ((h - 2 * RP) & 1 ? BX - 2 : 0);
        // beyond the last row and column that a cell of the box reads
        if (halo >= 0 && (jb - 1 + halo / BX > b.hi1 + 1 || kb - 2 + halo % BX > b.hi2 + 1)) halo = -1;
    }

    constexpr int MISSES = 3, PLAIN = 8, PLAIN_MAX = 64;  // (above)
    int E = fx::E_DEFAULT;  // the range's smallest exponent field
    auto splitPair = [&](const double *src, bool &ok) -> Limbs {
        const uint4 w = *reinterpret_cast<const uint4 *>(src);
        const uint32_t s0 = fx::place(w.y, E), s1 = fx::place(w.w, E);
        fx::Raw x = fx::split(w.y, w.x, s0), y = fx::split(w.w, w.z, s1);
        if (__builtin_expect(max(s0, s1) > 8u, 0)) {  // a zero, or a value outside the range
            x = fx::splitAny(w.y, w.x, s0, ok);
            y = fx::splitAny(w.w, w.z, s1, ok);
        }
        return fx::unbias(fx::pack(fx::ffrom(x.h), fx::ffrom(y.h)), fx::pack(fx::ffrom(x.m), fx::ffrom(y.m)),
                          fx::pack(fx::ffrom(x.l), fx::ffrom(y.l)));
    };
    struct Own {  // the own pairs' limbs in one plane, and whether all are in range
        Limbs v[JT];
        bool ok;
    };
    auto splitOwn = [&](const double *s, Own &o) -> bool {
        bool ok = true;
#pragma unroll
        for (int r = 0; r < JT; r++) o.v[r] = splitPair(s + own + r * BX, ok);
        o.ok = ok;
        return ok;
    };
    // a plane's limbs: the own pairs' to o and, with the halo pair's, to the ring
    auto splitPlane = [&](const double *s, float *l, Own &o) -> bool {
        bool ok = splitOwn(s, o);
#pragma unroll
        for (int r = 0; r < JT; r++) limb::stLimbs(l + own + r * BX, CELLS, o.v[r]);
        if (halo >= 0) limb::stLimbs(l + halo, CELLS, splitPair(s + halo, ok));
        return ok;
    };
    auto await = [&](uint32_t bar, uint32_t parity, int step) {
        if (!tma::mbarWait(bar, parity)) {
            if (status) atomicExch(status, DVMHGB_ERR_TMA_TIMEOUT);
            stopAt[step & 1] = 1;
        }
    };

    uint64_t mb = 0;    // the update's eps: Max(|B - A|) as a bit pattern (FP64-unit differences)
    uint64_t qmax = 0;  // ... and the largest exact difference in u units (range E)
    auto flushMax = [&]() {
        // RN(max |b - a|): RN is monotone, so the largest, rounded once
        const double d = __ull2double_rn(qmax) * 0x1p-64 * sf::from((uint64_t)(E - 1075 + 64 + 1023) << 52);
        if (sf::bits(d) > mb) mb = sf::bits(d);
        qmax = 0;
    };

    if (tid == 0) {
        stopAt[0] = stopAt[1] = 0;
        missAt = -1, missed = 2, nextPlain = PLAIN;
        seenMax = 0.0f;
        for (int s = 0; s < NS; s++) tma::mbarInit(tma::smemAddr(bars + s), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int q = 0; q < NS && q < nseq; q++) issue(q);
    }
    __syncthreads();
    Own oa, ob, oc;  // planes i - 1, i, i + 1, in turn
    await(barOf(0), 0, 0);
    splitOwn(slotOf(0), oa);
    await(barOf(1), 0, 0);
    bool planeOk = !__syncthreads_or(!splitPlane(slotOf(1), limbsOf(1), ob));
    bool stop = stopAt[0] != 0;
    // the slot, mbarrier and parity of the next plane to wait for (sequence number 2), and the limb slots
    const double *next = slotOf(2);
    uint32_t nextBar = barOf(2), nextPar = 0;
    float *lcur = limbsOf(1), *lnext = limbsOf(2);
    double *out = Out + ib * b.s0 + j * b.s1 + k;
    const long toOut2 = U ? (Out2 - Out) : 0;
    int t = 0;

    // plane t + 1 on the FP64 unit, from the doubles of the slots
    auto native = [&](double v[JT][2]) {
        const double *pm = slotOf(t) + own, *pc = slotOf(t + 1) + own, *pp = next + own;
        double2 ac[JT];
        // |B - A| of a cell after the next cell's sum, so that a division runs beside those additions (the pass at 512^3 with
        // values in [-1, 1) 1937 -> 1924 us, at 600 x 90 x 600 558 -> 549)
        auto diff = [&](int q) {
            const double d = sf::nadd(v[q >> 1][q & 1], -(q & 1 ? ac[q >> 1].y : ac[q >> 1].x));
            if (cells >> q & 1) mb = sf::absmax_bits(d, mb);
        };
#pragma unroll
        for (int q = 0; q < 2 * JT; q++) {
            const int r = q >> 1, e = q & 1;
            if (e == 0) ac[r] = *reinterpret_cast<const double2 *>(pc + r * BX);
            const double first = sf::nadd(sf::nadd(pm[r * BX + e], pc[(r - 1) * BX + e]), e ? ac[r].x : pc[r * BX - 1]);
            const double sum =
                sf::nadd(sf::nadd(sf::nadd(first, e ? pc[r * BX + 2] : ac[r].y), pc[(r + 1) * BX + e]), pp[r * BX + e]);
            if (U && q > 0) diff(q - 1);
            v[r][e] = sf::div3p2(sum, 1);
        }
        if (U) diff(2 * JT - 1);
    };
    auto store = [&](const double v[JT][2]) {
#pragma unroll
        for (int r = 0; r < JT; r++) {
            double *o = out + r * b.s1;
            if (__builtin_expect((cells >> 2 * r & 3) == 3, 1)) {
                st2cs(o, make_double2(v[r][0], v[r][1]));
                if (U) st2cs(o + toOut2, make_double2(v[r][0], v[r][1]));  // A = B into A's second buffer
            } else {
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    if (cells >> (2 * r + e) & 1) {
                        o[e] = v[r][e];
                        if (U) o[toOut2 + e] = v[r][e];
                    } else if (U && (cells >> (2 * r + e) & 16)) {
                        o[toOut2 + e] = slotOf(t + 1)[place + r * BX + e];
                    }
                }
            }
        }
    };
    // to the next step; `ok` of every thread's part of plane t + 2
    auto advance = [&](bool ok) -> bool {
        out += b.s0;
        next = reinterpret_cast<const double *>(reinterpret_cast<const unsigned char *>(next) + SLOT);
        nextBar += 8;
        if (next == reinterpret_cast<const double *>(base + NS * SLOT)) {
            next = reinterpret_cast<const double *>(base);
            nextBar -= 8 * NS;
            nextPar ^= 1;
        }
        float *const spare = lcur;
        lcur = lnext;
        lnext = spare;
        planeOk = !__syncthreads_or(!ok);
        stop = stopAt[t & 1] != 0;
        if (tid == 0 && !stop && t + NS < nseq) {  // every reader of plane c - 1 = t has passed the barrier
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            issue(t + NS);
        }
        t++;
        return t < nplanes && !stop;
    };
    int plain = 0;  // plain planes to do next

    // step t: plane c = t + 1 from planes m, c, p; false when the loop ends or plain planes are next
    auto step = [&](Own &m, Own &c, Own &p) -> bool {
        if (__builtin_expect(!planeOk, 0)) {  // move the range to the values of planes c - 1 and c (uniform)
            unsigned top = 0;
            // (written after the barriers below)
            const int in = t == missAt + 1 ? missed + 1 : 1, n = in > 1 ? nextPlain : PLAIN;
            for (int q = t; q <= t + 1; q++) {
                const uint2 *w = reinterpret_cast<const uint2 *>(slotOf(q));
#pragma unroll
                for (int r = 0; r < JT; r++)
                    top = max(top, max(w[own + r * BX].y >> 20, w[own + r * BX + 1].y >> 20));
                if (halo >= 0) top = max(top, max(w[halo].y >> 20, w[halo + 1].y >> 20));
            }
            top = __reduce_max_sync(0xffffffffu, top);
            if (tid == 0) topExp = 0;
            __syncthreads();
            if (lane == 0) atomicMax(&topExp, top);
            __syncthreads();
            const int e = (int)topExp - 8;
            if (e != E && e >= fx::E_MIN && e <= fx::E_MAX) {
                if (U) flushMax();
                if (tid == 0) seenMax = 0.0f;
                E = e;
                splitOwn(slotOf(t), m);
                planeOk = !__syncthreads_or(!splitPlane(slotOf(t + 1), lcur, c));
            }
            if (!planeOk) {
                if (tid == 0) {
                    missAt = t, missed = in;
                    nextPlain = in < MISSES ? n : n < PLAIN_MAX ? 2 * n : n;
                }
                plain = in >= MISSES ? n : 1;
                return false;
            }
        }
        await(nextBar, nextPar, t);
        const bool nextOk = splitPlane(next, lnext, p);

        double v[JT][2];
        float mags[JT][2], most = 0.0f;
        bool fast = planeOk && m.ok && p.ok;
        if (__builtin_expect(fast, 1)) {
            const float *l = lcur + own;
            Limbs up = limb::ldLimbs(l - BX, CELLS);
            float low = 0.0f;  // negative: a quotient is zero or too small for the assembly
#pragma unroll
            for (int r = 0; r < JT; r++) {
                const float *q = l + r * BX;
                const Limbs o = c.v[r];
                const Limbs dn = r + 1 < JT ? c.v[r + 1 < JT ? r + 1 : r] : limb::ldLimbs(q + BX, CELLS);
                // (((((A[i-1] + A[j-1]) + A[k-1]) + A[k+1]) + A[j+1]) + A[i+1]) / 6, left to right
                Limbs s = fx::add(m.v[r], up);
                s = fx::add(s, Limbs{fx::pack(q[-1], fx::lo(o.h)), fx::pack(q[CELLS - 1], fx::lo(o.m)),
                                     fx::pack(q[2 * CELLS - 1], fx::lo(o.l))});
                s = fx::add(s, Limbs{fx::pack(fx::hi(o.h), q[2]), fx::pack(fx::hi(o.m), q[CELLS + 2]),
                                     fx::pack(fx::hi(o.l), q[2 * CELLS + 2])});
                s = fx::add(s, dn);
                s = fx::add(s, p.v[r]);
                up = o;
                const f32x2 mag = fx::magnitude(s);
                mags[r][0] = fx::lo(mag), mags[r][1] = fx::hi(mag);
                low = fminf(low, fminf(mags[r][0] - tiny[r][0], mags[r][1] - tiny[r][1]));
                const fx::Quotient<f32x2> z = fx::div6(s);
                v[r][0] = fx::assemble(fx::lo(z.hm), fx::lo(z.mm), fx::lo(z.l), fx::lo(z.b), E);
                v[r][1] = fx::assemble(fx::hi(z.hm), fx::hi(z.mm), fx::hi(z.l), fx::hi(z.b), E);
                if (U) {
                    const f32x2 mtwo23 = fx::pack(-0x1p23f, -0x1p23f), m1 = fx::pack(-1.0f, -1.0f);
                    const f32x2 up20 = fx::pack(0x1p20f, 0x1p20f);
                    const f32x2 dh = fx::vfma(o.h, fx::pack(-0x1p-11f, -0x1p-11f), fx::vadd(z.hm, mtwo23));
                    const f32x2 dm = fx::vfma(o.m, m1, fx::vadd(z.mm, mtwo23)), dl = fx::vfma(o.l, m1, z.l);
                    const f32x2 d = fx::vmul(fx::vfma(fx::vfma(dh, up20, dm), up20, dl), mask[r]);
                    most = fmaxf(most, fmaxf(fabsf(fx::lo(d)), fabsf(fx::hi(d))));
                }
            }
            if (__builtin_expect(low < 0.0f, 0)) {
                fast = false;
            } else if (U && __builtin_expect(most > *(volatile float *)&seenMax, 0)) {
                // exact differences, as integers of u: both values are in range
                const double *pc = slotOf(t + 1) + own;
#pragma unroll
                for (int r = 0; r < JT; r++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const uint64_t x = fx::integer(v[r][e], E), y = fx::integer(pc[r * BX + e], E);
                        const uint64_t d = x > y ? x - y : y - x;
                        if ((cells >> (2 * r + e) & 1) && d > qmax) qmax = d;
                    }
                atomicMax(reinterpret_cast<int *>(&seenMax), __float_as_int(most * (1.0f - 0x1p-20f)));
            }
        } else {
#pragma unroll
            for (int r = 0; r < JT; r++) {
                mags[r][0] = mags[r][1] = 1.0f;
                if (!U) v[r][0] = v[r][1] = 0.0;
            }
        }
        if (__builtin_expect(!fast, 0)) {
            // values outside the range in the planes beside this one, or a quotient that is zero (all six neighbours are
            // +0) or small: on the FP64 unit, from the doubles of the slots.  Alone the stencil keeps the thread's other
            // quotients; with the update they are made again, since keeping them costs the common path 1 to 3 percent in
            // every form tried.  512^3, 2 percent of values among zeros: stencil 1703 -> 791 us (q61 kernels 1203), cross-step
            // pass 2582 -> 2205 (1572; 1300 where they were kept), 130^3 147 -> 67 (64); only zeros 922 -> 818.
            const double *pm = slotOf(t) + own, *pc = slotOf(t + 1) + own, *pp = next + own;
#pragma unroll
            for (int r = 0; r < JT; r++, pm += BX, pc += BX, pp += BX) {
                const double2 ac = *reinterpret_cast<const double2 *>(pc);
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    double d = e ? ac.y : ac.x;  // |B - A| of a zero
                    if (mags[r][e] == 0.0f) {
                        v[r][e] = 0.0;
                    } else if (U || mags[r][e] < tiny[r][e]) {
                        const double first = sf::nadd(sf::nadd(pm[e], pc[e - BX]), e ? ac.x : pc[-1]);
                        v[r][e] = sf::div3p2(
                            sf::nadd(sf::nadd(sf::nadd(first, e ? pc[2] : ac.y), pc[e + BX]), pp[e]), 1);
                        if (U) d = sf::nadd(v[r][e], -d);
                    }
                    if (U && (cells >> (2 * r + e) & 1)) mb = sf::absmax_bits(d, mb);
                }
            }
        }
        store(v);
        return advance(nextOk);
    };
    // three steps a trip, so that the limbs stay where they are
    if (!stop && nplanes > 0)
        while (true) {
            while (step(oa, ob, oc) && step(ob, oc, oa) && step(oc, oa, ob)) {
            }
            if (plain == 0) break;
            bool more = true;
            for (; plain > 0 && more; plain--) {
                await(nextBar, nextPar, t);
                if (cells & MINE) {
                    double v[JT][2];
                    native(v);
                    store(v);
                }
                more = advance(true);
            }
            if (!more) break;
            plain = 0;
            if (tid == 0) missAt = t - 1;
            splitOwn(slotOf(t), oa);
            planeOk = !__syncthreads_or(!splitPlane(slotOf(t + 1), lcur, ob));
        }
    if (U) {
        flushMax();
        double m = (cells & 15) ? sf::from(mb) : -__builtin_huge_val();
        m = ctaMax(m, shr);
        if (tid == 0) items[blockIdx.x + gridDim.x * ((long)blockIdx.y + (long)gridDim.y * blockIdx.z)] = m;
    }
    // after a timeout, the copies still in flight land before the CTA's shared memory is released
    if (stop && tid == 0)
        for (int q = issued - NS < 0 ? 0 : issued - NS; q < issued; q++) (void)tma::mbarWait(barOf(q), parityOf(q));
}

// The grid of kStencil3L with JT rows per thread and `ctas` CTAs resident per SM: the number of chunks of planes that
// costs least, a chunk of n planes taking about n + 4 steps (the first copies' latency and two planes split ahead),
// rounds of CTAs one after the other.  Of the counts that take the same rounds the largest costs least, so the rounds
// are gone through, not the counts: those took the host 130 us a call for a box of 60000 planes of 8 x 32.
St3Geom stLGeom(const long lo[3], const long hi[3], int jt, int ctas) {
    St3Geom g{};
    g.ok = hi[0] >= lo[0] && hi[1] >= lo[1] && hi[2] >= lo[2] && lo[2] >= 0;
    if (!g.ok) return g;
    g.p0 = lo[2] >> 1;
    const long gx = ((hi[2] >> 1) - g.p0 + TX) / TX, gy = (hi[1] - lo[1] + TY * jt) / (TY * jt);
    const long ni = hi[0] - lo[0] + 1, resident = (long)smCount() * ctas, tiles = gx * gy;
    const long most = ni < 65535 ? ni : 65535;  // chunks
    const long first = (tiles + resident - 1) / resident;
    long best = ni, bestCost = first * (ni + 4);
    // (64 rounds more: further chunks only add their first planes)
    for (long rounds = first; rounds * 5 < bestCost && rounds <= first + 64; rounds++) {
        const long fit = rounds * resident / tiles, n = (ni + (fit < most ? fit : most) - 1) / (fit < most ? fit : most);
        const long cost = (tiles * ((ni + n - 1) / n) + resident - 1) / resident * (n + 4);
        if (cost < bestCost) bestCost = cost, best = n;
    }
    g.ichunk = (int)best;
    const long gz = (ni + best - 1) / best;
    g.ok = gx < 65536 && gy < 65536 && gz < 65536;
    g.grid = dim3((unsigned)gx, (unsigned)gy, (unsigned)gz);
    return g;
}
