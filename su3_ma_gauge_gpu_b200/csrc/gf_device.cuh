// gf_device.cuh -- device-side building blocks of the B200 gauge-fixing sweep.
//
// SU(3) links live in registers as 3x3 complex matrices; only rows 0 and 1 travel to and from
// HBM, row 2 is rebuilt in registers (the reference's 12-parameter trick, lattice/SU3.hxx:639-676).
// A site update is done by FOUR lanes of a warp, one per direction mu: each lane holds the
// up link U_mu(x) and the down link U_mu(x-mu), so the 8 links of a site are spread over 4 lanes
// and the SU(2) subgroup sums are combined with two warp-shuffle butterflies (xor 8, xor 16)
// instead of the reference's shared-memory atomics and __syncthreads rounds
// (gaugefixing/GaugeFixingSubgroupStep.hxx:74-237).  The butterfly gives every lane of a site a
// bit-identical sum, so all four lanes compute the same SU(2) element without a broadcast.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gfb {

// gauge and algorithm codes: the gauge order is the reference's enum GaugeType
// (lattice/datatype/lattice_typedefs.h:43)
enum Gauge : int { LANDAU = 0, COULOMB = 1, MAG = 2, U1XU1 = 3 };
enum Algo : int { ALG_OR = 0, ALG_MICRO = 1, ALG_SA = 2, ALG_SR = 3, ALG_RANDOM = 4 };

template <typename R>
struct Cx {
    R x, y;
};

template <typename R>
__device__ __forceinline__ Cx<R> cx(R x, R y) { return Cx<R>{x, y}; }
template <typename R>
__device__ __forceinline__ Cx<R> cmul(Cx<R> a, Cx<R> b) { return cx<R>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
template <typename R>
__device__ __forceinline__ Cx<R> cmulcc(Cx<R> a, Cx<R> b)  // conj(a) * conj(b)
{
    return cx<R>(a.x * b.x - a.y * b.y, -(a.x * b.y + a.y * b.x));
}
template <typename R>
__device__ __forceinline__ R abs2(Cx<R> a) { return a.x * a.x + a.y * a.y; }

__device__ __forceinline__ float rsq(float x) { return rsqrtf(x); }
__device__ __forceinline__ double rsq(double x) { return rsqrt(x); }
__device__ __forceinline__ float sq(float x) { return sqrtf(x); }
__device__ __forceinline__ double sq(double x) { return sqrt(x); }
__device__ __forceinline__ float lg(float x) { return logf(x); }
__device__ __forceinline__ double lg(double x) { return log(x); }
__device__ __forceinline__ float cpi(float x) { return cospif(x); }
__device__ __forceinline__ double cpi(double x) { return cospi(x); }
__device__ __forceinline__ float spi(float x) { return sinpif(x); }
__device__ __forceinline__ double spi(double x) { return sinpi(x); }

template <typename R>
struct Link {
    Cx<R> e[3][3];
};

// row 2 = conj(row0 x row1), normalised (SU3::reconstructThirdLine, lattice/SU3.hxx:655-664)
template <typename R>
__device__ __forceinline__ void reconstruct(Link<R> &L)
{
    Cx<R> a = cmulcc(L.e[0][1], L.e[1][2]), a2 = cmulcc(L.e[0][2], L.e[1][1]);
    Cx<R> b = cmulcc(L.e[0][2], L.e[1][0]), b2 = cmulcc(L.e[0][0], L.e[1][2]);
    Cx<R> c = cmulcc(L.e[0][0], L.e[1][1]), c2 = cmulcc(L.e[0][1], L.e[1][0]);
    a.x -= a2.x; a.y -= a2.y;
    b.x -= b2.x; b.y -= b2.y;
    c.x -= c2.x; c.y -= c2.y;
    R n = rsq(abs2(a) + abs2(b) + abs2(c));
    L.e[2][0] = cx<R>(a.x * n, a.y * n);
    L.e[2][1] = cx<R>(b.x * n, b.y * n);
    L.e[2][2] = cx<R>(c.x * n, c.y * n);
}

template <typename R>
__device__ __forceinline__ void unpack12(Link<R> &L, const R r[12])
{
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) L.e[i][j] = cx<R>(r[2 * (3 * i + j)], r[2 * (3 * i + j) + 1]);
}

template <typename R>
__device__ __forceinline__ void pack12(const Link<R> &L, R r[12])
{
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            r[2 * (3 * i + j)] = L.e[i][j].x;
            r[2 * (3 * i + j) + 1] = L.e[i][j].y;
        }
}

// SU(2) quaternion q of the (I,J) 2x2 block, unnormalised (SU3::getSubgroupQuaternion,
// lattice/SU3.hxx:193-217); the SU(2) <-> 2x2 map is Quaternion::get (Quaternion.hxx:100-131):
// [[q0+i q3, q2+i q1], [-q2+i q1, q0-i q3]]
template <int I, int J, typename R>
__device__ __forceinline__ void subq(const Link<R> &L, R q[4])
{
    q[0] = L.e[I][I].x + L.e[J][J].x;
    q[3] = L.e[I][I].y - L.e[J][J].y;
    q[2] = L.e[I][J].x - L.e[J][I].x;
    q[1] = L.e[I][J].y + L.e[J][I].y;
}

// rows (I,J) <- g * rows (SU3::leftSubgroupMult, lattice/SU3.hxx:702-714)
template <int I, int J, typename R>
__device__ __forceinline__ void left_mult(Link<R> &L, const R g[4])
{
    const Cx<R> g00 = cx<R>(g[0], g[3]), g01 = cx<R>(g[2], g[1]);
    const Cx<R> g10 = cx<R>(-g[2], g[1]), g11 = cx<R>(g[0], -g[3]);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        Cx<R> a = cmul(g00, L.e[I][k]), b = cmul(g01, L.e[J][k]);
        Cx<R> c = cmul(g10, L.e[I][k]), d = cmul(g11, L.e[J][k]);
        L.e[I][k] = cx<R>(a.x + b.x, a.y + b.y);
        L.e[J][k] = cx<R>(c.x + d.x, c.y + d.y);
    }
}

// cols (I,J) <- cols * h (SU3::rightSubgroupMult, lattice/SU3.hxx:682-697)
template <int I, int J, typename R>
__device__ __forceinline__ void right_mult(Link<R> &L, const R h[4])
{
    const Cx<R> h00 = cx<R>(h[0], h[3]), h01 = cx<R>(h[2], h[1]);
    const Cx<R> h10 = cx<R>(-h[2], h[1]), h11 = cx<R>(h[0], -h[3]);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        Cx<R> a = cmul(h00, L.e[k][I]), b = cmul(h10, L.e[k][J]);
        Cx<R> c = cmul(h01, L.e[k][I]), d = cmul(h11, L.e[k][J]);
        L.e[k][I] = cx<R>(a.x + b.x, a.y + b.y);
        L.e[k][J] = cx<R>(c.x + d.x, c.y + d.y);
    }
}

// ---- Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11) ---------------------------------------
__device__ __forceinline__ uint4 philox4x32_10_inline(uint4 c, uint2 k)
{
#pragma unroll
    for (int r = 0; r < 10; r++) {
        if (r > 0) {
            k.x += 0x9E3779B9u;
            k.y += 0xBB67AE85u;
        }
        const uint32_t lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
        const uint32_t lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
        c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    }
    return c;
}
// Out of line for the draws off the common path and the rules that draw at several places: copies of
// the ten rounds at each of them make a kernel's code outgrow the instruction cache.
static __device__ __noinline__ uint4 philox4x32_10(uint4 c, uint2 k) { return philox4x32_10_inline(c, k); }

// The reference's per-thread generator (lattice/rng/PhiloxWrapper.hxx:92-137): key = (tid, seed),
// counter = (k, launch counter, 0x12345678, 0xabcdef09), the k = 0 block discarded; floats are
// drawn i[3], i[2], i[1], i[0] from each block, doubles i64[1], i64[0].
template <typename R>
struct Rng {
    uint2 key;
    uint4 ctr;
    uint4 res;
    int local;
    uint32_t drawn;  // numbers drawn so far, for the heat bath, which addresses its draws by index
    __device__ __forceinline__ void init(uint32_t tid, uint32_t seed, uint32_t counter)
    {
        key = make_uint2(tid, seed);
        ctr = make_uint4(0u, counter, 0x12345678u, 0xabcdef09u);
        local = 0;
        drawn = 0;
    }
    __device__ __forceinline__ R rand();
};

// u01_open_open_32_24 / _64_53 of Random123's u01.h: (1 + (i >> 8)) * 0x1.fffffep-25f and
// (1 + (i >> 11)) * 0x1.fffffffffffffp-54
template <>
__device__ __forceinline__ float Rng<float>::rand()
{
    if (local == 0) {
        local = 3;
        ctr.x++;
        res = philox4x32_10(ctr, key);
    } else {
        local--;
    }
    const uint32_t v = local == 3 ? res.w : (local == 2 ? res.z : (local == 1 ? res.y : res.x));
    return (float)(1u + (v >> 8)) * 0x1.fffffep-25f;
}

template <>
__device__ __forceinline__ double Rng<double>::rand()
{
    if (local == 0) {
        local = 1;
        ctr.x++;
        res = philox4x32_10(ctr, key);
    } else {
        local--;
    }
    const uint64_t v = local == 1 ? (((uint64_t)res.w << 32) | res.z) : (((uint64_t)res.y << 32) | res.x);
    return (double)(1ull + (v >> 11)) * 0x1.fffffffffffffp-54;
}

// ---- update rules on the accumulated 4-vector (gaugefixing/algorithms/*Update.hxx) ----------
struct AlgoParams {
    float param;      // OR omega, SA temperature, SR probability
    uint32_t seed;
    uint32_t counter;
    uint32_t counter_stride;  // batches: 0 = instance i draws key word seed + i; > 0 = every instance draws
                              // key word seed, instance i from launch counter counter + i * counter_stride
};

// Philox key word and launch counter of instance i of a batch.  By default every instance has a
// stream of its own (key word seed + i, the same counters).  With counter_stride > 0 the instances
// continue one stream, as the reference apps do when they fix gauge copies or timeslices one after
// the other (PhiloxWrapper::getNextCounter is one process-wide counter, lattice/rng/PhiloxWrapper.hxx:
// 90,142-145): key word seed, instance i starting counter_stride launches after instance i - 1.
__host__ __device__ __forceinline__ uint32_t inst_seed(const AlgoParams &p, int i)
{
    return p.counter_stride ? p.seed : p.seed + (uint32_t)i;
}
__host__ __device__ __forceinline__ uint32_t inst_counter(const AlgoParams &p, int i)
{
    return p.counter + (uint32_t)i * p.counter_stride;
}

// OrUpdate::calculateUpdate (OrUpdate.hxx:66-75)
template <typename R>
__device__ __forceinline__ void upd_or(R a[4], float omega)
{
    const R ai_sq = a[1] * a[1] + a[2] * a[2] + a[3] * a[3];
    const R a0_sq = a[0] * a[0];
    if (!(a0_sq + ai_sq > (R)0)) {  // no coupling (every contribution cancelled): leave the site
        a[0] = 1;
        a[1] = a[2] = a[3] = 0;
        return;
    }
    const R b = (omega * a0_sq + ai_sq) / (a0_sq + ai_sq);
    const R c = rsq(a0_sq + b * b * ai_sq);
    const R bc = b * c;
    a[0] *= c;
    a[1] *= bc;
    a[2] *= bc;
    a[3] *= bc;
}

// MicroUpdate::calculateUpdate (MicroUpdate.hxx:55-64)
template <typename R>
__device__ __forceinline__ void upd_micro(R a[4])
{
    const R ai_sq = a[1] * a[1] + a[2] * a[2] + a[3] * a[3];
    const R a0_sq = a[0] * a[0];
    const R n = a0_sq + ai_sq;
    if (!(n > (R)0)) {  // no coupling: the reflection is undefined, leave the site
        a[0] = 1;
        a[1] = a[2] = a[3] = 0;
        return;
    }
    const R b = (R)2. * a[0] / n;
    a[0] = (a0_sq - ai_sq) / n;
    a[1] *= b;
    a[2] *= b;
    a[3] *= b;
}

// ---- heat bath ---------------------------------------------------------------------------------
// Number n (0, 1, 2, ...) of a site's stream is word pair / word 3 - n % 4 (doubles: the upper, then
// the lower half) of Philox block 1 + n / (numbers per block), so any lane can draw any number.
__device__ __forceinline__ float draw_word(const uint4 &b, uint32_t j, float)
{
    const uint32_t v = j == 0 ? b.w : (j == 1 ? b.z : (j == 2 ? b.y : b.x));
    return (float)(1u + (v >> 8)) * 0x1.fffffep-25f;
}
__device__ __forceinline__ double draw_word(const uint4 &b, uint32_t j, double)
{
    const uint64_t v = j == 0 ? (((uint64_t)b.w << 32) | b.z) : (((uint64_t)b.y << 32) | b.x);
    return (double)(1ull + (v >> 11)) * 0x1.fffffffffffffp-54;
}
template <typename R>
struct PerBlock {
    static constexpr uint32_t log2 = sizeof(R) == 4 ? 2 : 1, mask = (1u << log2) - 1u;
};

// HOT: with the rounds in line.  The two-lane layout has one copy of the heat bath and gains from it
// (32^4, FP32 Landau / U1xU1: 146 / 234 us per pass against 150 / 258 us); the four-lane layout has
// three and waits for instructions then.
template <typename R, bool HOT = false>
__device__ __forceinline__ uint4 draw_block(uint2 key, uint32_t counter, uint32_t n)
{
    const uint4 c = make_uint4(1u + (n >> PerBlock<R>::log2), counter, 0x12345678u, 0xabcdef09u);
    return HOT ? philox4x32_10_inline(c, key) : philox4x32_10(c, key);
}
template <typename R>
__device__ __forceinline__ R draw_at(uint2 key, uint32_t counter, uint32_t n)
{
    return draw_word(draw_block<R>(key, counter, n), n & PerBlock<R>::mask, R());
}

// numbers n and n + 1; usually in one block
template <typename R, bool HOT = false>
__device__ __forceinline__ void draw_two(uint2 key, uint32_t counter, uint32_t n, R u[2])
{
    const uint4 b = draw_block<R, HOT>(key, counter, n);
    const uint32_t j = n & PerBlock<R>::mask;
    u[0] = draw_word(b, j, R());
    u[1] = j == PerBlock<R>::mask ? draw_at<R>(key, counter, n + 1) : draw_word(b, j + 1, R());
}

// numbers n .. n + 3: one or two blocks of floats, two (three for odd n) of doubles
template <bool HOT>
__device__ __forceinline__ void draw_four(uint2 key, uint32_t counter, uint32_t n, float u[4])
{
    const uint4 b = draw_block<float, HOT>(key, counter, n);
    const uint32_t j = n & 3u;
    uint4 c = b;
    if (j) c = draw_block<float>(key, counter, n + 4);
#pragma unroll
    for (uint32_t k = 0; k < 4; k++) u[k] = j + k < 4 ? draw_word(b, j + k, 0.f) : draw_word(c, j + k - 4, 0.f);
}
template <bool HOT>
__device__ __forceinline__ void draw_four(uint2 key, uint32_t counter, uint32_t n, double u[4])
{
    draw_two<double, HOT>(key, counter, n, u);
    draw_two<double, HOT>(key, counter, n + 2, u + 2);
}

// One trial of the Kennedy-Pendleton rejection loop, its draws starting at number n (SaUpdate.hxx:
// 103-128).  The literal types follow the reference (double constants, cospi of a double argument),
// so the FP32 variant promotes where the reference promotes.  Returns the acceptance; `used` is the
// number of draws, 4 unless a number below 0.0001 was drawn again (2e-4 of the trials).
template <typename R, bool HOT>
__device__ __forceinline__ bool kp_trial(uint2 key, uint32_t counter, uint32_t n, R p0, R &delta, uint32_t &used)
{
    R u[4];
    draw_four<HOT>(key, counter, n, u);
    used = 4;
    if (u[0] < 0.0001 || u[1] < 0.0001) {
        uint32_t q = n;
        int g1 = 0, g2 = 0;
        do { u[0] = draw_at<R>(key, counter, q++); } while (u[0] < 0.0001 && ++g1 < 65536);
        do { u[1] = draw_at<R>(key, counter, q++); } while (u[1] < 0.0001 && ++g2 < 65536);
        u[2] = draw_at<R>(key, counter, q++);
        u[3] = draw_at<R>(key, counter, q++);
        used = q - n;
    }
    const R r1 = -lg(u[0]) * p0;
    const R r2 = -lg(u[1]) * p0;
    R r3 = (R)cospi(2.0 * (double)u[2]);
    r3 = r3 * r3;
    delta = r2 + r1 * r3;
    const R r4 = u[3];
    return !(r4 * r4 > (1.0 - 0.5 * delta));
}

// position of set bit number g (0-based) of mask, g < popc(mask)
__device__ __forceinline__ int nth_bit(uint32_t mask, int g)
{
    int pos = 0;
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
        const int c = __popc((mask >> pos) & ((1u << w) - 1u));
        if (g >= c) {
            g -= c;
            pos += w;
        }
    }
    return pos;
}

constexpr uint32_t kMaxTrials = 65536;  // bound of a site's rejection loop
constexpr int kScreenRound = 8;         // rounds of shared trials before the sites left are screened

// The rest of the loop of one site, all arguments the same in every lane: rows of 32 trials, four at
// a time.  delta >= r2 = -ln(u1) p0, and delta > 2 is never accepted, so where p0 is large nearly
// every trial is decided by its second number alone: u1 < exp(-2 / p0) (less a margin that covers
// the rounding of r2) and neither of the first two numbers drawn again.  Only the other trials are
// evaluated, in order.  Such a site often runs into the bound, 2048 rows.
template <typename R, bool HOT>
__device__ __forceinline__ bool kp_screened(uint2 key, uint32_t counter, R p0, R &delta, uint32_t &n, uint32_t &trials)
{
    constexpr uint32_t full = 0xffffffffu;
    constexpr int rows = 4;
    const int lane = threadIdx.x & 31;
    const float bar = p0 > (R)1 && p0 < (R)1e30 ? expf(-2.f / (float)p0) - 1e-5f : 0.f;
    while (trials < kMaxTrials) {
        uint32_t open[rows];
#pragma unroll
        for (int q = 0; q < rows; q++) {
            const uint32_t k = 32u * q + lane;
            R u[2];
            draw_two<R, HOT>(key, counter, n + 4u * k, u);
            const bool rejected = !(u[0] < 0.0001) && !(u[1] < 0.0001) && (float)u[1] < bar;
            open[q] = __ballot_sync(full, !rejected && trials + k < kMaxTrials);
        }
        uint32_t steps = min(32u * rows, kMaxTrials - trials), drawn = 4u * steps;
        bool accepted = false, ended = false;
#pragma unroll 1
        for (int q = 0; q < rows && !ended; q++) {
            const uint32_t row = q == 0 ? open[0] : (q == 1 ? open[1] : (q == 2 ? open[2] : open[3]));
            if (!row) continue;
            R d = 0;
            uint32_t used = 4;
            bool acc = false;
            if ((row >> lane) & 1u) acc = kp_trial<R, HOT>(key, counter, n + 4u * (32u * q + lane), p0, d, used);
            const uint32_t ends = __ballot_sync(full, acc || used != 4);
            if (!ends) continue;
            const int f = __ffs(ends) - 1;
            ended = true;
            accepted = __shfl_sync(full, (int)acc, f);
            delta = __shfl_sync(full, d, f);
            steps = 32u * q + f + 1;
            drawn = 4u * (steps - 1) + __shfl_sync(full, used, f);
        }
        n += drawn;
        trials += steps;
        if (accepted) return true;
    }
    return false;
}

// The rejection loops of the S sites of a warp (site lane & (S - 1)), all 32 lanes together.  A
// site's trials are independent given where their draws start, and trial k starts 4 draws after trial
// k - 1 unless that one drew a number again.  So the lanes evaluate consecutive trials of the sites
// still looping, 32 / (such sites) each, and every site takes its first accepted trial; a trial that
// drew again ends the run of known starts, and the site goes on behind it.  The result is what one
// lane per site computes, draw for draw, but a warp loops for its total number of trials over 32
// instead of its slowest site's number.
// pending: this lane's site wants a trial.  Returns whether a trial was accepted within the bound;
// delta and n (draws used so far) are updated.
template <typename R, int S>
__device__ __forceinline__ bool kp_warp(bool pending, uint2 key, uint32_t counter, R p0, R &delta, uint32_t &n)
{
    static_assert(S == 8 || S == 16, "four or two lanes per site");
    constexpr uint32_t full = 0xffffffffu, sites = (1u << S) - 1u;
    const int lane = threadIdx.x & 31, site = lane & (S - 1);
    bool accepted = false;
    uint32_t trials = 0;
    uint32_t need = __ballot_sync(full, pending) & sites;
    for (int round = 0; need && round < kScreenRound; round++) {
        // this lane's trial: number m of the site whose draws these are.  In the first round every site
        // takes its own lanes; after it the lanes are shared out again.
        R ps = p0;
        uint2 ks = key;
        uint32_t cs = counter, ns = n, ts = trials;
        int m = lane / S, shift = 0;
        bool active = pending;
        if (round > 0) {
            const int count = __popc(need);
            shift = __clz(count - 1) - 27;  // 32 >> ceil(log2 count) lanes for each of them
            const int mine = lane >> shift, src = nth_bit(need, mine < count ? mine : 0);
            m = lane & ((1 << shift) - 1);
            ps = __shfl_sync(full, p0, src);
            ks = make_uint2(__shfl_sync(full, key.x, src), __shfl_sync(full, key.y, src));
            cs = __shfl_sync(full, counter, src);
            ns = __shfl_sync(full, n, src);
            ts = __shfl_sync(full, trials, src);
            active = mine < count && ts + m < kMaxTrials;
        }
        R d = 0;
        uint32_t used = 4;
        bool acc = false;
        if (active) acc = kp_trial<R, S == 16>(ks, cs, ns + 4u * m, ps, d, used);
        const uint32_t accs = __ballot_sync(full, acc), again = __ballot_sync(full, used != 4), ends = accs | again;
        // the first trial of this lane's site that ends its run, and the lane that evaluated it
        uint32_t seg, per;
        int first, from;
        if (round > 0) {
            const int base = (__popc(need & ((1u << site) - 1u)) << shift) & 31;  // (sites done: any lane)
            per = 1u << shift;
            seg = (ends >> base) & (per == 32 ? full : (1u << per) - 1u);
            first = seg ? __ffs(seg) - 1 : 0;
            from = base + first;
        } else {
            per = 32 / S;
            seg = (ends >> site) & (S == 16 ? 0x00010001u : 0x01010101u);
            const int bit = seg ? __ffs(seg) - 1 : 0;
            first = bit / S;
            from = site + bit;
        }
        const R df = __shfl_sync(full, d, from);
        const uint32_t uf = again ? __shfl_sync(full, used, from) : 4u;
        if (pending) {
            if (seg) {
                n += 4u * first + uf;
                trials += first + 1;
                if ((accs >> from) & 1u) {
                    accepted = true;
                    delta = df;
                }
            } else {
                const uint32_t done = min(per, kMaxTrials - trials);
                n += 4u * done;
                trials += done;
            }
            pending = !accepted && trials < kMaxTrials;
        }
        need = __ballot_sync(full, pending) & sites;
    }
    while (need) {
        const int src = __ffs(need) - 1;
        need &= need - 1;
        R d = 0;
        uint32_t ns = __shfl_sync(full, n, src), ts = __shfl_sync(full, trials, src);
        const bool acc = kp_screened<R, S == 16>(make_uint2(__shfl_sync(full, key.x, src), __shfl_sync(full, key.y, src)),
                                        __shfl_sync(full, counter, src), __shfl_sync(full, p0, src), d, ns, ts);
        if (site == src) {
            n = ns;
            accepted = acc;
            delta = d;
        }
    }
    return accepted;
}

// Kennedy-Pendleton heat bath, SaUpdate::calculateUpdate (SaUpdate.hxx:103-146), by all lanes of a
// warp that holds S sites.  A site's loop is bounded (2^16 trials): its acceptance is rare when
// p0 = T/|a| is large (a subgroup coupling |a| tiny against the temperature), and there the
// reference would keep drawing.  Such a site -- the bound exhausted, or |a| = 0 -- takes a0 from the
// p0 -> infinity limit of the same distribution, the Haar measure (density proportional to
// sqrt(1 - a0^2), sampled by rejection), instead of the unaccepted 1 - delta, whose square root below
// would be NaN for delta > 2.
template <typename R, int S>
__device__ __forceinline__ void upd_sa(R a[4], float temperature, Rng<R> &rng)
{
    const uint2 key = rng.key;
    const uint32_t counter = rng.ctr.y;
    uint32_t n = rng.drawn;
    R e0 = a[0], e1 = -a[1], e2 = -a[2], e3 = -a[3];
    const R nrm2 = e0 * e0 + e1 * e1 + e2 * e2 + e3 * e3;
    const bool flat = !(nrm2 > (R)0);  // no coupling: the local distribution is Haar
    const R dk = flat ? (R)1 : rsq(nrm2);
    if (flat) {
        e0 = 1;
        e1 = e2 = e3 = 0;
    }
    R delta = 0;
    const bool accepted = kp_warp<R, S>(!flat, key, counter, dk * temperature, delta, n);
    R a0 = (R)(1.0 - delta);
    if (!accepted) {
        int g = 0;
        R r4;
        do {
            a0 = (R)(2.0 * draw_at<R>(key, counter, n) - 1.0);
            r4 = draw_at<R>(key, counter, n + 1);
            n += 2;
        } while (r4 * r4 > (R)1 - a0 * a0 && ++g < 64);
    }
    R u[2];
    draw_two<R, S == 16>(key, counter, n, u);
    rng.drawn = n + 2;
    const R cos_theta = (R)(2.0 * u[0] - 1.0);
    const R sin_theta = (R)sqrt(1.0 - (double)(cos_theta * cos_theta));
    const R sin_alpha = sq((R)(1 - a0 * a0));
    const R phi = (R)(2.0 * u[1]);
    const R a1 = sin_alpha * sin_theta * cpi(phi);
    const R a2 = sin_alpha * sin_theta * spi(phi);
    const R a3 = sin_alpha * cos_theta;
    e0 *= dk;
    e1 *= dk;
    e2 *= dk;
    e3 *= dk;
    a[0] = a0 * e0 + a3 * e3 + a2 * e2 + e1 * a1;
    a[3] = e0 * a3 - e3 * a0 + a1 * e2 - a2 * e1;
    a[2] = a3 * e1 - a0 * e2 + a2 * e0 - a1 * e3;
    a[1] = a2 * e3 + a1 * e0 - a3 * e2 - e1 * a0;
}

// SrUpdate::calculateUpdate (SrUpdate.hxx:76-94): with probability p square the quaternion
template <typename R>
__device__ __forceinline__ void upd_sr(R a[4], float p, Rng<R> &rng)
{
    const R u = rng.rand();
    const R a0 = a[0], a1 = a[1], a2 = a[2], a3 = a[3];
    if (u < p) {
        a[0] = a0 * a0 - a1 * a1 - a2 * a2 - a3 * a3;
        a[1] = (R)(2.0 * a0 * a1);
        a[2] = (R)(2.0 * a0 * a2);
        a[3] = (R)(2.0 * a0 * a3);
    }
    const R c = rsq(a[0] * a[0] + a[1] * a[1] + a[2] * a[2] + a[3] * a[3]);
    a[0] *= c;
    a[1] *= c;
    a[2] *= c;
    a[3] *= c;
}

// RandomUpdate::calculateUpdate (RandomUpdate.hxx:47-59): uniform random SU(2) element
template <typename R>
__device__ __forceinline__ void upd_random(R a[4], Rng<R> &rng)
{
    const R alpha = rng.rand();
    const R phi = (R)(2.0 * rng.rand());
    const R cos_theta = (R)(2.0 * rng.rand() - 1.0);
    const R sin_theta = (R)sqrt(1.0 - (double)(cos_theta * cos_theta));
    const R sin_alpha = spi(alpha);
    a[0] = cpi(alpha);
    a[1] = sin_alpha * sin_theta * cpi(phi);
    a[2] = sin_alpha * sin_theta * spi(phi);
    a[3] = sin_alpha * cos_theta;
}

// S: sites per warp of the calling layout (the heat bath runs its sites' loops on all 32 lanes, so
// the whole warp must call it together)
template <int ALGO, int S, typename R>
__device__ __forceinline__ void apply_algo(R a[4], const AlgoParams &p, Rng<R> &rng)
{
    if constexpr (ALGO == ALG_OR) upd_or(a, p.param);
    else if constexpr (ALGO == ALG_MICRO) upd_micro(a);
    else if constexpr (ALGO == ALG_SA) upd_sa<R, S>(a, p.param, rng);
    else if constexpr (ALGO == ALG_SR) upd_sr(a, p.param, rng);
    else upd_random(a, rng);
}

// sum over the four lanes of one site (lanes l, l^8, l^16, l^24); the butterfly leaves the same
// bits in all four lanes
template <typename R>
__device__ __forceinline__ R site_sum(R v)
{
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 16);
    return v;
}

// One SU(2) subgroup step of GaugeFixingSubgroupStep::subgroup for the gauge GAUGE, done by the
// lane that holds direction mu of the site (LANDAU/COULOMB :99-237, U1xU1 :238-353, MAG :354-589).
// Refine mode: column k of D = W - 1, the deviation of the site's accumulated gauge
// transformation from the identity, under W <- g W:  D' = D + (g - 1)(1 + D) on rows (I, J).
// g - 1 is formed without cancellation (g0 - 1 = -|g_vec|^2 / (1 + g0)), so near convergence, where
// the folds keep W close to 1, D carries the small rotations to FP32 relative accuracy instead of
// rounding them against the unit diagonal.
template <int I, int J, typename R>
__device__ __forceinline__ void left_mult_dcolumn(Cx<R> (&col)[3], const R g[4], int k)
{
    const R v2 = g[1] * g[1] + g[2] * g[2] + g[3] * g[3];
    const R em = g[0] >= (R)0 ? -v2 / ((R)1 + g[0]) : g[0] - (R)1;
    const Cx<R> a = cx<R>(col[I].x + (k == I ? (R)1 : (R)0), col[I].y);
    const Cx<R> b = cx<R>(col[J].x + (k == J ? (R)1 : (R)0), col[J].y);
    const Cx<R> p0 = cmul(cx<R>(em, g[3]), a), p1 = cmul(cx<R>(g[2], g[1]), b);
    const Cx<R> q0 = cmul(cx<R>(-g[2], g[1]), a), q1 = cmul(cx<R>(em, -g[3]), b);
    col[I] = cx<R>(col[I].x + (p0.x + p1.x), col[I].y + (p0.y + p1.y));
    col[J] = cx<R>(col[J].x + (q0.x + q1.x), col[J].y + (q0.y + q1.y));
}

// Contribution of direction mu (its up link U_mu(x) and down link U_mu(x-mu)) to the subgroup
// quaternion w of the site, before the sum over mu (GaugeFixingSubgroupStep.hxx:99-237 Landau and
// Coulomb, :238-353 U1xU1, :354-589 MAG; MAG's factor 2 and square root follow the sum).
template <int GAUGE, int I, int J, typename R>
__device__ __forceinline__ void subgroup_contrib(const Link<R> &up, const Link<R> &dn, int mu, R v[4])
{
    if (GAUGE == MAG) {
        const Cx<R> u00 = up.e[I][I], u01 = up.e[I][J], u10 = up.e[J][I], u11 = up.e[J][J];
        const Cx<R> d00 = dn.e[I][I], d01 = dn.e[I][J], d10 = dn.e[J][I], d11 = dn.e[J][J];
        const R Du = abs2(u00) - abs2(u01) - abs2(u10) + abs2(u11);
        const R Dd = abs2(d00) - abs2(d01) - abs2(d10) + abs2(d11);
        // up:   c = m00 conj(m10) - m01 conj(m11);  down: c = conj(m00) m01 - conj(m10) m11
        const R cux = (u00.x * u10.x + u00.y * u10.y) - (u01.x * u11.x + u01.y * u11.y);
        const R cuy = (u00.y * u10.x - u00.x * u10.y) - (u01.y * u11.x - u01.x * u11.y);
        const R cdx = (d00.x * d01.x + d00.y * d01.y) - (d10.x * d11.x + d10.y * d11.y);
        const R cdy = (d00.x * d01.y - d00.y * d01.x) - (d10.x * d11.y - d10.y * d11.x);
        v[0] = Du + Dd;
        v[1] = cuy + cdy;
        v[2] = cux + cdx;
        v[3] = 0;
    } else {
        R qu[4], qd[4];
        subq<I, J>(up, qu);
        subq<I, J>(dn, qd);
        const bool skip = (GAUGE == COULOMB) && (mu == 0);  // Coulomb: mu = 0 not in the sum
        if (GAUGE == U1XU1) {
            v[0] = qu[0] + qd[0];
            v[1] = 0;
            v[2] = 0;
            v[3] = qd[3] - qu[3];
        } else {
            v[0] = skip ? (R)0 : qu[0] + qd[0];
            v[1] = skip ? (R)0 : qd[1] - qu[1];
            v[2] = skip ? (R)0 : qd[2] - qu[2];
            v[3] = skip ? (R)0 : qd[3] - qu[3];
        }
    }
}

// From the summed quaternion to the update g (in place): MAG's factor 2 and square root, the
// update rule, and the U1xU1 / MAG renormalisation.
template <int GAUGE, int ALGO, int S, typename R>
__device__ __forceinline__ void subgroup_finish(R w[4], const AlgoParams &p, Rng<R> &rng)
{
    if (GAUGE == MAG) {
        w[1] *= (R)2.;  // the factor 2 of GaugeFixingSubgroupStep.hxx:535-536
        w[2] *= (R)2.;
        w[3] = 0;
        w[0] = w[0] + sq(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
    } else if (GAUGE == U1XU1) {
        w[1] = 0;
        w[2] = 0;
    }
    apply_algo<ALGO, S>(w, p, rng);
    if (GAUGE == U1XU1) {
        w[1] = 0;
        w[2] = 0;
        const R n = rsq(w[0] * w[0] + w[3] * w[3]);
        w[0] *= n;
        w[3] *= n;
    } else if (GAUGE == MAG) {
        w[3] = 0;
        const R n = rsq(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
        w[0] *= n;
        w[1] *= n;
        w[2] *= n;
    }
}

template <int GAUGE, int ALGO, int I, int J, typename R, bool SITE_W = false>
__device__ __forceinline__ void subgroup_step(Link<R> &up, Link<R> &dn, int mu, const AlgoParams &p, Rng<R> &rng,
                                              Cx<R> (*wcol)[3] = nullptr)
{
    R v[4], w[4];
    subgroup_contrib<GAUGE, I, J>(up, dn, mu, v);
    w[0] = site_sum(v[0]);
    w[1] = (GAUGE == U1XU1) ? (R)0 : site_sum(v[1]);
    w[2] = (GAUGE == U1XU1) ? (R)0 : site_sum(v[2]);
    w[3] = (GAUGE == MAG) ? (R)0 : site_sum(v[3]);
    subgroup_finish<GAUGE, ALGO, 8>(w, p, rng);
    left_mult<I, J>(up, w);
    const R h[4] = {w[0], -w[1], -w[2], -w[3]};
    right_mult<I, J>(dn, h);
    if (SITE_W) left_mult_dcolumn<I, J>(*wcol, w, mu & 1);
}

// One thread per site: the same subgroup step with all 8 links of the site in the thread.  The
// sum over mu is taken in the order of the 4-lane butterfly, (v0 + v1) + (v2 + v3), so both
// layouts do the same arithmetic (the compiler may still contract a product differently in the
// two kernels).  With SITE_W the thread applies g to both tracked columns of D = W - 1.
template <int GAUGE, int ALGO, int I, int J, typename R, bool SITE_W = false>
__device__ __forceinline__ void subgroup_step_site(Link<R> (&up)[4], Link<R> (&dn)[4], const AlgoParams &p,
                                                   Rng<R> &rng, Cx<R> (*wcols)[2][3] = nullptr)
{
    static_assert(ALGO != ALG_SA, "the heat bath runs with two or four lanes per site");
    R v[4][4], w[4];
#pragma unroll
    for (int mu = 0; mu < 4; mu++) subgroup_contrib<GAUGE, I, J>(up[mu], dn[mu], mu, v[mu]);
#pragma unroll
    for (int k = 0; k < 4; k++) w[k] = (v[0][k] + v[1][k]) + (v[2][k] + v[3][k]);
    if (GAUGE == U1XU1) w[1] = w[2] = 0;
    if (GAUGE == MAG) w[3] = 0;
    subgroup_finish<GAUGE, ALGO, 32>(w, p, rng);
    const R h[4] = {w[0], -w[1], -w[2], -w[3]};
#pragma unroll
    for (int mu = 0; mu < 4; mu++) {
        left_mult<I, J>(up[mu], w);
        right_mult<I, J>(dn[mu], h);
    }
    if (SITE_W) {
        left_mult_dcolumn<I, J>((*wcols)[0], w, 0);
        left_mult_dcolumn<I, J>((*wcols)[1], w, 1);
    }
}

// Two lanes per site: lane `role` (0 or 1; its partner is lane ^ 16) holds directions 2*role and
// 2*role + 1, each as its up link U_mu(x) and down link U_mu(x - mu).  The quaternion sum is
// (v0 + v1) + (v2 + v3) -- the additions of the 4-lane butterfly, in the same order -- and both
// lanes compute the same g.  Each lane then updates its four links, and with SITE_W column `role`
// of the site's D = W - 1, so no lane repeats another's work except the SU(2) update itself.
template <int GAUGE, int I, int J, typename R>
__device__ __forceinline__ void subgroup_sum_pair(const Link<R> (&up)[2], const Link<R> (&dn)[2], int role, R w[4])
{
    R a[4], b[4];
    subgroup_contrib<GAUGE, I, J>(up[0], dn[0], 2 * role, a);
    subgroup_contrib<GAUGE, I, J>(up[1], dn[1], 2 * role + 1, b);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const bool zero = (GAUGE == U1XU1 && (k == 1 || k == 2)) || (GAUGE == MAG && k == 3);
        const R v = a[k] + b[k];
        w[k] = zero ? (R)0 : v + __shfl_xor_sync(0xffffffffu, v, 16);
    }
}
template <int I, int J, typename R, bool SITE_W>
__device__ __forceinline__ void subgroup_apply_pair(Link<R> (&up)[2], Link<R> (&dn)[2], int role, const R w[4],
                                                    Cx<R> (*wcol)[3])
{
    const R h[4] = {w[0], -w[1], -w[2], -w[3]};
#pragma unroll
    for (int j = 0; j < 2; j++) {
        left_mult<I, J>(up[j], w);
        right_mult<I, J>(dn[j], h);
    }
    if (SITE_W) left_mult_dcolumn<I, J>(*wcol, w, role);
}
template <int GAUGE, int ALGO, int I, int J, typename R, bool SITE_W>
__device__ __forceinline__ void subgroup_step_pair(Link<R> (&up)[2], Link<R> (&dn)[2], int role, const AlgoParams &p,
                                                   Rng<R> &rng, Cx<R> (*wcol)[3])
{
    R w[4];
    subgroup_sum_pair<GAUGE, I, J>(up, dn, role, w);
    subgroup_finish<GAUGE, ALGO, 16>(w, p, rng);
    subgroup_apply_pair<I, J, R, SITE_W>(up, dn, role, w, wcol);
}

template <int I_, int J_>
struct Pair {
    static constexpr int I = I_, J = J_;
};

// Calls f(Pair<I, J>()) for subgroup k in the reference order (0,2), (1,2), (0,1)
// (SU3::perSubgroup, SU3.hxx:762-771).
template <class F>
__device__ __forceinline__ void on_subgroup(int k, F f)
{
    if (k == 0) f(Pair<0, 2>());
    else if (k == 1) f(Pair<1, 2>());
    else f(Pair<0, 1>());
}

// The heat bath's code is larger than the rest of the update, so its three subgroup steps share one
// copy of it in a loop that is not unrolled; only the sums and the multiplications are there three times
// (three copies of the rejection loop made the pass wait for instructions more than for anything else).

template <int GAUGE, int ALGO, typename R, bool SITE_W = false>
__device__ __forceinline__ void site_update_pair(Link<R> (&up)[2], Link<R> (&dn)[2], int role, const AlgoParams &p,
                                                 Rng<R> &rng, Cx<R> (*wcol)[3] = nullptr)
{
    if constexpr (ALGO == ALG_SA) {
#pragma unroll 1
        for (int k = 0; k < 3; k++) {
            R w[4];
            on_subgroup(k, [&](auto s) { subgroup_sum_pair<GAUGE, s.I, s.J>(up, dn, role, w); });
            subgroup_finish<GAUGE, ALGO, 16>(w, p, rng);
            on_subgroup(k, [&](auto s) { subgroup_apply_pair<s.I, s.J, R, SITE_W>(up, dn, role, w, wcol); });
        }
        return;
    }
    subgroup_step_pair<GAUGE, ALGO, 0, 2, R, SITE_W>(up, dn, role, p, rng, wcol);
    subgroup_step_pair<GAUGE, ALGO, 1, 2, R, SITE_W>(up, dn, role, p, rng, wcol);
    subgroup_step_pair<GAUGE, ALGO, 0, 1, R, SITE_W>(up, dn, role, p, rng, wcol);
}

// the three subgroups in the reference order (0,2), (1,2), (0,1) (SU3::perSubgroup, SU3.hxx:762-771);
// with SITE_W the lane also applies every g to its column (mu & 1) of the site's D = W - 1
template <int GAUGE, int ALGO, typename R, bool SITE_W = false>
__device__ __forceinline__ void site_update(Link<R> &up, Link<R> &dn, int mu, const AlgoParams &p, Rng<R> &rng,
                                            Cx<R> (*wcol)[3] = nullptr)
{
    subgroup_step<GAUGE, ALGO, 0, 2, R, SITE_W>(up, dn, mu, p, rng, wcol);
    subgroup_step<GAUGE, ALGO, 1, 2, R, SITE_W>(up, dn, mu, p, rng, wcol);
    subgroup_step<GAUGE, ALGO, 0, 1, R, SITE_W>(up, dn, mu, p, rng, wcol);
}

template <int GAUGE, int ALGO, typename R, bool SITE_W = false>
__device__ __forceinline__ void site_update_thread(Link<R> (&up)[4], Link<R> (&dn)[4], const AlgoParams &p,
                                                   Rng<R> &rng, Cx<R> (*wcols)[2][3] = nullptr)
{
    subgroup_step_site<GAUGE, ALGO, 0, 2, R, SITE_W>(up, dn, p, rng, wcols);
    subgroup_step_site<GAUGE, ALGO, 1, 2, R, SITE_W>(up, dn, p, rng, wcols);
    subgroup_step_site<GAUGE, ALGO, 0, 1, R, SITE_W>(up, dn, p, rng, wcols);
}

// ---- two links at a time in packed FP32 arithmetic -------------------------------------------------
// The persistent FP32 passes with two lanes per site are bound by instruction issue (63 % of the issue
// slots, 1632 instructions per 16-site tile), and the multiplications of a lane's two up links, and
// of its two down links, by the same SU(2) element are the same instructions on different data.  Here
// the two links share float2 registers and every multiply and add of them is one packed instruction
// (FMUL2 / FFMA2 / FADD2): 39 M instructions per 32^4 pass instead of 53 M.  us per pass, scalar /
// packed: Coulomb 16 slices of 48^3 116.8 / 104.9, Landau 32^4 in FP32 storage 68.4 / 66.6 (6.05 TB/s).
// The persistent pass with W tracked gains nothing, 79.8 / 79.3 (MAG 48^4 393 / 415): there the register
// cap that buys 12 warps per SM leaves no room for the pairs, so it stays scalar; the direct pass with W, which
// holds no prefetched tile, is packed (87.9 / 78.3, 74.5 with the alternating walk).
// The products are added in the order the compiler gives the scalar functions
// above, (fma, product) + (fma, product), so the results are those of the other passes to the last bit.
struct Link2 {
    float2 x[3][3], y[3][3];  // .x: the link of direction 2 role, .y: that of 2 role + 1
};
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
// (a b + c d) + (e f + g h), each product pair as one fma on a rounded product
__device__ __forceinline__ float2 two_pairs(float2 a, float2 b, float2 c, float2 d, float2 e, float2 f, float2 g, float2 h)
{
    return add2(fma2(a, b, mul2(c, d)), fma2(e, f, mul2(g, h)));
}

__device__ __forceinline__ void pack_rows(Link2 &L, const float a[12], const float b[12])
{
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            L.x[i][j] = make_float2(a[2 * (3 * i + j)], b[2 * (3 * i + j)]);
            L.y[i][j] = make_float2(a[2 * (3 * i + j) + 1], b[2 * (3 * i + j) + 1]);
        }
}
// the rows of one of the two links (half = 0, 1)
__device__ __forceinline__ void unpack_rows(const Link2 &L, int half, float r[12])
{
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            r[2 * (3 * i + j)] = half ? L.x[i][j].y : L.x[i][j].x;
            r[2 * (3 * i + j) + 1] = half ? L.y[i][j].y : L.y[i][j].x;
        }
}
__device__ __forceinline__ void one_of(const Link2 &L, int half, Link<float> &o)
{
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++)
            o.e[i][j] = half ? cx<float>(L.x[i][j].y, L.y[i][j].y) : cx<float>(L.x[i][j].x, L.y[i][j].x);
}

// reconstruct() of both links
__device__ __forceinline__ void reconstruct2(Link2 &L)
{
    const float2 minus = both(-1.f);
    float2 nx[3], ny[3], cx_[3], cy_[3];  // -row1; the cross product
#pragma unroll
    for (int j = 0; j < 3; j++) {
        nx[j] = mul2(L.x[1][j], minus);
        ny[j] = mul2(L.y[1][j], minus);
    }
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const int p = (j + 1) % 3, q = (j + 2) % 3;
        cx_[j] = two_pairs(L.x[0][p], L.x[1][q], L.y[0][p], ny[q], L.x[0][q], nx[p], L.y[0][q], L.y[1][p]);
        cy_[j] = two_pairs(L.y[0][p], nx[q], L.x[0][p], ny[q], L.y[0][q], L.x[1][p], L.x[0][q], L.y[1][p]);
    }
    float2 n[3];
#pragma unroll
    for (int j = 0; j < 3; j++) n[j] = fma2(cx_[j], cx_[j], mul2(cy_[j], cy_[j]));
    const float2 sum = add2(add2(n[0], n[1]), n[2]);
    const float2 inv = make_float2(rsq(sum.x), rsq(sum.y));
#pragma unroll
    for (int j = 0; j < 3; j++) {
        L.x[2][j] = mul2(cx_[j], inv);
        L.y[2][j] = mul2(cy_[j], inv);
    }
}

// left_mult<I, J>(up, g) and right_mult<I, J>(dn, g^dagger) of two links each
template <int I, int J>
__device__ __forceinline__ void subgroup_mult2(Link2 &up, Link2 &dn, const float g[4])
{
    const float2 g0 = both(g[0]), g1 = both(g[1]), g2 = both(g[2]), g3 = both(g[3]);
    const float2 n1 = both(-g[1]), n2 = both(-g[2]), n3 = both(-g[3]);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float2 ax = up.x[I][k], ay = up.y[I][k], bx = up.x[J][k], by = up.y[J][k];
        up.x[I][k] = two_pairs(g0, ax, n3, ay, g2, bx, n1, by);
        up.y[I][k] = two_pairs(g3, ax, g0, ay, g1, bx, g2, by);
        up.x[J][k] = two_pairs(n2, ax, n1, ay, g0, bx, g3, by);
        up.y[J][k] = two_pairs(g1, ax, n2, ay, g0, by, n3, bx);
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float2 ax = dn.x[k][I], ay = dn.y[k][I], bx = dn.x[k][J], by = dn.y[k][J];
        dn.x[k][I] = two_pairs(g0, ax, g3, ay, g2, bx, g1, by);
        dn.y[k][I] = two_pairs(g0, ay, n3, ax, g2, by, n1, bx);
        dn.x[k][J] = two_pairs(g1, ay, n2, ax, g0, bx, n3, by);
        dn.y[k][J] = two_pairs(n1, ax, n2, ay, g3, bx, g0, by);
    }
}

template <int GAUGE, int I, int J>
__device__ __forceinline__ void subgroup_sum_pair2(const Link2 &up, const Link2 &dn, int role, float w[4])
{
    Link<float> u[2], d[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        one_of(up, h, u[h]);
        one_of(dn, h, d[h]);
    }
    subgroup_sum_pair<GAUGE, I, J>(u, d, role, w);
}
template <int GAUGE, int ALGO, int I, int J, bool SITE_W>
__device__ __forceinline__ void subgroup_step_pair2(Link2 &up, Link2 &dn, int role, const AlgoParams &p,
                                                    Rng<float> &rng, Cx<float> (*wcol)[3])
{
    float w[4];
    subgroup_sum_pair2<GAUGE, I, J>(up, dn, role, w);
    subgroup_finish<GAUGE, ALGO, 16>(w, p, rng);
    subgroup_mult2<I, J>(up, dn, w);
    if (SITE_W) left_mult_dcolumn<I, J>(*wcol, w, role);
}

// site_update_pair of a lane's links in packed form
template <int GAUGE, int ALGO, bool SITE_W>
__device__ __forceinline__ void site_update_pair2(Link2 &up, Link2 &dn, int role, const AlgoParams &p, Rng<float> &rng,
                                                  Cx<float> (*wcol)[3] = nullptr)
{
    if constexpr (ALGO == ALG_SA) {
#pragma unroll 1
        for (int k = 0; k < 3; k++) {
            float w[4];
            on_subgroup(k, [&](auto s) { subgroup_sum_pair2<GAUGE, s.I, s.J>(up, dn, role, w); });
            subgroup_finish<GAUGE, ALGO, 16>(w, p, rng);
            on_subgroup(k, [&](auto s) {
                subgroup_mult2<s.I, s.J>(up, dn, w);
                if (SITE_W) left_mult_dcolumn<s.I, s.J>(*wcol, w, role);
            });
        }
        return;
    }
    subgroup_step_pair2<GAUGE, ALGO, 0, 2, SITE_W>(up, dn, role, p, rng, wcol);
    subgroup_step_pair2<GAUGE, ALGO, 1, 2, SITE_W>(up, dn, role, p, rng, wcol);
    subgroup_step_pair2<GAUGE, ALGO, 0, 1, SITE_W>(up, dn, role, p, rng, wcol);
}

// The four links of a lane in the two-lanes-per-site layout: packed in FP32, scalar in FP64.
template <typename R>
struct PairLinks {
    Link<R> up[2], dn[2];
    __device__ __forceinline__ void set(const R (&ru)[2][12], const R (&rd)[2][12])
    {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            unpack12(up[j], ru[j]);
            unpack12(dn[j], rd[j]);
            reconstruct(up[j]);
            reconstruct(dn[j]);
        }
    }
    template <int GAUGE, int ALGO, bool SITE_W>
    __device__ __forceinline__ void update(int role, const AlgoParams &p, Rng<R> &rng, Cx<R> (*wcol)[3] = nullptr)
    {
        site_update_pair<GAUGE, ALGO, R, SITE_W>(up, dn, role, p, rng, wcol);
    }
    __device__ __forceinline__ void rows_up(int j, R r[12]) const { pack12(up[j], r); }
    __device__ __forceinline__ void rows_dn(int j, R r[12]) const { pack12(dn[j], r); }
};
template <>
struct PairLinks<float> {
    Link2 up, dn;
    __device__ __forceinline__ void set(const float (&ru)[2][12], const float (&rd)[2][12])
    {
        pack_rows(up, ru[0], ru[1]);
        pack_rows(dn, rd[0], rd[1]);
        reconstruct2(up);
        reconstruct2(dn);
    }
    template <int GAUGE, int ALGO, bool SITE_W>
    __device__ __forceinline__ void update(int role, const AlgoParams &p, Rng<float> &rng, Cx<float> (*wcol)[3] = nullptr)
    {
        site_update_pair2<GAUGE, ALGO, SITE_W>(up, dn, role, p, rng, wcol);
    }
    __device__ __forceinline__ void rows_up(int j, float r[12]) const { unpack_rows(up, j, r); }
    __device__ __forceinline__ void rows_dn(int j, float r[12]) const { unpack_rows(dn, j, r); }
};

// ---- lattice geometry -----------------------------------------------------------------------
// Division by a lattice extent without a divide instruction: for 0 <= n < 2^31 and d >= 1,
// q = (umulhi(n, m) + n) >> s with s = ceil(log2 d), m = floor(2^32 (2^s - d) / d) + 1
// (Granlund & Montgomery, "Division by invariant integers using multiplication", PLDI 1994).
struct FastDiv {
    uint32_t d, m, s;
    __host__ __device__ __forceinline__ uint32_t div(uint32_t n) const { return (__umulhi_any(n, m) + n) >> s; }

  private:
    __host__ __device__ static __forceinline__ uint32_t __umulhi_any(uint32_t a, uint32_t b)
    {
#ifdef __CUDA_ARCH__
        return __umulhi(a, b);
#else
        return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
    }
};

inline FastDiv make_fastdiv(uint32_t d)
{
    uint32_t s = 0;
    while ((1ull << s) < d) s++;
    const uint64_t m = ((uint64_t(1) << 32) * ((uint64_t(1) << s) - d)) / d + 1;
    return FastDiv{d, (uint32_t)m, s};
}

// Parity-split site order of the reference (SiteCoord.hxx:104-175): lexicographic l =
// ((t*Nx + x)*Ny + y)*Nz + z, s = l/2 (+V/2 for odd t+x+y+z).  All extents must be even and
// V < 2^31, so site arithmetic is 32-bit.
struct Geom {
    int32_t n[4];   // Nt, Nx, Ny, Nz
    int64_t V, Vh;
    FastDiv dx, dy, dz;
};

inline void geom_init_div(Geom &g)
{
    g.dx = make_fastdiv((uint32_t)g.n[1]);
    g.dy = make_fastdiv((uint32_t)g.n[2]);
    g.dz = make_fastdiv((uint32_t)g.n[3]);
}

__device__ __forceinline__ void site_coords(const Geom &g, int64_t h64, int parity, int32_t c[4])
{
    uint32_t l = 2u * (uint32_t)h64;
    uint32_t q = g.dz.div(l);
    c[3] = (int32_t)(l - q * g.dz.d);
    l = q;
    q = g.dy.div(l);
    c[2] = (int32_t)(l - q * g.dy.d);
    l = q;
    q = g.dx.div(l);
    c[1] = (int32_t)(l - q * g.dx.d);
    c[0] = (int32_t)q;
    if (((c[0] + c[1] + c[2] + c[3]) & 1) != parity) c[3] += 1;
}

__device__ __forceinline__ int64_t site_index(const Geom &g, const int32_t c[4])
{
    const uint32_t l = (((uint32_t)c[0] * g.n[1] + c[1]) * g.n[2] + c[2]) * g.n[3] + c[3];
    return (int64_t)(l >> 1) + (((c[0] + c[1] + c[2] + c[3]) & 1) ? g.Vh : 0);
}

// forward neighbour x + mu of the site with coordinates c
__device__ __forceinline__ int64_t neighbour_up(const Geom &g, const int32_t c[4], int mu)
{
    int32_t d[4];
#pragma unroll
    for (int k = 0; k < 4; k++) d[k] = (mu == k) ? ((c[k] + 1 == g.n[k]) ? 0 : c[k] + 1) : c[k];
    return site_index(g, d);
}

// backward neighbour x - mu of the site with coordinates c (mu is lane-dependent, so the
// coordinate arrays are only ever indexed with constants: no local-memory spill)
__device__ __forceinline__ int64_t neighbour_down(const Geom &g, const int32_t c[4], int mu)
{
    int32_t d[4];
#pragma unroll
    for (int k = 0; k < 4; k++) d[k] = (mu == k) ? ((c[k] == 0 ? g.n[k] : c[k]) - 1) : c[k];
    return site_index(g, d);
}

}  // namespace gfb
