// ism_moment.cu -- image-source forward kernel by fractional-delay moments, sm_103a.
//
// The early part of an RIR is y[t] = sum_i a_i W(t - tau_i), W the Hann-windowed sinc
// (src/gpuRIR_cuda.cu:110-121).  ism_forward.cu adds each image's Tw taps one by one;
// this kernel separates them.  Time is cut into cells of two samples; with tau = n + u, n
// the cell's centre and u in [-1, 1], each tap W(kappa - u), kappa = t - n, is a smooth
// function of u and a polynomial of degree 13 reproduces all of them (2 to 5e-8 relative L2, up to
// 6.5e-8 at windows below 80 samples; of an image whose window ends in the middle of a cell at
// most 7.3e-8, and 2.7e-7 below 80 samples, nearly all of it in the last tap):
//   y[t] = sum over cells n, sum_j c_j(t - n) A_j[n],   A_j[n] = sum over the cell's images of a T_j(u)
// with T_j the Chebyshev polynomials.  An image then costs its geometry and fourteen
// multiply-adds instead of Tw taps, and a sample costs a fixed filter whatever the number
// of images that reach it.
//
// The filter is made short by a basis F = S A of the moments in which taps away from the
// centre need few functions: the sinc's far taps are sin(pi tau)/(pi x) with 1/x nearly
// constant over a cell.  Functions 0..3 carry every tap beyond 12.6 samples, 0..5 every
// tap beyond 4.6, and twelve the nearest ones (moment_basis below).  Every basis function is
// even or odd in u, so a pair (even, odd) is one packed FP32 value all the way: moments
// are added, transformed and filtered two at a time, and at 16 kHz a sample takes 176 packed
// multiply-adds.
//
// Work item = one RIR x a run of its samples (x one of several interleaved sets of image
// rows), worked through in segments of at most T samples.  Per segment:
//   1. rows (m0, m1) of the image grid whose images can reach the segment: the range of
//      m2 between the segment's two spheres, one row per thread (an image outside the
//      segment's shell is never touched);
//   2. the rows' images, 32 per warp at a time without block barriers: float-float delay and
//      amplitude, cell and u, and the moments added to the cell's sums in shared memory;
//   3. sums -> basis, one thread per cell, then the filter: a warp takes 512 outputs (16 per
//      lane) and a range of taps; the warps' parts are added in order.
//
// The sums are integers, so that their order -- whichever warp comes first -- does not
// change a bit: a moment is scaled by a power of two (from a bound on the amplitudes) to at most
// 2^20, rounded to an integer, and its remainder to 2^-20 of that to a second one (both
// roundings by the addition of 1.5 2^23, whose bits are added up as they are and removed by the
// count): 41 bits below the bound.  T_8 to T_13, whose taps' coefficients are below 2e-3, have
// the first integer only.  Cells of up to 448 images need fewer guard bits and share words
// (kMPSums below): 17 words a cell instead of 23, 28 to 31 bits below the bound.  Either way an
// image adds an error of about 2e-10 of the bound.  Where a segment's loudest image is far above
// its quietest samples -- most first segments, any with dull walls -- the bound is that of every
// eight cells by themselves (16 samples, fewer than an image's taps reach), from a first pass
// over the images, so that the error stays below FP32's own.  A segment with cells of more
// images than the integers hold is done again with bounds that fit.
//
// What bounds it: the shared-memory atomics of the image loop (2.7 cycles per warp at random
// cells, 3.5 wavefronts; an FP32 atomicAdd takes 9.3 cycles) where images are many -- the
// load pipe is at 75 % on 128 rooms -- and issue with the phases' barriers where they are few
// (58 % of the slots on the array).  Per launch, ism_forward.cu and this kernel: one dense RIR of
// 6 million images 531 and 92 us, 64 x 32 array 490 and 321, 128 rooms 2680 and 642, 15 RIRs at
// 48 kHz 87 and 37 (with one scale per segment 90, 321, 617 and 37).  (Other ways that were built first: a counting sort by cell with one
// thread per cell adding in image order needed 8 barriers per 1024 images and ran at 228
// cycles per 32 images and SM, against 93 here.)
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <map>
#include <mutex>
#include <vector>

#include "gpurir_internal.cuh"
#include "ism_moment.cuh"
#include "tail_common.cuh"

namespace gpurir {

// The two shapes of a block: threads, blocks per SM, cells of one array (a constant, so that
// offsets are immediates), groups of 32 images per batch of rows.  A block's phases (image
// atomics, filter, output) wait for one another; three small blocks per SM overlap better
// than two large ones.  128 rooms: 660 us with two, 617 with three; 64 x 32 array 370 and 327.  The
// large one is for windows whose cells three blocks cannot hold and for launches of few
// segments, where each item's fixed cost counts (plan_moment).
template <int THREADS>
struct MomCfg {
    static constexpr int threads = THREADS, warps = THREADS / 32, rows = THREADS;   // rows: image rows per batch
    static constexpr int blocks = THREADS == kMomSmall ? 3 : 2;
    static constexpr int stride = THREADS == kMomSmall ? kMomSmallCells : kMomCells;
    static constexpr int groups = THREADS == kMomSmall ? 1024 : 2048;
    static constexpr int cells = (stride + THREADS - 1) / THREADS;                  // of one thread
    static_assert(kPowerThreads > THREADS && kPowerThreads <= 2 * THREADS,
                  "the fused tail sums the window power in the tail kernel's order");
};
constexpr int kMTwo = 4;                       // pairs of moments with two integers
constexpr int kMSums = 4 * kMTwo + 2 * (kMPairs - kMTwo) + 1;   // integers per cell, the last one the count
// Packed sums, for cells of fewer than 7/8 2^h images (h <= 9).  Amplitudes span 2^21 steps.
// T0..T7: two words of steps and, shared by a pair, one with what the rounding left, 16 bits
// each; T8..T10: a word each; T11 above a count of 10 bits; T12 (17 bits) above T13 (15 bits).
constexpr int kMPTwo = 4, kMPSums = 3 * kMPTwo + 2 + 3;
constexpr int kMPSpan = 21, kMPCount = 10, kMPMinBits = 6, kMPMaxBits = 9;
static_assert(kMPairs == 7, "the packed words are laid out for fourteen moments");
constexpr int kMScale = 3;                     // log2 of the cells that share a scale
constexpr int kMScales = kMomCells >> kMScale; // at most
static_assert(kMScales + kMomCells / 32 <= kMomSmall && kMomSmallCells <= kMomCells, "a thread for each scale and word of bits");
constexpr float kMMagic = 12582912.0f;         // 1.5 2^23
constexpr int kMMagicBits = 0x4b400000;

// Cell b of a basis pair: 16-byte chunks of two cells, rotated within groups of four so
// that 16-byte loads of lanes eight cells apart fall on distinct banks.
__device__ __forceinline__ int mchunk(int k) { return k ^ ((k >> 3) & 3); }

// Room, pair and work item of one item, copied to shared memory while the previous item
// is still being filtered.
struct MomCtx {
    IsmItem it;
    unsigned room[(offsetof(RoomDesc, pw) + 3) / 4];   // RoomDesc without its power tables
    float pos[6], ori[6];                               // source, receiver; their unit axes (zero: omni)
    float inv_L[3], ov[3], p2, q2, inv_k;               // reciprocals, source overhang, offsets along the last axis
    int reach;                                          // last sample an image of the pair can have
    int near2[3];                                       // bits of the least squared component along each axis
    int valid;
};
constexpr int kItemWords = sizeof(IsmItem) / 4, kRoomWords = offsetof(RoomDesc, pw) / 4;
static_assert(kItemWords <= 32 && kRoomWords <= 64 && kRoomWords > 32, "copied by one warp in one and two loads");

struct MomSmem {
    int *sum;                 // [kMSums][stride] moments as integers, and images, per cell;
                              // then [kMBasis][stride] float2 and, after those, the filter's parts
    float2 *coef;             // [8 * quads]: four taps x two output phases
    float4 *rows;             // [rows] rho^2 hi, lo, attenuation, m0 | m1 << 16
    int2 *range;              // [rows] first image, za | na << 9 | zb << 18
    unsigned short *group;    // [groups] row of a group's first image
    int *scale;               // [kMScales] bits of the loudest image of eight cells; then of their scale
    unsigned *bad;            // [kMomCells / 32] cells with an image of no finite amplitude, as bits
    MomCtx *ctx;              // [2]
    int *red;                 // scan scratch [32], control words [16]
    float4 *tab;              // [2][axis_cap] per-axis tables (or in global memory)
};

__host__ __device__ inline size_t mom_align16(size_t x) { return (x + 15) & ~(size_t)15; }

// Byte offsets of the arrays of MomSmem, in its order; returns the total.
template <class Cfg>
__host__ __device__ inline size_t mom_layout(int n_quads, int axis_cap, size_t o[10]) {
    const size_t sums = (size_t)kMSums * Cfg::stride * sizeof(int);
    const size_t filt = (size_t)kMBasis * Cfg::stride * sizeof(float2) + (size_t)Cfg::warps * 512 * sizeof(float);
    size_t b = 0;
    o[0] = b; b = mom_align16(b + (sums > filt ? sums : filt));
    o[1] = b; b = mom_align16(b + (size_t)n_quads * 8 * sizeof(float2));
    o[2] = b; b = b + Cfg::rows * sizeof(float4);
    o[3] = b; b = b + Cfg::rows * sizeof(int2);
    o[4] = b; b = b + Cfg::groups * sizeof(unsigned short);
    o[5] = b; b = b + kMScales * sizeof(int);
    o[6] = b; b = b + kMomCells / 32 * sizeof(int);
    o[7] = b; b = mom_align16(b + 2 * sizeof(MomCtx));
    o[8] = b; b = mom_align16(b + 48 * sizeof(int));
    o[9] = b; b += axis_cap <= kMomTabSmem ? 2 * (size_t)axis_cap * sizeof(float4) : 0;
    return b;
}

__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Exclusive block scan of one int per thread; `tot` is the block's sum.  red: WARPS ints, free
// again at the caller's next barrier.
template <int WARPS>
__device__ __forceinline__ int block_scan(int v, int *red, int &tot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) red[warp] = x;
    __syncthreads();
    int w = lane < WARPS ? red[lane] : 0;
#pragma unroll
    for (int o = 1; o < WARPS; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
    }
    tot = __shfl_sync(0xffffffffu, w, WARPS - 1);
    const int before = __shfl_sync(0xffffffffu, w, warp > 0 ? warp - 1 : 0);
    return x - v + (warp > 0 ? before : 0);
}

// Image indices of one axis whose coordinate range can come within [-hi, hi] of the
// receiver: the image of index k = m - N/2 lies in [k L - ov, (k + 1) L + ov], ov = how
// far the source lies outside the room along this axis (0 inside).
__device__ __forceinline__ void axis_range(int N, float inv_L, float ov, float r, float hi, int &a, int &b) {
    const float kmin = ceilf((r - hi - ov) * inv_L - 1.001f), kmax = floorf((r + hi + ov) * inv_L + 0.001f);
    a = max(0, (int)fmaxf(kmin, -1.0e6f) + N / 2);
    b = min(N, (int)fminf(kmax, 1.0e6f) + N / 2 + 1);
    if (b < a) b = a;
}

// Largest even (odd) k with k <= x, smallest with k >= x.
__device__ __forceinline__ float even_le(float x) { return 2.0f * floorf(0.5f * x); }
__device__ __forceinline__ float even_ge(float x) { return 2.0f * ceilf(0.5f * x); }
__device__ __forceinline__ float odd_le(float x) { return even_le(x - 1.0f) + 1.0f; }
__device__ __forceinline__ float odd_ge(float x) { return even_ge(x - 1.0f) + 1.0f; }

// Image indices m of one axis whose component v (receiver -> image) may have zl <= |v| <= zh:
// [za, ya) and [zb, yb).  Images of even k = m - N/2 lie at k L + s, those of odd k at
// (k + 1) L - s: each parity's first and last index within the outer bound and within
// the inner one follow by rounding; an index between the inner ones of both parities is
// surely nearer than zl.  (In units of L: p = (s - r) / L, q = 1 - (s + r) / L are the offsets
// of the even and odd images; eps covers the rounding of this arithmetic.)
__device__ __forceinline__ void shell_range(int N, float p, float q, float zl, float zh, int &za, int &ya, int &zb,
                                            int &yb) {
    const float eps = 1e-3f, big = 1.0e6f;
    const float lo = fminf(even_ge(-zh - p - eps), odd_ge(-zh - q - eps));
    const float hi = fmaxf(even_le(zh - p + eps), odd_le(zh - q + eps));
    const int c = N / 2;
    za = min(max((int)fminf(fmaxf(lo, -big), big) + c, 0), N);
    yb = min(max((int)fminf(fmaxf(hi, -big), big) + c + 1, za), N);
    const float g0 = fmaxf(even_ge(-zl - p + eps), odd_ge(-zl - q + eps)) - 1.0f;
    const float g1 = fminf(even_le(zl - p - eps), odd_le(zl - q - eps)) + 1.0f;
    const int gl = (int)fminf(fmaxf(g0, -big), big) + c, gh = (int)fminf(fmaxf(g1, -big), big) + c + 1;
    if (zl > 0.0f && gl < gh) {   // [gl, gh) is out
        ya = min(max(gl, za), yb);
        zb = min(max(gh, za), yb);
    } else {
        ya = zb = yb;
    }
}

// Packed FP32 sum, rounded by itself (the explicit rounding keeps ptxas from fusing it with a
// product before it).
__device__ __forceinline__ float2 add2_rn(float2 a, float2 b) {
    float2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<unsigned long long &>(r))
        : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)));
    return r;
}

// Four cell taps of one basis pair for 16 outputs: output (e, f) = sample 2 e + f of the lane's
// sixteen, acc[2 e + f] += X[j + e] c[j][f], X = eleven consecutive cells of three quads.
__device__ __forceinline__ void fir4(float2 (&acc)[16], const float2 (&q0)[4], const float2 (&q1)[4],
                                     const float2 (&q2)[4], const float2 *coef) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float4 c = *reinterpret_cast<const float4 *>(coef + 2 * j);
        const float2 c0 = make_float2(c.x, c.y), c1 = make_float2(c.z, c.w);
#pragma unroll
        for (int e = 0; e < 8; e++) {
            const int i = j + e;
            const float2 x = i < 4 ? q0[i & 3] : (i < 8 ? q1[i & 3] : q2[i & 3]);
            acc[2 * e] = __ffma2_rn(x, c0, acc[2 * e]);
            acc[2 * e + 1] = __ffma2_rn(x, c1, acc[2 * e + 1]);
        }
    }
}
__device__ __forceinline__ void load_quad(float2 (&q)[4], const float2 *pair, int quad) {
    const int x = (quad >> 2) & 3;   // mchunk(2 quad), mchunk(2 quad + 1)
    const float4 a = reinterpret_cast<const float4 *>(pair)[(2 * quad) ^ x],
                 b = reinterpret_cast<const float4 *>(pair)[(2 * quad + 1) ^ x];
    q[0] = make_float2(a.x, a.y); q[1] = make_float2(a.z, a.w);
    q[2] = make_float2(b.x, b.y); q[3] = make_float2(b.z, b.w);
}
// Place of the 16-byte chunk k (four samples) in a warp's part: the four chunks of a lane are
// rotated by its index, so that lanes 64 bytes apart fall on distinct banks.
__device__ __forceinline__ int part_chunk(int k) { return (k & ~3) | ((k + (k >> 3)) & 3); }

// Asynchronous 4-byte copy global -> shared (PTX cp.async); bytes = 0 writes a zero.
__device__ __forceinline__ void copy_async4(void *dst, const void *src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_done() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
}

// The copy of item `id`'s context by one warp, in three steps with other work in between:
// the item's words; then the room's words and the pair's positions; then what follows
// from them.
__device__ __forceinline__ void ctx_item(MomCtx &c, const MomLaunch &P, int id, int lane) {
    if (id < P.n_items && lane < kItemWords)
        copy_async4(reinterpret_cast<unsigned *>(&c.it) + lane, reinterpret_cast<const unsigned *>(P.items + id) + lane, 4);
}
__device__ __forceinline__ void ctx_pair(MomCtx &c, const MomLaunch &P, int id, int lane) {
    copies_done();
    if (id >= P.n_items) return;
    const unsigned *rw = reinterpret_cast<const unsigned *>(P.rooms + c.it.room);
    copy_async4(c.room + lane, rw + lane, 4);
    if (lane + 32 < kRoomWords) copy_async4(c.room + lane + 32, rw + lane + 32, 4);
    if (lane < 6) copy_async4(c.pos + lane, lane < 3 ? P.pos_src + 3 * c.it.src + lane : P.pos_rcv + 3 * c.it.rcv + lane - 3, 4);
}
__device__ __forceinline__ void ctx_finish(MomCtx &c, const MomLaunch &P, int id, int lane) {
    copies_done();
    if (lane == 0) c.valid = id < P.n_items;
    if (id >= P.n_items) return;
    const RoomDesc &R = *reinterpret_cast<const RoomDesc *>(c.room);
    float v2 = 0.0f, o = 0.0f;
    if (lane < 6 && (lane < 3 ? R.spkr : R.mic) != P_OMNI) {   // unit axes (only a directional pattern has one)
        const float *v = lane < 3 ? P.orv_src + 3 * c.it.src : P.orv_rcv + 3 * c.it.rcv;
        o = v[lane % 3] * rsqrtf(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    }
    if (lane < 6) c.ori[lane] = o;
    if (lane < 3) {
        const float L = R.L[lane], sa = c.pos[lane], ra = c.pos[3 + lane], inv = 1.0f / L;
        float v2min;
        axis_extent(R.nb[lane], L, sa, ra, v2min, v2);
        c.near2[lane] = 0x7f7fffff;
        c.inv_L[lane] = inv;
        c.ov[lane] = fmaxf(fmaxf(-sa, sa - L), 0.0f);
        if (lane == 2) {
            c.p2 = (sa - ra) * inv;
            c.q2 = 1.0f - (sa + ra) * inv;
        }
    }
    v2 = __shfl_sync(0xffffffffu, v2, 0) + __shfl_sync(0xffffffffu, v2, 1) + __shfl_sync(0xffffffffu, v2, 2);
    if (lane == 0) {
        // (a huge bound: no image is ruled out; of a position that is not a number no delay is one)
        const float far = sqrtf(v2) * (R.kh + R.kl) * 1.00001f + 4.0f;
        c.reach = far < 1.0e9f ? (int)far : 0x3fffffff;
        c.inv_k = 1.0f / R.kh;
    }
}

// Per-axis image terms of one item (as ism_forward.cu tabulates them): {v^2 hi, v^2 lo, v,
// attenuation} for m < N0, then N1, then N2 entries.  Wall powers come from the room in
// global memory, everything else from the item's context.
template <int THREADS>
__device__ __forceinline__ void axis_tables(const MomLaunch &P, MomCtx &c, float4 *tab, int tid) {
    const RoomDesc &R = *reinterpret_cast<const RoomDesc *>(c.room);
    const RoomDesc &G = P.rooms[c.it.room];
    const int N0 = R.nb[0], N1 = R.nb[1], N2 = R.nb[2];
    for (int e = tid; e < N0 + N1 + N2; e += THREADS) {
        const int a = e < N0 ? 0 : (e < N0 + N1 ? 1 : 2);
        const int m = e - (a == 0 ? 0 : (a == 1 ? N0 : N0 + N1));
        int ca, fa;
        image_axis(m, R.nb[a], ca, fa);
        const float att = G.pw[2 * a][abs(ca - fa)] * G.pw[2 * a + 1][abs(ca)];
        const float La = R.L[a], sa = c.pos[a], ra = c.pos[3 + a];
        if (R.ref_delay) {   // the reference's float32 component; its square only bounds
            const float v = ref_axis_component(ca, fa, La, sa, ra);
            tab[e] = make_float4(v * v, 0.0f, v, att);
            atomicMin(&c.near2[a], __float_as_int(v * v));
        } else {
            const ff v = ff_add(ff_two_prod((float)(2 * ca), La), ff_two_sum(fa ? -sa : sa, -ra));
            const ff sq = ff_sqr(v);
            tab[e] = make_float4(sq.hi, sq.lo, v.hi, att);
            atomicMin(&c.near2[a], __float_as_int(sq.hi));
        }
    }
}

// One image's moments, pair by pair: (a T_2k(u), a T_2k+1(u)) by x_k+1 = w x_k - x_k-1,
// w = 2 T_2(u); the signs + + - - + + - turn the subtraction into an addition (S carries them).
template <typename Put>
__device__ __forceinline__ void image_moments(float a, float u, Put put) {
    const float h = fmaf(2.0f * u, u, -1.0f), w = 2.0f * h;
    const float2 w2 = make_float2(w, w), v2 = make_float2(-w, -w);
    float2 x = make_float2(a, a * u);
    float2 y = make_float2(x.x * h, x.y * (w - 1.0f));
    put(0, x);
    put(1, y);
#pragma unroll
    for (int p = 2; p < kMPairs; p++) {
        const float2 z = __ffma2_rn(p & 1 ? w2 : v2, y, x);
        put(p, z);
        x = y;
        y = z;
    }
}

// Scale (its bits) of cells whose images have at most this peak / 4 pi (bits): 2^(e + 1) bounds them, with
// room for the peak's rounding, and the steps' span covers that.
__device__ __forceinline__ int scale_of(int peak, int span) {
    const int e = (__float_as_int(__int_as_float(peak) * 0.0797f) >> 23) - 127;
    return (127 + min(max(span - 1 - e, -120), 120)) << 23;
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS, MomCfg<THREADS>::blocks) ism_moment_kernel(const __grid_constant__ MomLaunch P) {
    using Cfg = MomCfg<THREADS>;
    constexpr int kMThreads = THREADS, kMWarps = Cfg::warps, kMStride = Cfg::stride;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    MomSmem s;
    {
        size_t o[10];
        mom_layout<Cfg>(P.n_quads, P.axis_cap, o);
        s.sum = reinterpret_cast<int *>(smem_raw + o[0]);
        s.coef = reinterpret_cast<float2 *>(smem_raw + o[1]);
        s.rows = reinterpret_cast<float4 *>(smem_raw + o[2]);
        s.range = reinterpret_cast<int2 *>(smem_raw + o[3]);
        s.group = reinterpret_cast<unsigned short *>(smem_raw + o[4]);
        s.scale = reinterpret_cast<int *>(smem_raw + o[5]);
        s.bad = reinterpret_cast<unsigned *>(smem_raw + o[6]);
        s.ctx = reinterpret_cast<MomCtx *>(smem_raw + o[7]);
        s.red = reinterpret_cast<int *>(smem_raw + o[8]);
        s.tab = P.axis_cap <= kMomTabSmem ? reinterpret_cast<float4 *>(smem_raw + o[9])
                                        : P.axis_tab + (size_t)(2 * blockIdx.x) * P.axis_cap;
    }
    float2 *basis = reinterpret_cast<float2 *>(s.sum);                 // [kMBasis][kMStride]
    float *part = reinterpret_cast<float *>(basis + kMBasis * kMStride);  // filter parts
    int *ctl = s.red + 32;   // [0] most images of a cell, [1] last cell with an image, [2] a cell is bad,
                             // [3] images not counted in a cell, [4..9] bounds of |attenuation| along the axes, [10, 11]
                             // an image's attenuation at the segment's ends
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned le_mask = 0xffffffffu >> (31 - lane);
    for (int i = tid; i < 8 * P.n_quads; i += kMThreads) s.coef[i] = P.coef[i];

    // the first item's context; later ones are fetched during the last segment before them
    int next = 0;      // (warp 0)
    if (warp == 0) {
        if (lane == 0) next = atomicAdd(P.work_counter, 1);
        next = __shfl_sync(0xffffffffu, next, 0);
        ctx_item(s.ctx[0], P, next, lane);
        ctx_pair(s.ctx[0], P, next, lane);
        ctx_finish(s.ctx[0], P, next, lane);
    }
    __syncthreads();
    if (s.ctx[0].valid) axis_tables<THREADS>(P, s.ctx[0], s.tab, tid);

    for (int par = 0;; par ^= 1) {
        const MomCtx &C = s.ctx[par];
        if (!C.valid) break;
        if (C.it.t_hi <= C.it.t_lo) {   // the host makes no such item
            if (tid == 0) atomicExch(P.status, DEV_BAD_ITEM);
            break;
        }
        const RoomDesc &R = *reinterpret_cast<const RoomDesc *>(C.room);
        const float4 *tab = s.tab + par * P.axis_cap;
        if (warp == 0) {
            if (lane == 0) next = atomicAdd(P.work_counter, 1);
            next = __shfl_sync(0xffffffffu, next, 0);
        }
        for (int t_lo = C.it.t_lo, t_hi; t_lo < C.it.t_hi; t_lo = t_hi) {
        // one segment; the last one of the item holds at least P.win samples, and samples past
        // every image are one segment of zeros
        t_hi = min(t_lo + P.T, C.it.t_hi);
        if (t_hi < C.it.t_hi && C.it.t_hi - t_hi < P.win) t_hi = (C.it.t_hi - P.win) & ~3;
        const int cell0 = t_lo - P.lead;                      // first sample of cell 0 (t_lo and lead are even)
        const bool empty = cell0 > C.reach;
        if (empty) t_hi = C.it.t_hi;
        const int len = t_hi - t_lo;
        const int tiles = (len + 511) >> 9;
        const int nb = ((len + 1) >> 1) + P.taps - 1;         // cells whose taps reach the segment
        const int nbe = min(kMStride, tiles * 256 + 4 * P.quads + 8);      // cells the filter reads
        const bool last = t_hi == C.it.t_hi;
        __syncthreads();   // tables written; the previous segment's output is done with the shared arrays
        if (last && warp == 0) ctx_item(s.ctx[par ^ 1], P, next, lane);

        int act = 0;       // tiles of 512 outputs that images reach
        if (!empty) {
            const int N0 = R.nb[0], N1 = R.nb[1], N2 = R.nb[2];
            // shell of the segment's cells: delays in [cell0 - 1, cell0 + 2 nb + 1]
            const float inv_L2 = C.inv_L[2];
            const float d_lo = fmaxf((float)(cell0 - 1) * C.inv_k - 0.01f, 0.0f);
            const float d_hi = (float)(cell0 + 2 * nb + 1) * C.inv_k * 1.00001f + 0.01f;
            const float dlo2 = d_lo * d_lo * 0.99999f, dhi2 = d_hi * d_hi;
            int a0, a1, W1, n_box, my_rows;
            {
                int b0, b1;
                axis_range(N0, C.inv_L[0], C.ov[0], C.pos[3], d_hi, a0, b0);
                axis_range(N1, C.inv_L[1], C.ov[1], C.pos[4], d_hi, a1, b1);
                W1 = b1 - a1;
                n_box = (b0 - a0) * W1;                       // rows of the bounding rectangle; part i_lo of i_hi
                my_rows = n_box > C.it.i_lo ? (n_box - C.it.i_lo + C.it.i_hi - 1) / C.it.i_hi : 0;
            }
            const float rW1 = 1.0f / (float)max(W1, 1);
            // (in registers: the atomics might alias the context, so that it would be read again per image)
            const int kind = R.spkr | R.mic << 8 | (R.ref_delay != 0) << 16;
            const ff k_samples = {R.kh, R.kl};
            const float k_scale = R.kh * (0.5f / (1 << kMScale)), g0 = (float)cell0 * (0.5f / (1 << kMScale));   // groups of cells
            const int batch = min(Cfg::rows, 32 * Cfg::groups / N2);   // rows at once: their images fill the groups at most
            // mean images per cell at the segment's end: a room's volume holds one; cells with few
            // have packed sums
            const float mean = 25.14f * d_hi * d_hi * C.inv_k * C.inv_L[0] * C.inv_L[1] * inv_L2 / (float)C.it.i_hi;
            int bits = kMPMinBits;
            while (bits < kMPMaxBits && 4.0f * mean + 24.0f > (float)(7 << bits >> 3)) bits++;
            bool packed = 2.0f * mean + 24.0f <= (float)(7 << bits >> 3);
            int shift = 0;     // bits given up to hold more images per cell
            int span = 0;      // log2 of the steps that cover an amplitude
            int n_rows = 0, n_img = 0;
            bool rows_ready = false;   // a segment's only batch of rows stays in place
            for (;;) {
                const int words = packed ? kMPSums : kMSums;
                for (int a = warp; a < words; a += kMWarps)
                    for (int i = lane; 4 * i < nbe; i += 32)
                        reinterpret_cast<int4 *>(s.sum + a * kMStride)[i] = make_int4(0, 0, 0, 0);
                if (tid < 4) ctl[tid] = tid == 1 ? -1 : 0;
                const int before = span;
                span = packed ? kMPSpan : 20 - shift;
                const float most = __int_as_float((127 + span) << 23);
                const float fine = packed ? __int_as_float((127 + 16 - bits) << 23) : most;   // steps of the second integer in one of the first
                if (before == 0) {
                    if (tid < kMScales) s.scale[tid] = 0;
                    else if (tid - kMScales < kMomCells / 32) s.bad[tid - kMScales] = 0;
                    if (warp < 3) {   // largest |attenuation| along one axis, and beyond d_lo / sqrt(3)
                        int a2, b2;
                        axis_range(N2, inv_L2, C.ov[2], C.pos[5], d_hi, a2, b2);
                        const int lo = warp == 0 ? a0 : (warp == 1 ? N0 + a1 : N0 + N1 + a2);
                        const int hi = warp == 0 ? a0 + (W1 > 0 ? n_box / W1 : 0) : (warp == 1 ? N0 + a1 + W1 : N0 + N1 + b2);
                        const float far2 = 0.3333f * dlo2;
                        int full = 0, far = 0;
                        for (int i = lo + lane; i < hi; i += 32) {
                            const int w = __float_as_int(fabsf(tab[i].w));
                            full = max(full, w);
                            if (!(tab[i].x < far2)) far = max(far, w);
                        }
                        full = __reduce_max_sync(0xffffffffu, full);
                        far = __reduce_max_sync(0xffffffffu, far);
                        if (lane == 0) {
                            ctl[4 + warp] = full;
                            ctl[7 + warp] = far;
                        }
                    } else if (warp == 3) {   // images d_lo and d_hi away in no special direction: half of that along each axis
                        const int axis = lane & 3;
                        float att = 1.0f;
                        if (lane < 8 && axis < 3) {
                            const int N = R.nb[axis], c = N / 2;
                            const int n = (int)fminf(0.5f * (lane < 4 ? d_lo : d_hi) * C.inv_L[axis], 1.0e6f) + (lane >> 2);
                            const float4 *t = tab + (axis > 0 ? N0 : 0) + (axis > 1 ? N1 : 0);
                            att = fminf(fabsf(t[max(c - n, 0)].w), fabsf(t[min(c + n, N - 1)].w));
                        }
                        att *= __shfl_xor_sync(0xffffffffu, att, 1);
                        att *= __shfl_xor_sync(0xffffffffu, att, 2);
                        if (lane == 0 || lane == 4) ctl[10 + (lane >> 2)] = __float_as_int(att);
                    }
                }
                __syncthreads();
                // One scale for the segment where its loudest image is not far above an image at either end: of an
                // image at least d_lo away one component is d_lo / sqrt(3) at least, which bounds its attenuation
                // (walls that amplify too), and amplitudes are at most that bound over 4 pi d with d the shell's
                // inner radius or the nearest image's distance.  An image's error of 2e-10 of that bound is then at
                // most 5e-8 of the quiet ones.  Else every eight cells (16 samples) have a scale of their own, from
                // the loudest of their images.  (With one scale always, 128 samples of a first segment were off by
                // 2e-4 at 16 kHz and 0.15 at 8 kHz with walls of 0.1, by 2e-6 and 1.5e-4 with walls of 0.3; now 4e-7
                // at most.  With a scale per eight cells always, 128 rooms take 887 us; with the line at 128, 673 us
                // and the same errors; here 642.)
                bool quiet = false;
                if (before == 0) {
                    const float f0 = __int_as_float(ctl[4]), f1 = __int_as_float(ctl[5]), f2 = __int_as_float(ctl[6]);
                    const float att_max = fmaxf(fmaxf(__int_as_float(ctl[7]) * (f1 * f2), __int_as_float(ctl[8]) * (f0 * f2)),
                                                __int_as_float(ctl[9]) * (f0 * f1));
                    const float first = sqrtf(__int_as_float(C.near2[0]) + __int_as_float(C.near2[1]) +
                                              __int_as_float(C.near2[2])) * 0.999f;
                    const float near = fmaxf(d_lo, first), peak = att_max * 1.001f / near;
                    quiet = max(max(ctl[4], ctl[5]), ctl[6]) >= 0x7f800000 ||   // (a factor that is not finite)
                            !(peak < 3.0e38f && peak * near <= 256.0f * __int_as_float(ctl[10]) &&
                              peak * d_hi <= 256.0f * __int_as_float(ctl[11]));
                    if (!quiet && tid < kMScales) s.scale[tid] = scale_of(__float_as_int(peak), span);
                } else if (tid < kMScales) {
                    s.scale[tid] += (span - before) * (1 << 23);
                }
                int placed = 0;
                // twice over the images of a quiet segment: the loudest of every eight cells, by an estimate of
                // distance and amplitude that is good to 1e-6; then the sums, at the scales that follow
                for (int sums = !quiet; sums < 2; sums++) {
                if (sums) {
                    if (quiet) {
                        __syncthreads();   // peaks complete
                        if (tid < kMScales) s.scale[tid] = scale_of(s.scale[tid], span);
                    }
                    if (rows_ready) __syncthreads();   // (else the rows' barriers come first)
                }
                for (int rbase = 0; rbase < my_rows; rbase += batch) {
                    if (!rows_ready) {
                    // ---- one row per thread: its m2 ranges [za, ya) and [zb, yb)
                    int za = 0, ya = 0, zb = 0, yb = 0;
                    float4 row = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (tid < batch && rbase + tid < my_rows) {
                        int q0, q1;
                        divmod_small(C.it.i_lo + C.it.i_hi * (rbase + tid), W1, rW1, q0, q1);
                        const int m0 = a0 + q0, m1 = a1 + q1;
                        const float4 tx = tab[m0], ty = tab[N0 + m1];
                        const ff rho = ff_add(ff{tx.x, tx.y}, ff{ty.x, ty.y});
                        row = make_float4(rho.hi, rho.lo, tx.w * ty.w, __int_as_float(m0 | (m1 << 16)));
                        const float h2 = dhi2 - rho.hi, l2 = dlo2 - rho.hi;
                        if (h2 > 0.0f)   // (square roots to ~1e-6: the shell has 0.01 m to spare)
                            shell_range(N2, C.p2, C.q2, l2 > 0.0f ? l2 * rsqrt_approx(l2) * inv_L2 : 0.0f,
                                        h2 * rsqrt_approx(h2) * inv_L2, za, ya, zb, yb);
                    }
                    const int na = ya - za, mine = na + (yb - zb);
                    int total;
                    const int scan = block_scan<kMWarps>(mine | (mine > 0 ? 1 << 20 : 0), s.red, total);
                    const int off = scan & 0xfffff, my_row = scan >> 20;   // images and rows with images before mine
                    if (mine > 0) {
                        s.rows[my_row] = row;
                        s.range[my_row] = make_int2(off, za | (na << 9) | (zb << 18));
                        for (int g = (off + 31) >> 5; 32 * g < off + mine; g++) s.group[g] = (unsigned short)my_row;
                    }
                    __syncthreads();
                    n_rows = total >> 20;
                    n_img = total & 0xfffff;
                    rows_ready = my_rows <= batch;
                    }
                    // ---- images, 32 of the batch per warp at a time
                    for (int base = 32 * warp; base < n_img; base += 32 * kMWarps) {
                        const int r0 = s.group[base >> 5], idx = base + lane;
                        // rows that begin inside this group, as bits
                        const int o = r0 + 1 + lane < n_rows ? s.range[r0 + 1 + lane].x - base : 32;
                        const int r = r0 + __popc(__reduce_or_sync(0xffffffffu, o < 32 ? 1u << o : 0u) & le_mask);
                        if (idx >= n_img) continue;
                        const float4 row = s.rows[r];
                        const int2 rg = s.range[r];
                        const int j = idx - rg.x, na = (rg.y >> 9) & 511;
                        const int m2 = j < na ? (rg.y & 511) + j : (rg.y >> 18) + (j - na);
                        const float4 t2 = tab[N0 + N1 + m2];
                        if (!sums) {
                            const float d2 = row.x + t2.x, rs = rsqrt_approx(d2), a = fabsf(row.z * t2.w) * rs;
                            const float g = d2 * rs * k_scale, room = fmaf(g, 2e-6f, 0.002f);   // groups from sample 0, the estimate's error
                            const float ga = floorf(g - g0 - room), gb = floorf(g - g0 + room);
                            if (!(gb >= 0.0f && ga < (float)kMScales) || !(a < 3.0e38f)) continue;
                            for (int k = max((int)ga, 0); k <= min((int)gb, kMScales - 1); k++) {
                                int *peak = s.scale + k;
                                if (__float_as_int(a) > *(volatile int *)peak) atomicMax(peak, __float_as_int(a));
                            }
                            continue;
                        }
                        ff d2 = ff_add(ff{row.x, row.y}, ff{t2.x, t2.y});
                        float v0h = 0.0f, v1h = 0.0f;
                        const int m0 = __float_as_int(row.w) & 0xffff, m1 = __float_as_int(row.w) >> 16;
                        const int spkr = kind & 255, mic = kind >> 8 & 255;
                        const bool ref_delay = kind >> 16 != 0, ref_dir = (kind & 0xffff) != (P_OMNI | P_OMNI << 8);
                        if (ref_dir || ref_delay) {
                            v0h = tab[m0].z;
                            v1h = tab[N0 + m1].z;
                            if (ref_delay) d2 = ff{ref_dist2(v0h, v1h, t2.z, ref_dir), 0.0f};
                        }
                        const float rs0 = rsqrt_approx(d2.hi);
                        float inv_d;
                        const ff dist = ff_dist_newton(d2, rs0, d2.hi * rs0, inv_d);
                        const ff tau = ref_delay ? ff{ref_tau(d2.hi, R.c, R.fs), 0.0f} : ff_mul(dist, k_samples);
                        float amp = row.z * t2.w * (0.0795774715459476679f * inv_d);   // attenuation / (4 pi dist)
                        if (spkr != P_OMNI) {
                            // doa = image -> receiver, axis mirrored per reflection (:357-362)
                            const float ct = -(((m0 - N0 / 2) & 1 ? -C.ori[0] : C.ori[0]) * v0h +
                                               ((m1 - N1 / 2) & 1 ? -C.ori[1] : C.ori[1]) * v1h +
                                               ((m2 - N2 / 2) & 1 ? -C.ori[2] : C.ori[2]) * t2.z) * inv_d;
                            amp *= pattern_gain(ct, spkr);
                        }
                        if (mic != P_OMNI)   // (:363)
                            amp *= pattern_gain((C.ori[3] * v0h + C.ori[4] * v1h + C.ori[5] * t2.z) * inv_d, mic);
                        // cell floor(tau / 2) of the whole time axis, by the rounding of an FP32 addition
                        // (at a boundary either neighbour will do); u from its centre.  A NaN or a
                        // huge delay fails the range test.
                        const float mg = (0.5f * tau.hi - 0.5f) + kMMagic;
                        const float u = (tau.hi - (2.0f * (mg - kMMagic) + 1.0f)) + tau.lo;
                        const int b = __float_as_int(mg) - kMMagicBits - (cell0 >> 1);
                        if (!(tau.hi < 4.0e6f) || b < 0 || b >= nb || amp == 0.0f) continue;
                        const float q = amp * __int_as_float(s.scale[b >> kMScale]);   // exact
                        if (!(fabsf(q) <= most)) {   // (finite amplitudes are covered)
                            atomicOr(&s.bad[b >> 5], 1u << (b & 31));
                            ctl[2] = 1;
                            continue;
                        }
                        int *cell = s.sum + b;
                        const float2 m2f = make_float2(kMMagic, kMMagic), n2f = make_float2(-kMMagic, -kMMagic);
                        const float2 fine2 = make_float2(fine, fine), minus = make_float2(-1.0f, -1.0f);
                        if (packed) {
                            placed++;
                            const float f11 = __int_as_float((127 - bits) << 23);
                            image_moments(q, u, [&](int p, float2 v) {
                                int *c = cell + (p < kMPTwo ? 3 * p : 3 * kMPTwo + 2 * (p - kMPTwo)) * kMStride;
                                const float2 f = p == 5 ? make_float2(1.0f, f11)
                                                        : make_float2(f11 * 0.03125f, f11 * 0.0078125f);
                                const float2 t = p < 5 ? add2_rn(v, m2f) : __ffma2_rn(v, f, m2f);
                                const unsigned x = __float_as_uint(t.x), y = __float_as_uint(t.y);
                                // (the constant's bits are zero below bit 22: shifted by ten or more they vanish)
                                atomicAdd(c, (int)(p == 6 ? (x << 15) + y : x));
                                if (p < 6) atomicAdd(c + kMStride, (int)(p == 5 ? (y << kMPCount) + 1 : y));
                                if (p < kMPTwo) {   // what the rounding left, in steps of 1 / fine
                                    const float2 w = __ffma2_rn(__ffma2_rn(add2_rn(t, n2f), minus, v), fine2, m2f);
                                    atomicAdd(c + 2 * kMStride, (int)((__float_as_uint(w.x) << 16) + __float_as_uint(w.y)));
                                }
                            });
                            continue;
                        }
                        atomicAdd(cell + (kMSums - 1) * kMStride, 1);
                        image_moments(q, u, [&](int p, float2 v) {
                            const float2 t = add2_rn(v, m2f);
                            int *c = cell + (p < kMTwo ? 4 * p : 4 * kMTwo + 2 * (p - kMTwo)) * kMStride;
                            atomicAdd(c, __float_as_int(t.x));
                            atomicAdd(c + kMStride, __float_as_int(t.y));
                            if (p < kMTwo) {
                                const float2 w = __ffma2_rn(__ffma2_rn(add2_rn(t, n2f), minus, v), fine2, m2f);
                                atomicAdd(c + 2 * kMStride, __float_as_int(w.x));
                                atomicAdd(c + 3 * kMStride, __float_as_int(w.y));
                            }
                        });
                    }
                }
                }
                __syncthreads();   // sums complete
                int n_max = 0, top = -1;
                const int *count = s.sum + (packed ? 3 * kMPTwo + 3 : kMSums - 1) * kMStride;
                for (int b = tid; b < nbe; b += kMThreads) {
                    const int n = packed ? count[b] & ((1 << kMPCount) - 1) : count[b];
                    n_max = max(n_max, n);
                    placed -= n;
                    if (n > 0 || (ctl[2] && s.bad[b >> 5] >> (b & 31) & 1)) top = b;
                }
                n_max = __reduce_max_sync(0xffffffffu, n_max);
                top = __reduce_max_sync(0xffffffffu, top);
                placed = __reduce_add_sync(0xffffffffu, placed);
                if (lane == 0) {
                    atomicMax(&ctl[0], n_max);
                    atomicMax(&ctl[1], top);
                    atomicAdd(&ctl[3], placed);
                }
                __syncthreads();
                if (packed) {   // too many images in a cell, or more than its count holds: unpacked sums
                    if (ctl[0] <= (7 << bits >> 3) && ctl[3] == 0) break;
                    packed = false;
                } else {        // a cell's sums hold 2^(11 + shift) images
                    if (ctl[0] >> (11 + shift) == 0) break;
                    while (ctl[0] >> (11 + shift)) shift++;
                }
                __syncthreads();
            }
            const bool any_bad = ctl[2] != 0;
            act = ctl[1] >= 0 ? min((ctl[1] >> 8) + 1, tiles) : 0;
            // ---- sums -> basis, each cell by one thread
            const float fine = __int_as_float((127 - (packed ? 16 - bits : 20 - shift)) << 23);
            float2 F[Cfg::cells][kMBasis];
#pragma unroll
            for (int i = 0; i < Cfg::cells; i++) {
                const int b = tid + i * kMThreads;
#pragma unroll
                for (int p = 0; p < kMBasis; p++) F[i][p] = make_float2(0.0f, 0.0f);
                const int *sum = s.sum + b;
                const int tc = b < nbe ? sum[(packed ? 3 * kMPTwo + 3 : kMSums - 1) * kMStride] : 0;
                const int n = packed ? tc & ((1 << kMPCount) - 1) : tc;
                if (b >= nbe || (n == 0 && !any_bad)) continue;
                const float unit = __int_as_float((254 << 23) - s.scale[b >> kMScale]);   // of a step, one over the scale
                const int bias = n * kMMagicBits;   // (modulo 2^32, as the sums)
                float2 A[kMPairs];
                if (packed) {
#pragma unroll
                    for (int p = 0; p < kMPTwo; p++) {
                        const int *c = sum + 3 * p * kMStride;
                        const int w = c[2 * kMStride] - bias, y = (short)w;
                        A[p] = make_float2(fmaf((float)((w - y) >> 16), fine, (float)(c[0] - bias)),
                                           fmaf((float)y, fine, (float)(c[kMStride] - bias)));
                    }
                    const int *c = sum + 3 * kMPTwo * kMStride;
                    const float f11 = __int_as_float((127 + bits) << 23);
                    A[4] = make_float2((float)(c[0] - bias), (float)(c[kMStride] - bias));
                    A[5] = make_float2((float)(c[2 * kMStride] - bias), (float)(tc >> kMPCount) * f11);
                    const int w = c[4 * kMStride] - bias, y = (int)((unsigned)w << 17) >> 17;
                    A[6] = make_float2((float)((w - y) >> 15) * (f11 * 32.0f), (float)y * (f11 * 128.0f));
#pragma unroll
                    for (int p = 0; p < kMPairs; p++) A[p] = __fmul2_rn(A[p], make_float2(unit, unit));
                } else {
#pragma unroll
                    for (int p = 0; p < kMPairs; p++) {
                        const int *c = sum + (p < kMTwo ? 4 * p : 4 * kMTwo + 2 * (p - kMTwo)) * kMStride;
                        A[p] = make_float2((float)(c[0] - bias), (float)(c[kMStride] - bias));
                        if (p < kMTwo) {
                            A[p].x = fmaf((float)(c[2 * kMStride] - bias), fine, A[p].x);
                            A[p].y = fmaf((float)(c[3 * kMStride] - bias), fine, A[p].y);
                        }
                        A[p].x *= unit;
                        A[p].y *= unit;
                    }
                }
                if (any_bad && s.bad[b >> 5] >> (b & 31) & 1) A[0].x = A[0].y = __int_as_float(0x7fffffff);
#pragma unroll
                for (int p = 0; p < kMBasis; p++) {
                    // (high orders first: the small terms, so that fewer roundings are of full size)
                    F[i][p] = __fmul2_rn(P.S[p][kMPairs - 1], A[kMPairs - 1]);
#pragma unroll
                    for (int k = kMPairs - 2; k >= 0; k--) F[i][p] = __ffma2_rn(P.S[p][k], A[k], F[i][p]);
                }
            }
            __syncthreads();   // sums read: the basis takes their place
#pragma unroll
            for (int i = 0; i < Cfg::cells; i++) {
                const int b = tid + i * kMThreads;
                if (b < nbe)
#pragma unroll
                    for (int p = 0; p < kMBasis; p++) basis[p * kMStride + 2 * mchunk(b >> 1) + (b & 1)] = F[i][p];
            }
            __syncthreads();
        }

        // ---- filter: warp = (tile of 512 outputs, range of tap quads), over the tiles that cells
        // with images reach (outputs past the last such cell are zero)
        const int G = act > 0 ? kMWarps / act : 1;
        if (last && warp == 0) ctx_pair(s.ctx[par ^ 1], P, next, lane);
        {
            const int tile = warp / G, g = warp - tile * G;
            if (tile < act) {
                float2 acc[16];
#pragma unroll
                for (int e = 0; e < 16; e++) acc[e] = make_float2(0.0f, 0.0f);
                const unsigned char *cut = P.cut[act == 1 ? 0 : 1];
                int q = cut[g];
                const int q_end = cut[g + 1];
                int r = 0, base = 0;
                while (q < q_end) {
                    while (q >= base + P.run[r].quads) base += P.run[r++].quads;
                    const int run = min(q_end, base + P.run[r].quads) - q;
                    const float2 *pair = basis + P.run[r].pair * kMStride;
                    const float2 *cf = s.coef + 8 * q;
                    int quad = 2 * (32 * tile + lane) + P.run[r].first + (q - base);
                    float2 qa[4], qb[4], qc[4];
                    load_quad(qa, pair, quad);
                    load_quad(qb, pair, quad + 1);
                    int n = run;
                    for (; n >= 3; n -= 3, quad += 3, cf += 24) {
                        load_quad(qc, pair, quad + 2);
                        fir4(acc, qa, qb, qc, cf);
                        load_quad(qa, pair, quad + 3);
                        fir4(acc, qb, qc, qa, cf + 8);
                        load_quad(qb, pair, quad + 4);
                        fir4(acc, qc, qa, qb, cf + 16);
                    }
                    if (n > 0) {
                        load_quad(qc, pair, quad + 2);
                        fir4(acc, qa, qb, qc, cf);
                        if (n > 1) {
                            load_quad(qa, pair, quad + 3);
                            fir4(acc, qb, qc, qa, cf + 8);
                        }
                    }
                    q += run;
                }
                float4 *dst = reinterpret_cast<float4 *>(part + (g * act + tile) * 512);
#pragma unroll
                for (int e = 0; e < 4; e++)
                    dst[part_chunk(4 * lane + e)] = make_float4(acc[4 * e].x + acc[4 * e].y, acc[4 * e + 1].x + acc[4 * e + 1].y,
                                                                acc[4 * e + 2].x + acc[4 * e + 2].y,
                                                                acc[4 * e + 3].x + acc[4 * e + 3].y);
            }
        }
        if (last && warp == 0) ctx_finish(s.ctx[par ^ 1], P, next, lane);
        __syncthreads();
        if (last && s.ctx[par ^ 1].valid)
            axis_tables<THREADS>(P, s.ctx[par ^ 1], s.tab + (par ^ 1) * P.axis_cap, tid);
        // ---- output: four samples per thread and round; round v of thread j takes the groups
        // t/4 = j + v kMThreads (mod kPowerThreads): the order in which the tail kernel sums the
        // window power
        float *orow = C.it.part_off >= 0 ? P.partial + C.it.part_off - C.it.t_lo : P.out + C.it.out_row;
        const bool fuse = P.fuse_tail && C.it.part_off < 0 && t_hi == R.n_ism && R.n_total > R.n_ism;
        float tau_dp = 0.0f;
        int w_start = t_hi;
        if (fuse) {
            tau_dp = direct_tau(R, C.pos, C.pos + 3);
            w_start = envelope_start(R, tau_dp);
        }
        float pw[2] = {0.0f, 0.0f};
#pragma unroll
        for (int v = 0; v < 2; v++)
            for (int i4 = tid + v * kMThreads < kPowerThreads
                              ? 4 * ((tid + v * kMThreads - (t_lo >> 2)) & (kPowerThreads - 1)) : len;
                 i4 < len; i4 += 4 * kPowerThreads) {
                float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (i4 < act * 512) {
                    const float4 *src = reinterpret_cast<const float4 *>(part) + (i4 >> 9) * 128 + part_chunk((i4 & 511) >> 2);
                    for (int g = 0; g < G; g++) {
                        const float4 y = src[g * act * 128];
                        x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
                    }
                }
                float *dst = orow + t_lo + i4;
                const uintptr_t al = reinterpret_cast<uintptr_t>(dst);
                const int left = len - i4;
                if (left >= 4 && (al & 15) == 0) {
                    *reinterpret_cast<float4 *>(dst) = x;
                } else if (left >= 4 && (al & 7) == 0) {   // rows of an even length: 8-byte aligned
                    *reinterpret_cast<float2 *>(dst) = make_float2(x.x, x.y);
                    *reinterpret_cast<float2 *>(dst + 2) = make_float2(x.z, x.w);
                } else {
                    dst[0] = x.x;
                    if (left > 1) dst[1] = x.y;
                    if (left > 2) dst[2] = x.z;
                    if (left > 3) dst[3] = x.w;
                }
                if (fuse) {
                    const float e4[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        if (t_lo + i4 + e >= w_start && e < left) pw[v] = fmaf(e4[e], e4[e], pw[v]);
                }
            }
        if (fuse) {
            float *red = reinterpret_cast<float *>(s.red);
#pragma unroll
            for (int v = 0; v < 2; v++) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) pw[v] += __shfl_xor_sync(0xffffffffu, pw[v], o);
                if (lane == 0 && warp + v * kMWarps < kPowerThreads / 32) red[warp + v * kMWarps] = pw[v];
            }
            __syncthreads();
            if (tid == 0) {
                float tot = 0.0f;
                for (int w = 0; w < kPowerThreads / 32; w++) tot += red[w];
                const TailEnv e = tail_envelope(R, tot, w_start, tau_dp);
                red[kPowerThreads / 32] = e.ea;
                red[kPowerThreads / 32 + 1] = e.eb;
                if (P.env_out) {
                    P.env_out[3 * C.it.rir] = e.A;
                    P.env_out[3 * C.it.rir + 1] = e.alpha;
                    P.env_out[3 * C.it.rir + 2] = tau_dp;
                }
            }
            __syncthreads();
            if (!(P.tail_pre && P.tail_pre[C.it.rir])) {   // (else silent, and written by the caller)
                const uint64_t offset = P.offset_ptr ? *P.offset_ptr : P.offset;
                tail_fill(orow + R.n_ism, R.n_total - R.n_ism, 0, R.n_total - R.n_ism, tid, kMThreads,
                          red[kPowerThreads / 32], red[kPowerThreads / 32 + 1], P.seed, offset, (uint32_t)C.it.rir, P.noise_kind);
            }
        }
        }   // segments
    }
}

// ---------------------------------------------------------------------------
// Host side: the basis and the filter of one window length
// ---------------------------------------------------------------------------
namespace {

// Gauss-Legendre nodes and weights on [-1, 1] (Newton's method on P_n).
void gauss_legendre(int n, std::vector<double> &x, std::vector<double> &w) {
    x.resize(n);
    w.resize(n);
    for (int i = 0; i < n; i++) {
        double z = std::cos(M_PI * (i + 0.75) / (n + 0.5)), dp = 1.0;
        for (int k = 0; k < 100; k++) {
            double p0 = 1.0, p1 = z;
            for (int j = 2; j <= n; j++) {
                const double p2 = ((2 * j - 1) * z * p1 - (j - 1) * p0) / j;
                p0 = p1;
                p1 = p2;
            }
            dp = n * (z * p1 - p0) / (z * z - 1);
            const double dz = p1 / dp;
            z -= dz;
            if (std::fabs(dz) < 1e-16) break;
        }
        x[i] = z;
        w[i] = 2.0 / ((1 - z * z) * dp * dp);
    }
}

typedef double Mat[kMPairs][kMPairs];

// Eigenvectors of a symmetric n x n matrix (cyclic Jacobi), columns of V by falling eigenvalue.
void jacobi(Mat A, int n, Mat V) {
    for (int i = 0; i < n; i++)
        for (int j = 0; j < n; j++) V[i][j] = i == j;
    for (int sweep = 0; sweep < 60; sweep++) {
        double off = 0.0, diag = 0.0;
        for (int i = 0; i < n; i++) {
            diag += A[i][i] * A[i][i];
            for (int j = 0; j < i; j++) off += A[i][j] * A[i][j];
        }
        if (off <= 1e-40 * diag) break;
        for (int p = 0; p < n; p++)
            for (int q = p + 1; q < n; q++) {
                if (A[p][q] == 0.0) continue;
                const double th = 0.5 * (A[q][q] - A[p][p]) / A[p][q];
                const double t = (th >= 0 ? 1.0 : -1.0) / (std::fabs(th) + std::sqrt(th * th + 1));
                const double c = 1 / std::sqrt(t * t + 1), s = t * c;
                for (int k = 0; k < n; k++) {
                    const double x = A[k][p], y = A[k][q];
                    A[k][p] = c * x - s * y;
                    A[k][q] = s * x + c * y;
                }
                for (int k = 0; k < n; k++) {
                    const double x = A[p][k], y = A[q][k];
                    A[p][k] = c * x - s * y;
                    A[q][k] = s * x + c * y;
                }
                for (int k = 0; k < n; k++) {
                    const double x = V[k][p], y = V[k][q];
                    V[k][p] = c * x - s * y;
                    V[k][q] = s * x + c * y;
                }
            }
    }
    for (int i = 0; i < n; i++)   // selection sort by falling eigenvalue
        for (int j = i + 1; j < n; j++)
            if (A[j][j] > A[i][i]) {
                std::swap(A[i][i], A[j][j]);
                for (int k = 0; k < n; k++) std::swap(V[k][i], V[k][j]);
            }
}

}  // namespace

// Basis and filter of one window length.  Each tap (cell j of an output, output phase f) is
// expanded in orthonormal Legendre polynomials of u (degree < 14; Gauss-Legendre quadrature,
// split where the window ends inside the cell), by parity.  In each parity's seven
// coefficients the basis vectors are found in three steps, each the leading eigenvectors of
// a Gram matrix in what the steps before it leave: two for the taps beyond kMomFar samples,
// one for those beyond kMomNear, the others for all taps (the last of those is not needed:
// kMBasis).  Taps count by their relative error down to 2 / H^2, so that the far taps of a lone
// image are as good as its near ones (2e-7 of their size; unweighted the same 3e-8 of the whole,
// but 2e-6 at 50 samples of a window of 128).  Taps on which a pair's coefficients are below 2e-8 are left out of its runs.
// The vectors are orthonormal, so S and the coefficients are of order one; S is rounded to
// FP32 first and the coefficients fitted to the rounded functions (with monomial moments
// and plain rounding, the FP32 tables cost 2e-7).
void moment_basis(int tw, MomBasis &B) {
    const double H = 0.5 * tw;
    const int n = 2 * kMPairs, lead = 2 * (int)std::ceil(H / 2);
    const int J = (int)std::ceil((lead + H + 1) / 2);
    std::vector<double> x, w;
    gauss_legendre(48, x, w);
    std::vector<double> kap(2 * J);
    std::vector<std::vector<double>> C(2 * J, std::vector<double>(n, 0.0));
    for (int j = 0; j < J; j++)
        for (int f = 0; f < 2; f++) {
            const int m = 2 * j + f;
            kap[m] = lead - 2 * j + f - 1;
            double cut[4] = {-1.0, kap[m] - H, kap[m] + H, 1.0};   // pieces between the window's ends
            for (int c = 1; c < 3; c++) cut[c] = std::min(1.0, std::max(-1.0, cut[c]));
            for (int c = 0; c < 3; c++) {
                const double mid = 0.5 * (cut[c] + cut[c + 1]), half = 0.5 * (cut[c + 1] - cut[c]);
                if (half <= 0.0 || std::fabs(kap[m] - mid) >= H) continue;
                for (size_t k = 0; k < x.size(); k++) {
                    const double u = mid + half * x[k], t = kap[m] - u;
                    const double h = 0.5 * (1 + std::cos(M_PI * t / H)) *
                                     (std::fabs(t) < 1e-14 ? 1.0 : std::sin(M_PI * t) / (M_PI * t));
                    double p0 = 1.0, p1 = u;   // Legendre polynomials at u
                    for (int i = 0; i < n; i++) {
                        C[m][i] += half * w[k] * h * p0 * std::sqrt((2 * i + 1) / 2.0);
                        const double p2 = ((2 * i + 3) * u * p1 - (i + 1) * p0) / (i + 2);
                        p0 = p1;
                        p1 = p2;
                    }
                }
            }
        }
    // Chebyshev coefficients of the orthonormal Legendre polynomials (projection at Chebyshev nodes)
    std::vector<std::vector<double>> L(n, std::vector<double>(n, 0.0));
    for (int k = 0; k < 2 * n; k++) {
        const double th = M_PI * (k + 0.5) / (2 * n), u = std::cos(th);
        double p0 = 1.0, p1 = u;
        for (int i = 0; i < n; i++) {
            for (int j = 0; j < n; j++)
                L[i][j] += (j == 0 ? 1.0 : 2.0) / (2 * n) * std::cos(j * th) * p0 * std::sqrt((2 * i + 1) / 2.0);
            const double p2 = ((2 * i + 3) * u * p1 - (i + 1) * p0) / (i + 2);
            p0 = p1;
            p1 = p2;
        }
    }
    std::vector<std::vector<double>> F(2 * J, std::vector<double>(n, 0.0));   // (even, odd) per pair
    const double beyond[3] = {kMomFar, kMomNear, -1.0};
    const double quiet = 2.0 / (H * H);   // taps below this are weighted alike
    const int take[3] = {2, 1, kMPairs - 3};
    for (int par = 0; par < 2; par++) {
        Mat Q, rest;   // columns found so far; columns spanning what they leave
        int nq = 0, nr = kMPairs;
        for (int i = 0; i < kMPairs; i++)
            for (int j = 0; j < kMPairs; j++) rest[i][j] = i == j;
        for (int step = 0; step < 3; step++) {
            Mat G = {}, V, next;
            for (int m = 0; m < 2 * J; m++) {
                if (std::fabs(kap[m]) <= beyond[step] || std::fabs(kap[m]) > H - 1.01) continue;   // (whole cells)
                double y[kMPairs], size2 = 0.0;
                for (int a = 0; a < kMPairs; a++) size2 += C[m][2 * a + par] * C[m][2 * a + par];
                const double weight = 1.0 / (size2 + quiet * quiet);
                for (int j = 0; j < nr; j++) {
                    y[j] = 0.0;
                    for (int a = 0; a < kMPairs; a++) y[j] += C[m][2 * a + par] * rest[a][j];
                }
                for (int i = 0; i < nr; i++)
                    for (int j = 0; j < nr; j++) G[i][j] += weight * y[i] * y[j];
            }
            jacobi(G, nr, V);
            for (int a = 0; a < kMPairs; a++)
                for (int j = 0; j < nr; j++) {
                    next[a][j] = 0.0;
                    for (int i = 0; i < nr; i++) next[a][j] += rest[a][i] * V[i][j];
                }
            for (int j = 0; j < take[step]; j++, nq++)
                for (int a = 0; a < kMPairs; a++) Q[a][nq] = next[a][j];
            for (int j = take[step]; j < nr; j++)
                for (int a = 0; a < kMPairs; a++) rest[a][j - take[step]] = next[a][j];
            nr -= take[step];
        }
        for (int p = 0; p < kMPairs; p++) {
            for (int k = 0; k < kMPairs; k++) {
                double v = 0.0;
                for (int a = 0; a < kMPairs; a++) v += Q[a][p] * L[2 * a + par][2 * k + par];
                if (k & 2) v = -v;   // the sign of the kernel's recurrence
                if (p < kMBasis) (par ? B.S[p][k].y : B.S[p][k].x) = (float)v;
            }
            for (int m = 0; m < 2 * J; m++)
                for (int a = 0; a < kMPairs; a++) F[m][2 * p + par] += Q[a][p] * C[m][2 * a + par];
        }
    }
    // quads (four taps) on which each pair is used
    B.tw = tw;
    B.lead = lead;
    B.taps = J;
    B.quads = (J + 3) / 4;
    std::vector<char> used(B.quads * kMBasis, 1);
    for (int q = 0; q < B.quads; q++)
        for (int p = 2; p < kMBasis; p++) {
            double big = 0.0;
            for (int m = 8 * q; m < std::min(8 * q + 8, 2 * J); m++)
                big = std::max(big, std::max(std::fabs(F[m][2 * p]), std::fabs(F[m][2 * p + 1])));
            used[q * kMBasis + p] = big >= 2e-8;
        }
    // The coefficients are fitted to the basis as it is in FP32 (S rounded): least squares by
    // Gram-Schmidt in Legendre coordinates, over the pairs used on the tap's quad.
    std::vector<std::vector<double>> T(n, std::vector<double>(n, 0.0));   // Legendre coordinates of T_k
    for (size_t k = 0; k < x.size(); k++) {
        double p0 = 1.0, p1 = x[k];
        for (int i = 0; i < n; i++) {
            for (int j = 0; j < n; j++) T[j][i] += w[k] * std::cos(j * std::acos(x[k])) * p0 * std::sqrt((2 * i + 1) / 2.0);
            const double p2 = ((2 * i + 3) * x[k] * p1 - (i + 1) * p0) / (i + 2);
            p0 = p1;
            p1 = p2;
        }
    }
    for (int par = 0; par < 2; par++) {
        double f[kMBasis][kMPairs];   // the rounded basis
        for (int p = 0; p < kMBasis; p++)
            for (int a = 0; a < kMPairs; a++) {
                f[p][a] = 0.0;
                for (int k = 0; k < kMPairs; k++)
                    f[p][a] += (k & 2 ? -1.0 : 1.0) * (double)(par ? B.S[p][k].y : B.S[p][k].x) * T[2 * k + par][2 * a + par];
            }
        for (int m = 0; m < 2 * J; m++) {
            int at[kMBasis], nu = 0;
            for (int p = 0; p < kMBasis; p++) {
                F[m][2 * p + par] = 0.0;
                if (used[m / 8 * kMBasis + p]) at[nu++] = p;
            }
            double q[kMBasis][kMPairs], r[kMBasis][kMBasis], c[kMBasis];
            for (int i = 0; i < nu; i++) {
                for (int a = 0; a < kMPairs; a++) q[i][a] = f[at[i]][a];
                for (int k = 0; k < i; k++) {
                    r[k][i] = 0.0;
                    for (int a = 0; a < kMPairs; a++) r[k][i] += q[k][a] * f[at[i]][a];
                    for (int a = 0; a < kMPairs; a++) q[i][a] -= r[k][i] * q[k][a];
                }
                double d = 0.0;
                for (int a = 0; a < kMPairs; a++) d += q[i][a] * q[i][a];
                r[i][i] = std::sqrt(d);
                for (int a = 0; a < kMPairs; a++) q[i][a] /= r[i][i];
                c[i] = 0.0;
                for (int a = 0; a < kMPairs; a++) c[i] += q[i][a] * C[m][2 * a + par];
            }
            for (int i = nu - 1; i >= 0; i--) {
                for (int k = i + 1; k < nu; k++) c[i] -= r[i][k] * c[k];
                c[i] /= r[i][i];
                F[m][2 * at[i] + par] = c[i];
            }
        }
    }
    // runs of consecutive quads of one pair
    B.n_runs = B.n_quads = 0;
    B.coef.clear();
    for (int p = kMBasis - 1; p >= 0; p--)   // (the smaller terms of a sample first)
        for (int q = 0; q < B.quads; q++) {
            if (!used[q * kMBasis + p]) continue;
            if (B.n_runs > 0 && B.run[B.n_runs - 1].pair == p && B.run[B.n_runs - 1].first + B.run[B.n_runs - 1].quads == q)
                B.run[B.n_runs - 1].quads++;
            else
                B.run[B.n_runs++] = {p, q, 1};   // (the centre and both ends of the window: at most three per pair)
            B.n_quads++;
            for (int m = 8 * q; m < 8 * q + 8; m++)
                B.coef.push_back(m < 2 * J ? make_float2((float)F[m][2 * p], (float)F[m][2 * p + 1])
                                           : make_float2(0.0f, 0.0f));
        }
}

// Cuts of the filter's quads into G ranges of about equal time: a quad, and a good one more
// for every run that a range touches (its first cells are loaded before it starts).
static void cut_filter(const MomBasis &B, int G, unsigned char *cut) {
    std::vector<int> begin(B.n_quads, 0);   // 1: a run begins at this quad
    for (int r = 0, q = 0; r < B.n_runs; q += B.run[r++].quads) begin[q] = 1;
    for (double most = (double)B.n_quads / G;; most += 0.1) {
        int g = 0;
        double c = 0.0;
        cut[0] = 0;
        for (int q = 0; q < B.n_quads; q++) {
            const double add = 1.0 + (begin[q] || q == cut[g] ? 1.3 : 0.0);
            if (q > cut[g] && c + add > most) {
                if (++g == G) break;
                cut[g] = (unsigned char)q;
                c = 2.3;
            } else {
                c += add;
            }
        }
        if (g < G) {
            while (g < G) cut[++g] = (unsigned char)B.n_quads;
            return;
        }
    }
}

// Bases of the window lengths in use, built once each (about 1 ms).
const MomBasis &moment_basis_cached(int tw) {
    static std::mutex mu;
    static std::map<int, MomBasis> known;   // kMomMinTw <= tw <= kMomMaxTw: bounded
    std::lock_guard<std::mutex> lock(mu);
    auto it = known.find(tw);
    if (it == known.end()) {
        it = known.emplace(tw, MomBasis{}).first;
        moment_basis(tw, it->second);
        for (int v = 0; v < 2; v++)
            for (int tiles = 1; tiles <= 2; tiles++)
                cut_filter(it->second, (v ? kMomSmall : kMomLarge) / 32 / tiles, it->second.cut[v][tiles - 1]);
    }
    return it->second;
}

// cells of a launch: the longest segment's outputs and the filter's reach past them
int moment_cells(int T, const MomBasis &B) { return (T / 2 + 4 * B.quads + 8 + 7) / 8 * 8; }

size_t moment_smem_bytes(int threads, int axis_cap, const MomBasis &B) {
    size_t o[10];
    return threads == kMomSmall ? mom_layout<MomCfg<kMomSmall>>(B.n_quads, axis_cap, o)
                                : mom_layout<MomCfg<kMomLarge>>(B.n_quads, axis_cap, o);
}

static const void *moment_function(int threads) {
    return threads == kMomSmall ? reinterpret_cast<const void *>(ism_moment_kernel<kMomSmall>)
                                : reinterpret_cast<const void *>(ism_moment_kernel<kMomLarge>);
}

int moment_blocks_per_sm(int threads, size_t smem) {
    static std::mutex mu;
    static std::map<std::pair<int, size_t>, int> known;
    std::lock_guard<std::mutex> lock(mu);
    auto it = known.find({threads, smem});
    if (it != known.end()) return it->second;
    int n = 0;
    cudaFuncSetAttribute(moment_function(threads), cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, moment_function(threads), threads, smem);
    known[{threads, smem}] = n;
    return n;
}

cudaError_t moment_launch(const MomLaunch &p, int threads, size_t smem, int grid, cudaStream_t st) {
    static bool attr_set = false;   // per process; the attribute is per function
    if (!attr_set) {
        for (int t : {kMomSmall, kMomLarge}) {
            cudaError_t e = cudaFuncSetAttribute(moment_function(t), cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
            if (e != cudaSuccess) return e;
        }
        attr_set = true;
    }
    if (threads == kMomSmall) ism_moment_kernel<kMomSmall><<<grid, kMomSmall, smem, st>>>(p);
    else ism_moment_kernel<kMomLarge><<<grid, kMomLarge, smem, st>>>(p);
    return cudaGetLastError();
}

}  // namespace gpurir
