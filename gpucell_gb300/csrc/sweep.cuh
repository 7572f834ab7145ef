// sweep.cuh -- the neighbour sweep of the boundary entry points that need the
// pairs of a cube grid (density, SDPD force, wall repulsion, wall velocity).
//
// One block takes one cube at a time: all particles of a cube share the same
// 27 cubes of candidates (about 760 at 27 particles per rc^3), which are
// staged once in shared memory.  Eight lanes take two particles: they first
// only mark the candidates within the cut-off (a bit each; one shared-memory
// load serves both particles), then four lanes each evaluate the marked
// candidates of one of the two in even shares.  About 15 % of the candidates
// are partners: with one thread per particle testing and evaluating in one
// loop, nearly every iteration ran the pair physics for one or two lanes of
// a warp (17.5 of 32 lanes active, 4240 warp instructions per particle in
// the SDPD sweep).  The lanes also give a small system enough warps: an 83
// thousand particle channel is 650 blocks of one thread per particle, each a
// serial chain of 750 candidates.
//
// Bound by instruction issue (81 % of the slots in the density sweep, 72 % in
// the SDPD sweep, where shared memory holds six blocks a SM).  Measured on
// one GB300: a million-particle suspension's step 6.73 -> 3.16 ms, an 83
// thousand particle channel with walls of both kinds 1.55 -> 0.42 ms; at 524
// thousand particles the density sweep takes 0.39 ms and the SDPD sweep 0.75
// (2.50 before).  On an earlier form of it, 0.66 and 1.32 ms for a million
// particles, one particle per four lanes testing for itself took 0.86 and 1.51
// ms (a shared-memory load per test), without even shares 0.99 and 2.26 ms.
//
// Candidates are taken in the order of the cubes (z, y, x) and of their
// slots, and the partial sums of the lanes are added by a fixed tree, so
// results repeat bit for bit.
#pragma once

#include "gc_internal.cuh"

#include <type_traits>

namespace gcsweep {

constexpr int kBlock = 128;              // threads per block
constexpr int kGroup = 8;                // lanes that test candidates together, for two particles
constexpr int kLanes = 4;                // lanes that evaluate a particle's partners
constexpr int kPart = kBlock / kLanes;   // particles of a cube taken together
constexpr int kCap = 896;                // candidates staged together
constexpr int kWord = 32 * kGroup;       // candidates of one word of every lane's marks
constexpr int kWords = (kCap + kWord - 1) / kWord;
constexpr float kFar = 3.0e38f;          // coordinate of a candidate that takes no part (its r^2 is infinite)

// Cubes a block takes one after the other: one where cubes hold eight
// particles or more on average (a fluid has 27), more in a sparse grid, so
// that a block has about eight particles to work on and the empty cubes do
// not each cost a block.
inline int cubes_per_block(long long n, long long K) {
    long long c = n > 0 ? (8 * K + n - 1) / n : 1;
    return c < 1 ? 1 : (c > 128 ? 128 : (int)c);
}

// A block takes every gridDim-th cube, so that a crowd of particles in a
// corner of a sparse grid is shared out over the blocks.  From an empty cube
// on, the block's next 32 are looked at together, as the empty cubes of such a
// grid would otherwise be a serial chain of loads: last_empty gives the last
// of the empty ones.  Density of 10 / 80 / 27 thousand particles crowded into 0.04
// / 0.3 / 0.8 % of a box: 301 / 315 / 200 us with runs of consecutive cubes per
// block, 199 / 322 / 69 with every gridDim-th cube, 48 / 172 / 58 with both.
// Called by whole warps.
__device__ __forceinline__ int last_empty(int cube, int K, const int2* __restrict__ bec) {
    const long long step = gridDim.x, c = cube + ((threadIdx.x & 31) + 1) * step;
    const int2 be = c < K ? bec[c] : make_int2(0, 0);
    const unsigned full = __ballot_sync(0xffffffffu, be.y > be.x);
    const long long last = cube + (full ? __ffs(full) - 1 : 32) * step;
    return last < K ? (int)last : K;
}

struct Shared {
    float4 x[kCap];                      // position, id bits
    unsigned mark[2][kWords * kBlock];   // per particle of the group: word w of thread t at w * kBlock + t
    int beg[27], off[28];                // first slot of each cube of the stencil, their scanned sizes
};

// First slots and scanned sizes (sh.off[27] is the number of candidates) of
// the 27 cubes around cube c.  Cubes beyond a wall axis are empty; periodic
// axes have at least three cubes, so none is taken twice.
__device__ __forceinline__ void stencil(const GcGrid& g, int3 c, const int2* __restrict__ bec, Shared& sh) {
    if (threadIdx.x < 32) {
        const int t = threadIdx.x;
        int cnt = 0, b = 0;
        if (t < 27) {
            const int z = cube_step(c.z, t / 9 - 1, 2, g), y = cube_step(c.y, t / 3 % 3 - 1, 1, g),
                      x = cube_step(c.x, t % 3 - 1, 0, g);
            if (x >= 0 && y >= 0 && z >= 0) {
                const int2 be = bec[cube_key(x, y, z, g)];
                b = be.x;
                cnt = max(be.y - be.x, 0);
            }
        }
        int sum = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, sum, o);
            if (t >= o) sum += v;
        }
        if (t < 27) {
            sh.beg[t] = b;
            sh.off[t + 1] = sum;
        }
        if (t == 0) sh.off[0] = 0;
    }
    __syncthreads();
}

// How the candidates of a cube are tested: bits 1, 2, 4 for the image along
// x, y, z, or kAny.  kAny also takes positions that are no numbers: a NaN
// distance counts as within, as in the oracle's test, so that a lost particle
// shows in its neighbours.
constexpr int kAny = 8;

// The positions for which the plain difference along an axis decides as the
// minimum image does: of the cube's own particles within A of the cube's
// centre, of the candidates within B, where A + B = L - rc.  (A pair more
// than L/2 apart is then farther than rc either way.)  Particles in the cube
// they were sorted into keep to that with (L - rc - 2 w) / 2 to spare, w the
// cube's width, at least 3e-5 rc.  It is tested on the positions: one that
// the caller has moved since, that lies outside the box, or whose cube came
// out on the other side of a face by rounding makes its block take images.
// No limit along wall axes and where the stencil crosses a face (those take
// the image in any case).
struct Limits {
    float3 centre, own, cand;
    int cross;   // periodic axes along which the stencil crosses a face
};

__device__ __forceinline__ Limits limits(const GcGrid& g, int3 c, float rc) {
    Limits l;
    l.cross = 0;
    auto axis = [&](int a, int cc, float& centre, float& own, float& cand) {
        const float w = 1.f / g.invw[a];
        centre = g.origin[a] + ((float)cc + 0.5f) * w;
        own = cand = kFar;
        if (!(g.pmask & (1 << a))) return;
        if (cc == 0 || cc == g.n[a] - 1) {
            l.cross |= 1 << a;
            return;
        }
        const float spare = 0.5f * (g.L[a] * 0.99999f - rc) - w;
        own = 0.5f * w + spare;
        cand = 1.5f * w + spare;
    };
    axis(0, c.x, l.centre.x, l.own.x, l.cand.x);
    axis(1, c.y, l.centre.y, l.own.y, l.cand.y);
    axis(2, c.z, l.centre.z, l.own.z, l.cand.z);
    return l;
}

// The form that a position asks for beyond l.cross.
__device__ __forceinline__ int form_of(float3 x, const Limits& l, float3 lim) {
    const float3 d = f3(fabsf(x.x - l.centre.x), fabsf(x.y - l.centre.y), fabsf(x.z - l.centre.z));
    if (d.x <= lim.x && d.y <= lim.y && d.z <= lim.z) return 0;
    return d.x < kFar && d.y < kFar && d.z < kFar ? 7 : kAny;
}

// Difference along an axis; with IMAGE the minimum image, the same as
// min_image_1's (half: half the box, infinite along wall axes).  One comparison
// instead of two per axis: the cubes at the faces are the last blocks to end in a
// small box (density of 13.8 thousand particles 66 -> 52 us, 614 thousand 471 -> 456).
template <bool IMAGE>
__device__ __forceinline__ float diff_1(float a, float b, float half, float L) {
    const float d = __fsub_rn(a, b);
    return IMAGE && fabsf(d) > half ? __fsub_rn(d, copysignf(L, d)) : d;
}

template <bool IMAGE>
__device__ __forceinline__ float3 diff(float3 a, float4 b, float3 half, const GcGrid& g) {
    return f3(diff_1<IMAGE>(a.x, b.x, half.x, g.L[0]), diff_1<IMAGE>(a.y, b.y, half.y, g.L[1]),
              diff_1<IMAGE>(a.z, b.z, half.z, g.L[2]));
}

__device__ __forceinline__ float3 half_box(const GcGrid& g) {
    return f3(g.pmask & 1 ? g.halfL[0] : INFINITY, g.pmask & 2 ? g.halfL[1] : INFINITY, g.pmask & 4 ? g.halfL[2] : INFINITY);
}

// Marks the staged candidates [0, m) (m a multiple of 4 kGroup, padded with
// far ones) within cutm of xa and of xb that lane s tests; returns their
// numbers (xa's in the low half).  Bit 31 - u of word w is the candidate
// w * kWord + u * kGroup + s.
//
// The test takes seven instructions a candidate and particle, two more for an
// axis with the image: r^2 - cutm by fused multiply-adds, where the image's
// distance is the smaller of |d| and L - |d|, and its sign shifted into the
// word.  cutm is the cut-off with a margin above its rounding; evaluate()
// applies the predicate itself.
template <int FORM>
__device__ __forceinline__ int mark(Shared& sh, float3 xa, float3 xb, int s, int m, float cutm, const GcGrid& g) {
    const float3 L = f3(g.pmask & 1 ? g.L[0] : INFINITY, g.pmask & 2 ? g.L[1] : INFINITY,
                        g.pmask & 4 ? g.L[2] : INFINITY);
    const float3 half = half_box(g);
    auto beyond = [&](float3 x, float4 y) {
        float dx = __fsub_rn(x.x, y.x), dy = __fsub_rn(x.y, y.y), dz = __fsub_rn(x.z, y.z);
        if constexpr (FORM & 1) dx = fminf(fabsf(dx), L.x - fabsf(dx));
        if constexpr (FORM & 2) dy = fminf(fabsf(dy), L.y - fabsf(dy));
        if constexpr (FORM & 4) dz = fminf(fabsf(dz), L.z - fabsf(dz));
        return fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, -cutm)));
    };
    int count = 0;
    for (int w = 0, q0 = 0; q0 < m; ++w, q0 += kWord) {
        const int it = min(32, (m - q0) / kGroup);
        const float4* x = sh.x + q0 + s;
        unsigned a = 0, b = 0;
        for (int u0 = 0; u0 < it; u0 += 4) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float4 xj = x[(u0 + u) * kGroup];
                if constexpr (FORM == kAny) {
                    const bool none = xj.x == kFar;
                    a = (a << 1) | (none || norm2_rn(diff<true>(xa, xj, half, g)) >= cutm ? 0u : 1u);
                    b = (b << 1) | (none || norm2_rn(diff<true>(xb, xj, half, g)) >= cutm ? 0u : 1u);
                } else {
                    a = __funnelshift_l(__float_as_uint(beyond(xa, xj)), a, 1);
                    b = __funnelshift_l(__float_as_uint(beyond(xb, xj)), b, 1);
                }
            }
        }
        a <<= 32 - it;
        b <<= 32 - it;
        sh.mark[0][w * kBlock + threadIdx.x] = a;
        sh.mark[1][w * kBlock + threadIdx.x] = b;
        count += __popc(a) + (__popc(b) << 16);
    }
    return count;
}

// Evaluates op.pair(acc, ...) for an even share of the marked candidates of
// this thread's particle (particle h of the group): lane s of its four takes
// the ranks total s / 4 to total (s + 1) / 4 of the marks in the order of
// lanes, words and bits.  (The marks found by four lanes differ by a third,
// and the largest of a warp's shares sets its time.)  The marked candidates
// within cut2 by the oracle's predicate, bit for bit, are the pairs.  `count`
// as mark() returned it.  Called by whole warps.
template <bool IMAGE, class Op>
__device__ __forceinline__ void evaluate(const Op& op, const typename Op::Extra& ex, const typename Op::Self& self,
                                         typename Op::Acc& acc, const Shared& sh, float3 xi, int m, int count,
                                         float cut2, const GcParams& p) {
    const int t = threadIdx.x % kGroup, h = t / kLanes, s = t % kLanes;
    int end = count;   // inclusive scan over the group's lanes
#pragma unroll
    for (int o = 1; o < kGroup; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, end, o, kGroup);
        if (t >= o) end += v;
    }
    auto of = [&](int v) { return (v >> (16 * h)) & 0xffff; };
    const int total = of(__shfl_sync(0xffffffffu, end, kGroup - 1, kGroup));
    int r = total * s / kLanes, n = total * (s + 1) / kLanes - r;
    int lane = 0, base = 0;   // the lane whose marks hold rank r, and the marks before it
#pragma unroll
    for (int l = 0; l + 1 < kGroup; ++l) {
        const int e = of(__shfl_sync(0xffffffffu, end, l, kGroup));
        if (e <= r) {
            lane = l + 1;
            base = e;
        }
    }
    if (n <= 0) return;
    const unsigned* col = sh.mark[h] + (threadIdx.x & ~(kGroup - 1));
    int w = 0;
    unsigned bits = col[lane];
    r -= base;
    for (int c = __popc(bits); r >= c; c = __popc(bits)) {   // the word
        r -= c;
        bits = col[++w * kBlock + lane];
    }
    for (; r > 0; --r) bits &= ~(0x80000000u >> __clz(bits));   // the bit
    const int words = (m + kWord - 1) / kWord;
    const float3 half = half_box(p.g);
    for (; n > 0; --n) {
        while (!bits) {   // ends: n marks are left
            if (++w == words) {
                w = 0;
                ++lane;
            }
            bits = col[w * kBlock + lane];
        }
        const int u = __clz(bits);
        bits &= ~(0x80000000u >> u);
        const int q = w * kWord + u * kGroup + lane;
        const float4 xj = sh.x[q];
        const float3 d = diff<IMAGE>(xi, xj, half, p.g);
        const float r2 = norm2_rn(d);
        if (!(r2 >= cut2)) op.pair(acc, self, ex, q, __float_as_uint(xj.w), d, r2, p);
    }
}

// The sweep.  Op says which particles it is for (active), which candidates
// take part (keep), what else of a candidate is staged (Extra, stage), the
// cut-off, the pair function, what to do with the sum (finish) and with a
// particle that it is not for (idle).
//
// Positions are staged as they are; whether a cube's pairs need the minimum
// image follows from its place in the grid and from the positions (Limits),
// one form per cube.
template <class Op>
__global__ void __launch_bounds__(kBlock, Op::kBlocks) k_sweep(int K, GcParams p, Op op,
                                                  const float3* __restrict__ coor, const int* __restrict__ sortpart,
                                                  const int2* __restrict__ bec) {
    __shared__ Shared sh;
    __shared__ typename Op::Extra ex;
    const GcGrid& g = p.g;
    const int grp = threadIdx.x / kGroup, t = threadIdx.x % kGroup, h = t / kLanes;
    const float cut2 = op.cut2(p), cutm = cut2 * 1.00001f;
    for (int cube = blockIdx.x; cube < K; cube += gridDim.x) {
        const int2 be = bec[cube];
        if (be.y <= be.x) {
            cube = last_empty(cube, K, bec);
            continue;
        }
        const int3 c = make_int3(cube % g.n[0], cube / g.n[0] % g.n[1], cube / g.n[0] / g.n[1]);
        const Limits lim = limits(g, c, p.rc);
        bool any = false;
        int own_form = 0;
        for (int i = be.x + threadIdx.x; i < be.y; i += kBlock) {
            const unsigned id = (unsigned)sortpart[i];
            if (op.active(id, p)) {
                any = true;
                own_form |= form_of(coor[i], lim, lim.own);
            } else {
                op.idle(i);
            }
        }
        if (!__syncthreads_or(any)) continue;
        stencil(g, c, bec, sh);
        const int total = sh.off[27];
        int form = 0;
        bool some = false;
        // stages the candidates [q0, q0 + cnt), padded with far ones to m
        auto stage = [&](int q0, int cnt, int m, int& need) {
            bool kept = false;
            for (int r = threadIdx.x / 32; r < 27; r += kBlock / 32) {
                const int o = sh.off[r] - q0, e = min(sh.off[r + 1] - q0, cnt), j0 = sh.beg[r] - o;
                for (int q = max(o, 0) + (int)threadIdx.x % 32; q < e; q += 32) {
                    const int j = j0 + q;
                    const unsigned idj = (unsigned)sortpart[j];
                    float4 x = make_float4(kFar, kFar, kFar, 0.f);
                    if (op.keep(idj, p)) {
                        const float3 y = coor[j];
                        need |= form_of(y, lim, lim.cand);
                        x = make_float4(y.x, y.y, y.z, __uint_as_float(idj));
                        kept = true;
                        op.stage(ex, q, j, p);
                    }
                    sh.x[q] = x;
                }
            }
            for (int q = cnt + threadIdx.x; q < m; q += kBlock) sh.x[q] = make_float4(kFar, kFar, kFar, 0.f);
            return kept;
        };
        for (int b0 = be.x; b0 < be.y; b0 += kPart) {
            // the group's two particles, and the one of them this thread evaluates
            const int ia = b0 + 2 * grp, i = ia + h;
            const unsigned id = i < be.y ? (unsigned)sortpart[i] : 0u;
            const bool act = i < be.y && op.active(id, p);
            const float3 xi = act ? coor[i] : f3(-kFar, -kFar, -kFar);
            typename Op::Acc acc;
            typename Op::Self self;
            op.begin(acc, self, i, id, act, p);
            for (int q0 = 0; q0 < total; q0 += kCap) {
                const int cnt = min(kCap, total - q0);
                const int m = (cnt + 4 * kGroup - 1) / (4 * kGroup) * (4 * kGroup);
                if (b0 == be.x || total > kCap) {   // the candidates stay staged for the cube's next particles
                    __syncthreads();
                    int need = own_form;
                    const bool kept = stage(q0, cnt, m, need);
                    some = __syncthreads_or(kept);
                    form = lim.cross;
                    if (__syncthreads_or(need)) form = __syncthreads_or(need & kAny) ? kAny : 7;
                }
                if (!some || !__any_sync(0xffffffffu, act)) continue;
                const float3 xo = f3(__shfl_xor_sync(0xffffffffu, xi.x, kLanes), __shfl_xor_sync(0xffffffffu, xi.y, kLanes),
                                     __shfl_xor_sync(0xffffffffu, xi.z, kLanes));
                const float3 xa = h ? xo : xi, xb = h ? xi : xo;
                int count;
                switch (form) {
                case 0: count = mark<0>(sh, xa, xb, t, m, cutm, g); break;
                case 1: count = mark<1>(sh, xa, xb, t, m, cutm, g); break;
                case 2: count = mark<2>(sh, xa, xb, t, m, cutm, g); break;
                case 4: count = mark<4>(sh, xa, xb, t, m, cutm, g); break;
                case kAny: count = mark<kAny>(sh, xa, xb, t, m, cutm, g); break;
                default: count = mark<7>(sh, xa, xb, t, m, cutm, g);
                }
                __syncwarp();
                if (form == 0) evaluate<false>(op, ex, self, acc, sh, xi, m, count, cut2, p);
                else evaluate<true>(op, ex, self, acc, sh, xi, m, count, cut2, p);
                __syncwarp();   // the marks are written again for the next candidates
            }
            op.reduce(acc);
            if (act && t % kLanes == 0) op.finish(acc, self, i, p);
        }
    }
}

// Adds v over the lanes of a particle (a fixed tree).
__device__ __forceinline__ float lane_sum(float v) {
#pragma unroll
    for (int o = kLanes / 2; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, kLanes);
    return v;
}

}  // namespace gcsweep
