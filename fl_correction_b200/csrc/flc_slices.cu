// The emission projector with the slices as lanes, for volumes of square
// slices (sm_100a).
//
// The sample points of an angle are the same in every slice.  The kernels here
// work on slice-fastest copies -- attenuation (A, N, N, Bp), projections
// (A, N, Bp), images (N, N, Bp), Bp = B rounded up to 32 -- so that a warp
// handles one sample or pixel of 32 NS slices: the geometry (rotation, clamp,
// bilinear weights, addresses) is worked out once and applied to all of them,
// every load is a whole run of 128 NS bytes, and shared memory has no bank
// conflicts to avoid.  Making the copy costs about one read and one write of
// the attenuation, so it pays where the attenuation is used several times (an
// MLEM call) or where the backward is called.
//
//   forward   a warp walks one detector column of one angle along the beam;
//             per sample one load of the attenuation (each byte read once,
//             from HBM) and four of the image (from L1).
//   backward  a warp owns a few pixels and sums, angle by angle, the samples
//             whose bilinear footprint covers them -- about four per pixel,
//             among the 3 x 3 samples around the pixel's inverse image -- into
//             registers: no atomics, no phases, no barriers.
//
// 120 angles x 128 slices of 128^2 (1 GB of attenuation, 0.15 ms at the measured
// copy rate): copy 0.31 ms, forward 0.23 ms (lean kernel 0.42), backward 0.42 + 0.08 ms
// (lean kernel 1.37); flc_mlem with 5 iterations 4.4 ms (10.3).  180 angles x 32
// slices of 256^2: forward 0.63 ms (2.71), backward 1.37 + 0.17 ms (4.96 in row bands).
//
// Reference semantics as in flc_project.cu (atten_cuda_kernel.cu:91-446).

#include <cooperative_groups.h>

#include "flc_common.cuh"
#include "flc_geom.cuh"

namespace flc {

int check_proj_sizes(int64_t A, int64_t B, int64_t R, int64_t H, int64_t W);
int bwd_emission_launch(const float* atten, const float* ratio, const float* em,
                        const float* theta, float* out, int64_t A, int64_t B, int64_t R,
                        int64_t H, int64_t W, float clamp_min, cudaStream_t st);

// Gather backward for few slices (flc_few.cu).
bool use_few(int64_t A, int64_t B, int64_t R, int64_t H, int64_t W);
int64_t few_floats(int64_t A, int64_t B, int64_t R, int64_t N);
int bwd_few_launch(const float* atten, const float* ratio, const float* em, const float* theta,
                   float* out, const float* Cin, const float* sens, float* frame, int64_t A, int64_t B,
                   int64_t R, int64_t N, float clamp_min, int mode, float beta, float delta,
                   cudaStream_t st);

namespace {

namespace cg = cooperative_groups;

constexpr int kSThreads = 256;
constexpr int kSWarps = kSThreads / 32;

// Paired FP32 arithmetic: one instruction works on both halves of a 64-bit
// register pair, each rounded as the scalar instruction would round it.
typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pk2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk2(f32x2 r, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// acc += w * v and v *= r over NS slices
template <int NS>
__device__ __forceinline__ void axpy(float w, const float (&v)[NS], float (&acc)[NS]) {
    if constexpr (NS == 1) {
        acc[0] = fmaf(w, v[0], acc[0]);
    } else {
        const f32x2 ww = pk2(w, w);
#pragma unroll
        for (int n = 0; n < NS; n += 2)
            upk2(fma2(ww, pk2(v[n], v[n + 1]), pk2(acc[n], acc[n + 1])), acc[n], acc[n + 1]);
    }
}
template <int NS>
__device__ __forceinline__ void scale(float (&v)[NS], const float (&r)[NS]) {
    if constexpr (NS == 1) {
        v[0] *= r[0];
    } else {
#pragma unroll
        for (int n = 0; n < NS; n += 2)
            upk2(mul2(pk2(v[n], v[n + 1]), pk2(r[n], r[n + 1])), v[n], v[n + 1]);
    }
}

template <int NS>
struct Vec;
template <>
struct Vec<1> { using type = float; };
template <>
struct Vec<2> { using type = float2; };
template <>
struct Vec<4> { using type = float4; };

// The lane's NS slices at byte offset `off` from a base that is the same in
// the whole block.
template <int NS>
__device__ __forceinline__ void load_slices(const float* __restrict__ base, uint32_t off,
                                            float (&v)[NS]) {
    using T = typename Vec<NS>::type;
    const T t = __ldg(reinterpret_cast<const T*>(reinterpret_cast<const char*>(base) + off));
    if constexpr (NS == 1) {
        v[0] = t;
    } else if constexpr (NS == 2) {
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
}
// ... and at position p of `pitch` floats from the lane's base.
template <int NS>
__device__ __forceinline__ void load_at(const float* __restrict__ base, uint32_t p, uint32_t pitch,
                                        float (&v)[NS]) {
    using T = typename Vec<NS>::type;
    const T t = __ldg(reinterpret_cast<const T*>(base + (uint64_t)p * pitch));
    if constexpr (NS == 1) {
        v[0] = t;
    } else if constexpr (NS == 2) {
        v[0] = t.x; v[1] = t.y;
    } else {
        v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
}
template <int NS>
__device__ __forceinline__ void store_slices(float* p, const float (&v)[NS]) {
    using T = typename Vec<NS>::type;
    if constexpr (NS == 1) *p = v[0];
    else if constexpr (NS == 2) *reinterpret_cast<T*>(p) = make_float2(v[0], v[1]);
    else *reinterpret_cast<T*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}

// ---------------------------------------------------------------------------
// Copies between (n, B, M) and slice-fastest (n, M, Bp): tiles of 64 x 64
// through shared memory, 256 threads.  Grid (ceil(M/64), ceil(Bp/64), n).
// ---------------------------------------------------------------------------
constexpr int kTr = 64;

__global__ void __launch_bounds__(256)
slices_in_kernel(const float* __restrict__ src, float* __restrict__ dst, int B, int Bp, int M,
                 float fill) {
    __shared__ float t[kTr][kTr + 1];
    const int m0 = blockIdx.x * kTr, b0 = blockIdx.y * kTr;
    const float* s = src + (int64_t)blockIdx.z * B * M;
    float* d = dst + (int64_t)blockIdx.z * M * Bp;
    const int x = threadIdx.x & 63, y = threadIdx.x >> 6;
    float v[kTr / 4];
#pragma unroll
    for (int k = 0; k < kTr / 4; ++k) {
        const int b = b0 + y + 4 * k;
        v[k] = (b < B && m0 + x < M) ? __ldg(s + (int64_t)b * M + m0 + x) : fill;
    }
#pragma unroll
    for (int k = 0; k < kTr / 4; ++k) t[y + 4 * k][x] = v[k];
    __syncthreads();
    if (b0 + x >= Bp) return;
#pragma unroll
    for (int k = 0; k < kTr / 4; ++k) {
        const int m = m0 + y + 4 * k;
        if (m < M) d[(int64_t)m * Bp + b0 + x] = t[x][y + 4 * k];
    }
}

__global__ void __launch_bounds__(256)
slices_out_kernel(const float* __restrict__ src, float* __restrict__ dst, int B, int Bp, int M) {
    __shared__ float t[kTr][kTr + 1];
    const int m0 = blockIdx.x * kTr, b0 = blockIdx.y * kTr;
    const float* s = src + (int64_t)blockIdx.z * M * Bp;
    float* d = dst + (int64_t)blockIdx.z * B * M;
    const int x = threadIdx.x & 63, y = threadIdx.x >> 6;
    float v[kTr / 4];
#pragma unroll
    for (int k = 0; k < kTr / 4; ++k) {
        const int m = m0 + y + 4 * k;
        v[k] = (m < M && b0 + x < Bp) ? __ldg(s + (int64_t)m * Bp + b0 + x) : 0.f;
    }
#pragma unroll
    for (int k = 0; k < kTr / 4; ++k) t[y + 4 * k][x] = v[k];
    __syncthreads();
    if (m0 + x >= M) return;
#pragma unroll
    for (int k = 0; k < kTr / 4; ++k) {
        const int b = b0 + y + 4 * k;
        if (b < B) d[(int64_t)b * M + m0 + x] = t[x][y + 4 * k];
    }
}

// ---------------------------------------------------------------------------
// Forward: grid (ceil(N / 8), A, slice groups); warp = detector column.  The
// lanes work out the weights of 32 samples of the column at a time.  out =
// em * sum, or I / max(that, 1e-6) when I != nullptr.  Bound by the L1 (71% busy) and the
// latency of the attenuation it streams (1.05 GB in 0.23 ms, 4.5 TB/s); the eight columns
// of a CTA walk the beam side by side, so the taps of one are mostly in L1 from another.
// ---------------------------------------------------------------------------
constexpr int kFU = 4;     // samples whose loads are issued together

// bilerp's interpolation, f = (fx, fy).
__device__ __forceinline__ float lerp2(float2 f, float p00, float p01, float p10, float p11) {
    const float t = fmaf(f.y, p01 - p00, p00), b = fmaf(f.y, p11 - p10, p10);
    return fmaf(f.x, b - t, t);
}

template <int NS>
__global__ void __launch_bounds__(kSThreads, 3)
slices_fwd_kernel(const float* __restrict__ at, const float* __restrict__ C,
                  const float* __restrict__ em, const float* __restrict__ theta,
                  const float* __restrict__ I, float* __restrict__ out, int N, int Bp) {
    __shared__ float2 swt[kSWarps][32];
    __shared__ uint32_t soff[kSWarps][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int w = blockIdx.x * kSWarps + warp, a = blockIdx.y;
    if (w >= N) return;
    const int b0 = blockIdx.z * 32 * NS;
    const Geo g = make_geo(__ldg(theta + a), N, N);
    const float bx = col_bx(g, w), by = col_by(g, w);
    // bases that are the same in the whole block, 32-bit offsets per warp / lane
    const float* c00 = C + b0;
    const float* c01 = c00 + Bp;
    const float* c10 = c00 + (int64_t)N * Bp;
    const float* c11 = c10 + Bp;
    const float* ab = at + (int64_t)a * N * N * Bp + b0;
    const uint32_t row = (uint32_t)N * (uint32_t)Bp * 4u;
    const uint32_t lane_off = lane * (4 * NS);
    uint32_t aoff = (uint32_t)w * (uint32_t)Bp * 4u + lane_off;
    float acc[2][NS];          // even and odd samples: shorter sums
#pragma unroll
    for (int n = 0; n < NS; ++n) acc[0][n] = acc[1][n] = 0.f;
    for (int h0 = 0; h0 < N; h0 += 32) {
        {
            const float hf = (float)(h0 + lane) - g.cy;
            const Smp s = sample_xy(g, fmaf(g.c, hf, bx), fmaf(g.s, hf, by));
            __syncwarp();
            swt[warp][lane] = make_float2(s.fx, s.fy);
            soff[warp][lane] = (uint32_t)(s.i0 * N + s.j0) * (uint32_t)Bp * 4u;
            __syncwarp();
        }
        const int n_h = min(32, N - h0);
        int k0 = 0;
        for (; k0 + kFU <= n_h; k0 += kFU) {
            float av[kFU][NS], v0[kFU][NS], v1[kFU][NS], v2[kFU][NS], v3[kFU][NS];
#pragma unroll
            for (int k = 0; k < kFU; ++k) {
                load_slices<NS>(ab, aoff, av[k]);
                aoff += row;
            }
#pragma unroll
            for (int k = 0; k < kFU; ++k) {
                const uint32_t o = soff[warp][k0 + k] + lane_off;
                load_slices<NS>(c00, o, v0[k]);
                load_slices<NS>(c01, o, v1[k]);
                load_slices<NS>(c10, o, v2[k]);
                load_slices<NS>(c11, o, v3[k]);
            }
#pragma unroll
            for (int k = 0; k < kFU; ++k) {
                const float2 f = swt[warp][k0 + k];
#pragma unroll
                for (int n = 0; n < NS; ++n)
                    acc[k & 1][n] =
                        fmaf(av[k][n], lerp2(f, v0[k][n], v1[k][n], v2[k][n], v3[k][n]), acc[k & 1][n]);
            }
        }
        for (; k0 < n_h; ++k0) {
            float av[NS], v0[NS], v1[NS], v2[NS], v3[NS];
            load_slices<NS>(ab, aoff, av);
            aoff += row;
            const uint32_t o = soff[warp][k0] + lane_off;
            load_slices<NS>(c00, o, v0);
            load_slices<NS>(c01, o, v1);
            load_slices<NS>(c10, o, v2);
            load_slices<NS>(c11, o, v3);
            const float2 f = swt[warp][k0];
#pragma unroll
            for (int n = 0; n < NS; ++n)
                acc[0][n] = fmaf(av[n], lerp2(f, v0[n], v1[n], v2[n], v3[n]), acc[0][n]);
        }
    }
    const float e = __ldg(em + a);
    const int64_t o = ((int64_t)a * N + w) * Bp + b0 + lane * NS;
    float r[NS];
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        r[n] = (acc[0][n] + acc[1][n]) * e;
        if (I) r[n] = I[o + n] / fmaxf(r[n], 1e-6f);
    }
    store_slices<NS>(out + o, r);
}

// ---------------------------------------------------------------------------
// Backward
// ---------------------------------------------------------------------------
constexpr int kSlots = 16;       // list entries per block of 2 x 2 pixels (the open square of
                                 // side 3 that they cover holds at most 13 lattice points, or
                                 // 4 x 4 where it is aligned to within rounding)
constexpr int kAlways = 10;      // entries that are always added, without branches
constexpr int kSub = 4;          // lanes that build one list together
constexpr int kFlush = 32;       // angles summed in registers before they are added to the
                                 // tile's image: short sums, for their rounding error
constexpr float kRectPad = 0.01f;  // widening of a sample range, in pixels: far above the
                                   // rounding of the sample coordinates

// Pixel tile of a CTA: 32 sums per thread.
template <int NS>
struct STile;
template <>
struct STile<1> { static constexpr int TH = 16, TW = 16; };
template <>
struct STile<2> { static constexpr int TH = 8, TW = 16; };
template <>
struct STile<4> { static constexpr int TH = 8, TW = 8; };

template <int NS>
struct SSmem {
    static constexpr int SL = 32 * NS;
    static constexpr int BPW = 8 / NS;                               // blocks per warp
    static constexpr int NA = 32 / (kSub * BPW);                     // angles listed at once
    static constexpr int kLists = kSWarps * BPW * NA;
    static constexpr int WP = kSlots + 1, OP = kSlots + 2;           // list pitches (bank spread)
    static constexpr int wlist = 0;                                  // float4 [lists][WP] weights
    static constexpr int olist = wlist + kLists * WP * 16;           // uint2 [lists][OP] position, column
    static constexpr int img = olist + kLists * OP * 8;              // float [block][4][SL]
    static constexpr int bytes = img + kSWarps * BPW * 4 * SL * 4;
};

struct SArgs {
    const float* at;
    const float* ratio;    // nullptr: 1
    const float* em;
    const float* theta;
    float* out;
    const float* Cin;
    const float* sens;
    float* frame;          // border sums [split][edge][N][Bp]
    int splits;            // border sums: angles s, s + splits, ... in sum s
    int em_stride;         // floats per angle of em
    int A, N, Bp, apc, G, nty, ntx;
    float clamp_min;
    int mode;              // 0 store (clamped below), 1 MLEM update, 2 add to out
    float beta, delta;
};

// Lists the unclamped samples that cover the block of pixels (i, j), (i, j+1),
// (i+1, j), (i+1, j+1): the samples in the open square of side 3 around it, from
// the 5 x 5 around the block's inverse image, with their weights (times
// `scale`) for the four pixels, position and column.  kSub adjacent lanes take
// the candidates in turn.  Sample points are computed by the forward's
// expressions.  A list is filled up to kAlways entries, and to an even number,
// with its first sample at weight 0.  Returns the number of samples.
__device__ __forceinline__ int list_samples(const Geo& g, int N, float i, float j, float scale,
                                            bool live, int lane, float4* wl, uint2* ol) {
    const int sub = lane & (kSub - 1), lead = lane & ~(kSub - 1);
    const float xi = i + 0.5f - g.cy, yj = j + 0.5f - g.cx;
    const float ext = 1.5f * (fabsf(g.c) + fabsf(g.s)) + kRectPad;   // half-width of the square
    const int hs = (int)ceilf(fmaf(g.c, xi, fmaf(g.s, yj, g.cy)) - ext);
    const int ws = (int)ceilf(fmaf(-g.s, xi, fmaf(g.c, yj, g.cx)) - ext);
    int n = 0;
#pragma unroll
    for (int t = 0; t < (25 + kSub - 1) / kSub; ++t) {
        const int cand = t * kSub + sub;
        const int da = (cand * 13) >> 6, db = cand - da * 5;         // cand / 5 for cand < 28
        const int h = hs + da, w = ws + db;
        const float hf = (float)h - g.cy;
        const float x = fmaf(g.c, hf, col_bx(g, w)), y = fmaf(g.s, hf, col_by(g, w));
        const float dx = x - i, dy = y - j;
        const bool in = live && cand < 25 && (unsigned)h < (unsigned)N && (unsigned)w < (unsigned)N &&
                        x >= 0.f && x <= g.rmax && y >= 0.f && y <= g.cmax && dx > -1.f &&
                        dx < 2.f && dy > -1.f && dy < 2.f;
        const unsigned m = __ballot_sync(0xffffffffu, in) >> lead & ((1u << kSub) - 1u);
        const int at = n + __popc(m & ((1u << sub) - 1u));
        if (in && at < kSlots) {
            if (near_axis(g, N)) {
                wl[at] = make_float4(part_code(x, i), part_code(x, i + 1.f), part_code(y, j),
                                     part_code(y, j + 1.f));
            } else {
                const float s0 = fmaxf(1.f - fabsf(dx), 0.f) * scale;
                const float s1 = fmaxf(1.f - fabsf(dx - 1.f), 0.f) * scale;
                const float wy0 = fmaxf(1.f - fabsf(dy), 0.f), wy1 = fmaxf(1.f - fabsf(dy - 1.f), 0.f);
                wl[at] = make_float4(s0 * wy0, s0 * wy1, s1 * wy0, s1 * wy1);
            }
            ol[at] = make_uint2((uint32_t)(h * N + w), (uint32_t)w);
        }
        n = min(n + __popc(m), kSlots);
    }
    __syncwarp();
    if (n > 0 || !live) {
        const uint2 f = live ? ol[0] : make_uint2(0u, 0u);
        const int upto = n <= kAlways ? kAlways : (n + 1) & ~1;
        for (int e = n + sub; e < upto; e += kSub) {
            wl[e] = make_float4(0.f, 0.f, 0.f, 0.f);
            ol[e] = f;
        }
    }
    return n;
}

// acc[pixel] += list entries [e0, e1) of a block.  `ab`, `rb`: the lane's slices
// of position 0 and column 0; a position takes `pitch` floats.
template <int NS, bool RATIO, int E>
__device__ __forceinline__ void add_block(const float* ab, const float* rb, uint32_t pitch,
                                          const float4* wl, const uint2* ol, float (*acc)[NS]) {
    float v[E][NS];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint2 o = ol[e];
        load_at<NS>(ab, o.x, pitch, v[e]);
        if constexpr (RATIO) {
            float r[NS];
            load_at<NS>(rb, o.y, pitch, r);
            scale<NS>(v[e], r);
        }
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const float4 w = wl[e];
        axpy<NS>(w.x, v[e], acc[0]);
        axpy<NS>(w.y, v[e], acc[1]);
        axpy<NS>(w.z, v[e], acc[2]);
        axpy<NS>(w.w, v[e], acc[3]);
    }
}

// add_block at an angle near an axis: the entries are (row 0, row 1, column 0,
// column 1) codes.
template <int NS, bool RATIO, int E>
__device__ __forceinline__ void add_parts(const float* ab, const float* rb, uint32_t pitch, float em,
                                          const float4* wl, const uint2* ol, float (*acc)[NS]) {
    float v[E][NS], r[E][NS];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint2 o = ol[e];
        load_at<NS>(ab, o.x, pitch, v[e]);
        if constexpr (RATIO) load_at<NS>(rb, o.y, pitch, r[e]);
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const float4 w = wl[e];
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            const float t = __fmul_rn(v[e][n], RATIO ? __fmul_rn(r[e][n], em) : em);
            const float t0 = part_row(t, w.x), t1 = part_row(t, w.y);
            acc[0][n] += part_col(t0, w.z);
            acc[1][n] += part_col(t0, w.w);
            acc[2][n] += part_col(t1, w.z);
            acc[3][n] += part_col(t1, w.w);
        }
    }
}

// ---------------------------------------------------------------------------
// Border sums.  Samples clamped to the border (atten_cuda_kernel.cu:116-133)
// lie outside the slice by up to (sqrt(2) - 1)/2 of its side; each adds to one
// or two positions of a border line: edge 0 row 0, 1 the last rows, 2 column
// 0, 3 the last columns (samples clamped in both coordinates belong to the
// rows).  frame[split][edge][q] is the sum for position q; the far edges are
// split over the last two rows (columns) by the clamp's constant fraction when
// the sums are added to the image.
//
// Grid (warps of [edge][position pair] / 8, splits, slice groups).  A warp
// walks the strip of samples outside its two positions, six sample lines of
// five samples at a time, compacts the clamped ones into a list that runs on
// over the angles, and adds them eight at a time.
// ---------------------------------------------------------------------------
constexpr int kFrameList = 40;   // up to 7 waiting, and 30 more

template <int NS, bool RATIO, int E>
__device__ __forceinline__ void add_frame(const float* ab, const float* rb, uint32_t pitch,
                                          const uint4* lst, float (&acc)[2][NS]) {
    float v[E][NS];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint4 t = lst[e];
        load_at<NS>(ab, t.z, pitch, v[e]);
        if constexpr (RATIO) {
            float r[NS];
            load_at<NS>(rb, t.w, pitch, r);
            scale<NS>(v[e], r);
        }
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint4 t = lst[e];
        // (a value that is not finite stays with the positions it covers)
        if (__uint_as_float(t.x) != 0.f) axpy<NS>(__uint_as_float(t.x), v[e], acc[0]);
        if (__uint_as_float(t.y) != 0.f) axpy<NS>(__uint_as_float(t.y), v[e], acc[1]);
    }
}

template <int NS, bool RATIO>
__global__ void __launch_bounds__(kSThreads)
slices_frame_kernel(SArgs P) {
    __shared__ uint4 slist[kSWarps][kFrameList];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int N = P.N, nq = (N + 1) / 2;
    const int id = blockIdx.x * kSWarps + warp;
    if (id >= 4 * nq) return;
    const int e = id / nq, q = 2 * (id - e * nq);
    const bool row = e < 2, low = !(e & 1);
    const int b0 = blockIdx.z * 32 * NS + lane * NS;
    const uint32_t pitch = (uint32_t)P.Bp;
    const float* ab = P.at + b0;
    const float* rb = RATIO ? P.ratio + b0 : nullptr;
    uint4* lst = slist[warp];
    const int line = lane / 5, cell = lane - line * 5;      // lanes 30, 31 idle
    float acc[2][NS];
#pragma unroll
    for (int n = 0; n < NS; ++n) acc[0][n] = acc[1][n] = 0.f;
    int n = 0;                                              // entries waiting
    for (int a = blockIdx.y; a < P.A; a += P.splits) {
        const Geo g = make_geo(__ldg(P.theta + a), N, N);
        const float em = __ldg(P.em + (int64_t)a * P.em_stride);
        const float depth = g.cy * (fabsf(g.c) + fabsf(g.s) - 1.f) + 0.5f;   // farthest outside
        const float edge = low ? 0.f : g.rmax;
        // sample coordinates (h, w) of the strip's axis: outward distance t at
        // the middle of the two positions is (h, w) = (hm, wm) + t (uh, uw)
        const float om = edge - g.cy, pm = (float)q + 0.5f - g.cy, sg = low ? -1.f : 1.f;
        const float xm = row ? om : pm, ym = row ? pm : om;
        const float hm = g.c * xm + g.s * ym + g.cy, wm = g.c * ym - g.s * xm + g.cy;
        const float uh = sg * (row ? g.c : g.s), uw = sg * (row ? -g.s : g.c);
        // lines along the axis' steeper coordinate (m), five samples across (k)
        const bool hmaj = fabsf(uh) >= fabsf(uw);
        const float mm = hmaj ? hm : wm, km = hmaj ? wm : hm;
        const float um = hmaj ? uh : uw, slope = (hmaj ? uw : uh) / um;
        const float half = 1.5f * fabsf(hmaj ? uw : uh) + kRectPad;   // the strip's half-width, along m
        const float m1 = mm + depth * um;
        const int mlo = max(0, (int)ceilf(fminf(mm, m1) - half));
        const int mhi = min(N - 1, (int)floorf(fmaxf(mm, m1) + half));
        const float across = 1.5f / fabsf(um) + kRectPad;
        for (int l0 = mlo; l0 <= mhi; l0 += 6) {
            const int m = l0 + line;
            const int k = (int)ceilf(km + ((float)m - mm) * slope - across) + cell;
            const int h = hmaj ? m : k, w = hmaj ? k : m;
            const float hf = (float)h - g.cy;
            const float x = fmaf(g.c, hf, col_bx(g, w)), y = fmaf(g.s, hf, col_by(g, w));
            const float o = row ? x : y;
            const float z = row ? fminf(fmaxf(y, 0.f), g.cmax) : x;
            const float w0 = tap_weight(z, (float)q), w1 = tap_weight(z, (float)(q + 1));
            const bool in = lane < 30 && m <= mhi && (unsigned)k < (unsigned)N &&
                            (low ? o < 0.f : o > edge) && (row || (x >= 0.f && x <= g.rmax)) &&
                            (w0 > 0.f || w1 > 0.f);
            const unsigned mask = __ballot_sync(0xffffffffu, in);
            if (mask == 0) continue;
            if (in)
                lst[n + __popc(mask & ((1u << lane) - 1u))] =
                    make_uint4(__float_as_uint(w0 * em), __float_as_uint(w1 * em),
                               ((uint32_t)a * N + h) * N + w, (uint32_t)a * N + w);
            n += __popc(mask);
            __syncwarp();
            int k0 = 0;
            for (; k0 + 8 <= n; k0 += 8) add_frame<NS, RATIO, 8>(ab, rb, pitch, lst + k0, acc);
            if (k0 > 0) {
                const uint4 t = lst[min(k0 + lane, kFrameList - 1)];
                __syncwarp();
                if (lane < n - k0) lst[lane] = t;
                n -= k0;
                __syncwarp();
            }
        }
    }
    for (int k = 0; k < n; ++k) add_frame<NS, RATIO, 1>(ab, rb, pitch, lst + k, acc);
    float* f = P.frame + (((int64_t)blockIdx.y * 4 + e) * N + q) * P.Bp + b0;
    store_slices<NS>(f, acc[0]);
    if (q + 1 < N) store_slices<NS>(f + P.Bp, acc[1]);
}

// Sum of the unclamped samples that cover pixel (i, j) of slice sl, each on its own.  A
// block's samples go to its four pixels alike, at weight 0 where they don't cover one, so a
// value that is not finite makes all four sums so; such a sum is made again here.  (Weights
// of 0 left out in add_block: 4 and 13% on the kernel for NS = 4 and 1.)
__device__ __noinline__ float covered_sum(const float* __restrict__ at, const float* __restrict__ ratio,
                                          const float* __restrict__ em, const float* __restrict__ theta,
                                          int em_stride, int A, int N, int Bp, int sl, int i, int j) {
    const float fi = (float)i, fj = (float)j;
    double sum = 0.0;
    for (int a = 0; a < A; ++a) {
        const Geo g = make_geo(__ldg(theta + a), N, N);
        const float e = __ldg(em + (int64_t)a * em_stride), xi = fi - g.cy, yj = fj - g.cx;
        const int h0 = (int)rintf(fmaf(g.c, xi, fmaf(g.s, yj, g.cy))) - 1;
        const int w0 = (int)rintf(fmaf(-g.s, xi, fmaf(g.c, yj, g.cx))) - 1;
        for (int k = 0; k < 9; ++k) {
            const int h = h0 + k / 3, w = w0 + k % 3;
            if ((unsigned)h >= (unsigned)N || (unsigned)w >= (unsigned)N) continue;
            const float hf = (float)h - g.cy;
            const float x = fmaf(g.c, hf, col_bx(g, w)), y = fmaf(g.s, hf, col_by(g, w));
            if (!(x >= 0.f && x <= g.rmax && y >= 0.f && y <= g.cmax)) continue;
            const float cr = part_code(x, fi), cc = part_code(y, fj);
            if (cr == 0.f || cc == 0.f) continue;
            float v = __ldg(at + (((int64_t)a * N + h) * N + w) * Bp + sl);
            v = __fmul_rn(v, ratio ? __fmul_rn(__ldg(ratio + ((int64_t)a * N + w) * Bp + sl), e) : e);
            sum += (double)part_col(part_row(v, cr), cc);
        }
    }
    return (float)sum;
}

// The backward: unclamped samples, then the border sums.  Grid (G * tiles, slice
// groups), cluster (G, 1, 1): CTA g of a tile sums angles [g * apc, ...).
// Bound by the latency of its loads (two 128 NS byte runs, attenuation and ratio, per
// sample and block of pixels; 16 warps an SM issue in 37% of the slots and wait for these,
// the L1 is 44% busy, and each byte comes from HBM once).  What brought the 120
// angles x 128 slices of 128^2 down: one pixel at a time, the list's loads behind
// a branch per pixel 0.68 ms (NS = 4; 1.33 and 2.75 ms with NS = 2 and 1); loads
// of several pixels in flight 0.59; blocks of 2 x 2 pixels, nine samples instead
// of four times four 0.52; ten samples without a branch 0.51; the border sums in
// a kernel of their own instead of in the border tiles 0.39 + 0.08.
template <int NS, bool RATIO>
__global__ void __launch_bounds__(kSThreads, 2)
slices_bwd_kernel(SArgs P) {
    using L = SSmem<NS>;
    constexpr int SL = L::SL, BPW = L::BPW, NA = L::NA;
    constexpr unsigned kAll = (1u << BPW) - 1u;
    extern __shared__ __align__(128) char smem[];
    cg::cluster_group cluster = cg::this_cluster();
    const int G = P.G, rank = blockIdx.x % G;        // clusters run along x
    float4* swl = reinterpret_cast<float4*>(smem + L::wlist);
    uint2* sol = reinterpret_cast<uint2*>(smem + L::olist);
    const int N = P.N, NB = (N + 1) / 2;             // blocks per side
    const int ty = blockIdx.x / G / P.ntx, tx = blockIdx.x / G - ty * P.ntx;
    const int r0 = 2 * (ty * NB / P.nty), r1 = min(N, 2 * ((ty + 1) * NB / P.nty));
    const int c0 = 2 * (tx * NB / P.ntx), c1 = min(N, 2 * ((tx + 1) * NB / P.ntx));
    const int th = r1 - r0, tw = c1 - c0, npx = th * tw;
    const int bw = (tw + 1) / 2, nblk = (th + 1) / 2 * bw;
    const int b0 = blockIdx.y * SL;
    const int a0 = rank * P.apc, a1 = min(P.A, a0 + P.apc);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t pitch = (uint32_t)P.Bp;
    // lists are built for NA angles at once, kSub lanes per block and angle
    const int bblk = lane / kSub % BPW, bang = lane / (kSub * BPW);
    const int blk = warp * BPW + bblk;               // tile block, row-major
    const int brow = blk / bw, bcol = blk - brow * bw;
    // the sums of this thread's slices: in registers, and in its own words of the
    // tile's image [block][pixel][lane]
    float* simg = reinterpret_cast<float*>(smem + L::img);
    float* own = simg + warp * BPW * 4 * SL + lane * NS;
    float acc[BPW][4][NS];
#pragma unroll
    for (int k = 0; k < BPW; ++k)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
#pragma unroll
            for (int n = 0; n < NS; ++n) acc[k][q][n] = 0.f;
            store_slices<NS>(own + (k * 4 + q) * SL, acc[k][q]);
        }
    auto flush = [&]() {
#pragma unroll
        for (int k = 0; k < BPW; ++k)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float* p = own + (k * 4 + q) * SL;
#pragma unroll
                for (int n = 0; n < NS; ++n) {
                    acc[k][q][n] += p[n];
                }
                store_slices<NS>(p, acc[k][q]);
#pragma unroll
                for (int n = 0; n < NS; ++n) acc[k][q][n] = 0.f;
            }
    };
    int cnt = 0;                                     // this lane's block and angle: samples
    unsigned dead = 0;                               // the warp's blocks past the tile
#pragma unroll
    for (int k = 0; k < BPW; ++k) dead |= warp * BPW + k >= nblk ? 1u << k : 0u;
    for (int a = a0; a < a1; ++a) {
        const Geo g = make_geo(__ldg(P.theta + a), N, N);
        const float* ab = P.at + (int64_t)a * N * N * P.Bp + b0 + lane * NS;
        const float* rb = RATIO ? P.ratio + (int64_t)a * N * P.Bp + b0 + lane * NS : nullptr;
        const float em = __ldg(P.em + (int64_t)a * P.em_stride);
        // ---- the tile's pixels, from the unclamped samples ----
        const int par = (a - a0) % NA;
        if (par == 0) {
            const int al = min(a + bang, a1 - 1);
            const Geo gl = NA == 1 ? g : make_geo(__ldg(P.theta + al), N, N);
            const int l = (warp * NA + bang) * BPW + bblk;
            __syncwarp();                            // the last lists have been read
            cnt = list_samples(gl, N, (float)(r0 + 2 * brow), (float)(c0 + 2 * bcol),
                               NA == 1 ? em : __ldg(P.em + (int64_t)al * P.em_stride), blk < nblk, lane, swl + l * L::WP,
                               sol + l * L::OP);
            __syncwarp();
        }
        // per block of this angle (its lanes: par * BPW * kSub + k * kSub ...)
        int cnts[BPW];
        unsigned some = dead;
#pragma unroll
        for (int k = 0; k < BPW; ++k) {
            cnts[k] = __shfl_sync(0xffffffffu, cnt, (par * BPW + k) * kSub);
            some |= cnts[k] > 0 ? 1u << k : 0u;
        }
        const int l0 = (warp * NA + par) * BPW;
        const float4* wl = swl + l0 * L::WP;
        const uint2* ol = sol + l0 * L::OP;
        // the first kAlways of every block, without branches so that many loads
        // are in flight; a block that no sample reaches (outside the rotated
        // slice) has no list
        if (near_axis(g, N)) {
#pragma unroll
            for (int k = 0; k < BPW; ++k) {
                if (!(some >> k & 1u)) continue;
#pragma unroll 1
                for (int e = 0; e < cnts[k]; e += 2)
                    add_parts<NS, RATIO, 2>(ab, rb, pitch, em, wl + k * L::WP + e, ol + k * L::OP + e, acc[k]);
            }
            if ((a - a0) % kFlush == kFlush - 1) flush();
            continue;
        }
        if (some == kAll) {
#pragma unroll
            for (int k = 0; k < BPW; ++k) {
                add_block<NS, RATIO, kAlways / 2>(ab, rb, pitch, wl + k * L::WP, ol + k * L::OP, acc[k]);
                add_block<NS, RATIO, kAlways / 2>(ab, rb, pitch, wl + k * L::WP + kAlways / 2,
                                                  ol + k * L::OP + kAlways / 2, acc[k]);
            }
        } else {
#pragma unroll
            for (int k = 0; k < BPW; ++k) {
                if (!(some >> k & 1u)) continue;
                add_block<NS, RATIO, kAlways / 2>(ab, rb, pitch, wl + k * L::WP, ol + k * L::OP, acc[k]);
                add_block<NS, RATIO, kAlways / 2>(ab, rb, pitch, wl + k * L::WP + kAlways / 2,
                                                  ol + k * L::OP + kAlways / 2, acc[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < BPW; ++k)
            for (int e = kAlways; e < cnts[k]; e += 2)
                add_block<NS, RATIO, 2>(ab, rb, pitch, wl + k * L::WP + e, ol + k * L::OP + e, acc[k]);
        if ((a - a0) % kFlush == kFlush - 1) flush();
    }
    // ---- sum over the cluster, epilogue ----
    flush();
    cluster.sync();
    const int n = npx * SL, share = (npx + G - 1) / G * SL;
    const int i1 = min(n, (rank + 1) * share);
    for (int i = rank * share + threadIdx.x; i < i1; i += kSThreads) {
        const int p = i / SL, sl = i - p * SL;
        const int pr = p / tw, pc = p - pr * tw, r = r0 + pr, c = c0 + pc;
        float s = 0.f;
        const int k = ((pr >> 1) * bw + (pc >> 1)) * 4 + (pr & 1) * 2 + (pc & 1);
        for (int q = 0; q < G; ++q) s += cluster.map_shared_rank(simg, q)[k * SL + sl];
        if (!(fabsf(s) <= 3.4e38f))
            s = covered_sum(P.at, P.ratio, P.em, P.theta, P.em_stride, P.A, N, P.Bp, b0 + sl, r, c);
        if (r == 0 || c == 0 || r >= N - 2 || c >= N - 2) {
            const Geo g0 = make_geo(0.f, N, N);
            const float fr = r == N - 1 ? g0.fxh : 1.f - g0.fxh, fc = c == N - 1 ? g0.fyh : 1.f - g0.fyh;
            for (int q = 0; q < P.splits; ++q) {
                const float* f = P.frame + (int64_t)q * 4 * N * P.Bp + b0 + sl;
                if (r == 0) s += f[(int64_t)c * P.Bp];
                if (r >= N - 2) s += f[(int64_t)(N + c) * P.Bp] * fr;
                if (c == 0) s += f[(int64_t)(2 * N + r) * P.Bp];
                if (c >= N - 2) s += f[(int64_t)(3 * N + r) * P.Bp] * fc;
            }
        }
        const int64_t o = ((int64_t)r * N + c) * P.Bp + b0 + sl;
        if (P.mode == 2) {
            P.out[o] += s;
        } else if (P.mode == 0) {
            P.out[o] = P.clamp_min > 0.f ? fmaxf(s, P.clamp_min) : s;
        } else {
            const float* ci = P.Cin + o;
            const float cp = *ci;
            float den = P.sens[o];
            if (P.beta > 0.f) {
                const int64_t up = (int64_t)N * P.Bp;
                float hg = 0.f;
                if (r > 0) { const float d = cp - ci[-up]; hg += fabsf(d) <= P.delta ? d : copysignf(P.delta, d); }
                if (r + 1 < N) { const float d = cp - ci[up]; hg += fabsf(d) <= P.delta ? d : copysignf(P.delta, d); }
                if (c > 0) { const float d = cp - ci[-P.Bp]; hg += fabsf(d) <= P.delta ? d : copysignf(P.delta, d); }
                if (c + 1 < N) { const float d = cp - ci[P.Bp]; hg += fabsf(d) <= P.delta ? d : copysignf(P.delta, d); }
                den = __fadd_rn(den, __fmul_rn(P.beta, hg));
            }
            P.out[o] = fmaxf(__fmul_rn(cp, s) / den, 0.f);
        }
    }
    cluster.sync();
}

// Tiles per side, whole blocks each.
int tiles(int64_t N, int T) { return (int)ceil_div((N + 1) / 2, T / 2); }

// Angle sets of the border sums: a warp's loads wait for one another, so few
// angles each.
int frame_splits(int64_t A) { return (int)(A < 16 ? A : 16); }

template <int NS, bool RATIO>
int bwd_groups(SArgs P, int groups, cudaStream_t st) {
    slices_frame_kernel<NS, RATIO>
        <<<dim3((unsigned)ceil_div(4 * ((P.N + 1) / 2), kSWarps), (unsigned)P.splits, (unsigned)groups),
           kSThreads, 0, st>>>(P);
    FLC_TRY(check_launch("slices_frame_kernel"));
    P.nty = tiles(P.N, STile<NS>::TH);
    P.ntx = tiles(P.N, STile<NS>::TW);
    const void* fn = (const void*)slices_bwd_kernel<NS, RATIO>;
    const ClusterPlan p = plan_cluster(fn, P.A, (int64_t)P.nty * P.ntx * groups, SSmem<NS>::bytes, kSThreads);
    P.apc = p.apc;
    P.G = p.G;
    void* args[] = {&P};
    return launch_cluster(fn, dim3((unsigned)(p.G * P.nty * P.ntx), (unsigned)groups), p.G,
                          SSmem<NS>::bytes, st, args, kSThreads);
}

template <int NS>
int fwd_groups(const float* at, const float* C, const float* em, const float* theta, const float* I,
               float* out, int64_t A, int64_t N, int64_t Bp, int groups, cudaStream_t st) {
    slices_fwd_kernel<NS><<<dim3((unsigned)ceil_div(N, kSWarps), (unsigned)A, (unsigned)groups),
                            kSThreads, 0, st>>>(at, C, em, theta, I, out, (int)N, (int)Bp);
    return check_launch("slices_fwd_kernel");
}

// Slices per lane for a padded slice count (slices_pad), so that one launch
// covers all of them.
int slices_per_lane(int64_t Bp) { return Bp % 128 == 0 ? 4 : Bp % 64 == 0 ? 2 : 1; }

int64_t frame_floats(int64_t A, int64_t N, int64_t Bp) { return (int64_t)frame_splits(A) * 4 * N * Bp; }

}  // namespace

// Slice count of the copies: a multiple of 32, 64 or 128, whichever takes the
// least time in groups of that many slices (forward + backward of 120 angles of
// 128^2: 0.36, 0.42 and 0.64 ms a group).
int64_t slices_pad(int64_t B) {
    const int64_t n1 = ceil_div(B, 32), n2 = ceil_div(B, 64), n4 = ceil_div(B, 128);
    const int64_t t1 = 36 * n1, t2 = 42 * n2, t4 = 64 * n4;
    return t1 <= t2 && t1 <= t4 ? 32 * n1 : t2 <= t4 ? 64 * n2 : 128 * n4;
}

// Whether the slice-lane kernels take the shape (32-bit byte offsets within one
// angle, 32-bit positions over all).
bool slices_takes(int64_t A, int64_t B, int64_t H, int64_t W) {
    return H == W && H >= 16 && H <= 4096 && A <= 65535 && slices_pad(B) <= 65535 &&
           4 * slices_pad(B) * H * W < (1LL << 32) && A * H * W < (1LL << 32);
}

// Whether a call that has the scratch goes to the slice-lane kernels (the
// "proj.slices" knob: 1 wherever they take the shape, 2 never).  A group of 32
// slices costs the same however many of them exist (33 to 37 are padded to 64, which
// below 112^2 the splats still beat), and the copies and the five launches of a backward
// have to be paid for.  Up to ten slices the kernels of flc_few.cu are the others, above
// the lean or band kernels.  Microseconds, others / these:
//   MLEM, 5 iterations: 60 angles 64^2 x 16 slices 617 / 598; 90 x 96^2: 8 899 / 1252,
//   24 1368 / 1245, 33 1478 / 1624, 48 1821 / 1619; 120 x 128^2: 8 1743 / 2599, 12
//   2896 / 2600 (the one side of the line where the other would be a little faster), 16
//   3202 / 2597, 128 10341 / 4440; 180 x 256^2: 8 8991 / 12963, 32 36790 / 12944.
//   One backward: 120 x 128^2: 8 slices 245 / 430, 16 463 / 432, 128 1369 / 903; 90 x
//   96^2: 48 234 / 286, 96 411 / 378; 60 x 64^2: 48 104 / 110, 64 123 / 115; 30 x 48^2:
//   64 51 / 69, 128 90 / 79 (by the line at 8 million samples 64 stay with the others);
//   180 x 256^2: 8 1202 / 2344, 16 2764 / 2346, 32 4986 / 2379.
// Where the lean splats run with three CTAs an SM (small_image), a backward whose slices
// fill their group badly, or with few angles, loses: 60 x 64^2: 72 slices (of 128) 130 /
// 157, 136 (of 192) 214 / 252, 96 171 / 158; 40 x 80^2: 65 110 / 168; 90 x 96^2: 72 305 /
// 370, 136 506 / 758, 96 410 / 372; 40 x 128^2: 16 154 / 175, 48 198 / 224, 72 302 / 332,
// 96 365 / 334; 120 x 128^2: 33 481 / 529, 40 548 / 531, 65 717 / 889, 96 1047 / 891; two
// references, 60 x 64^2: 70 230 / 265, 100 333 / 264.
bool use_slices(int64_t A, int64_t B, int64_t R, int64_t H, int64_t W, bool mlem) {
    const int64_t knob = tune(kTuneProjSlices);
    if (tune(kTuneProjLegacy) != 0 || tune(kTuneProjBand) != 0 || knob == 2) return false;
    if (!slices_takes(A, B, H, W)) return false;
    if (knob == 1) return true;
    const int64_t work = A * B * H * W;
    if (mlem) return B >= 16 && work >= 3000000 && !(H < 112 && B > 32 && B < 38);
    if (B < (H >= 128 ? 16 : 64) || work < 8000000) return false;
    if (!small_image(R, H, W)) return true;
    return B > 64 ? 4 * B >= 3 * slices_pad(B) : A >= 48 && (B <= 32 || B >= 40);
}

int slices_in(const float* src, float* dst, int64_t n, int64_t B, int64_t M, cudaStream_t st) {
    const int64_t Bp = slices_pad(B);
    for (int64_t i = 0; i < n; i += 65535) {
        const int64_t k = n - i < 65535 ? n - i : 65535;
        slices_in_kernel<<<dim3((unsigned)ceil_div(M, kTr), (unsigned)ceil_div(Bp, kTr), (unsigned)k),
                           256, 0, st>>>(src + i * B * M, dst + i * Bp * M, (int)B, (int)Bp, (int)M, 0.f);
        FLC_TRY(check_launch("slices_in_kernel"));
    }
    return FLC_OK;
}

int slices_out(const float* src, float* dst, int64_t n, int64_t B, int64_t M, cudaStream_t st) {
    const int64_t Bp = slices_pad(B);
    for (int64_t i = 0; i < n; i += 65535) {
        const int64_t k = n - i < 65535 ? n - i : 65535;
        slices_out_kernel<<<dim3((unsigned)ceil_div(M, kTr), (unsigned)ceil_div(Bp, kTr), (unsigned)k),
                            256, 0, st>>>(src + i * Bp * M, dst + i * B * M, (int)B, (int)Bp, (int)M);
        FLC_TRY(check_launch("slices_out_kernel"));
    }
    return FLC_OK;
}

// Forward on slice-fastest data: out (A, N, Bp) = em * P C, or I / max(that, 1e-6).
int slices_fwd(const float* at, const float* C, const float* em, const float* theta, const float* I,
               float* out, int64_t A, int64_t N, int64_t Bp, cudaStream_t st) {
    switch (slices_per_lane(Bp)) {
        case 4: return fwd_groups<4>(at, C, em, theta, I, out, A, N, Bp, (int)(Bp / 128), st);
        case 2: return fwd_groups<2>(at, C, em, theta, I, out, A, N, Bp, (int)(Bp / 64), st);
        default: return fwd_groups<1>(at, C, em, theta, I, out, A, N, Bp, (int)(Bp / 32), st);
    }
}

// Backward on slice-fastest data, em with em_stride floats per angle (mode:
// SArgs); frame: frame_floats floats of scratch.
int slices_bwd(const float* at, const float* ratio, const float* em, int em_stride,
               const float* theta, float* out, const float* Cin, const float* sens, float* frame,
               int64_t A, int64_t N, int64_t Bp, float clamp_min, int mode, float beta, float delta,
               cudaStream_t st) {
    SArgs P = {};
    P.at = at;
    P.ratio = ratio;
    P.em = em;
    P.em_stride = em_stride;
    P.theta = theta;
    P.out = out;
    P.Cin = Cin;
    P.sens = sens;
    P.frame = frame;
    P.splits = frame_splits(A);
    P.A = (int)A;
    P.N = (int)N;
    P.Bp = (int)Bp;
    P.clamp_min = clamp_min;
    P.mode = mode;
    P.beta = beta;
    P.delta = delta;
    switch (slices_per_lane(Bp)) {
        case 4: return ratio ? bwd_groups<4, true>(P, (int)(Bp / 128), st) : bwd_groups<4, false>(P, (int)(Bp / 128), st);
        case 2: return ratio ? bwd_groups<2, true>(P, (int)(Bp / 64), st) : bwd_groups<2, false>(P, (int)(Bp / 64), st);
        default: return ratio ? bwd_groups<1, true>(P, (int)(Bp / 32), st) : bwd_groups<1, false>(P, (int)(Bp / 32), st);
    }
}

namespace {

size_t al256(size_t n) { return (n + 255) & ~(size_t)255; }

// Buffers of an MLEM call on slice-fastest data.
struct SliceBufs {
    float *at, *I, *ratio, *sens, *C[2], *frame;
    size_t bytes;
};

SliceBufs mlem_bufs(int64_t A, int64_t N, int64_t Bp, char* base) {
    SliceBufs b = {};
    size_t off = 0;
    auto take = [&](int64_t n) {
        char* p = base ? base + off : nullptr;
        off += al256(sizeof(float) * (size_t)n);
        return (float*)p;
    };
    b.at = take(A * N * N * Bp);
    b.I = take(A * N * Bp);
    b.ratio = take(A * N * Bp);
    b.sens = take(N * N * Bp);
    b.C[0] = take(N * N * Bp);
    b.C[1] = take(N * N * Bp);
    b.frame = take(frame_floats(A, N, Bp));
    b.bytes = off;
    return b;
}

// Angles per pass of a single backward: about 512 MB of copied attenuation.
int64_t bwd_chunk(int64_t A, int64_t N, int64_t Bp) {
    int64_t c = (512LL << 20) / (4 * N * N * Bp);
    c = c < 1 ? 1 : (c > A ? A : c);
    return ceil_div(A, ceil_div(A, c));              // evened
}

size_t bwd_bytes(int64_t A, int64_t R, int64_t N, int64_t Bp) {
    return al256(sizeof(float) * (size_t)(bwd_chunk(A, N, Bp) * N * N * Bp)) +
           al256(sizeof(float) * (size_t)(A * N * Bp)) + al256(sizeof(float) * (size_t)(R * N * N * Bp)) +
           al256(sizeof(float) * (size_t)frame_floats(A, N, Bp));
}

}  // namespace

// Scratch of mlem_slices, 0 where it does not take the call.
size_t mlem_slices_bytes(int64_t A, int64_t B, int64_t R, int64_t H, int64_t W) {
    if (R != 1 || !use_slices(A, B, R, H, W, true)) return 0;
    return mlem_bufs(A, H, slices_pad(B), nullptr).bytes;
}

// flc_mlem (R = 1) on slice-fastest copies: the copies and the sensitivity, then
// two launches per iteration.  n_iter >= 1.
int mlem_slices(float* C, const float* atten, const float* em, const float* theta, const float* I,
                int64_t n_iter, float beta, float delta, int64_t A, int64_t B, int64_t N, void* ws,
                cudaStream_t st) {
    const int64_t Bp = slices_pad(B);
    const SliceBufs b = mlem_bufs(A, N, Bp, (char*)ws);
    FLC_TRY(slices_in(atten, b.at, A, B, N * N, st));
    FLC_TRY(slices_in(I, b.I, A, B, N, st));
    FLC_TRY(slices_in(C, b.C[0], 1, B, N * N, st));
    // sens = max(P^T 1, 1e-6)   (atten_cuda.cpp:308-314)
    FLC_TRY(slices_bwd(b.at, nullptr, em, 1, theta, b.sens, nullptr, nullptr, b.frame, A, N, Bp, 1e-6f,
                       0, 0.f, 0.f, st));
    for (int64_t it = 0; it < n_iter; ++it) {
        const float* cur = b.C[it & 1];
        FLC_TRY(slices_fwd(b.at, cur, em, theta, b.I, b.ratio, A, N, Bp, st));
        FLC_TRY(slices_bwd(b.at, b.ratio, em, 1, theta, b.C[~it & 1], cur, b.sens, b.frame, A, N, Bp,
                           0.f, 1, beta, delta, st));
    }
    return slices_out(b.C[n_iter & 1], C, 1, B, N * N, st);
}

// flc_bwd_emission on slice-fastest copies, a part of the angles at a time.
int bwd_slices(const float* atten, const float* ratio, const float* em, const float* theta,
               float* out, int64_t A, int64_t B, int64_t R, int64_t N, void* ws, cudaStream_t st) {
    const int64_t Bp = slices_pad(B), chunk = bwd_chunk(A, N, Bp);
    float* at = (float*)ws;
    float* q = (float*)((char*)at + al256(sizeof(float) * (size_t)(chunk * N * N * Bp)));
    float* img = (float*)((char*)q + al256(sizeof(float) * (size_t)(A * N * Bp)));
    float* frame = (float*)((char*)img + al256(sizeof(float) * (size_t)(R * N * N * Bp)));
    FLC_TRY(slices_in(ratio, q, A, B, N, st));
    for (int64_t a0 = 0; a0 < A; a0 += chunk) {
        const int64_t n = A - a0 < chunk ? A - a0 : chunk;
        FLC_TRY(slices_in(atten + a0 * B * N * N, at, n, B, N * N, st));
        for (int64_t r = 0; r < R; ++r)
            FLC_TRY(slices_bwd(at, q + a0 * N * Bp, em + a0 * R + r, (int)R, theta + a0,
                               img + r * N * N * Bp, nullptr, nullptr, frame, n, N, Bp, 0.f, a0 ? 2 : 0,
                               0.f, 0.f, st));
    }
    return slices_out(img, out, R, B, N * N, st);
}

}  // namespace flc

using namespace flc;

extern "C" size_t flc_bwd_emission_workspace_bytes(int64_t A, int64_t B, int64_t R, int64_t H,
                                                   int64_t W) {
    if (A < 1 || B < 1 || R < 1 || H < 2 || W < 2) return 0;
    if (use_slices(A, B, R, H, W, false)) return bwd_bytes(A, R, H, slices_pad(B));
    return use_few(A, B, R, H, W) ? sizeof(float) * (size_t)few_floats(A, B, R, H) : 0;
}

extern "C" int flc_bwd_emission_ws(const float* atten, const float* ratio, const float* em,
                                   const float* theta, float* out, int64_t A, int64_t B, int64_t R,
                                   int64_t H, int64_t W, void* workspace, size_t workspace_bytes,
                                   void* stream) {
    clear_error();
    FLC_REQUIRE(atten && ratio && em && theta && out, "flc_bwd_emission_ws: null pointer argument");
    FLC_TRY(check_proj_sizes(A, B, R, H, W));
    if (workspace && ((uintptr_t)workspace & 255) != 0) {
        set_error("flc_bwd_emission_ws: workspace must be 256-byte aligned");
        return FLC_ERR_ALIGNMENT;
    }
    const size_t need = flc_bwd_emission_workspace_bytes(A, B, R, H, W);
    if (workspace && need && workspace_bytes >= need) {
        if (use_slices(A, B, R, H, W, false))
            return bwd_slices(atten, ratio, em, theta, out, A, B, R, H, workspace, as_stream(stream));
        return bwd_few_launch(atten, ratio, em, theta, out, nullptr, nullptr, (float*)workspace, A, B, R, H,
                              0.f, 0, 0.f, 0.f, as_stream(stream));
    }
    return bwd_emission_launch(atten, ratio, em, theta, out, A, B, R, H, W, 0.f, as_stream(stream));
}
