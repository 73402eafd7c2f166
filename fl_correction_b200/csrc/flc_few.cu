// Backward emission projector in gather form for a few square slices (sm_100a).
//
// With few slices the splats of flc_project.cu leave the GPU idle: one slice is
// one cluster of at most eight CTAs, each behind six barriers an angle.  Here a
// thread owns a pixel and, for its share of the angles, sums the samples whose
// bilinear footprint covers it, among the 3 x 3 samples around the pixel's inverse
// image: no barriers and no shared image, and as many threads as pixels times
// angle shares.  About 130 instructions per pixel and angle against 92 per sample
// of the splat, but with every lane of the chip at work.
//
// Samples clamped to the border (atten_cuda_kernel.cu:116-133) are summed first, by
// few_frame_kernel: a warp per border line and pair of positions walks the strip of
// samples outside them (as slices_frame_kernel in flc_slices.cu), a lane a sample.
//
// 90 angles of one 96^2 slice: 22 us (8 border, 14 pixels) against 155 us.

#include "flc_common.cuh"
#include "flc_geom.cuh"

namespace flc {

// Whether the lean forward takes the slice (flc_project.cu).
bool fwd2_takes(int64_t R, int64_t H, int64_t W);
// ... and whether it is compiled for the width.
bool fwd2_fixed_width(int64_t W);

namespace {

constexpr int kFewWarps = 16;    // angle shares of a CTA
constexpr int kFewR = 8;         // references at most
constexpr int kTrig = 128;       // angles whose cosines and sines a CTA keeps at a time
constexpr float kPad = 0.01f;    // widening of a sample range: far above the rounding of
                                 // the sample coordinates

struct FewArgs {
    const float* atten;
    const float* ratio;    // nullptr: 1
    const float* em;
    const float* theta;
    float* out;
    const float* Cin;
    const float* sens;
    float* frame;          // border sums [split][R][edge][B][N]
    int splits;            // angles s, s + splits, ... in sum s
    int A, B, R, N;
    float clamp_min;
    int mode;              // bwd_epilogue
    float beta, delta;
};

// make_geo with the angle's cosine and sine from a table (they are make_geo's).
__device__ __forceinline__ float2 trig_of(const float* __restrict__ theta, int a) {
    const float th = __ldg(theta + a);
    return make_float2(cosf(-th), sinf(-th));
}
__device__ __forceinline__ Geo geo_of(float2 cs, int H, int W) {
    Geo g = make_geo(0.f, H, W);
    g.c = cs.x;
    g.s = cs.y;
    return g;
}

// Grid (position pairs of the four edges / 8, splits, B), 8 warps.
__global__ void __launch_bounds__(256)
few_frame_kernel(FewArgs P) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int N = P.N, nq = (N + 1) / 2;
    const int id = blockIdx.x * 8 + warp;
    __shared__ float2 trig[kTrig];
    const int e = id / nq, q = 2 * (id - e * nq), b = blockIdx.z;
    const bool row = e < 2, low = !(e & 1);
    const int line = lane / 5, cell = lane - line * 5;      // lanes 30, 31 idle
    float acc[kFewR][2];
#pragma unroll
    for (int r = 0; r < kFewR; ++r) acc[r][0] = acc[r][1] = 0.f;
    for (int a = blockIdx.y, n = 0; a < P.A; a += P.splits, ++n) {
        if (n % kTrig == 0) {
            __syncthreads();
            for (int t = threadIdx.x; t < kTrig && a + t * P.splits < P.A; t += 256)
                trig[t] = trig_of(P.theta, a + t * P.splits);
            __syncthreads();
        }
        if (id >= 4 * nq) continue;
        const Geo g = geo_of(trig[n % kTrig], N, N);
        const float* at = P.atten + ((int64_t)a * P.B + b) * N * N;
        const float* rt = P.ratio ? P.ratio + ((int64_t)a * P.B + b) * N : nullptr;
        const float depth = g.cy * (fabsf(g.c) + fabsf(g.s) - 1.f) + 0.5f;   // farthest outside
        const float edge = low ? 0.f : g.rmax;
        // the strip's axis in sample coordinates, from (hm, wm) along (uh, uw)
        const float om = edge - g.cy, pm = (float)q + 0.5f - g.cy, sg = low ? -1.f : 1.f;
        const float xm = row ? om : pm, ym = row ? pm : om;
        const float hm = g.c * xm + g.s * ym + g.cy, wm = g.c * ym - g.s * xm + g.cy;
        const float uh = sg * (row ? g.c : g.s), uw = sg * (row ? -g.s : g.c);
        const bool hmaj = fabsf(uh) >= fabsf(uw);
        const float mm = hmaj ? hm : wm, km = hmaj ? wm : hm;
        const float um = hmaj ? uh : uw, slope = (hmaj ? uw : uh) / um;
        const float half = 1.5f * fabsf(hmaj ? uw : uh) + kPad;
        const float m1 = mm + depth * um;
        const int mlo = max(0, (int)ceilf(fminf(mm, m1) - half));
        const int mhi = min(N - 1, (int)floorf(fmaxf(mm, m1) + half));
        const float across = 1.5f / fabsf(um) + kPad;
        float t0 = 0.f, t1 = 0.f;
        for (int l0 = mlo; l0 <= mhi; l0 += 6) {
            const int m = l0 + line;
            const int k = (int)ceilf(km + ((float)m - mm) * slope - across) + cell;
            const int h = hmaj ? m : k, w = hmaj ? k : m;
            const float hf = (float)h - g.cy;
            const float x = fmaf(g.c, hf, col_bx(g, w)), y = fmaf(g.s, hf, col_by(g, w));
            const float o = row ? x : y;
            const float z = row ? fminf(fmaxf(y, 0.f), g.cmax) : x;
            const float w0 = tap_weight(z, (float)q), w1 = tap_weight(z, (float)(q + 1));
            // samples clamped in both coordinates belong to the rows
            if (lane < 30 && m <= mhi && (unsigned)k < (unsigned)N && (low ? o < 0.f : o > edge) &&
                (row || (x >= 0.f && x <= g.rmax)) && (w0 > 0.f || w1 > 0.f)) {
                const float v = __ldg(at + h * N + w) * (rt ? __ldg(rt + w) : 1.f);
                // (a value that is not finite stays with the positions it covers)
                if (w0 > 0.f) t0 = fmaf(w0, v, t0);
                if (w1 > 0.f) t1 = fmaf(w1, v, t1);
            }
        }
#pragma unroll
        for (int r = 0; r < kFewR; ++r)
            if (r < P.R) {
                const float em = __ldg(P.em + (int64_t)a * P.R + r);
                acc[r][0] = fmaf(em, t0, acc[r][0]);
                acc[r][1] = fmaf(em, t1, acc[r][1]);
            }
    }
    if (id >= 4 * nq) return;
    for (int r = 0; r < P.R; ++r) {
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int k = 0; k < kFewR; ++k)
            if (k == r) { s0 = acc[k][0]; s1 = acc[k][1]; }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s0 += __shfl_xor_sync(0xffffffffu, s0, o);
            s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        }
        float* f = P.frame + ((((int64_t)blockIdx.y * P.R + r) * 4 + e) * P.B + b) * N + q;
        if (lane == 0) f[0] = s0;
        if (lane == 1 && q + 1 < N) f[1] = s1;
    }
}

// Sum of atten * ratio * weight over the unclamped samples that cover pixel (i, j),
// among the 3 x 3 around its inverse image.  EDGE: the pixel is within two of the
// border, where samples in reach may be clamped (those are in the border sums; the
// test is the forward's own).  Attenuation and ratio count only where a sample covers
// the pixel, also when they are not finite.
template <bool EDGE>
__device__ __forceinline__ float gather9(const Geo& g, const float* __restrict__ at,
                                         const float* __restrict__ rt, int N, float fi, float fj) {
    const float xi = fi - g.cy, yj = fj - g.cx;
    const float hr = rintf(fmaf(g.c, xi, fmaf(g.s, yj, g.cy)));
    const float wr = rintf(fmaf(-g.s, xi, fmaf(g.c, yj, g.cx)));
    const int h0 = (int)hr - 1, w0 = (int)wr - 1;
    const float* p = at + h0 * N + w0;
    bool hin[3];
    float hf[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        hin[d] = (unsigned)(h0 + d) < (unsigned)N;
        hf[d] = hr + (float)(d - 1) - g.cy;
    }
    float t = 0.f, v[3][3], wt[3][3], rr[3];
#pragma unroll
    for (int db = 0; db < 3; ++db) {
        const bool win = (unsigned)(w0 + db) < (unsigned)N;
        const float wf = wr + (float)(db - 1) - g.cx;
        const float bx = fmaf(-g.s, wf, g.cy), by = fmaf(g.c, wf, g.cx);   // col_bx, col_by
        bool any = false;
#pragma unroll
        for (int da = 0; da < 3; ++da) {
            const float x = fmaf(g.c, hf[da], bx), y = fmaf(g.s, hf[da], by);
            const float wx = 1.f - fabsf(x - fi), wy = 1.f - fabsf(y - fj);
            bool in = win && hin[da] && fminf(wx, wy) > 0.f;
            if (EDGE) in = in && x >= 0.f && x <= g.rmax && y >= 0.f && y <= g.cmax;
            v[da][db] = in ? __ldg(p + da * N + db) : 0.f;
            wt[da][db] = wx * wy;
            any = any || in;
        }
        rr[db] = any ? (rt ? __ldg(rt + w0 + db) : 1.f) : 0.f;
    }
#pragma unroll
    for (int db = 0; db < 3; ++db) {
        float c = v[0][db] * wt[0][db];
        c = fmaf(v[1][db], wt[1][db], c);
        c = fmaf(v[2][db], wt[2][db], c);
        t = fmaf(rr[db], c, t);
    }
    return t;
}

// gather9 with em at an angle near an axis, in the splats' steps (near_axis).
__device__ __noinline__ float gather_parts(float2 cs, const float* __restrict__ at,
                                           const float* __restrict__ rt, float em, int N, float fi,
                                           float fj) {
    const Geo g = geo_of(cs, N, N);
    const float xi = fi - g.cy, yj = fj - g.cx;
    const int h0 = (int)rintf(fmaf(g.c, xi, fmaf(g.s, yj, g.cy))) - 1;
    const int w0 = (int)rintf(fmaf(-g.s, xi, fmaf(g.c, yj, g.cx))) - 1;
    float t = 0.f;
    for (int k = 0; k < 9; ++k) {
        const int db = k / 3, h = h0 + k - 3 * db, w = w0 + db;
        if ((unsigned)h >= (unsigned)N || (unsigned)w >= (unsigned)N) continue;
        const float hf = (float)h - g.cy;
        const float x = fmaf(g.c, hf, col_bx(g, w)), y = fmaf(g.s, hf, col_by(g, w));
        if (!(x >= 0.f && x <= g.rmax && y >= 0.f && y <= g.cmax)) continue;
        const float cr = part_code(x, fi), cc = part_code(y, fj);
        if (cr == 0.f || cc == 0.f) continue;
        const float v = __fmul_rn(__ldg(at + h * N + w), rt ? __fmul_rn(__ldg(rt + w), em) : em);
        t += part_col(part_row(v, cr), cc);
    }
    return t;
}

// Grid (ceil(N / 8), ceil(N / 4), B): a patch of 8 x 4 pixels, whose samples lie in
// few lines at every angle; warp k takes angles k, k + 16, ...  Bound by the latency of
// the reads behind the footprint tests: all nine in flight before the first sum, and no
// clamp tests away from the border, 14.3 us for 90 angles of 96^2 and 149 for 120 of
// 8 x 128^2; a row of 32 pixels a warp, one read at a time, 16.4 and 192.  The warps'
// sums are added in order (deterministic), then the border sums and the epilogue.
template <int RC>
__global__ void __launch_bounds__(kFewWarps * 32)
few_bwd_kernel(FewArgs P) {
    constexpr int RM = RC > 0 ? RC : kFewR;
    __shared__ float part[RM][kFewWarps][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int N = P.N, R = RC > 0 ? RC : P.R;
    const int i = blockIdx.y * 4 + (lane >> 3), j = blockIdx.x * 8 + (lane & 7), b = blockIdx.z;
    const float fi = (float)i, fj = (float)j;
    const int i0 = blockIdx.y * 4, j0 = blockIdx.x * 8;      // (the same in the whole block)
    const bool edge = i0 < 2 || j0 < 2 || i0 + 4 > N - 2 || j0 + 8 > N - 2;
    float acc[RM];
#pragma unroll
    for (int r = 0; r < RM; ++r) acc[r] = 0.f;
    __shared__ float2 trig[kTrig];
    for (int a = warp; a - warp < P.A; a += kFewWarps) {
        const int ta = (a - warp) % kTrig;
        if (ta == 0) {
            __syncthreads();
            const int t = threadIdx.x;
            if (t < kTrig && a - warp + t < P.A) trig[t] = trig_of(P.theta, a - warp + t);
            __syncthreads();
        }
        if (a >= P.A) continue;
        const Geo g = geo_of(trig[ta + warp], N, N);
        const float* at = P.atten + ((int64_t)a * P.B + b) * N * N;
        const float* rt = P.ratio ? P.ratio + ((int64_t)a * P.B + b) * N : nullptr;
        if (near_axis(g, N)) {
            for (int r = 0; r < R; ++r) {
                const float t =
                    gather_parts(trig[ta + warp], at, rt, __ldg(P.em + (int64_t)a * R + r), N, fi, fj);
#pragma unroll
                for (int k = 0; k < RM; ++k)
                    if (k == r) acc[k] += t;
            }
            continue;
        }
        const float t = edge ? gather9<true>(g, at, rt, N, fi, fj) : gather9<false>(g, at, rt, N, fi, fj);
        if (RC == 1) {
            acc[0] = fmaf(__ldg(P.em + a), t, acc[0]);
        } else {
#pragma unroll
            for (int r = 0; r < RM; ++r)
                if (r < R) acc[r] = fmaf(__ldg(P.em + (int64_t)a * R + r), t, acc[r]);
        }
    }
#pragma unroll
    for (int r = 0; r < RM; ++r) part[r][warp][lane] = acc[r];
    __syncthreads();
    if (warp >= R || i >= N || j >= N) return;
    const int r = warp;
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < kFewWarps; ++k) s += part[RC == 1 ? 0 : r][k][lane];
    if (i == 0 || j == 0 || i >= N - 2 || j >= N - 2) {
        const Geo g0 = make_geo(0.f, N, N);
        const float fr = i == N - 1 ? g0.fxh : 1.f - g0.fxh, fc = j == N - 1 ? g0.fyh : 1.f - g0.fyh;
        const int64_t es = (int64_t)P.B * N;
        for (int q = 0; q < P.splits; ++q) {
            const float* f = P.frame + (((int64_t)q * P.R + r) * 4 * P.B + b) * N;
            if (i == 0) s += f[j];
            if (i >= N - 2) s += f[es + j] * fr;
            if (j == 0) s += f[2 * es + i];
            if (j >= N - 2) s += f[3 * es + i] * fc;
        }
    }
    bwd_epilogue(P.mode, P.out, P.Cin, P.sens, P.clamp_min, P.beta, P.delta, r, b, P.B, N, N, i, j, s);
}

// Forward: grid (ceil(N / 32), A, B), 32 detector columns of one angle; warp k takes
// the beam steps k, k + 16, ...  The taps of the image come from L1 and L2.
template <int RC>
__global__ void __launch_bounds__(kFewWarps * 32)
few_fwd_kernel(const float* __restrict__ atten, const float* __restrict__ C, const float* __restrict__ em,
               const float* __restrict__ theta, const float* __restrict__ I, float* __restrict__ out,
               int B, int Rrt, int H, int W) {
    __shared__ float part[kFewWarps][32];
    __shared__ float2 cs;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int R = RC > 0 ? RC : Rrt;
    const int w = blockIdx.x * 32 + lane, a = blockIdx.y, b = blockIdx.z;
    if (threadIdx.x == 0) cs = trig_of(theta, a);
    __syncthreads();
    const Geo g = geo_of(cs, H, W);
    const int64_t HW = (int64_t)H * W;
    const float* at = atten + ((int64_t)a * B + b) * HW + w;
    const float* Cb = C + (int64_t)b * HW;
    float acc = 0.f;
    if (w < W) {
        const float bx = col_bx(g, w), by = col_by(g, w);
#pragma unroll 4
        for (int h = warp; h < H; h += kFewWarps) {
            const float hf = (float)h - g.cy;
            const Smp s = sample_xy(g, fmaf(g.c, hf, bx), fmaf(g.s, hf, by));
            const float* p = Cb + s.i0 * W + s.j0;
            const float av = __ldg(at + (int64_t)h * W);
            float v = 0.f;
            for (int r = 0; r < R; ++r) {
                const float* q = p + (int64_t)r * B * HW;
                const float t0 = __ldg(q), t1 = __ldg(q + 1), u0 = __ldg(q + W), u1 = __ldg(q + W + 1);
                const float t = fmaf(s.fy, t1 - t0, t0), u = fmaf(s.fy, u1 - u0, u0);
                const float c = fmaf(s.fx, u - t, t);
                v = RC == 1 ? c : fmaf(__ldg(em + (int64_t)a * R + r), c, v);
            }
            acc = fmaf(av, v, acc);
        }
    }
    part[warp][lane] = acc;
    __syncthreads();
    if (warp != 0 || w >= W) return;
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < kFewWarps; ++k) s += part[k][lane];
    if (RC == 1) s *= __ldg(em + a);
    const int64_t o = ((int64_t)a * B + b) * W + w;
    if (I) s = I[o] / fmaxf(s, 1e-6f);
    out[o] = s;
}

int few_splits(int64_t A, int64_t B, int64_t N) {
    // warps enough for the chip, few angles each; the sums fit R B N^2 floats
    int64_t s = ceil_div(2368 * 2, 2 * N * B);
    s = s < 4 ? 4 : s > 32 ? 32 : s;
    if (s > N / 4) s = N / 4;
    return (int)(s > A ? A : s);
}

}  // namespace

// Whether a backward of these sizes goes to the gather kernels for few slices, with
// few_floats(...) floats of scratch (the "proj.few" knob: 1 wherever they take the
// shape, 2 never).  Their time goes with the slices, the splats' has a floor; more
// references cost the splats in proportion and these next to nothing.  One backward
// with its allocation, us, splats / these: 90 angles of 96^2 161 / 36 for 1 slice, 163 /
// 141 for 10, 163 / 165 for 12; 120 of 128^2 405 / 233 for 8; 40 of 24^2 40 / 33 for 10.
// Two references: 75 of 33 x 101^2 512 / 510, 30 of 31 x 64^2 89 / 97; past 128^2
// the splats take one reference at a time: 60 of 64 x 192^2 4216 / 1984.  Three: 120 of
// 33 x 101^2 1512 / 657, 60 of 31 x 48^2 155 / 109; where the splats run with three CTAs
// an SM (small_image) they are ahead again from some slices on: 40 of 24^2: 33 slices 74 /
// 50, 70 79 / 87, 150 104 / 164; 60 of 48^2: 33 150 / 143, 70 184 / 280; 60 of 64^2: 33 212 /
// 221; MLEM of 60 x 48^2, 5 iterations: 70 1606 / 2207, 150 3709 / 4770; five references: 40
// of 24^2: 30 97 / 52, 100 109 / 136; 60 of 48^2: 30 213 / 155, 100 399 / 464.
bool use_few(int64_t A, int64_t B, int64_t R, int64_t H, int64_t W) {
    const int64_t knob = tune(kTuneProjFew);
    if (tune(kTuneProjLegacy) != 0 || tune(kTuneProjBand) != 0 || knob == 2) return false;
    if (H != W || H < 16 || R > kFewR || B > 65535 || H * W > (1 << 30)) return false;
    if (knob == 1) return true;
    if (R > 2) return !small_image(R, H, W) || B * W < 400 * R + 400;
    return B <= (R == 1 ? 10 : 26) || (R == 2 && W > 128);
}

int64_t few_floats(int64_t A, int64_t B, int64_t R, int64_t N) {
    return (int64_t)few_splits(A, B, N) * R * 4 * B * N;
}

// Whether a forward of these sizes goes to few_fwd_kernel (the "proj.few" knob).
bool use_few_fwd(int64_t A, int64_t B, int64_t R, int64_t H, int64_t W) {
    const int64_t knob = tune(kTuneProjFew);
    if (tune(kTuneProjLegacy) != 0 || knob == 2 || A > 65535 || B > 65535) return false;
    // (the lean forward where it takes the slice, us / these: 90 angles of 96^2 15.4 /
    // 9.9 for 1 slice, 120 of 128^2 26.1 / 23.7 for 2, 31.3 / 37.0 for 4; 75 of 101^2
    // with 2 references 48.5 / 35.4 for 4, 227 / 258 for 33.  Where it does not, the
    // first forward, us: 180 of 256^2 141 / 51 for 1 slice, 2694 / 1346 for 32; 60 of
    // 512^2 554 / 73 for 1)
    if (knob == 1 || !fwd2_takes(R, H, W)) return true;
    // (tall slices have few columns to share out: 60 of 200 x 64, 1 and 2 slices, 24 / 21
    // and 21 / 27, with two references 34 / 31 and 35 / 50)
    if (H > 2 * W) return B == 1;
    if (R == 1) return B <= 2;
    // (up to 128^2 the lean forward is at its best at its compile-time widths: two
    // references, 60 of 64^2: 2 slices 21 / 21, 6 20 / 25, 8 21 / 29, 120 of 128^2: 4 86 / 79, 6
    // 100 / 111, 8 129 / 144; at others 60 of 101^2: 6 52 / 42, 8 53 / 54; above, 30 of 160^2:
    // 8 107 / 69)
    return B <= (H * W > 128 * 128 || !fwd2_fixed_width(W) ? 8 : small_image(R, H, W) ? 2 : 4);
}

// Forward: out (A, B, W) = P C, or I / max(P C, 1e-6) when I != nullptr.
int fwd_few_launch(const float* atten, const float* C, const float* em, const float* theta, float* out,
                   const float* I, int64_t A, int64_t B, int64_t R, int64_t H, int64_t W,
                   cudaStream_t st) {
    const dim3 grid((unsigned)ceil_div(W, 32), (unsigned)A, (unsigned)B);
    if (R == 1)
        few_fwd_kernel<1><<<grid, kFewWarps * 32, 0, st>>>(atten, C, em, theta, I, out, (int)B, (int)R,
                                                           (int)H, (int)W);
    else
        few_fwd_kernel<0><<<grid, kFewWarps * 32, 0, st>>>(atten, C, em, theta, I, out, (int)B, (int)R,
                                                           (int)H, (int)W);
    return check_launch("few_fwd_kernel");
}

// Backward with its epilogue (bwd_epilogue); frame: few_floats floats of scratch.
int bwd_few_launch(const float* atten, const float* ratio, const float* em, const float* theta,
                   float* out, const float* Cin, const float* sens, float* frame, int64_t A, int64_t B,
                   int64_t R, int64_t N, float clamp_min, int mode, float beta, float delta,
                   cudaStream_t st) {
    FewArgs P{atten, ratio, em, theta, out, Cin, sens, frame, few_splits(A, B, N), (int)A, (int)B, (int)R,
              (int)N, clamp_min, mode, beta, delta};
    few_frame_kernel<<<dim3((unsigned)ceil_div(4 * ((N + 1) / 2), 8), (unsigned)P.splits, (unsigned)B), 256,
                       0, st>>>(P);
    FLC_TRY(check_launch("few_frame_kernel"));
    const dim3 grid((unsigned)ceil_div(N, 8), (unsigned)ceil_div(N, 4), (unsigned)B);
    if (R == 1)
        few_bwd_kernel<1><<<grid, kFewWarps * 32, 0, st>>>(P);
    else
        few_bwd_kernel<0><<<grid, kFewWarps * 32, 0, st>>>(P);
    return check_launch("few_bwd_kernel");
}

}  // namespace flc
