// Spectral cone path sum with line transforms in registers (sm_100a).
//
// The algorithm is that of flc_cone_fft.cu: the depth sum of 2-D correlations as
// pointwise products of (z, y) spectra, R_x = sum_d G_d P_{x+d} for every frequency.
// The depth is summed directly, as there: a transform along it (22 instead of 66 kFLOP
// per frequency of a 128^3 volume, the middle kernel below 0.59 ms) would spread the
// rounding error of the strongest planes, and a value that is not finite, over all of
// them, where a plane depends on those in front of the detector only: planes 1e4 times
// weaker in front of strong ones came out with an error of 1e-3.
//
// Two rows of the same volume travel through the transforms along y together, as the
// real and imaginary part of one, and are taken apart into half spectra (ky = 0 ..
// Ny/2) before the transforms along z, so that volumes do not mix.  Every transform has
// a length N = R1 R2 and runs in two steps of R1- and R2-point DFTs, one line segment per
// thread in registers, in place: element n = R2 n1 + n2 becomes A(k1, n2) at R2 k1 + n2,
// that becomes X(k1 + R1 k2) at R2 k1 + k2.  The spectra along z stay in that order (the
// filter is made in it), and the inverse takes the same steps back.
//
//   line_roots, line_filter : twiddles, the mask's line spectra, G
//   line_rows   : mu -> S[ky][x][z]; 64 rows of one plane x per CTA, transforms
//                 along y
//   line_mid    : per (ky, volume), the whole (x, z) plane in shared memory:
//                 transform along z; the depth sums in place; back along z;
//                 S[ky][z][x] over the same memory
//   line_out    : transforms back along y, 32 x of two slices z per CTA, and
//                 writes exp(-res) into the beam layout (x is its fastest axis,
//                 so no transpose is left) or res into the reference layout
//
// 36 volumes of 128^3 with a 29 x 128 x 29 mask: rows 0.16, middle 0.86, out 0.18,
// filter 0.01 ms, against 2.2 ms in five kernels of the plane form.  Rows and out move
// the bytes they must at about half the copy rate, four CTAs an SM (three: 0.17 and 0.21;
// two volumes as one complex one, with no half spectra to take apart, three CTAs: 0.15
// and 0.20, but each volume then has the rounding error of the other, and its NaN); of
// the middle (one CTA of 16 warps per SM: the plane takes 148 KB) 0.6 ms are the depth
// sums.  The line form is the faster one for few volumes too (planes / lines, us: 1
// volume of 64^3 39 / 38, of 128^3 94 / 84, of 30 x 200^2 130 / 91; 2 of 48 x 64^2 42 /
// 36, of 128^3 146 / 97; 3 of 96^3 101 / 87), so it runs wherever it takes the shape, and
// a volume's bits do not depend on how many volumes are in the call.

#include <algorithm>

#include "flc_common.cuh"

namespace flc {

size_t cone_fft_ws_bytes(int64_t Vn, int64_t Z, int64_t X, int64_t Y, int64_t Mz, int64_t Mx,
                         int64_t My, int mode);

namespace {

typedef unsigned long long c32;   // complex FP32 in a register pair

__device__ __forceinline__ c32 mk(float a, float b) {
    c32 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void un(c32 r, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
// PK: one paired instruction instead of two scalar ones.  The paired form costs
// registers; it is the faster one in line_mid (0.60 against 0.63 ms for 30 volumes
// of 128^3), the scalar one in line_out (0.28 against 0.23 ms).
template <bool PK>
__device__ __forceinline__ c32 cadd(c32 a, c32 b) {
    if constexpr (PK) {
        c32 d;
        asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
        return d;
    } else {
        float x, y, u, v;
        un(a, x, y);
        un(b, u, v);
        return mk(x + u, y + v);
    }
}
template <bool PK>
__device__ __forceinline__ c32 csub(c32 a, c32 b) {
    if constexpr (PK) {
        c32 d;
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(b), "l"(mk(-1.f, -1.f)), "l"(a));
        return d;
    } else {
        float x, y, u, v;
        un(a, x, y);
        un(b, u, v);
        return mk(x - u, y - v);
    }
}
__device__ __forceinline__ c32 cmul2(c32 a, c32 b) {   // halves apart
    c32 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ c32 cfma2(c32 a, c32 b, c32 c) {
    c32 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// z (c + i s): four scalar instructions (paired ones would need the halves swapped)
__device__ __forceinline__ c32 cturn(c32 z, float c, float s) {
    float x, y;
    un(z, x, y);
    return mk(fmaf(c, x, -s * y), fmaf(c, y, s * x));
}
// z * i^{SG}
template <int SG>
__device__ __forceinline__ c32 crot(c32 z) {
    float x, y;
    un(z, x, y);
    return SG > 0 ? mk(-y, x) : mk(y, -x);
}

// cos and sin of 2 pi m / n at compile time, by their power series.
constexpr double series(double x, bool sine) {
    double t = sine ? x : 1.0, sum = t;
    for (int k = sine ? 2 : 1; k < 40; k += 2) {
        t *= -x * x / (double)(k * (k + 1));
        sum += t;
    }
    return sum;
}
constexpr double kTwoPi = 6.283185307179586476925286766559;
constexpr double angle(int m, int n) {
    m %= n;
    if (2 * m > n) m -= n;
    return kTwoPi * (double)m / (double)n;
}
constexpr float cos_of(int m, int n) { return (float)series(angle(m, n), false); }
constexpr float sin_of(int m, int n) { return (float)series(angle(m, n), true); }

// v[k] = sum_n v[n] e^{SG 2 pi i n k / R}, in place, natural order.
template <int R, int SG, bool PK>
__device__ __forceinline__ void dft(c32 (&v)[R]);

template <int P, int Q, int SG, bool PK>
__device__ __forceinline__ void dft_pq(c32 (&v)[P * Q]) {
    constexpr int R = P * Q;
    c32 y[Q][P];
#pragma unroll
    for (int n2 = 0; n2 < Q; ++n2) {
        c32 t[P];
#pragma unroll
        for (int n1 = 0; n1 < P; ++n1) t[n1] = v[Q * n1 + n2];
        dft<P, SG, PK>(t);
#pragma unroll
        for (int k1 = 0; k1 < P; ++k1) {
            const int m = n2 * k1;
            y[n2][k1] = m == 0 ? t[k1]
                      : 4 * m == R ? crot<SG>(t[k1])
                                   : cturn(t[k1], cos_of(m, R), SG * sin_of(m, R));
        }
    }
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) {
        c32 u[Q];
#pragma unroll
        for (int n2 = 0; n2 < Q; ++n2) u[n2] = y[n2][k1];
        dft<Q, SG, PK>(u);
#pragma unroll
        for (int k2 = 0; k2 < Q; ++k2) v[k1 + P * k2] = u[k2];
    }
}

template <int R, int SG, bool PK>
__device__ __forceinline__ void dft(c32 (&v)[R]) {
    if constexpr (R == 2) {
        const c32 a = v[0], b = v[1];
        v[0] = cadd<PK>(a, b);
        v[1] = csub<PK>(a, b);
    } else if constexpr (R == 3) {
        const c32 a = cadd<PK>(v[1], v[2]);
        const c32 t = cfma2(mk(-0.5f, -0.5f), a, v[0]);
        const c32 d = csub<PK>(v[1], v[2]);
        constexpr float s3 = 0.866025403784438647f;
        const c32 u = cmul2(mk(s3, s3), crot<SG>(d));
        v[0] = cadd<PK>(v[0], a);
        v[1] = cadd<PK>(t, u);
        v[2] = csub<PK>(t, u);
    } else if constexpr (R == 4) {
        const c32 s02 = cadd<PK>(v[0], v[2]), d02 = csub<PK>(v[0], v[2]);
        const c32 s13 = cadd<PK>(v[1], v[3]), w13 = crot<SG>(csub<PK>(v[1], v[3]));
        v[0] = cadd<PK>(s02, s13);
        v[2] = csub<PK>(s02, s13);
        v[1] = cadd<PK>(d02, w13);
        v[3] = csub<PK>(d02, w13);
    } else if constexpr (R == 5) {
        constexpr float c1 = 0.309016994374947424f, c2 = -0.809016994374947424f;
        constexpr float s1 = 0.951056516295153572f, s2 = 0.587785252292473129f;
        const c32 a1 = cadd<PK>(v[1], v[4]), b1 = crot<SG>(csub<PK>(v[1], v[4]));
        const c32 a2 = cadd<PK>(v[2], v[3]), b2 = crot<SG>(csub<PK>(v[2], v[3]));
        const c32 t1 = cfma2(mk(c2, c2), a2, cfma2(mk(c1, c1), a1, v[0]));
        const c32 t2 = cfma2(mk(c1, c1), a2, cfma2(mk(c2, c2), a1, v[0]));
        const c32 u1 = cfma2(mk(s2, s2), b2, cmul2(mk(s1, s1), b1));
        const c32 u2 = cfma2(mk(-s1, -s1), b2, cmul2(mk(s2, s2), b1));
        v[0] = cadd<PK>(v[0], cadd<PK>(a1, a2));
        v[1] = cadd<PK>(t1, u1);
        v[4] = csub<PK>(t1, u1);
        v[2] = cadd<PK>(t2, u2);
        v[3] = csub<PK>(t2, u2);
    } else if constexpr (R == 6) {
        dft_pq<2, 3, SG, PK>(v);
    } else if constexpr (R == 8) {
        dft_pq<2, 4, SG, PK>(v);
    } else if constexpr (R == 9) {
        dft_pq<3, 3, SG, PK>(v);
    } else if constexpr (R == 10) {
        dft_pq<2, 5, SG, PK>(v);
    } else if constexpr (R == 12) {
        dft_pq<3, 4, SG, PK>(v);
    } else if constexpr (R == 16) {
        dft_pq<4, 4, SG, PK>(v);
    } else if constexpr (R == 18) {
        dft_pq<2, 9, SG, PK>(v);
    } else {
        static_assert(R == 20, "radix");
        dft_pq<4, 5, SG, PK>(v);
    }
}

// v[k] *= e^{SG 2 pi i m k / N}, k = 1 .. R-1; tw[j] = e^{-2 pi i j / N}.
template <int R, int SG>
__device__ __forceinline__ void twiddle(c32 (&v)[R], const float2* tw, int m) {
#pragma unroll
    for (int k = 1; k < R; ++k) {
        const float2 t = tw[m * k];
        v[k] = cturn(v[k], t.x, SG < 0 ? t.y : -t.y);
    }
}

struct Len {
    int n, r1, r2, id;
};

struct LineGeom {
    int Z, X, Y, Mz, Mx, My;
    Len z, y;
    int Nyh;        // y.n / 2 + 1
};

// Transform lengths R1 R2, as F(index, R1, R2), shortest first.  The steps
// are compiled for each, so that strides and pitches are immediates.
#define FLC_LENS(F)                                                                         \
    F(0, 4, 4) F(1, 6, 4) F(2, 8, 4) F(3, 8, 5) F(4, 8, 6) F(5, 9, 6) F(6, 8, 8) F(7, 9, 8) \
    F(8, 10, 8) F(9, 10, 9) F(10, 12, 8) F(11, 12, 9) F(12, 12, 10) F(13, 16, 8)            \
    F(14, 12, 12) F(15, 16, 10) F(16, 18, 10) F(17, 16, 12) F(18, 18, 12) F(19, 20, 12)     \
    F(20, 16, 16) F(21, 18, 16) F(22, 20, 16) F(23, 20, 20)

#define FLC_CASE(i, A, B) case i: CALL(A, B); break;
#define FLC_LEN(l) switch ((l).id) { FLC_LENS(FLC_CASE) }

constexpr int kRowsT = 256;      // threads of line_rows / line_out
constexpr int kLines = 32;       // pairs of rows per CTA of line_rows / line_out
constexpr int kMidT = 512;
constexpr int kTeam = 256;       // threads of a team of line_mid

// floor(a / b) for 0 <= a < 2^22 from b's reciprocal.
__device__ __forceinline__ int div_small(int a, float rb) { return (int)(((float)a + 0.5f) * rb); }

// ---------------------------------------------------------------------------
// Twiddles T[m] = e^{-2 pi i m / N} of the two lengths, and the line spectra
// Uf_d(kz) = sum_dz u[d][dz] e^{+2 pi i kz (dz - hz) / Nz} (Vf likewise) in FP64, kz
// in the transforms' order.  Grid Mx + 1: block d < Mx its spectra, block Mx the
// twiddles.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
line_roots_kernel(const float* __restrict__ U, const float* __restrict__ V, double2* __restrict__ Uf,
                  double2* __restrict__ Vf, float2* __restrict__ Tz, float2* __restrict__ Ty,
                  LineGeom g) {
    extern __shared__ double2 root[];      // e^{2 pi i m / N} of z, then y
    const int d = blockIdx.x, Nz = g.z.n, Ny = g.y.n;
    if (d == g.Mx) {
        for (int m = threadIdx.x; m < Nz + Ny; m += blockDim.x) {
            double s, c;
            sincospi(m < Nz ? -2.0 * (double)m / (double)Nz : -2.0 * (double)(m - Nz) / (double)Ny, &s, &c);
            (m < Nz ? Tz[m] : Ty[m - Nz]) = make_float2((float)c, (float)s);
        }
        return;
    }
    for (int m = threadIdx.x; m < Nz + Ny; m += blockDim.x) {
        double s, c;
        sincospi(m < Nz ? 2.0 * (double)m / (double)Nz : 2.0 * (double)(m - Nz) / (double)Ny, &s, &c);
        root[m] = make_double2(c, s);
    }
    __syncthreads();
    const int hz = g.Mz / 2, hy = g.My / 2;
    for (int p = threadIdx.x; p < Nz + g.Nyh; p += blockDim.x) {
        const bool zk = p < Nz;
        const int pos = zk ? p : p - Nz, n = zk ? Nz : Ny, M = zk ? g.Mz : g.My, h = zk ? hz : hy;
        const int k = zk ? pos / g.z.r2 + g.z.r1 * (pos % g.z.r2) : pos;   // frequency at this place
        const float* w = zk ? U + (int64_t)d * g.Mz : V + (int64_t)d * g.My;
        const double2* rt = zk ? root : root + Nz;
        int m = (int)(((int64_t)k * (n - h % n)) % n);
        double re = 0.0, im = 0.0;
        for (int t = 0; t < M; ++t) {
            const double wt = (double)__ldg(w + t);
            re += wt * rt[m].x;
            im += wt * rt[m].y;
            m += k;
            if (m >= n) m -= n;
        }
        (zk ? Uf + (int64_t)d * Nz : Vf + (int64_t)d * g.Nyh)[pos] = make_double2(re, im);
    }
}

// Filter spectra G[ky][d][kz] = Uf_d(kz) Vf_d(ky), d < min(Mx, X) (kz in the transforms'
// order), rounded from FP64.  Grid (D, Nyh).
__global__ void __launch_bounds__(128)
line_filter_kernel(const double2* __restrict__ Uf, const double2* __restrict__ Vf, c32* __restrict__ G,
                   LineGeom g) {
    const int d = blockIdx.x, ky = blockIdx.y;
    const double2 b = Vf[(int64_t)d * g.Nyh + ky];
    c32* Gd = G + ((int64_t)ky * gridDim.x + d) * g.z.n;
    for (int k = threadIdx.x; k < g.z.n; k += blockDim.x) {
        const double2 a = Uf[(int64_t)d * g.z.n + k];
        Gd[k] = mk((float)(a.x * b.x - a.y * b.y), (float)(a.x * b.y + a.y * b.x));
    }
}

// ---------------------------------------------------------------------------
// Rows forward: grid (ceil(Z / 64), X, volumes).  Row 2l is the real part, 2l + 1 (if
// it exists) the imaginary part.
// ---------------------------------------------------------------------------
// Place of frequency k in the transforms' order.
template <int R1, int R2>
__device__ __forceinline__ int place(int k) { return R2 * (k % R1) + k / R1; }

template <int R, int R2>
__device__ __forceinline__ void rows_a(const float* mu, c32* sm, const float2* tw, const LineGeom& g,
                                       int nz) {
    constexpr int r2 = R2, P = R * R2 + 1;
    const int64_t zs = (int64_t)g.X * g.Y;
    for (int i = threadIdx.x; i < (nz + 1) / 2 * r2; i += kRowsT) {
        const int l = i / r2, n2 = i - l * r2;
        const float* ma = mu + 2 * l * zs;
        const bool two = 2 * l + 1 < nz;
        float a[R], b[R];
#pragma unroll
        for (int n1 = 0; n1 < R; ++n1) {
            const int y = r2 * n1 + n2;
            a[n1] = y < g.Y ? __ldg(ma + y) : 0.f;
            b[n1] = y < g.Y && two ? __ldg(ma + zs + y) : 0.f;
        }
        c32 v[R];
#pragma unroll
        for (int n1 = 0; n1 < R; ++n1) v[n1] = mk(a[n1], b[n1]);
        dft<R, -1, false>(v);
        twiddle<R, -1>(v, tw, n2);
#pragma unroll
        for (int k1 = 0; k1 < R; ++k1) sm[l * P + r2 * k1 + n2] = v[k1];
    }
}

// Step 2, then the rows' own half spectra: of the pair's W, twice the first is
// W(k) + conj W(-k), twice the second -i (W(k) - conj W(-k)).
template <int R1, int R>
__device__ __forceinline__ void rows_b(c32* sm, c32* S, const LineGeom& g, int nz) {
    constexpr int N = R1 * R, P = N + 1;
    const int64_t ks = (int64_t)g.X * g.Z;
    const int l = threadIdx.x & 31;
    const bool live = 2 * l < nz;
    if (live) {
        for (int k1 = threadIdx.x >> 5; k1 < R1; k1 += kRowsT / 32) {
            c32 v[R];
#pragma unroll
            for (int n2 = 0; n2 < R; ++n2) v[n2] = sm[l * P + R * k1 + n2];
            dft<R, -1, false>(v);
#pragma unroll
            for (int k2 = 0; k2 < R; ++k2) sm[l * P + R * k1 + k2] = v[k2];
        }
    }
    __syncthreads();
    if (!live) return;
    const bool vec = (g.Z & 1) == 0;
#pragma unroll 4
    for (int k = threadIdx.x >> 5; k <= N / 2; k += kRowsT / 32) {
        float x, y, u, v;
        un(sm[l * P + place<R1, R>(k)], x, y);
        un(sm[l * P + place<R1, R>(k ? N - k : 0)], u, v);
        const c32 a = mk(x + u, y - v), b = mk(y + v, u - x);
        c32* s = S + k * ks + 2 * l;
        if (vec) {
            *reinterpret_cast<ulonglong2*>(s) = make_ulonglong2(a, b);
        } else {
            s[0] = a;
            if (2 * l + 1 < nz) s[1] = b;
        }
    }
}

__global__ void __launch_bounds__(kRowsT, 4)
line_rows_kernel(const float* __restrict__ mu, const float2* __restrict__ Ty, c32* __restrict__ S,
                 LineGeom g) {
    extern __shared__ __align__(16) c32 sm[];                       // [32][Ny + 1], twiddles
    float2* tw = reinterpret_cast<float2*>(sm + kLines * (g.y.n + 1));
    for (int m = threadIdx.x; m < g.y.n; m += kRowsT) tw[m] = Ty[m];
    __syncthreads();
    const int z0 = blockIdx.x * 2 * kLines, x = blockIdx.y, v = blockIdx.z;
    const int nz = min(2 * kLines, g.Z - z0);
    const float* src = mu + (((int64_t)v * g.Z + z0) * g.X + x) * g.Y;
#define CALL(A, B) rows_a<A, B>(src, sm, tw, g, nz)
    FLC_LEN(g.y)
#undef CALL
    __syncthreads();
    c32* Sv = S + ((int64_t)v * g.Nyh * g.X + x) * g.Z + z0;
#define CALL(A, B) rows_b<A, B>(sm, Sv, g, nz)
    FLC_LEN(g.y)
#undef CALL
}

// ---------------------------------------------------------------------------
// Middle: grid (Nyh, volumes), one CTA per SM with the (x, z) plane of one ky.  In the
// transforms along z the threads work in teams, each on its own x lines, with barriers of
// the team only.
// ---------------------------------------------------------------------------
struct Team {
    int t, n, id;     // thread in the team, threads, team
    int x0, x1;       // its x lines
    __device__ __forceinline__ void sync() const {
        asm volatile("bar.sync %0, %1;" ::"r"(id + 1), "r"(n) : "memory");
    }
};

// z step 1 (adjacent threads along x: the pitch Nz + 1 is odd or spreads over the
// banks, and a warp reads one twiddle); samples z >= Z are zero.
template <int R, int R2>
__device__ __forceinline__ void mid_za(c32* pl, const float2* tw, const LineGeom& g, const Team& tm) {
    constexpr int r2 = R2, P = R * R2 + 1;
    const int nx = tm.x1 - tm.x0;
    const float rX = 1.f / (float)nx;
    for (int i = tm.t; i < nx * r2; i += tm.n) {
        const int n2 = div_small(i, rX), x = tm.x0 + i - n2 * nx;
        c32* row = pl + x * P + n2;
        c32 v[R];
#pragma unroll
        for (int n1 = 0; n1 < R; ++n1) v[n1] = r2 * n1 + n2 < g.Z ? row[r2 * n1] : 0ull;
        dft<R, -1, true>(v);
        twiddle<R, -1>(v, tw, n2);
#pragma unroll
        for (int k1 = 0; k1 < R; ++k1) row[r2 * k1] = v[k1];
    }
}

// z step 2 (SG = -1) and its inverse (+1, with the twiddles after): adjacent
// threads along x.
template <int R1, int R, int SG>
__device__ __forceinline__ void mid_zb(c32* pl, const float2* tw, const LineGeom& g, const Team& tm) {
    constexpr int P = R1 * R + 1;
    const int nx = tm.x1 - tm.x0;
    const float rX = 1.f / (float)nx;
    for (int i = tm.t; i < nx * R1; i += tm.n) {
        const int k1 = div_small(i, rX), x = tm.x0 + i - k1 * nx;
        c32* row = pl + x * P + R * k1;
        c32 v[R];
#pragma unroll
        for (int n2 = 0; n2 < R; ++n2) v[n2] = row[n2];
        dft<R, SG, true>(v);
        if constexpr (SG > 0) twiddle<R, 1>(v, tw, k1);
#pragma unroll
        for (int k2 = 0; k2 < R; ++k2) row[k2] = v[k2];
    }
}

// inverse z step 1, straight to S[z][x].
template <int R, int R2>
__device__ __forceinline__ void mid_zo(const c32* pl, c32* S, const LineGeom& g, const Team& tm) {
    constexpr int r2 = R2, P = R * R2 + 1;
    const int nx = tm.x1 - tm.x0;
    const float rX = 1.f / (float)nx;
    for (int i = tm.t; i < nx * r2; i += tm.n) {
        const int n2 = div_small(i, rX), x = tm.x0 + i - n2 * nx;
        const c32* row = pl + x * P + n2;
        c32 v[R];
#pragma unroll
        for (int k1 = 0; k1 < R; ++k1) v[k1] = row[r2 * k1];
        dft<R, 1, true>(v);
#pragma unroll
        for (int n1 = 0; n1 < R; ++n1)
            if (r2 * n1 + n2 < g.Z) S[(int64_t)(r2 * n1 + n2) * g.X + x] = v[n1];
    }
}

// ---------------------------------------------------------------------------
// The depth: R_x = sum_d G_d P_{x+d} for every line kz, in place.  A thread sums a tile
// of kTile planes of one line with a window of the line in registers: per d one load
// of the window's next plane and one of G for kTile complex products, each two paired
// FMAs into sums of G.x P and G.y P that are put together every kRun depths.  Tiles go in
// rounds of a thread each, lowest planes first: a tile reads its own planes and later
// ones, so what a round writes nobody reads any more.  Middle kernel, 36 volumes of 128^3:
// tiles of 12 planes 1.00 ms, 10 0.94, 8 0.82, 6 0.89 (four warps a scheduler, and what
// the registers leave for loads in flight; 768 threads of 80 registers 1.06); the sums cut
// at 32 depths and G four steps ahead instead of eight 0.86 (cut at 64 0.85, with G two steps
// ahead 0.86, eight 0.92; the depths in halves on two lanes 0.94).
// ---------------------------------------------------------------------------
constexpr int kTile = 8;
constexpr int kAhead = 4;        // steps that G is loaded ahead of its use
constexpr int kRun = 32;         // depths summed in one go: short sums, for their rounding error

struct DepthSum {
    c32 p[kTile], q[kTile], w[kTile], gv[kAhead], sum[kTile];
    // Steps d .. d + nd - 1, the planes x0 + d + t in w[(d + t) % kTile]; each place of
    // w and gv is refilled as soon as it has been used (`more` depths from `G` on exist,
    // `left` planes from `line` on).
    template <bool FULL>
    __device__ __forceinline__ void steps(const c32* __restrict__ G, int gs, int more, const c32* line, int P,
                                          int left, int nd) {
#pragma unroll
        for (int e = 0; e < kTile; ++e) {
            if (!FULL && e >= nd) break;
            float a, b;
            un(gv[e % kAhead], a, b);
            if (e < more) gv[e % kAhead] = __ldg(G + (int64_t)e * gs);
            const c32 ga = mk(a, a), gb = mk(b, b);
#pragma unroll
            for (int t = 0; t < kTile; ++t) {
                p[t] = cfma2(ga, w[(e + t) % kTile], p[t]);
                q[t] = cfma2(gb, w[(e + t) % kTile], q[t]);
            }
            w[e] = e < left ? line[e * P] : 0ull;
        }
    }
    __device__ __forceinline__ void flush() {
#pragma unroll
        for (int t = 0; t < kTile; ++t) {
            float px, py, qx, qy;
            un(p[t], px, py);
            un(q[t], qx, qy);
            sum[t] = cadd<true>(sum[t], mk(px - qy, py + qx));
            p[t] = q[t] = 0ull;
        }
    }
};

__device__ __forceinline__ void mid_depth(c32* pl, const c32* __restrict__ Gk, const LineGeom& g) {
    const int Nz = g.z.n, P = Nz + 1, D = min(g.Mx, g.X);
    const int items = Nz * ((g.X + kTile - 1) / kTile);
    const float rN = 1.f / (float)Nz;
    for (int i0 = 0; i0 < items; i0 += kMidT) {
        const int i = i0 + threadIdx.x, tile = div_small(i, rN), kz = i - tile * Nz, x0 = tile * kTile;
        const int n = i < items ? g.X - x0 : 0, dmax = min(D, n);   // planes from x0 on, depths
        c32* line = pl + x0 * P + kz;
        const c32* G = Gk + kz;
        DepthSum s;
#pragma unroll
        for (int t = 0; t < kTile; ++t) {
            s.p[t] = s.q[t] = s.sum[t] = 0ull;
            s.w[t] = t < n ? line[t * P] : 0ull;
            if (t < kAhead) s.gv[t] = t < dmax ? __ldg(G + (int64_t)t * Nz) : 0ull;
        }
        const c32* src = line + kTile * P;
        int left = n - kTile, d = dmax;
#pragma unroll 1
        for (; d >= kTile; d -= kTile) {
            s.steps<true>(G + (int64_t)kAhead * Nz, Nz, d - kAhead, src, P, left, kTile);
            G += (int64_t)kTile * Nz;
            src += kTile * P;
            left -= kTile;
            if ((dmax - d) % kRun == kRun - kTile) s.flush();
        }
        s.steps<false>(G + (int64_t)kAhead * Nz, Nz, d - kAhead, src, P, left, d);
        s.flush();
        __syncthreads();
#pragma unroll
        for (int t = 0; t < kTile; ++t)
            if (t < n) line[t * P] = s.sum[t];
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kMidT, 1)
line_mid_kernel(c32* __restrict__ S, const c32* __restrict__ G, const float2* __restrict__ Tz, LineGeom g) {
    extern __shared__ __align__(16) c32 sp[];
    const int P = g.z.n + 1;
    c32* pl = sp;                                                   // [X][Nz + 1]
    float2* tz = reinterpret_cast<float2*>(pl + g.X * P);
    for (int m = threadIdx.x; m < g.z.n; m += kMidT) tz[m] = Tz[m];
    const int ky = blockIdx.x;
    c32* Sk = S + ((int64_t)blockIdx.y * g.Nyh + ky) * g.X * g.Z;
    // the plane, eight bytes a copy, all of it in flight at once
    const int n = g.X * g.Z;
    const float rZ = 1.f / (float)g.Z;
    for (int i = threadIdx.x; i < n; i += kMidT) {
        const int x = div_small(i, rZ);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                         (unsigned)__cvta_generic_to_shared(pl + x * P + i - x * g.Z)), "l"(Sk + i));
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    Team tm;
    tm.n = kTeam;
    tm.id = threadIdx.x / kTeam;
    tm.t = threadIdx.x - tm.id * kTeam;
    tm.x0 = tm.id * g.X / (kMidT / kTeam);
    tm.x1 = (tm.id + 1) * g.X / (kMidT / kTeam);
#define CALL(A, B) mid_za<A, B>(pl, tz, g, tm)
    FLC_LEN(g.z)
#undef CALL
    tm.sync();
#define CALL(A, B) mid_zb<A, B, -1>(pl, tz, g, tm)
    FLC_LEN(g.z)
#undef CALL
    __syncthreads();
    mid_depth(pl, G + (int64_t)ky * min(g.Mx, g.X) * g.z.n, g);
#define CALL(A, B) mid_zb<A, B, 1>(pl, tz, g, tm)
    FLC_LEN(g.z)
#undef CALL
    tm.sync();
#define CALL(A, B) mid_zo<A, B>(pl, Sk, g, tm)
    FLC_LEN(g.z)
#undef CALL
}

// ---------------------------------------------------------------------------
// Rows inverse: grid (ceil(X / 32), ceil(Z / 2), volumes).  Slices z and z + 1 (if it
// exists) are the real and the imaginary part.
// ---------------------------------------------------------------------------
// Where the results go: the reference layout; the beam layout; the beam layout, multiplying
// an attenuation that is loaded before the last DFTs.  The loads ahead take registers, three
// CTAs an SM instead of four; they pay up to DFTs of kAheadR points (us, ahead / not: 36
// volumes of 128^3, 12 points, 243 / 442; 24 of 96^3, 12, 89 / 163; 40 of 61 x 111^2, 16,
// 262 / 185; 12 of 150^3, 18, 401 / 322).
enum { kRef, kBeam, kBeamAhead };
constexpr int kAheadR = 12;

struct OutArgs {
    float* out;
    int mode;                // 0 res, 1 exp(-res) in the reference layout;
                             // 2 multiplies, 3 stores exp(-res) in the beam layout
    int L, a_base, v0;       // first volume of this launch
    int64_t a_stride, l_stride;
    float scale;
};

// The slices' half spectra as one spectrum, then step 1.
template <int R1, int R>
__device__ __forceinline__ void out_b(const c32* S, c32* sm, const float2* tw, const LineGeom& g, int nl,
                                      bool two) {
    constexpr int N = R1 * R, P = N + 1;
    const int64_t ks = (int64_t)g.X * g.Z;
    const int l = threadIdx.x & 31;
    if (l < nl) {
#pragma unroll 4
        for (int k = threadIdx.x >> 5; k <= N / 2; k += kRowsT / 32) {
            float x, y, u = 0.f, v = 0.f;
            un(S[k * ks + l], x, y);
            if (two) un(S[k * ks + g.X + l], u, v);
            if (k == 0 || 2 * k == N) y = v = 0.f;       // (real rows)
            sm[l * P + place<R1, R>(k)] = mk(x - v, y + u);
            if (k != 0 && 2 * k != N) sm[l * P + place<R1, R>(N - k)] = mk(x + v, u - y);
        }
    }
    __syncthreads();
    if (l >= nl) return;
    for (int k1 = threadIdx.x >> 5; k1 < R1; k1 += kRowsT / 32) {
        c32 v[R];
#pragma unroll
        for (int k2 = 0; k2 < R; ++k2) v[k2] = sm[l * P + R * k1 + k2];
        dft<R, 1, false>(v);
        twiddle<R, 1>(v, tw, k1);
#pragma unroll
        for (int n2 = 0; n2 < R; ++n2) sm[l * P + R * k1 + n2] = v[n2];
    }
}

template <int R, int R2, int TO>
__device__ __forceinline__ void out_a(c32* sm, const LineGeom& g, const OutArgs& o, float* oa, float* ob,
                                      int nl) {
    constexpr int r2 = R2, P = R * R2 + 1;
    const int l = threadIdx.x & 31;
    if (l >= nl) return;
    for (int n2 = threadIdx.x >> 5; n2 < r2; n2 += kRowsT / 32) {
        c32 v[R];
        float pa[R], pb[R];
        constexpr bool ahead = TO == kBeamAhead && R <= kAheadR;
        // (the mode is known to be 2: the branch keeps the loads from being moved down
        // to their use, 243 against 352 us)
        if (ahead && o.mode == 2) {
#pragma unroll
            for (int n1 = 0; n1 < R; ++n1) {
                const int y = r2 * n1 + n2;
                pa[n1] = y < g.Y ? oa[(int64_t)(g.Y - 1 - y) * g.X + l] : 0.f;
                pb[n1] = y < g.Y && ob ? ob[(int64_t)(g.Y - 1 - y) * g.X + l] : 0.f;
            }
        }
#pragma unroll
        for (int k1 = 0; k1 < R; ++k1) v[k1] = sm[l * P + r2 * k1 + n2];
        dft<R, 1, false>(v);
#pragma unroll
        for (int n1 = 0; n1 < R; ++n1) {
            const int y = r2 * n1 + n2;
            float ra, rb;
            un(v[n1], ra, rb);
            ra *= o.scale;
            rb *= o.scale;
            if constexpr (TO == kRef) {
                sm[l * P + y] = mk(o.mode ? expf(-ra) : ra, o.mode ? expf(-rb) : rb);
            } else if (y < g.Y) {
                const int64_t at = (int64_t)(g.Y - 1 - y) * g.X + l;
                const float ea = expf(-ra), eb = expf(-rb);
                oa[at] = o.mode == 2 ? (ahead ? pa[n1] : oa[at]) * ea : ea;
                if (ob) ob[at] = o.mode == 2 ? (ahead ? pb[n1] : ob[at]) * eb : eb;
            }
        }
    }
}

template <int TO>
__global__ void __launch_bounds__(kRowsT, TO == kBeamAhead ? 3 : 4)
line_out_kernel(const c32* __restrict__ S, const float2* __restrict__ Ty, OutArgs o, LineGeom g) {
    extern __shared__ __align__(16) c32 sm[];                       // [32][Ny + 1], twiddles
    const int P = g.y.n + 1;
    float2* tw = reinterpret_cast<float2*>(sm + kLines * P);
    for (int m = threadIdx.x; m < g.y.n; m += kRowsT) tw[m] = Ty[m];
    __syncthreads();
    const int x0 = blockIdx.x * kLines, z = 2 * blockIdx.y;
    const bool two = z + 1 < g.Z;
    const int nl = min(kLines, g.X - x0);
    const c32* Sv = S + ((int64_t)blockIdx.z * g.Nyh * g.Z + z) * g.X + x0;
#define CALL(A, B) out_b<A, B>(Sv, sm, tw, g, nl, two)
    FLC_LEN(g.y)
#undef CALL
    __syncthreads();
    const int v = o.v0 + blockIdx.z;
    float* oa;
    if constexpr (TO != kRef) {
        const int al = v / o.L, l = v - al * o.L;
        oa = o.out + l * o.l_stride + (int64_t)(o.a_base + al) * o.a_stride + (int64_t)z * g.Y * g.X + x0;
    } else {
        oa = o.out + (((int64_t)v * g.Z + z) * g.X + x0) * g.Y;
    }
    float* ob = two ? oa + (int64_t)g.X * g.Y : nullptr;
#define CALL(A, B) out_a<A, B, TO>(sm, g, o, oa, ob, nl)
    FLC_LEN(g.y)
#undef CALL
    if constexpr (TO != kRef) return;
    __syncthreads();
    const float rY = 1.f / (float)g.Y;
    for (int i = threadIdx.x; i < nl * g.Y; i += kRowsT) {
        const int l = div_small(i, rY), y = i - l * g.Y;
        float ra, rb;
        un(sm[l * P + y], ra, rb);
        oa[i] = ra;
        if (ob) ob[i] = rb;
    }
}

#define FLC_ENTRY(i, A, B) {(A) * (B), A, B, i},
const Len kLens[] = {FLC_LENS(FLC_ENTRY)};

bool pick_len(int need, Len* l) {
    for (const Len& c : kLens)
        if (c.n >= need) { *l = c; return true; }
    return false;
}

size_t al256(size_t n) { return (n + 255) & ~(size_t)255; }

size_t mid_smem(const LineGeom& g) { return sizeof(c32) * ((size_t)g.X * (g.z.n + 1) + g.z.n); }
size_t rows_smem(const LineGeom& g) { return sizeof(c32) * ((size_t)kLines * (g.y.n + 1) + g.y.n); }

bool line_geom(int64_t Z, int64_t X, int64_t Y, int64_t Mz, int64_t Mx, int64_t My, LineGeom* g) {
    if (Z < 1 || X < 1 || Y < 1 || Mz < 1 || Mx < 1 || My < 1) return false;
    if (Z > 4096 || Y > 4096 || X > 4096 || Mx > 4096 || Mz > 4096 || My > 4096) return false;
    const int hz = (int)Mz / 2, hy = (int)My / 2;
    g->Z = (int)Z; g->X = (int)X; g->Y = (int)Y;
    g->Mz = (int)Mz; g->Mx = (int)Mx; g->My = (int)My;
    if (!pick_len((int)Z + std::max(hz, (int)Mz - 1 - hz), &g->z) ||
        !pick_len((int)Y + std::max(hy, (int)My - 1 - hy), &g->y))
        return false;
    g->Nyh = g->y.n / 2 + 1;
    const size_t cap = (size_t)max_smem_optin();
    return mid_smem(*g) <= cap && rows_smem(*g) <= cap;
}

// Spectra held at a time: volumes are taken in batches of at most this much scratch.
constexpr size_t kBatchBytes = 512u << 20;

struct LineWs {
    double2 *Uf, *Vf;
    float2 *Tz, *Ty;
    c32 *G, *S;
    int64_t batch;    // volumes whose spectra S holds
    size_t bytes;
};

// The scratch that is asked for has room for min(Vn, the most of a batch) volumes, so a
// call over fewer volumes never needs more; a call takes what it is given, `have` bytes,
// for batches of one volume on (batch 0: not even that).
LineWs line_ws(const LineGeom& g, int64_t Vn, char* base, size_t have) {
    LineWs w{};
    size_t off = 0;
    auto take = [&](size_t n) { char* p = base ? base + off : nullptr; off += al256(n); return p; };
    const size_t vol = sizeof(c32) * (size_t)g.Nyh * g.X * g.Z;
    w.Uf = (double2*)take(sizeof(double2) * (size_t)g.Mx * g.z.n);
    w.Vf = (double2*)take(sizeof(double2) * (size_t)g.Mx * g.Nyh);
    w.Tz = (float2*)take(sizeof(float2) * g.z.n);
    w.Ty = (float2*)take(sizeof(float2) * g.y.n);
    w.G = (c32*)take(sizeof(c32) * (size_t)g.Nyh * std::min(g.Mx, g.X) * g.z.n);
    w.batch = std::max<int64_t>(1, std::min<int64_t>(Vn, (int64_t)(kBatchBytes / vol)));
    if (base) w.batch = have < off ? 0 : std::min<int64_t>(w.batch, (int64_t)((have - off) / vol));
    w.S = (c32*)take(vol * (size_t)w.batch);
    w.bytes = off;
    return w;
}

template <class K>
int allow_smem(K kernel, size_t bytes) {
    FLC_TRY_CUDA(cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)bytes));
    return FLC_OK;
}

}  // namespace

// Scratch bytes of the line form for Vn volumes, 0 if it does not take the shape.
size_t cone_line_ws_bytes(int64_t Vn, int64_t Z, int64_t X, int64_t Y, int64_t Mz, int64_t Mx,
                          int64_t My) {
    LineGeom g;
    if (tune(kTuneConeVariant) == 5 || !line_geom(Z, X, Y, Mz, Mx, My, &g)) return 0;
    return line_ws(g, Vn, nullptr, 0).bytes;
}

// Scratch bytes of the spectral cone, whichever form takes the shape.
size_t cone_spec_ws_bytes(int64_t Vn, int64_t Z, int64_t X, int64_t Y, int64_t Mz, int64_t Mx,
                          int64_t My, int mode) {
    const size_t line = cone_line_ws_bytes(Vn, Z, X, Y, Mz, Mx, My);
    return line ? line : cone_fft_ws_bytes(Vn, Z, X, Y, Mz, Mx, My, mode);
}

// The path sum in the line form; arguments, modes and FLC_ERR_UNSUPPORTED as
// cone_fft_launch.
int cone_line_launch(const float* mu, const float* U, const float* Vw, float* out, int64_t Vn,
                     int64_t Z, int64_t X, int64_t Y, int64_t Mz, int64_t Mx, int64_t My, int mode,
                     int L, int a_base, int64_t out_a_stride, int64_t out_l_stride, void* workspace,
                     size_t ws_bytes, cudaStream_t st) {
    LineGeom g;
    if (!workspace || Vn < 1 || Vn > 65535 || tune(kTuneConeVariant) == 5 ||
        !line_geom(Z, X, Y, Mz, Mx, My, &g) || ((uintptr_t)workspace & 255) != 0)
        return FLC_ERR_UNSUPPORTED;
    const LineWs w = line_ws(g, Vn, (char*)workspace, ws_bytes);
    if (w.batch < 1) return FLC_ERR_UNSUPPORTED;
    const size_t rsm = rows_smem(g), msm = mid_smem(g);
    FLC_TRY(allow_smem(line_rows_kernel, rsm));
    FLC_TRY(allow_smem(line_mid_kernel, msm));
    const auto out_kernel = mode < 2 ? line_out_kernel<kRef>
                            : mode == 2 && g.y.r1 <= kAheadR ? line_out_kernel<kBeamAhead>
                                                             : line_out_kernel<kBeam>;
    FLC_TRY(allow_smem(out_kernel, rsm));
    line_roots_kernel<<<(unsigned)g.Mx + 1, 256, sizeof(double2) * (size_t)(g.z.n + g.y.n), st>>>(
        U, Vw, w.Uf, w.Vf, w.Tz, w.Ty, g);
    FLC_TRY(check_launch("line_roots_kernel"));
    line_filter_kernel<<<dim3((unsigned)std::min(g.Mx, g.X), (unsigned)g.Nyh), 128, 0, st>>>(w.Uf, w.Vf, w.G,
                                                                                             g);
    FLC_TRY(check_launch("line_filter_kernel"));
    OutArgs o{out, mode, L, a_base, 0, out_a_stride, out_l_stride,
              (float)(0.5 / ((double)g.y.n * (double)g.z.n))};      // (line_rows leaves twice the spectra)
    const int64_t vol = Z * X * Y, batch = ceil_div(Vn, ceil_div(Vn, w.batch));   // evened
    for (int64_t v0 = 0; v0 < Vn; v0 += batch) {
        const unsigned n = (unsigned)std::min<int64_t>(batch, Vn - v0);
        line_rows_kernel<<<dim3((unsigned)ceil_div(Z, 2 * kLines), (unsigned)X, n), kRowsT, rsm, st>>>(
            mu + v0 * vol, w.Ty, w.S, g);
        FLC_TRY(check_launch("line_rows_kernel"));
        line_mid_kernel<<<dim3((unsigned)g.Nyh, n), kMidT, msm, st>>>(w.S, w.G, w.Tz, g);
        FLC_TRY(check_launch("line_mid_kernel"));
        o.v0 = (int)v0;
        out_kernel<<<dim3((unsigned)ceil_div(X, kLines), (unsigned)ceil_div(Z, 2), n), kRowsT, rsm, st>>>(
            w.S, w.Ty, o, g);
        FLC_TRY(check_launch("line_out_kernel"));
    }
    return FLC_OK;
}

}  // namespace flc
