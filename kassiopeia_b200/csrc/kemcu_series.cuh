// Far-field series of an element: what the cubature bands of a distant pair sum up to, as a
// multipole expansion about the element's centroid instead of 7, 12 or 33 nodes.
//
// With d = P - centroid, R = |d|, an orthonormal frame (e1, e2) of the element's plane, X = d.e1 / R,
// Y = d.e2 / R and t = s / R (s: the largest distance of the element's rim from its centroid),
//   phi = pre / R (1 + sum_n t^n G_n(X, Y)),   G_n = < |o|^n P_n(cos(o, d)) > / s^n
// where < > is the mean over the element: G_n is a polynomial of degree and parity n whose
// coefficients are the element's exact moments (n = 1 vanishes at the centroid). The rules of the
// numeric policy integrate these polynomials exactly up to their degree and agree with the series
// far below rounding beyond the cuts used here, whatever band the pair has, so no band decision
// is needed either. The field follows from the value, the value weighted by n + 1 and the two
// derivatives:
//   E = pre / R^2 { (d/R) [W + X S_X + Y S_Y] - e1 S_X - e2 S_Y },  W = sum_n (n + 1) t^n G_n.
// By parity a G_n splits into p(X^2, Y^2) and q(X^2, Y^2): p + XY q for even n, X p + Y q for odd n;
// elements with two mirror axes (rectangles, wires) have the p of even n only.
//
// What bounds it: an FP64 instruction holds the issue port of its scheduler for two cycles (16 lanes),
// an FP32 one for one, so the cost of a pair is 2 x FP64 + the rest in issue cycles (measured within
// 20 %: 250 cycles per 32 pairs for 67 FP64 and 81 other instructions). A 33-node pair of the rules
// takes ~440 FP64 operations, a 12-node one ~190; the series of a symmetric element 54 to 88 and 45 to
// 75 others. (Two points per lane would share the coefficient loads, but take 131 to 168 registers and spill:
// 193 instead of 147 ms for 400,000 points of a coaxial electrode pair.)
//
// Precision. FP64 form: n <= 4 in FP64, nearer elements also n = 5 (general) or 6 (symmetric); the
// tail of higher orders is at most ~3e-9 of the term where it is used. The cuts bound the first orders
// left out by 5e-16 of the pair's field in the worst direction at the cut, and the rounding of order 6 in FP32 by
// 1e-15 (in the nearest tier of general elements, where orders 7 to 10 add theirs, 2.5e-16). Measured against
// exact integrals, a pair's field at most 2.1e-15 and 2.5e-16 in the mean, a rule's 2.2e-15 and 2.4e-16. MIXED
// form: n = 4 (symmetric elements' farthest tier) and 5 (general) in FP32 too, orders left out 1e-14, the FP32
// orders 3e-13: at most 2.5e-13, where the rules' nodes give 1.4e-12. Wires keep FP64's precision in both.
//
// Included after kemcu_device.cuh (element records, V3, irsq); the functions here are plain C++
// apart from their decorations, and tests/cxx/series_host.cc runs them on the CPU.
#pragma once

namespace kemcu
{

// Far records, in tiles: a tile holds up to kFarSym elements that all have two mirror axes, or up
// to kFarGen others, in element order. Layout in doubles (16-byte groups, as the kernel loads them;
// the strides put consecutive elements' headers into different banks for the per-lane tier test):
constexpr int kFarSym = 16, kFarGen = 8;
constexpr int kFarSymStride = 66, kFarGenStride = 130;
constexpr int kFarStage = kFarSym * kFarSymStride > kFarGen * kFarGenStride ? kFarSym * kFarSymStride
                                                                            : kFarGen * kFarGenStride;
// Every polynomial's coefficients start on a 16-byte boundary (far_pad).
enum Far : int
{
    fCen = 0,   // centroid (3)
    fSize = 3,  // s
    fE1 = 4,    // frame (6)
    fCut = 10,  // distances beyond which tiers 3, 2, 1 hold: FP64 form (3)
    fCutM = 13, // and MIXED form (3)
    fD2 = 16,   // FP64: p of n = 2 (3), and at fD2 + 3 the q of n = 2 (general, 1)
    fD4 = 20,   // p of n = 4 (6)
    fSymD6 = 26,  // symmetric: p of n = 6 (10); FP32 from fSymF: p of n = 4, 6, 8, 10
    fSymF = 36,
    fGenD3 = 26,  // general: X p and Y q of n = 3 (3 + 3), q of n = 4 (3), n = 5 (6 + 6)
    fGenQ4 = 32,
    fGenD5 = 36,
    fGenF = 48,  // FP32: n = 5 (p, q), 6 (p, q), ..., 10
};
template<class T> __host__ __device__ constexpr int far_pad(int k)
{
    return (k + 16 / (int) sizeof(T) - 1) / (16 / (int) sizeof(T)) * (16 / (int) sizeof(T));
}
__host__ __device__ constexpr int far_terms(int deg)
{
    return (deg + 1) * (deg + 2) / 2;
}
// offsets (in floats) of the FP32 polynomials
constexpr int kS4 = 0, kS6 = kS4 + far_pad<float>(far_terms(2)), kS8 = kS6 + far_pad<float>(far_terms(3)), kS10 = kS8 + far_pad<float>(far_terms(4)),
              kSEnd = kS10 + far_pad<float>(far_terms(5));
constexpr int kG5p = 0, kG5q = kG5p + far_pad<float>(far_terms(2)), kG6p = kG5q + far_pad<float>(far_terms(2)),
              kG6q = kG6p + far_pad<float>(far_terms(3)), kG7p = kG6q + far_pad<float>(far_terms(2)),
              kG7q = kG7p + far_pad<float>(far_terms(3)), kG8p = kG7q + far_pad<float>(far_terms(3)),
              kG8q = kG8p + far_pad<float>(far_terms(4)), kG9p = kG8q + far_pad<float>(far_terms(3)),
              kG9q = kG9p + far_pad<float>(far_terms(4)), kG10p = kG9q + far_pad<float>(far_terms(4)),
              kG10q = kG10p + far_pad<float>(far_terms(5)), kGEnd = kG10q + far_pad<float>(far_terms(4));
static_assert(2 * fSymF + kSEnd <= 2 * kFarSymStride && 2 * fGenF + kGEnd <= 2 * kFarGenStride, "far record layout");

// one tile: elements [first, first + count), doubles offset of its records, general or symmetric
struct FarTile
{
    int first, count, general;
    long long off16;  // offset in 16-byte units
};
// where an element's far record is: the low 32 bits of its offset, the high bits and whether it is general
__host__ __device__ inline int2 far_where(long long off16, bool general)
{
    return make_int2((int) (unsigned) off16, (int) (off16 >> 32) * 2 + (general ? 1 : 0));
}
__host__ __device__ inline size_t far_offset(int2 at)
{
    return 2 * (((size_t) (at.y >> 1) << 32) | (unsigned) at.x);
}

// ------------------------------------------------------------------------- building
constexpr int kFarOrder = 12;  // moments: up to the first order that any tier leaves out
constexpr int kFarQ = 7;       // Gauss-Legendre points a direction: degree 13 on the collapsed square
struct FarTables
{
    double x[kFarQ], w[kFarQ];          // Gauss-Legendre rule on [0, 1]
    double bin[kFarOrder + 1][kFarOrder + 1];
    double leg[kFarOrder + 1][kFarOrder / 2 + 1];  // P_n(x) = sum_m leg[n][m] x^(n - 2m)
    double ca[12], sa[12];              // directions in the plane, every 15 degrees
};
inline void far_tables(FarTables& t)  // all but the quadrature rule
{
    for (int n = 0; n <= kFarOrder; n++) {
        for (int k = 0; k <= kFarOrder; k++)
            t.bin[n][k] = k > n ? 0. : k == 0 ? 1. : t.bin[n][k - 1] * (n - k + 1) / k;
        // leg = (-1)^m (2n - 2m)! / (2^n m! (n - m)! (n - 2m)!), with (2k)! / (k! 2^k) = (2k - 1)!!
        for (int m = 0; m <= n / 2; m++) {
            double v = (m & 1) ? -1. : 1.;
            for (int k = 2 * (n - m) - 1; k > 1; k -= 2)
                v *= k;
            for (int k = 2; k <= n - 2 * m; k++)
                v /= k;
            for (int k = 1; k <= m; k++)
                v /= 2. * k;
            t.leg[n][m] = v;
        }
    }
    for (int k = 0; k < 12; k++) {
        t.ca[k] = cos(k * 0.261799387799149436);
        t.sa[k] = sin(k * 0.261799387799149436);
    }
}

// One warp builds a record; as plain C++ one lane does.
#ifdef __CUDACC__
constexpr int kFarLanes = 32;
__device__ __forceinline__ double far_max(double v)
{
    for (int o = 16; o > 0; o >>= 1)
        v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
#else
#define __shared__ static
constexpr int kFarLanes = 1;
inline double far_max(double v)
{
    return v;
}
inline void __syncwarp() {}
inline void __syncthreads() {}
#endif
constexpr int kFarBuild = 4 * kFarLanes;  // threads of a CTA
constexpr int kFarDirs = 25;              // directions that |G_n| is looked at in

// coefficients of G_n, n <= kFarOrder: those of X^i Y^j with i + j = n, n - 2, ...
__host__ __device__ constexpr int far_count(int n)
{
    return (n + 2) * (n + 2) / 4;
}
__host__ __device__ constexpr int far_base(int n)  // orders 2, 3, ..., n - 1 come first
{
    int s = 0;
    for (int q = 2; q < n; q++)
        s += far_count(q);
    return s;
}
constexpr int kFarCoefs = far_base(kFarOrder + 1);
__device__ __forceinline__ int far_index(int n, int i, int j)  // within order n
{
    const int m = (n - i - j) / 2;
    return m * (n + 1) - m * (m - 1) + i;
}

// a warp's workspace
struct FarWork
{
    double M[kFarOrder + 1][kFarOrder + 1];  // < x^a y^b > / s^(a + b), a + b <= kFarOrder
    double c[kFarCoefs];
    double g[kFarOrder + 1];  // largest |G_n|
    double r[16];
    alignas(16) double f[kFarGenStride];
};
struct FarBinLeg
{
    double bin[kFarOrder + 1][kFarOrder + 1], leg[kFarOrder + 1][kFarOrder / 2 + 1];
};

// the coefficients of the class (px, py) of G_n, X^px Y^py poly(X^2, Y^2) of degree `deg`, in
// the order far_poly reads them (powers of X^2 descending; within one, powers of Y^2 descending)
template<int N, int PX, int PY, int DEG, class T> __device__ __forceinline__ void far_class(const FarWork& W, int lane, T* out)
{
    for (int k = lane; k < far_terms(DEG); k += kFarLanes) {
        int row = 0, first = 0;  // row: DEG - i, of row + 1 terms
        while (first + row + 1 <= k)
            first += ++row;
        const int i = DEG - row, j = row - (k - first);
        out[k] = (T) W.c[far_base(N) + far_index(N, 2 * i + PX, 2 * j + PY)];
    }
}

// Far record of every element from its element record, one warp per slot of the tiles; the moments of
// rectangles and wires in symmetric tiles are closed forms, the others' an exact cubature. (One
// thread per element was a chain of 0.96 ms whatever their number.)
__global__ void far_build_kernel(const double* __restrict__ rec, const FarTile* __restrict__ tiles, int ntiles,
                                 const __grid_constant__ FarTables gl, double* __restrict__ far, double* __restrict__ pre, int2* __restrict__ where)
{
    __shared__ FarBinLeg s_t;
    __shared__ FarWork s_w[kFarBuild / kFarLanes];
    for (int i = threadIdx.x; i < (kFarOrder + 1) * (kFarOrder + 1); i += blockDim.x)
        s_t.bin[i / (kFarOrder + 1)][i % (kFarOrder + 1)] = gl.bin[i / (kFarOrder + 1)][i % (kFarOrder + 1)];
    for (int i = threadIdx.x; i < (kFarOrder + 1) * (kFarOrder / 2 + 1); i += blockDim.x)
        s_t.leg[i / (kFarOrder / 2 + 1)][i % (kFarOrder / 2 + 1)] = gl.leg[i / (kFarOrder / 2 + 1)][i % (kFarOrder / 2 + 1)];
    __syncthreads();
    const int lane = threadIdx.x % kFarLanes;
    const size_t q = (blockIdx.x * (size_t) blockDim.x + threadIdx.x) / kFarLanes;
    const int ti = (int) (q / kFarSym), k = (int) (q % kFarSym);
    if (ti >= ntiles || k >= tiles[ti].count)
        return;
    FarWork& W = s_w[threadIdx.x / kFarLanes];
    const FarTile T = tiles[ti];
    const double* e = rec + (size_t) (T.first + k) * rRecSize;
    const int stride = T.general ? kFarGenStride : kFarSymStride;
    double* f = W.f;
    for (int i = lane; i < stride; i += kFarLanes)
        f[i] = 0.;
    const int type = (int) e[rType];
    const V3 a = ld3(e + rEa), b = ld3(e + rEb), c = ld3(e + rCen);
    const double la = norm(a);
    const V3 e1 = (1. / la) * a;
    V3 e2 = b - dot(b, e1) * e1;
    if (type == kLineSegment) {  // any direction across the wire
        const V3 x = fabs(e1.x) < 0.6 ? v3(1., 0., 0.) : v3(0., 1., 0.);
        e2 = x - dot(x, e1) * e1;
    }
    e2 = (1. / norm(e2)) * e2;
    const double bx = dot(b, e1), by = dot(b, e2);
    // s and the moments over s
    double s;
    // the corner (x0, y0) and the sides that its nodes (u, v) in [0, 1]^2 run along
    const bool triangle = type == kTriangle, wire = type == kLineSegment;
    const double wx = type == kLineSegment ? 0. : bx, wy = type == kLineSegment ? 0. : by;
    double x0, y0;
    if (triangle) {
        x0 = -(la + bx) / 3., y0 = -by / 3.;
        const double x1 = la + x0, y1 = y0, x2 = bx + x0, y2 = by + y0;
        s = sqrt(fmax(x0 * x0 + y0 * y0, fmax(x1 * x1 + y1 * y1, x2 * x2 + y2 * y2)));
    }
    else {  // the parallelogram u a + v b, u, v in [-1/2, 1/2] (wires: b = 0)
        const double cx1 = 0.5 * (la + wx), cx2 = 0.5 * (la - wx), cy = 0.5 * wy;
        s = sqrt(fmax(cx1 * cx1 + cy * cy, cx2 * cx2 + cy * cy));
        x0 = -cx1, y0 = -cy;
    }
    const double is = 1. / s;
    if (!T.general) {
        const double hx = 0.5 * la * is, hy = 0.5 * wy * is;
        for (int m = lane; m < (kFarOrder / 2 + 1) * (kFarOrder / 2 + 1); m += kFarLanes) {
            const int i = m / (kFarOrder / 2 + 1), j = m % (kFarOrder / 2 + 1);
            double v = 1. / ((2. * i + 1.) * (2. * j + 1.));
            for (int p = 0; p < i; p++)
                v *= hx * hx;
            for (int p = 0; p < j; p++)
                v *= hy * hy;
            if (i + j <= kFarOrder / 2)
                W.M[2 * i][2 * j] = v;
        }
    }
    else
        for (int ax = lane; ax <= kFarOrder; ax += kFarLanes) {  // a lane per power of x
            double m[kFarOrder + 1];
#pragma unroll
            for (int ay = 0; ay <= kFarOrder; ay++)
                m[ay] = 0.;
#pragma unroll 1
            for (int i = 0; i < kFarQ; i++)
#pragma unroll 1
                for (int j = 0; j < kFarQ; j++) {
                    const double u = gl.x[i], h = triangle ? 1. - u : 1., v = gl.x[j] * h;
                    const double x = (x0 + u * la + v * wx) * is, y = (y0 + v * wy) * is;
                    double p = (triangle ? 2. : 1.) * gl.w[i] * gl.w[j] * h, x2 = x;
#pragma unroll
                    for (int bit = 1; bit <= kFarOrder; bit <<= 1) {
                        if (ax & bit)
                            p *= x2;
                        x2 *= x2;
                    }
#pragma unroll
                    for (int ay = 0; ay <= kFarOrder; ay++) {
                        m[ay] += p;
                        p *= y;
                    }
                }
#pragma unroll
            for (int ay = 0; ay <= kFarOrder; ay++)
                if (ax + ay <= kFarOrder)
                    W.M[ax][ay] = m[ay];
        }
    __syncwarp();
    // coefficient of X^i Y^j in G_n (i + j = p = n - 2m); two mirror axes leave even n, i and j
    for (int w = lane; w < kFarCoefs; w += kFarLanes) {
        int n = 2, t = w;
        while (t >= far_count(n))
            t -= far_count(n++);
        int p = n;
        while (t > p) {
            t -= p + 1;
            p -= 2;
        }
        const int i = t, j = p - t, m = (n - p) / 2;
        double v = 0.;
        if (T.general || !(i & 1 || j & 1)) {
            for (int z = 0; z <= m; z++)
                v += s_t.bin[m][z] * W.M[i + 2 * z][j + 2 * (m - z)];
            v *= s_t.leg[n][m] * s_t.bin[p][i];
        }
        W.c[w] = v;
    }
    __syncwarp();
    // largest |G_n| over directions in the plane (every 15 degrees), at 60 degrees from its normal and along it
    for (int n = 4; n <= kFarOrder; n++) {
        if (n == 5 || (!T.general && n & 1)) {
            if (lane == 0)
                W.g[n] = 0.;
            continue;
        }
        double big = 0.;
        for (int z = lane; z < kFarDirs; z += kFarLanes) {
            const double x = z < 24 ? gl.ca[z % 12] * (z < 12 ? 1. : 0.8660254037844386) : 0.;
            const double y = z < 24 ? gl.sa[z % 12] * (z < 12 ? 1. : 0.8660254037844386) : 0.;
            const double* cn = W.c + far_base(n);
            double v = 0.;
            for (int p = n; p >= 0; p -= 2) {
                double yp = 1., h = 0.;
                for (int i = p; i >= 0; i--) {  // sum over i of c x^i y^(p - i)
                    h = fma(h, x, cn[i] * yp);
                    yp *= y;
                }
                v += h;
                cn += p + 1;
            }
            big = fmax(big, fabs(v));
        }
        big = far_max(big);
        if (lane == 0)
            W.g[n] = big;
    }
    __syncwarp();
    if (lane == 0) {
        f[fCen] = c.x, f[fCen + 1] = c.y, f[fCen + 2] = c.z;
        f[fSize] = s;
        f[fE1] = e1.x, f[fE1 + 1] = e1.y, f[fE1 + 2] = e1.z;
        f[fE1 + 3] = e2.x, f[fE1 + 4] = e2.y, f[fE1 + 5] = e2.z;
    }
    far_class<2, 0, 0, 1>(W, lane, f + fD2);
    far_class<4, 0, 0, 2>(W, lane, f + fD4);
    if (T.general) {
        far_class<2, 1, 1, 0>(W, lane, f + fD2 + 3);
        far_class<3, 1, 0, 1>(W, lane, f + fGenD3);
        far_class<3, 0, 1, 1>(W, lane, f + fGenD3 + 3);
        far_class<4, 1, 1, 1>(W, lane, f + fGenQ4);
        far_class<5, 1, 0, 2>(W, lane, f + fGenD5);
        far_class<5, 0, 1, 2>(W, lane, f + fGenD5 + 6);
        float* g = reinterpret_cast<float*>(f + fGenF);
        far_class<5, 1, 0, 2>(W, lane, g + kG5p);
        far_class<5, 0, 1, 2>(W, lane, g + kG5q);
        far_class<6, 0, 0, 3>(W, lane, g + kG6p);
        far_class<6, 1, 1, 2>(W, lane, g + kG6q);
        far_class<7, 1, 0, 3>(W, lane, g + kG7p);
        far_class<7, 0, 1, 3>(W, lane, g + kG7q);
        far_class<8, 0, 0, 4>(W, lane, g + kG8p);
        far_class<8, 1, 1, 3>(W, lane, g + kG8q);
        far_class<9, 1, 0, 4>(W, lane, g + kG9p);
        far_class<9, 0, 1, 4>(W, lane, g + kG9q);
        far_class<10, 0, 0, 5>(W, lane, g + kG10p);
        far_class<10, 1, 1, 4>(W, lane, g + kG10q);
    }
    else {
        float* g = reinterpret_cast<float*>(f + fSymF);
        far_class<4, 0, 0, 2>(W, lane, g + kS4);
        far_class<6, 0, 0, 3>(W, lane, f + fSymD6);
        far_class<6, 0, 0, 3>(W, lane, g + kS6);
        far_class<8, 0, 0, 4>(W, lane, g + kS8);
        far_class<10, 0, 0, 5>(W, lane, g + kS10);
    }
    // Cuts: the first order left out, n, contributes t^n G_n to the value and (n + 1) times that to
    // the field, held to `eps` of the term at the cut; sampled directions and the later orders
    // (R >= 5 s) are covered by the factor 1.5. Odd and even orders are looked at (parallelograms have
    // no odd ones). An order n evaluated in FP32 rounds by at most ~4e-7 (n + 1) t^n G_n. Never near
    // the analytic band.
    for (int z = lane; z < 15; z += kFarLanes) {
        // FP64, MIXED; FP32 orders (the last: of general elements' nearest tier, whose orders 7 to 10 are FP32 too).
        // Wires are FP64 in every form
        const double eps = z < 6 || (wire && z < 12) ? 5e-16 : z < 12 ? 1e-14
                           : z == 12 && !wire        ? 3e-13 : z < 14 ? 1e-15 : 2.5e-16;
        const int n = z < 12 ? 7 + z % 6 : z == 12 ? 4 : 6;
        W.r[z] = pow((z < 12 ? 1.5 : 4e-7) * (n + 1) * W.g[n] / eps, 1. / n);
    }
    __syncwarp();
    if (lane == 0) {
        for (int form = 0; form < 2; form++) {
            // half of MIXED's cuts, the FP32 form's, lie outside the analytic band too
            auto distance = [&](double r) { return fmax(s * fmax(5., r), sqrt((form ? 4.0001 : 2.) * e[rCut])); };
            const double* r = W.r + 6 * form;
            double* cut = f + (form ? fCutM : fCut);
            // symmetric: n <= 6, 8, 10; general: n <= 6, 8, 10
            double r1 = fmax(r[4], r[5]), r2 = fmax(r[2], r[3]), r3 = fmax(r[0], r[1]);
            if (form && !T.general)  // n = 4 in FP32 beyond the first cut
                r3 = fmax(r3, W.r[12]);
            if (!form || T.general || wire) {
                if (form || T.general)
                    r1 = fmax(r1, W.r[form ? 13 : 14]);
                r2 = fmax(r2, W.r[13]);
            }
            r2 = fmax(r2, r1);
            r3 = fmax(r3, r2);
            const double twice = form && wire ? 2. : 1.;  // the FP32 form takes half of these cuts
            cut[0] = twice * distance(r3), cut[1] = twice * distance(r2), cut[2] = twice * distance(r1);
        }
        // a degenerate element (no plane, no extent) keeps the cubature everywhere
        const double chk = e1.x + e1.y + e1.z + e2.x + e2.y + e2.z + f[fCut] + f[fCut + 2] + f[fCutM] + f[fCutM + 2];
        if (!(s > 0.) || !isfinite(chk))
            for (int i = 0; i < 6; i++)
                f[fCut + i] = CUDART_INF;
        where[T.first + k] = far_where(T.off16 + k * stride / 2, T.general);
        pre[T.first + k] = type == kLineSegment ? e[rPrefac] * e[rA] : e[rPrefac];
    }
    __syncwarp();
    double* out = far + 2 * (size_t) T.off16 + (size_t) k * stride;
    for (int i = lane; i < stride; i += kFarLanes)
        out[i] = f[i];
}

// ------------------------------------------------------------------------- evaluation
// g = sum c x^i y^j, i + j <= DEG (coefficients in far_class's order) and its derivatives
template<int DEG, bool GRAD, class T>
__device__ __forceinline__ void far_poly(const T* c, T x, T y, T& g, T& gx, T& gy)
{
    int k = 0;
    g = c[k++];
    gx = gy = (T) 0;
#pragma unroll
    for (int i = DEG - 1; i >= 0; i--) {
        T a = c[k++], da = (T) 0;
#pragma unroll
        for (int j = DEG - i; j > 0; j--) {
            if (GRAD)
                da = j == DEG - i ? a : fma(da, y, a);
            a = fma(a, y, c[k++]);
        }
        if (GRAD) {
            gx = i == DEG - 1 ? g : fma(gx, x, g);
            gy = i == DEG - 1 ? da : fma(gy, x, da);
        }
        g = fma(g, x, a);
    }
}

// accumulators of one class: value, value weighted by n + 1, derivatives to X^2 and Y^2
template<class T> struct FarAcc
{
    T v, w, x, y;
};

// the coefficients of one polynomial, in 16-byte loads
template<int N> __device__ __forceinline__ void far_load(const float* p, float (&c)[N])
{
#pragma unroll
    for (int k = 0; k < N / 4; k++) {
        const float4 v = reinterpret_cast<const float4*>(p)[k];
        c[4 * k] = v.x, c[4 * k + 1] = v.y, c[4 * k + 2] = v.z, c[4 * k + 3] = v.w;
    }
}
template<int N> __device__ __forceinline__ void far_load(const double* p, double (&c)[N])
{
#pragma unroll
    for (int k = 0; k < N / 2; k++) {
        const double2 v = reinterpret_cast<const double2*>(p)[k];
        c[2 * k] = v.x, c[2 * k + 1] = v.y;
    }
}

// one more order of a class at NP points: A = (A h) + the polynomial (TOP: A = the polynomial); the
// coefficients are read once for all points
template<int DEG, bool GRAD, bool TOP, int NP, class T>
__device__ __forceinline__ void far_step(FarAcc<T> (&A)[NP], const T* c, const T (&x)[NP], const T (&y)[NP],
                                         const T (&h)[NP], T n1)
{
    T k[far_pad<T>(far_terms(DEG))];
    far_load(c, k);
#pragma unroll
    for (int p = 0; p < NP; p++) {
        T g, gx, gy;
        far_poly<DEG, GRAD>(k, x[p], y[p], g, gx, gy);
        if (TOP)
            A[p] = FarAcc<T>{g, GRAD ? n1 * g : (T) 0, gx, gy};
        else {
            A[p].v = fma(A[p].v, h[p], g);
            if (GRAD) {
                A[p].w = fma(A[p].w, h[p], n1 * g);
                A[p].x = fma(A[p].x, h[p], gx);
                A[p].y = fma(A[p].y, h[p], gy);
            }
        }
    }
}
template<bool GRAD, int NP> __device__ __forceinline__ void far_up(const FarAcc<float> (&B)[NP], FarAcc<double> (&A)[NP])
{
#pragma unroll
    for (int p = 0; p < NP; p++)
        A[p] = FarAcc<double>{(double) B[p].v, GRAD ? (double) B[p].w : 0., GRAD ? (double) B[p].x : 0.,
                              GRAD ? (double) B[p].y : 0.};
}

// One far pair per unit charge: S with phi = pre S / R (POT) and the field's three coefficients,
// E = pre / R^2 (cd d / R - c1 e1 - c2 e2) (FIELD).
struct FarSum
{
    double ir, S, cd, c1, c2;
};

// elements with two mirror axes. TIER 3: n <= 6, of them n = 6 in FP32 (MIXED: 4, 6). TIER 2: n <= 8,
// n = 6, 8 in FP32. TIER 1: n <= 10, n = 8, 10 in FP32 (MIXED: 6, 8, 10).
template<int TIER, bool FIELD, bool FAST, int NP>
__device__ __forceinline__ void far_sym(const double* f, const double (&X)[NP], const double (&Y)[NP], double s,
                                        FarSum (&F)[NP])
{
    const float* g = reinterpret_cast<const float*>(f + fSymF);
    double x2[NP], y2[NP], h[NP];
    float xf[NP], yf[NP], hf[NP];
#pragma unroll
    for (int p = 0; p < NP; p++) {
        const double t = s * F[p].ir;
        x2[p] = X[p] * X[p], y2[p] = Y[p] * Y[p], h[p] = t * t;
        xf[p] = (float) x2[p], yf[p] = (float) y2[p], hf[p] = (float) h[p];
    }
    FarAcc<float> B[NP];
    if (TIER == 1) {
        far_step<5, FIELD, true>(B, g + kS10, xf, yf, hf, 11.f);
        far_step<4, FIELD, false>(B, g + kS8, xf, yf, hf, 9.f);
        if (FAST)
            far_step<3, FIELD, false>(B, g + kS6, xf, yf, hf, 7.f);
    }
    else {
        if (TIER == 2)
            far_step<4, FIELD, true>(B, g + kS8, xf, yf, hf, 9.f);
        far_step<3, FIELD, TIER == 3>(B, g + kS6, xf, yf, hf, 7.f);
        if (TIER == 3 && FAST)
            far_step<2, FIELD, false>(B, g + kS4, xf, yf, hf, 5.f);
    }
    FarAcc<double> A[NP];
    far_up<FIELD>(B, A);
    if (TIER == 1 && !FAST)
        far_step<3, FIELD, false>(A, f + fSymD6, x2, y2, h, 7.);
    if (TIER != 3 || !FAST)
        far_step<2, FIELD, false>(A, f + fD4, x2, y2, h, 5.);
    far_step<1, FIELD, false>(A, f + fD2, x2, y2, h, 3.);
#pragma unroll
    for (int p = 0; p < NP; p++) {
        F[p].S = fma(A[p].v, h[p], 1.);
        if (FIELD) {
            const double h2 = 2. * h[p];
            F[p].c1 = (h2 * X[p]) * A[p].x;
            F[p].c2 = (h2 * Y[p]) * A[p].y;
            F[p].cd = fma(X[p], F[p].c1, fma(Y[p], F[p].c2, fma(A[p].w, h[p], 1.)));
        }
    }
}

// other elements. n = 2, 3, 4 in FP64, in the FP64 form also n = 5 unless TIER == 3; the rest to
// n = 6, 8, 10 (TIER 3, 2, 1) in FP32. The FP32 tail is put together in FP32 (X Po + Y Qo + t (Pe + XY Qe))
// and joins as four numbers: sixteen conversions of its classes' accumulators cost more than that.
template<int TIER, bool FIELD, bool FAST, int NP>
__device__ __forceinline__ void far_gen(const double* f, const double (&X)[NP], const double (&Y)[NP], double s,
                                        FarSum (&F)[NP])
{
    constexpr bool d5 = TIER != 3 && !FAST;  // n = 5 in FP64
    const float* g = reinterpret_cast<const float*>(f + fGenF);
    double x2[NP], y2[NP], h[NP], t[NP];
    float xf[NP], yf[NP], hf[NP];
    // the tail over t^5, and its gradient's three sums
    float Sf[NP], Wf[NP], Gx[NP], Gy[NP];
#pragma unroll
    for (int p = 0; p < NP; p++) {
        t[p] = s * F[p].ir;
        x2[p] = X[p] * X[p], y2[p] = Y[p] * Y[p], h[p] = t[p] * t[p];
    }
    {
        float Xs[NP], Ys[NP], ts[NP];
#pragma unroll
        for (int p = 0; p < NP; p++) {
            Xs[p] = (float) X[p], Ys[p] = (float) Y[p], ts[p] = (float) t[p];
            xf[p] = Xs[p] * Xs[p], yf[p] = Ys[p] * Ys[p], hf[p] = ts[p] * ts[p];
        }
        FarAcc<float> po[NP], qo[NP], pe[NP], qe[NP];
        if (TIER == 1) {
            far_step<4, FIELD, true>(po, g + kG9p, xf, yf, hf, 10.f);
            far_step<4, FIELD, true>(qo, g + kG9q, xf, yf, hf, 10.f);
        }
        if (TIER <= 2) {
            far_step<3, FIELD, TIER == 2>(po, g + kG7p, xf, yf, hf, 8.f);
            far_step<3, FIELD, TIER == 2>(qo, g + kG7q, xf, yf, hf, 8.f);
        }
        if (!d5) {
            far_step<2, FIELD, TIER == 3>(po, g + kG5p, xf, yf, hf, 6.f);
            far_step<2, FIELD, TIER == 3>(qo, g + kG5q, xf, yf, hf, 6.f);
        }
        // odd part: n = 5 first (n = 7 first where 5 is in FP64: one more h)
#pragma unroll
        for (int p = 0; p < NP; p++) {
            const float u = d5 ? hf[p] : 1.f;
            Sf[p] = u * fmaf(Xs[p], po[p].v, Ys[p] * qo[p].v);
            if (FIELD) {
                const float xy2 = 2.f * Xs[p] * Ys[p];
                Wf[p] = u * fmaf(Xs[p], po[p].w, Ys[p] * qo[p].w);
                Gx[p] = u * fmaf(xy2, qo[p].x, fmaf(2.f * xf[p], po[p].x, po[p].v));
                Gy[p] = u * fmaf(xy2, po[p].y, fmaf(2.f * yf[p], qo[p].y, qo[p].v));
            }
        }
        if (TIER == 1) {
            far_step<5, FIELD, true>(pe, g + kG10p, xf, yf, hf, 11.f);
            far_step<4, FIELD, true>(qe, g + kG10q, xf, yf, hf, 11.f);
        }
        if (TIER <= 2) {
            far_step<4, FIELD, TIER == 2>(pe, g + kG8p, xf, yf, hf, 9.f);
            far_step<3, FIELD, TIER == 2>(qe, g + kG8q, xf, yf, hf, 9.f);
        }
        far_step<3, FIELD, TIER == 3>(pe, g + kG6p, xf, yf, hf, 7.f);
        far_step<2, FIELD, TIER == 3>(qe, g + kG6q, xf, yf, hf, 7.f);
#pragma unroll
        for (int p = 0; p < NP; p++) {
            const float xy = Xs[p] * Ys[p];
            Sf[p] = fmaf(ts[p], fmaf(xy, qe[p].v, pe[p].v), Sf[p]);
            if (FIELD) {
                Wf[p] = fmaf(ts[p], fmaf(xy, qe[p].w, pe[p].w), Wf[p]);
                Gx[p] = fmaf(ts[p], fmaf(2.f * Xs[p], pe[p].x, Ys[p] * fmaf(2.f * xf[p], qe[p].x, qe[p].v)), Gx[p]);
                Gy[p] = fmaf(ts[p], fmaf(2.f * Ys[p], pe[p].y, Xs[p] * fmaf(2.f * yf[p], qe[p].y, qe[p].v)), Gy[p]);
            }
        }
    }
    // FP64: X Po + Y Qo of n = 3 (and 5), Pe + XY Qe of n = 2, 4
    FarAcc<double> A[NP], C[NP];
    if (d5) {
        far_step<2, FIELD, true>(A, f + fGenD5, x2, y2, h, 6.);
        far_step<2, FIELD, true>(C, f + fGenD5 + 6, x2, y2, h, 6.);
    }
    double So[NP], Wo[NP], ox[NP], oy[NP];
    {
        double k3[6];
        far_load(f + fGenD3, k3);
#pragma unroll
        for (int p = 0; p < NP; p++) {
            double v, vx, vy;
            auto add = [&](FarAcc<double>& Q, const double* c) {
                far_poly<1, FIELD>(c, x2[p], y2[p], v, vx, vy);
                if (d5) {
                    Q.v = fma(Q.v, h[p], v);
                    if (FIELD) {
                        Q.w = fma(Q.w, h[p], 4. * v);
                        Q.x = fma(Q.x, h[p], vx);
                        Q.y = fma(Q.y, h[p], vy);
                    }
                }
                else
                    Q = FarAcc<double>{v, 4. * v, vx, vy};
            };
            add(A[p], k3);
            add(C[p], k3 + 3);
            So[p] = fma(X[p], A[p].v, Y[p] * C[p].v);
            if (FIELD) {
                const double XY2 = 2. * X[p] * Y[p];
                Wo[p] = fma(X[p], A[p].w, Y[p] * C[p].w);
                ox[p] = fma(XY2, C[p].x, fma(2. * x2[p], A[p].x, A[p].v));
                oy[p] = fma(XY2, A[p].y, fma(2. * y2[p], C[p].y, C[p].v));
            }
        }
    }
    far_step<2, FIELD, true>(A, f + fD4, x2, y2, h, 5.);
    far_step<1, FIELD, true>(C, f + fGenQ4, x2, y2, h, 5.);
    double k2[4];
    far_load(f + fD2, k2);
#pragma unroll
    for (int p = 0; p < NP; p++) {
        double v, vx, vy;
        far_poly<1, FIELD>(k2, x2[p], y2[p], v, vx, vy);
        const double q = fma(C[p].v, h[p], k2[3]);  // Qe of n = 2: a constant
        // t^2 (even + t (odd + t^2 tail)): the tail starts at t^5
        const double XY = X[p] * Y[p], th = t[p] * h[p];
        const double h1 = h[p];
        F[p].S = fma(fma(t[p], fma(h1, (double) Sf[p], So[p]), fma(XY, q, fma(A[p].v, h1, v))), h1, 1.);
        if (FIELD) {
            const double qw = fma(C[p].w, h1, 3. * k2[3]), qx = C[p].x * h1, qy = C[p].y * h1;
            const double pw = fma(A[p].w, h1, 3. * v), px = fma(A[p].x, h1, vx), py = fma(A[p].y, h1, vy);
            const double W = fma(t[p], fma(h1, (double) Wf[p], Wo[p]), fma(XY, qw, pw));
            // d/dX: 2X Pe_x + Y (Qe + 2 x2 Qe_x) + t (Po + 2 x2 Po_x + 2 XY Qo_x), d/dY alike
            const double ex = fma(2. * X[p], px, Y[p] * fma(2. * x2[p], qx, q));
            const double ey = fma(2. * Y[p], py, X[p] * fma(2. * y2[p], qy, q));
            F[p].c1 = fma(th, fma(h1, (double) Gx[p], ox[p]), h1 * ex);
            F[p].c2 = fma(th, fma(h1, (double) Gy[p], oy[p]), h1 * ey);
            F[p].cd = fma(X[p], F[p].c1, fma(Y[p], F[p].c2, fma(W, h1, 1.)));
        }
    }
}

// the pairs of far record f with NP points; FAST: the MIXED form's orders. f is 16-byte aligned. The reciprocal
// distance is FP64's in both forms: one Newton step's error, which 7 to 33 nodes average, would go into every
// pair whole (single pairs' field 5.2e-13 instead of 3.2e-13 in the mean, 3.1e-12 instead of 1.4e-12 at most).
template<bool GENERAL, int TIER, bool FIELD, bool FAST, int NP>
__device__ __forceinline__ void far_pairs(const double* f, const V3 (&P)[NP], V3 (&d)[NP], FarSum (&F)[NP])
{
    double hd[10];
    far_load(f, hd);
    const V3 e1 = v3(hd[fE1], hd[fE1 + 1], hd[fE1 + 2]), e2 = v3(hd[fE1 + 3], hd[fE1 + 4], hd[fE1 + 5]);
    double X[NP], Y[NP];
#pragma unroll
    for (int p = 0; p < NP; p++) {
        d[p] = v3(P[p].x - hd[fCen], P[p].y - hd[fCen + 1], P[p].z - hd[fCen + 2]);
        F[p].ir = kPotScale<false> * irsq<false>(dot(d[p], d[p]));
        X[p] = F[p].ir * dot(d[p], e1);
        Y[p] = F[p].ir * dot(d[p], e2);
    }
    if (GENERAL)
        far_gen<TIER, FIELD, FAST>(f, X, Y, hd[fSize], F);
    else
        far_sym<TIER, FIELD, FAST>(f, X, Y, hd[fSize], F);
}

// ------------------------------------------------------------------------- tiers of a warp
// The tier of one element (far record f) for all points within `wr` of `wc`: the largest of 3, 2, 1
// whose cut every point's centre distance exceeds (with a 1e-9 margin for the rounding of either
// side), or 0: some point may need the cubature or the analytic integrals.
// F32, whose cubature nodes are good to 1e-7: the farther two tiers from half of MIXED's cuts on, where the orders
// left out grow by at most 2^10 from 1e-14 and the FP32 ones round to below 1e-10 (the nearest tier costs more
// than FP32 nodes: 4,000 scattered points and 28,800 slivers 6.3 ms with it, 5.6 without). 20,000 points and the
// slivers, ms: 14.8 without the series, 20.7 with MIXED's cuts, 12.7 with half of them; their product 17.6, 16.4, 11.3.
template<bool F32> constexpr double kFarCut = F32 ? 0.5 : 1.;
template<bool FAST, bool F32> __device__ __forceinline__ int far_tier(const double* f, V3 wc, double wr)
{
    const double dx = f[fCen] - wc.x, dy = f[fCen + 1] - wc.y, dz = f[fCen + 2] - wc.z;
    const double d2 = (dx * dx + dy * dy + dz * dz) * (1. - 1e-9);
    const double* c = f + (FAST ? fCutM : fCut);
    constexpr double h = kFarCut<F32>;
    const double r3 = h * c[0] + wr, r2 = h * c[1] + wr, r1 = h * c[2] + wr;
    return d2 > r3 * r3 ? 3 : d2 > r2 * r2 ? 2 : !F32 && d2 > r1 * r1 ? 1 : 0;
}
// one point: the series holds (tier 1; F32: tier 2)
template<bool FAST, bool F32> __device__ __forceinline__ bool far_point(const double* f, V3 P)
{
    const double dx = P.x - f[fCen], dy = P.y - f[fCen + 1], dz = P.z - f[fCen + 2];
    const double r1 = kFarCut<F32> * f[(FAST ? fCutM : fCut) + (F32 ? 1 : 2)];
    return (dx * dx + dy * dy + dz * dz) * (1. - 1e-9) > r1 * r1;
}

}  // namespace kemcu
