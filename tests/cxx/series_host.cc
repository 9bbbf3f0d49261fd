// The far-field series of kemcu_series.cuh as plain C++, for tests/test_cpu_series.py: what the
// header takes from the device code is restated here, and its build kernel runs as a loop.
#include <cmath>
#include <cstddef>
using std::fabs;
using std::fmax;
using std::isfinite;
#define __device__
#define __host__
#define __global__ static
#define __forceinline__ inline
#define __noinline__
#define __grid_constant__
#define CUDART_INF INFINITY
namespace kemcu
{
enum Shape : int { kTriangle = 0, kRectangle = 1, kLineSegment = 2 };
enum Rec : int { rA = 0, rEa = 11, rEb = 14, rCen = 17, rPrefac = 24, rType = 25, rCut = 29, rRecSize = 32 };
struct V3 { double x, y, z; };
inline V3 v3(double x, double y, double z) { return V3{x, y, z}; }
inline V3 operator-(V3 a, V3 b) { return v3(a.x - b.x, a.y - b.y, a.z - b.z); }
inline V3 operator*(double s, V3 a) { return v3(s * a.x, s * a.y, s * a.z); }
inline double dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
inline double norm(V3 a) { return std::sqrt(dot(a, a)); }
inline V3 ld3(const double* p) { return v3(p[0], p[1], p[2]); }
template<bool FAST> double irsq(double x) { return 2. / std::sqrt(x); }
template<bool FAST> constexpr double kPotScale = 0.5;
struct float4 { float x, y, z, w; };
struct double2 { double x, y; };
struct int2 { int x, y; };
inline int2 make_int2(int x, int y) { return int2{x, y}; }
struct Dim { int x; };
static Dim blockIdx, blockDim{1}, threadIdx;
}  // namespace kemcu
using std::fma;
using std::fmaf;
using std::pow;
using std::sqrt;
using std::cos;
using std::sin;
#include "../../kassiopeia_b200/csrc/kemcu_series.cuh"
using namespace kemcu;

template<bool GENERAL, int TIER, bool FAST> static void eval(const double* f, double pre, const double* P, double* out)
{
    const V3 p[2] = {ld3(P), ld3(P + 3)};
    V3 d[2];
    const V3 e1 = ld3(f + fE1), e2 = ld3(f + fE1 + 3);
    FarSum F[2], G[2];
    far_pairs<GENERAL, TIER, true, FAST>(f, p, d, F);
    far_pairs<GENERAL, TIER, false, FAST>(f, p, d, G);
    for (int i = 0; i < 2; i++, out += 4) {
        const double k = pre * F[i].ir * F[i].ir, a = k * F[i].ir * F[i].cd;
        out[0] = a * d[i].x - k * F[i].c1 * e1.x - k * F[i].c2 * e2.x;
        out[1] = a * d[i].y - k * F[i].c1 * e1.y - k * F[i].c2 * e2.y;
        out[2] = a * d[i].z - k * F[i].c1 * e1.z - k * F[i].c2 * e2.z;
        out[3] = pre * G[i].ir * G[i].S;
    }
}

// one element record (32 doubles), n points at which the series of `tier` is evaluated; cuts: the
// squared distances of the record (tiers 3, 2, 1)
extern "C" void series_host(const double* rec, int general, int mixed, int tier, const double* gx, const double* gw, int n,
                            const double* P, double* out, double* cuts)
{
    alignas(16) double far[kFarGenStride];
    double pre;
    FarTile T{0, 1, general, 0};
    FarTables gl;
    far_tables(gl);
    for (int i = 0; i < kFarQ; i++)
        gl.x[i] = gx[i], gl.w[i] = gw[i];
    int2 where;
    far_build_kernel(rec, &T, 1, gl, far, &pre, &where);
    for (int k = 0; k < 3; k++)
        cuts[k] = far[(mixed ? fCutM : fCut) + k];
    for (int i = 0; i < n; i += 2) {  // pairs of points, n even
        const double* p = P + 3 * i;
        double* o = out + 4 * i;
        using Fn = void (*)(const double*, double, const double*, double*);
        const Fn fn[2][2][3] = {{{eval<false, 1, false>, eval<false, 2, false>, eval<false, 3, false>},
                                 {eval<false, 1, true>, eval<false, 2, true>, eval<false, 3, true>}},
                                {{eval<true, 1, false>, eval<true, 2, false>, eval<true, 3, false>},
                                 {eval<true, 1, true>, eval<true, 2, true>, eval<true, 3, true>}}};
        fn[general][mixed][tier - 1](far, pre, p, o);
    }
}
