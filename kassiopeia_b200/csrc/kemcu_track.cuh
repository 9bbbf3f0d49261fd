// K4: persistent batched RK8 tracker for charged particles in the electrostatic field of the
// charged elements (exact trajectory, B = 0).
//
// Reference path: KSRoot -> KSTrajTrajectoryExact::CalculateTrajectory -> KSMathRK8::Integrate
// (Kassiopeia/Math/Include/KSMathRK8.h:45-137, Butcher table :139-226) with the derivative of
// KSTrajTrajectoryExact::Differentiate + KSTrajTermPropagation::Differentiate
// (Kassiopeia/Trajectories/Source/KSTrajTrajectoryExact.cxx:302-316, KSTrajTermPropagation.cxx:25-35):
//   d/dt (t, s, x, p) = (1, |v|, v, q E(x)),  v = p / (m gamma),  gamma = sqrt(1 + p^2 / (m c)^2)
// with E(x) the Kahan-summed direct sum of KIntegratingFieldSolver::ElectricField.
//
// Layout: a CTA owns 32 slots, one per lane, and W warps that share the elements: part c of kTrackParts
// is elements c, c + kTrackParts, ..., warp w sums parts w, w + W, ... one after another for all 32
// slots, and warp 0 adds the parts' sums in order and advances the slots. The parts do not depend on W,
// which follows the number of tracks. The element records come a warp at a time through its own piece of shared memory, the next
// one's loads in flight during the pairs of this one, so a stage has no CTA barrier but the two around
// it. (One thread per track left 4 warps on an SM at 16,384 tracks, waiting for FP64 latencies.) Slots
// take tracks in Morton order of their positions, so that a warp's lanes agree on an element's form;
// each lane takes the form its own distance asks for, whoever its neighbours are, so a track does not
// depend on the others. The 13 stage derivatives of each slot live in shared memory. A slot whose
// track ends (electrode hit, leaving the volume, step limit, non-finite state) or has taken `budget`
// steps in this launch writes it back and takes the next track of the list from a global work counter,
// so tracks of very different lengths keep every slot busy and one launch advances every listed track
// by at most `budget` steps; unfinished tracks stay active for the next launch.
#pragma once

#include "kemcu_kernels.cuh"

namespace kemcu
{

constexpr int kTrackSlots = 32;  // per CTA: a lane each
constexpr int kTrackParts = 16;  // sums over the elements, the most warps of a CTA
constexpr int kStages = 13;
constexpr int kTrackK = 6;     // stored per stage and slot: v (3), q E (3)

// Butcher coefficients a[s][k] (row s gives stage value s from derivatives 0..s; row 12 is
// the final combination), the 13-stage eighth-order scheme of KSMathRK8.h:139-226
__constant__ double c_rk8[kStages][kStages];

inline void rk8_table(double a[kStages][kStages])
{
    for (int i = 0; i < kStages; i++)
        for (int j = 0; j < kStages; j++)
            a[i][j] = 0.;
    a[0][0] = 1. / 4.;
    a[1][0] = 5. / 72.; a[1][1] = 1. / 72.;
    a[2][0] = 1. / 32.; a[2][2] = 3. / 32.;
    a[3][0] = 106. / 125.; a[3][2] = -408. / 125.; a[3][3] = 352. / 125.;
    a[4][0] = 1. / 48.; a[4][3] = 8. / 33.; a[4][4] = 125. / 528.;
    a[5][0] = -1263. / 2401.; a[5][3] = 39936. / 26411.; a[5][4] = -64125. / 26411.; a[5][5] = 5520. / 2401.;
    a[6][0] = 37. / 392.; a[6][4] = 1625. / 9408.; a[6][5] = -2. / 15.; a[6][6] = 61. / 6720.;
    a[7][0] = 17176. / 25515.; a[7][3] = -47104. / 25515.; a[7][4] = 1325. / 504.; a[7][5] = -41792. / 25515.;
    a[7][6] = 20237. / 145800.; a[7][7] = 4312. / 6075.;
    a[8][0] = -23834. / 180075.; a[8][3] = -77824. / 1980825.; a[8][4] = -636635. / 633864.;
    a[8][5] = 254048. / 300125.; a[8][6] = -183. / 7000.; a[8][7] = 8. / 11.; a[8][8] = -324. / 3773.;
    a[9][0] = 12733. / 7600.; a[9][3] = -20032. / 5225.; a[9][4] = 456485. / 80256.; a[9][5] = -42599. / 7125.;
    a[9][6] = 339227. / 912000.; a[9][7] = -1029. / 4180.; a[9][8] = 1701. / 1408.; a[9][9] = 5145. / 2432.;
    a[10][0] = -27061. / 204120.; a[10][3] = 40448. / 280665.; a[10][4] = -1353775. / 1197504.;
    a[10][5] = 17662. / 25515.; a[10][6] = -71687. / 1166400.; a[10][7] = 98. / 225.; a[10][8] = 1. / 16.;
    a[10][9] = 3773. / 11664.;
    a[11][0] = 11203. / 8680.; a[11][3] = -38144. / 11935.; a[11][4] = 2354425. / 458304.;
    a[11][5] = -84046. / 16275.; a[11][6] = 673309. / 1636800.; a[11][7] = 4704. / 8525.; a[11][8] = 9477. / 10912.;
    a[11][9] = -1029. / 992.; a[11][11] = 729. / 341.;
    a[12][0] = 31. / 720.; a[12][5] = 16. / 75.; a[12][6] = 16807. / 79200.; a[12][7] = 16807. / 79200.;
    a[12][8] = 243. / 1760.; a[12][11] = 243. / 1760.; a[12][12] = 31. / 720.;
}

struct TrackParams
{
    double dt, charge, mass, c2;  // c2 = (speed of light)^2
    double hit_r2, max_r2;        // squared radii (0 disables)
    int max_steps, budget;
    int n_list;                   // number of track indices in list
    unsigned live;                // bit s: stage s's derivative has a nonzero weight somewhere
};

// Stages whose derivative no later stage and not the final combination uses (zero column of the
// Butcher table; stage 10 of this scheme: a[10][10] = a[11][10] = a[12][10] = 0). Their field
// sums cannot change the result, so the tracker does not evaluate them.
inline unsigned rk8_live_stages(const double a[kStages][kStages])
{
    unsigned live = 0u;
    for (int k = 0; k < kStages; k++)
        for (int r = k; r < kStages; r++)
            if (a[r][k] != 0.)
                live |= 1u << k;
    return live;
}

// the field of one element at X per unit charge density, by the form the lane's distance asks for: the
// series wherever one holds, in its nearest tier (the farther ones are cheaper, but the lanes of a warp
// lie on both sides of their cuts and would run both), else the cubature bands or the analytic integrals. f: far record, e: element record, w: near record.
template<bool MIXED> __device__ __forceinline__ V3 track_pair(const double* f, bool general, const double* e,
                                                              const double* __restrict__ w, double pre, V3 X)
{
    const double* c = f + (MIXED ? fCutM : fCut);
    const V3 d0 = v3(X.x - f[fCen], X.y - f[fCen + 1], X.z - f[fCen + 2]);
    const double d2 = dot(d0, d0) * (1. - 1e-9);
    if (d2 > c[2] * c[2]) {
        const V3 P[1] = {X};
        V3 d[1];
        FarSum F[1];
        if (general)
            far_pairs<true, 1, true, MIXED>(f, P, d, F);
        else
            far_pairs<false, 1, true, MIXED>(f, P, d, F);
        const double k = pre * F[0].ir * F[0].ir, a = (k * F[0].ir) * F[0].cd, b = -k * F[0].c1, q = -k * F[0].c2;
        const V3 e1 = ld3(f + fE1), e2 = ld3(f + fE1 + 3);
        return v3(fma(a, d[0].x, fma(b, e1.x, q * e2.x)), fma(a, d[0].y, fma(b, e1.y, q * e2.y)),
                  fma(a, d[0].z, fma(b, e1.z, q * e2.z)));
    }
    const Out4 r = epi<MIXED, false, true>(e, w, X);
    return v3(r.ex, r.ey, r.ez);
}

// the elements as the tracker takes them
struct TrackElems
{
    FarView V;
    const double* rec;
    const int2* where;  // per element: its far record (far_where)
    const double* sigma;
    int n;
};

// state: n x 8; steps, status: n; list: n_list track indices to work on; next: work counter;
// done_steps: total steps taken (for statistics); dpsum (n, may be null): per track the sum over
// its steps of |p_after - p_before|, accumulated.
template<bool MIXED, int W>
__global__ void __launch_bounds__(32 * W, 16 / W) rk8_tracker_kernel(TrackElems el, double* __restrict__ state,
                                                                     int* __restrict__ steps, int* __restrict__ status,
                                                                     const int* __restrict__ list,
                                                                     unsigned* __restrict__ next,
                                                                     unsigned long long* __restrict__ done_steps,
                                                                     double* __restrict__ dpsum, TrackParams prm)
{
    __shared__ double s_k[kStages][kTrackK][kTrackSlots];
    __shared__ double s_x[3][kTrackSlots];
    __shared__ __align__(16) double s_far[W][kFarGenStride], s_rec[W][rRecSize];
    // the parts' sums (a warp with one part leaves them where its records were)
    static_assert(W <= kTrackParts && kTrackParts % W == 0 && kFarGenStride >= 3 * kTrackSlots, "parts of the sum");
    __shared__ double s_part[W < kTrackParts ? kTrackParts : 1][3 * kTrackSlots];
    auto part = [&](int c) { return W < kTrackParts ? s_part[c] : s_far[c]; };
    __shared__ int s_any;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int track = -1, tsteps = 0;
    double y[8];
    double dps = 0.;
    int nstep = 0;
    auto pull = [&]() {
        track = -1;
        tsteps = 0;
        const unsigned w = atomicAdd(next, 1u);
        if (w < (unsigned) prm.n_list) {
            track = list[w];
            for (int c = 0; c < 8; c++)
                y[c] = state[(size_t) track * 8 + c];
            nstep = steps[track];
            dps = dpsum ? dpsum[track] : 0.;
        }
    };
    // this warp's share of the field at the 32 slot positions
    auto field = [&]() {
        const V3 X = v3(s_x[0][lane], s_x[1][lane], s_x[2][lane]);
        constexpr int NV = (kFarGenStride + 31) / 32;
        double v[NV], r = 0., pre_next = 0., sg_next = 0.;
        int2 at = make_int2(0, 0);
        auto fetch = [&](int j) {
            at = el.where[j];
            const double* f = el.V.far + far_offset(at);
            const int len = at.y & 1 ? kFarGenStride : kFarSymStride;
#pragma unroll
            for (int k = 0; k < NV; k++)
                if (lane + 32 * k < len)
                    v[k] = __ldg(f + lane + 32 * k);
            r = __ldg(el.rec + (size_t) j * rRecSize + lane);
            pre_next = __ldg(el.V.pre + j);
            sg_next = __ldg(el.sigma + j);
        };
        if (warp < el.n)
            fetch(warp);
#pragma unroll 1
        for (int c = warp; c < kTrackParts; c += W) {
            Kahan ex, ey, ez;
#pragma unroll 1
            for (int j = c; j < el.n; j += kTrackParts) {
                __syncwarp();
                const bool general = at.y & 1;
                const int len = general ? kFarGenStride : kFarSymStride;
#pragma unroll
                for (int k = 0; k < NV; k++)
                    if (lane + 32 * k < len)
                        s_far[warp][lane + 32 * k] = v[k];
                s_rec[warp][lane] = r;
                __syncwarp();
                const double pre = pre_next, sg = sg_next;
                const int next = j + kTrackParts < el.n ? j + kTrackParts : c + W < kTrackParts ? c + W : el.n;
                if (next < el.n)
                    fetch(next);
                const V3 E = track_pair<MIXED>(s_far[warp], general, s_rec[warp], el.V.rwg + (size_t) j * wRecSize, pre, X);
                ex.add(E.x * sg);
                ey.add(E.y * sg);
                ez.add(E.z * sg);
            }
            __syncwarp();
            part(c)[lane] = ex.s;
            part(c)[kTrackSlots + lane] = ey.s;
            part(c)[2 * kTrackSlots + lane] = ez.s;
        }
    };
    if (warp == 0)
        pull();
    unsigned long long my_steps = 0;
    // every iteration is one RK8 step of all busy slots; ends when the list is exhausted
    while (true) {
        if (warp == 0) {
            const bool any = __any_sync(0xffffffffu, track >= 0);
            // slots without a track sit where some busy slot is: they take its elements' forms
            const unsigned busy = __ballot_sync(0xffffffffu, track >= 0);
            if (any) {
                const int src = track >= 0 ? lane : __ffs(busy) - 1;
                for (int c = 0; c < 8; c++) {
                    const double q = __shfl_sync(0xffffffffu, y[c], src);
                    if (track < 0)
                        y[c] = q;
                }
            }
            if (lane == 0)
                s_any = any;
        }
        __syncthreads();
        if (!s_any)
            break;
        double ds = 0.;  // sum over stages of a[12][k] |v_k|
        for (int st = 0; st < kStages; st++) {
            if (!((prm.live >> st) & 1u))
                continue;  // unused derivative (its column of the table is zero): not evaluated
            V3 Pm = v3(0., 0., 0.);
            if (warp == 0) {
                // stage position and momentum: value_{st-1} = y0 + dt sum_k a[st-1][k] k_k
                V3 X = v3(y[2], y[3], y[4]);
                Pm = v3(y[5], y[6], y[7]);
                if (st > 0) {
                    double sx = 0., sy = 0., sz = 0., px = 0., py = 0., pz = 0.;
                    for (int k = 0; k < st; k++) {
                        if (!((prm.live >> k) & 1u))
                            continue;
                        const double a = c_rk8[st - 1][k];
                        sx += a * s_k[k][0][lane];
                        sy += a * s_k[k][1][lane];
                        sz += a * s_k[k][2][lane];
                        px += a * s_k[k][3][lane];
                        py += a * s_k[k][4][lane];
                        pz += a * s_k[k][5][lane];
                    }
                    X = v3(y[2] + prm.dt * sx, y[3] + prm.dt * sy, y[4] + prm.dt * sz);
                    Pm = v3(y[5] + prm.dt * px, y[6] + prm.dt * py, y[7] + prm.dt * pz);
                }
                s_x[0][lane] = X.x;
                s_x[1][lane] = X.y;
                s_x[2][lane] = X.z;
            }
            __syncthreads();
            field();
            __syncthreads();
            if (warp == 0) {
                Kahan ex, ey, ez;
                for (int c = 0; c < kTrackParts; c++) {
                    ex.add(part(c)[lane]);
                    ey.add(part(c)[kTrackSlots + lane]);
                    ez.add(part(c)[2 * kTrackSlots + lane]);
                }
                const double p2 = dot(Pm, Pm);
                const double gam = sqrt(1. + p2 / (prm.mass * prm.mass * prm.c2));
                const double inv = 1. / (prm.mass * gam);
                const double vx = inv * Pm.x, vy = inv * Pm.y, vz = inv * Pm.z;
                s_k[st][0][lane] = vx;
                s_k[st][1][lane] = vy;
                s_k[st][2][lane] = vz;
                s_k[st][3][lane] = prm.charge * ex.s;
                s_k[st][4][lane] = prm.charge * ey.s;
                s_k[st][5][lane] = prm.charge * ez.s;
                ds += c_rk8[kStages - 1][st] * sqrt(vx * vx + vy * vy + vz * vz);
            }
        }
        if (warp == 0 && track >= 0) {
            // final combination (row 12) for t (derivative 1), s (|v|), x and p
            double dtt = 0., d[6] = {0., 0., 0., 0., 0., 0.};
            for (int k = 0; k < kStages; k++) {
                const double a = c_rk8[kStages - 1][k];
                dtt += a;
                if (!((prm.live >> k) & 1u))
                    continue;
                for (int c = 0; c < 6; c++)
                    d[c] += a * s_k[k][c][lane];
            }
            y[0] += prm.dt * dtt;
            y[1] += prm.dt * ds;
            double dp2 = 0.;
            for (int c = 0; c < 6; c++) {
                const double before = y[2 + c];
                y[2 + c] += prm.dt * d[c];
                if (c >= 3)
                    dp2 += (y[2 + c] - before) * (y[2 + c] - before);
            }
            dps += sqrt(dp2);  // KSStep::ContinuousMomentumChange (KSRootTrajectory.cxx:217-218)
            nstep++;
            my_steps++;
            const double r2 = y[2] * y[2] + y[3] * y[3] + y[4] * y[4];
            int stat = 0;
            bool finite = true;
            for (int c = 0; c < 8; c++)
                finite = finite && isfinite(y[c]);
            if (!finite)
                stat = 4;
            else if (prm.hit_r2 > 0. && r2 <= prm.hit_r2)
                stat = 1;
            else if (prm.max_r2 > 0. && r2 >= prm.max_r2)
                stat = 3;
            else if (nstep >= prm.max_steps)
                stat = 2;
            tsteps++;
            if (stat != 0 || tsteps >= prm.budget) {
                for (int c = 0; c < 8; c++)
                    state[(size_t) track * 8 + c] = y[c];
                steps[track] = nstep;
                if (dpsum)
                    dpsum[track] = dps;
                if (stat != 0)
                    status[track] = stat;
                pull();
            }
        }
        __syncthreads();  // s_any is read before warp 0 writes it again
    }
    if (warp == 0)
        atomicAdd(done_steps, my_steps);
}

// positions of the listed tracks (for their Morton order), and the list in that order
__global__ void track_points_kernel(const double* __restrict__ state, const int* __restrict__ list, int n,
                                    double* __restrict__ P)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        for (int c = 0; c < 3; c++)
            P[3 * i + c] = state[(size_t) list[i] * 8 + 2 + c];
}
__global__ void track_permute_kernel(const int* __restrict__ list, const int* __restrict__ perm, int n,
                                     int* __restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        out[i] = list[perm[i]];
}

// list of ACTIVE tracks: list[atomicAdd(count)] = i for status[i] == 0
__global__ void active_list_kernel(const int* __restrict__ status, int n, int* __restrict__ list, unsigned* __restrict__ count)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && status[i] == 0)
        list[atomicAdd(count, 1u)] = i;
}

}  // namespace kemcu
