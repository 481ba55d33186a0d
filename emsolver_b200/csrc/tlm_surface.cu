// tlm_surface.cu -- surface monitors of the TLM step and the far field.
//
// The reference's monitors beyond ports, probes and energy
// (TlmSolver::monitors, TlmSolver.cpp:616-675 and 715-763):
//   * PEC-surface currents: for every face between a PEC cell and a non-PEC
//     neighbour (Geometry.cpp:402-436), the circulations ZI of the two
//     tangential axes at the neighbour (|Js| = sqrt(h1^2 + h2^2) each step,
//     and a running DFT at f0 from settle_steps on);
//   * Huygens-box phasors: on the air cells of a box inset huy_offset cells
//     (TlmSolver.cpp:310-348), running DFTs of -V_t and -ZI_t of the two
//     tangential axes, input of the near-to-far-field transform;
//   * the |E| cut plane (every second step) and playback frames.
// Each runs on the incident pulses after injection of step n. Those are not
// stored (the state between steps is the reflected pulses), so the monitor
// kernel recomputes them for the cells it needs from the same input buffer
// the step kernel of step n reads: the gather of connect, then the soft
// sources of the cell in the reference's order. Every accumulator belongs to
// one thread and is updated in step order in the storage's real type, so
// FP32 results are bitwise the reference's.
//
// The far field (ComputeFarFieldFromHuygens, TlmSolver.cpp:805-916) is summed on
// the device in FP64, a few directions per block.
#include "tlm_b200.h"
#include "tlm_internal.h"

#include "tlm_host_math.h"
#include "tlm_step_kernel.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

using namespace tlmi;

namespace tlmk {

constexpr int kSurfaceThreads = 128;

template <class S> struct SurfaceArgs
{
    using R = typename Traits<S>::R;
    const S *in;            // state before step n (reflected pulses, or incident if `incident`)
    int incident;
    const uint8_t *mat;
    long long P;
    int nx, ny, nz, px;
    R rho, scale;
    const SpecEntry *spec;  // node-sorted sources and samples
    int nspec;
    long long injLo, injHi; // first and last node with a source (injLo > injHi: none)
    R sv;                   // source value of step n
    // PEC-surface faces
    const long long *jsNode;  // face code: padded node * 8 + axis * 2 + (normal sign < 0)
    int njs;
    R *jsInst;              // |Js| per face
    R *jsAcc;               // per face: Re1 Im1 Re2 Im2
    // Huygens faces
    const long long *huyNode;
    int nhuy;
    R *huyAcc;              // per face: E1 re/im, E2 re/im, eta0 H1 re/im, eta0 H2 re/im
    int doDft;
    R cph, sph;
    // cut plane
    int planeAxis, planeIndex, planeN1, planeN2;
    R *plane;
};

// The 12 incident pulses of node `node` (cell i, j, k) at step n: the gather
// of connect (TlmSolver.cpp:551-613) from the reflected pulses of step n-1,
// then the soft sources of the node (TlmSolver.cpp:487-505).
template <class S>
__device__ void incidentAt(const SurfaceArgs<S> &a, long long node, int i, int j, int k,
                           typename Traits<S>::R (&inc)[12])
{
    using R = typename Traits<S>::R;
    const long long stride[3] = { 1, a.px, (long long)a.px * a.ny };
    const int co[3] = { i, j, k };
    const int dims[3] = { a.nx, a.ny, a.nz };
    // loads first, all independent: the pulse that arrives on each slot (the
    // node's own one from an outer wall) and the neighbours' materials
    uint8_t mat[6];
#pragma unroll
    for (int s = 0; s < 12; ++s)
    {
        const int ax = s >> 2, side = (s >> 1) & 1;
        const int q = co[ax] + (side ? 1 : -1);
        const bool in = !a.incident && q >= 0 && q < dims[ax];
        const long long nb = in ? node + (side ? stride[ax] : -stride[ax]) : node;
        inc[s] = loadOne<S>(a.in, (in ? s ^ 2 : s) * a.P + nb, a.scale);
        if (!(s & 1)) mat[s >> 1] = in ? a.mat[nb] : 0;
    }
    if (!a.incident)
    {
#pragma unroll
        for (int s = 0; s < 12; ++s)
        {
            const int ax = s >> 2, side = (s >> 1) & 1;
            const int q = co[ax] + (side ? 1 : -1);
            if (q < 0 || q >= dims[ax])
                inc[s] = a.rho * inc[s];
            else if (mat[s >> 1] == kPec)
                inc[s] = -loadOne<S>(a.in, s * a.P + node, a.scale);
        }
    }
    if (node < a.injLo || node > a.injHi) return;
    // soft sources of this node, in the order the step kernel applies them
    int lo = 0, hi = a.nspec;
    while (lo < hi)
    {
        const int mid = (lo + hi) >> 1;
        if (a.spec[mid].node < node) lo = mid + 1; else hi = mid;
    }
    for (int e = lo; e < a.nspec && a.spec[e].node == node; ++e)
    {
        const SpecEntry se = a.spec[e];
        if (se.kind != kInject) continue;
        const R qv = (R(0.5) * R(se.amp)) * a.sv;
#pragma unroll
        for (int s = 0; s < 12; ++s)
            if ((s >> 2) != se.arg && fieldOfSlot(s) == se.arg) inc[s] = inc[s] + qv;
    }
}

// (32-bit divisions for nodes below 2^32, as on every grid that fits 180 GB)
__device__ __forceinline__ void cellOfNode(long long node, int px, int ny, int *i, int *j, int *k)
{
    if (node >> 32)
    {
        const long long r = node / px;
        *i = (int)(node - r * px);
        *j = (int)(r % ny);
        *k = (int)(r / ny);
        return;
    }
    const unsigned n = (unsigned)node, r = n / (unsigned)px;
    *i = (int)(n - r * (unsigned)px);
    *j = (int)(r % (unsigned)ny);
    *k = (int)(r / (unsigned)ny);
}

// N accumulators of a face, 16-byte loads and stores (N * sizeof(R) is a
// multiple of 16, and so is every face's offset).
template <class R, int N> __device__ __forceinline__ void loadAcc(const R *p, R (&v)[N])
{
#pragma unroll
    for (int q = 0; q < N * (int)sizeof(R) / 16; ++q)
        reinterpret_cast<int4 *>(v)[q] = reinterpret_cast<const int4 *>(p)[q];
}
template <class R, int N> __device__ __forceinline__ void storeAcc(R *p, const R (&v)[N])
{
#pragma unroll
    for (int q = 0; q < N * (int)sizeof(R) / 16; ++q)
        reinterpret_cast<int4 *>(p)[q] = reinterpret_cast<const int4 *>(v)[q];
}

// One thread per face or cut-plane point. Bound by the chain of dependent
// loads (a face touches 12 pulses, 6 materials and its accumulators, scattered
// for x faces, and the 38,688 faces of a 104x96x101 grid fill an eighth of the
// card's threads), so the chain is kept at two: the face's code and
// accumulators, then everything else; only a PEC neighbour and a face among the
// sources add one.
// On a B200, those faces, FP32, caches cold: 20.0 -> 8.5 us per step.
template <class S> __global__ void __launch_bounds__(kSurfaceThreads) surfaceMonitorKernel(const SurfaceArgs<S> a)
{
    using R = typename Traits<S>::R;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int nh = a.doDft ? a.nhuy : 0;
    const long long nplane = a.planeAxis >= 0 ? (long long)a.planeN1 * a.planeN2 : 0;
    R inc[12];
    if (t < a.njs)
    {
        // TlmSolver.cpp:632-646
        const long long code = a.jsNode[t];
        alignas(16) R acc[4];
        if (a.doDft) loadAcc<R, 4>(a.jsAcc + t * 4, acc);
        const long long node = code >> 3;
        const int ax = (int)((code >> 1) & 3);
        int i, j, k;
        cellOfNode(node, a.px, a.ny, &i, &j, &k);
        incidentAt<S>(a, node, i, j, k, inc);
        const R h1 = circulation(inc, ax == 0 ? 1 : 0), h2 = circulation(inc, ax == 2 ? 1 : 2);
        a.jsInst[t] = sqrt(h1 * h1 + h2 * h2);
        if (a.doDft)
        {
            acc[0] = acc[0] + h1 * a.cph;
            acc[1] = acc[1] - h1 * a.sph;
            acc[2] = acc[2] + h2 * a.cph;
            acc[3] = acc[3] - h2 * a.sph;
            storeAcc<R, 4>(a.jsAcc + t * 4, acc);
        }
        return;
    }
    long long u = t - a.njs;
    if (u < nh)
    {
        // TlmSolver.cpp:660-671: E_t ~ -V_t, eta0 H_t ~ -ZI_t
        const long long code = a.huyNode[u];
        alignas(16) R acc[8];
        loadAcc<R, 8>(a.huyAcc + u * 8, acc);
        const long long node = code >> 3;
        const int ax = (int)((code >> 1) & 3);
        int i, j, k;
        cellOfNode(node, a.px, a.ny, &i, &j, &k);
        incidentAt<S>(a, node, i, j, k, inc);
        const int t1 = ax == 0 ? 1 : 0, t2 = ax == 2 ? 1 : 2;
        const R e1 = -nodeVoltage(inc, t1), e2 = -nodeVoltage(inc, t2);
        const R m1 = -circulation(inc, t1), m2 = -circulation(inc, t2);
        acc[0] = acc[0] + e1 * a.cph;
        acc[1] = acc[1] - e1 * a.sph;
        acc[2] = acc[2] + e2 * a.cph;
        acc[3] = acc[3] - e2 * a.sph;
        acc[4] = acc[4] + m1 * a.cph;
        acc[5] = acc[5] - m1 * a.sph;
        acc[6] = acc[6] + m2 * a.cph;
        acc[7] = acc[7] - m2 * a.sph;
        storeAcc<R, 8>(a.huyAcc + u * 8, acc);
        return;
    }
    u -= nh;
    if (u < nplane)
    {
        // TlmSolver.cpp:716-743: |E| = sqrt(V_x^2 + V_y^2 + V_z^2), 0 on PEC
        const int q1 = (int)(u % a.planeN1), q2 = (int)(u / a.planeN1);
        const int pa = a.planeAxis;
        const int a1 = pa == 0 ? 1 : 0, a2 = pa == 2 ? 1 : 2;
        int co[3];
        co[pa] = a.planeIndex;
        co[a1] = q1;
        co[a2] = q2;
        const long long node = ((long long)co[2] * a.ny + co[1]) * a.px + co[0];
        R v = R(0);
        if (a.mat[node] != kPec)
        {
            incidentAt<S>(a, node, co[0], co[1], co[2], inc);
            R e2 = R(0);
#pragma unroll
            for (int jj = 0; jj < 3; ++jj)
            {
                const R vj = nodeVoltage(inc, jj);
                e2 = e2 + vj * vj;
            }
            v = sqrt(e2);
        }
        a.plane[u] = v;
    }
}

// Far field: a block takes kFarDirs directions (theta index d / nPhi, phi index
// d % nPhi) and one of gridDim.y slices of the faces. Per face the equivalent
// currents are J' = n x (eta0 H), M = -(n x E) (TlmSolver.cpp:829-848); summed
// with e^{+j k0 r.pos} they give N and L (TlmSolver.cpp:860-890), here as world
// components, FP64 throughout, and projected on theta and phi after the sum:
// U = |L_phi + N_theta|^2 + |L_theta - N_phi|^2. A face has only two components
// of each, so that costs the same 16 fused multiply-adds as summing projections,
// and a face is read, signed and widened once for all the block's directions.
// Sums run in a fixed order: a thread's faces, lanes, warps, slices. With more
// than one slice the blocks leave their sums in `part` for farFieldFinish.
// Bound by issue (sine, cosine and 16 FP64 operations per face and direction).
// 37 x 73 directions of 38,688 FP32 faces on a B200: 1584 -> 421 us (one block of
// 256 threads per direction, its projections summed, before).
constexpr int kFarDirs = 4, kFarThreads = 128;

template <class R> __device__ __forceinline__ void sinCos(R x, R *s, R *c)
{
    if constexpr (std::is_same<R, float>::value)
        sincosf(x, s, c);
    else
        sincos(x, s, c);
}

// Unit vectors of direction d: r, theta and (x and y of) phi.
template <class R>
__device__ __forceinline__ void farDirection(int d, int nTheta, int nPhi, R (&rh)[3], R (&tv)[3], R (&pv)[2])
{
    const R pi = R(3.14159265358979323846);
    const R th = pi * R(d / nPhi) / R(nTheta - 1);
    const R ph = R(2) * pi * R(d % nPhi) / R(nPhi - 1);
    const R st = sin(th), ct = cos(th), cp = cos(ph), sp = sin(ph);
    rh[0] = st * cp, rh[1] = st * sp, rh[2] = ct;
    tv[0] = ct * cp, tv[1] = ct * sp, tv[2] = -st;
    pv[0] = -sp, pv[1] = cp;
}

// U of direction d from its sums: N (re, im per component), then L.
template <class R>
__device__ __forceinline__ R farIntensity(const double (&v)[12], int d, int nTheta, int nPhi)
{
    R rh[3], tv[3], pv[2];
    farDirection(d, nTheta, nPhi, rh, tv, pv);
    double t[2][2], p[2][2];  // [N, L][re, im]
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int c = 0; c < 2; ++c)
        {
            const double x = v[q * 6 + c], y = v[q * 6 + 2 + c], z = v[q * 6 + 4 + c];
            t[q][c] = x * (double)tv[0] + y * (double)tv[1] + z * (double)tv[2];
            p[q][c] = x * (double)pv[0] + y * (double)pv[1];
        }
    const double aR = p[1][0] + t[0][0], aI = p[1][1] + t[0][1];
    const double bR = t[1][0] - p[0][0], bI = t[1][1] - p[0][1];
    return (R)(aR * aR + aI * aI + bR * bR + bI * bI);
}

template <class R>
__global__ void __launch_bounds__(kFarThreads, 3)
    farFieldKernel(const R *__restrict__ acc, const long long *__restrict__ code, const float *__restrict__ pos,
                   int nh, R k0, int nTheta, int nPhi, R *__restrict__ U, double *__restrict__ part)
{
    __shared__ double red[kFarThreads / 32][kFarDirs * 12];
    const int nd = nTheta * nPhi, d0 = blockIdx.x * kFarDirs;
    R rh[kFarDirs][3];
#pragma unroll
    for (int q = 0; q < kFarDirs; ++q)
    {
        R tv[3], pv[2];
        farDirection(min(d0 + q, nd - 1), nTheta, nPhi, rh[q], tv, pv);
    }
    double s[kFarDirs][12] = {};
    const int f0 = (int)((long long)nh * blockIdx.y / gridDim.y), f1 = (int)((long long)nh * (blockIdx.y + 1) / gridDim.y);
    for (int f = f0 + (int)threadIdx.x; f < f1; f += kFarThreads)
    {
        alignas(16) R a[8];
        loadAcc<R, 8>(acc + (long long)f * 8, a);
        const int c = (int)(code[f] & 7), ax = c >> 1;
        const R sa = ax == 1 ? R(-1) : R(1);
        const R sg = (c & 1) ? R(-1) : R(1);  // outward normal sign
        const R w = sg * sa;
        // J'[t2] = w H1, J'[t1] = -w H2, M[t2] = -w E1, M[t1] = w E2
        const double j1R = (double)(-w * a[6]), j1I = (double)(-w * a[7]);
        const double j2R = (double)(w * a[4]), j2I = (double)(w * a[5]);
        const double m1R = (double)(w * a[2]), m1I = (double)(w * a[3]);
        const double m2R = (double)(-w * a[0]), m2I = (double)(-w * a[1]);
        const R x = R(pos[3 * f]), y = R(pos[3 * f + 1]), z = R(pos[3 * f + 2]);
        double cs[kFarDirs], sn[kFarDirs];
#pragma unroll
        for (int q = 0; q < kFarDirs; ++q)
        {
            R sr, cr;
            sinCos(k0 * (rh[q][0] * x + rh[q][1] * y + rh[q][2] * z), &sr, &cr);
            cs[q] = (double)cr;
            sn[q] = (double)sr;
        }
        auto add = [&](auto T1, auto T2) {
            constexpr int t1 = decltype(T1)::value, t2 = decltype(T2)::value;
#pragma unroll
            for (int q = 0; q < kFarDirs; ++q)
            {
                auto rotate = [&](int at, double re, double im) {
                    s[q][at] = fma(re, cs[q], fma(-im, sn[q], s[q][at]));
                    s[q][at + 1] = fma(re, sn[q], fma(im, cs[q], s[q][at + 1]));
                };
                rotate(2 * t1, j1R, j1I);
                rotate(2 * t2, j2R, j2I);
                rotate(6 + 2 * t1, m1R, m1I);
                rotate(6 + 2 * t2, m2R, m2I);
            }
        };
        using I0 = std::integral_constant<int, 0>;
        using I1 = std::integral_constant<int, 1>;
        using I2 = std::integral_constant<int, 2>;
        if (ax == 0)  // faces are listed by axis: a warp takes one way
            add(I1{}, I2{});
        else if (ax == 1)
            add(I0{}, I2{});
        else
            add(I0{}, I1{});
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < kFarDirs; ++q)
#pragma unroll
        for (int c = 0; c < 12; ++c)
        {
            double v = s[q][c];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) red[warp][q * 12 + c] = v;
        }
    __syncthreads();
    if (threadIdx.x < kFarDirs * 12)
    {
        double v = 0;
        for (int w = 0; w < kFarThreads / 32; ++w) v += red[w][threadIdx.x];
        red[0][threadIdx.x] = v;
    }
    __syncthreads();
    const int q = threadIdx.x, d = d0 + q;
    if (q >= kFarDirs || d >= nd) return;
    double v[12];
#pragma unroll
    for (int c = 0; c < 12; ++c) v[c] = red[0][q * 12 + c];
    if (part != nullptr)
    {
#pragma unroll
        for (int c = 0; c < 12; ++c) part[((long long)blockIdx.y * 12 + c) * nd + d] = v[c];
    }
    else
        U[d] = farIntensity<R>(v, d, nTheta, nPhi);
}

template <class R>
__global__ void __launch_bounds__(128)
    farFieldFinish(const double *__restrict__ part, int slices, int nTheta, int nPhi, R *__restrict__ U)
{
    const int nd = nTheta * nPhi, d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= nd) return;
    double v[12] = {};
    for (int y = 0; y < slices; ++y)
#pragma unroll
        for (int c = 0; c < 12; ++c) v[c] += part[((long long)y * 12 + c) * nd + d];
    U[d] = farIntensity<R>(v, d, nTheta, nPhi);
}

} // namespace tlmk

namespace tlmi {

namespace {

size_t realSize(const tlm_solver *h) { return realBytes(h->storage); }

} // namespace

// Face lists in the reference's order: PEC faces by the scan of
// BuildPecSurfaceFaces (Geometry.cpp:402-436; cell, then axis, then side -1
// before +1), Huygens faces by TlmSolver::buildHuygens (TlmSolver.cpp:310-348;
// x faces over (k, j), y faces over (k, i), z faces over (j, i), low first).
void buildFaceLists(int nx, int ny, int nz, const float origin[3], float dl, const uint8_t *mat, bool surfaceOn,
                    int huyOffset, SurfaceState &s)
{
    s.jsCell.clear();
    s.jsAxis.clear();
    s.jsSign.clear();
    s.jsCenter.clear();
    s.huyCell.clear();
    s.huyAxis.clear();
    s.huySign.clear();
    s.huyPos.clear();
    if (!surfaceOn) return;
    auto center = [&](int i, int j, int k, float c[3]) {
        // origin + (i + 0.5) dl per axis, in float (Geometry.h:100-105)
        c[0] = origin[0] + ((float)i + 0.5f) * dl;
        c[1] = origin[1] + ((float)j + 0.5f) * dl;
        c[2] = origin[2] + ((float)k + 0.5f) * dl;
    };
    const long long stride[3] = { 1, nx, (long long)nx * ny };
    const int dims[3] = { nx, ny, nz };
    for (int k = 0; k < nz; ++k)
        for (int j = 0; j < ny; ++j)
        {
            // the row's PEC cells by memchr: a loop over its bytes took 300 or
            // 440 us for 1 M cells, by where the linker put it
            const uint8_t *row = mat + ((size_t)k * ny + j) * nx;
            for (const uint8_t *m = row; (m = static_cast<const uint8_t *>(std::memchr(m, tlmk::kPec, row + nx - m)));
                 ++m)
            {
                const int i = (int)(m - row);
                const size_t c = m - mat;
                const int co[3] = { i, j, k };
                for (int a = 0; a < 3; ++a)
                    for (int sd = -1; sd <= 1; sd += 2)
                    {
                        const int q = co[a] + sd;
                        if (q < 0 || q >= dims[a]) continue;
                        const size_t nb = c + (size_t)((long long)sd * stride[a]);
                        if (mat[nb] == tlmk::kPec) continue;
                        float cc[3];
                        center(i, j, k, cc);
                        cc[a] = cc[a] + (float)sd * dl * 0.5f;
                        s.jsCell.push_back(nb);
                        s.jsAxis.push_back(a);
                        s.jsSign.push_back(sd);
                        s.jsCenter.insert(s.jsCenter.end(), cc, cc + 3);
                    }
            }
        }
    const int o = huyOffset;
    if (o < 2 || 2 * o + 2 >= nx || 2 * o + 2 >= ny || 2 * o + 2 >= nz) return;
    const float half[3] = { ((float)nx * dl) * 0.5f, ((float)ny * dl) * 0.5f, ((float)nz * dl) * 0.5f };
    float dom[3];
    for (int a = 0; a < 3; ++a) dom[a] = origin[a] + half[a];
    auto add = [&](int i, int j, int k, int axis, int outSign) {
        const size_t c = ((size_t)k * ny + j) * nx + i;
        if (mat[c] != tlmk::kAir) return;
        float cc[3];
        center(i, j, k, cc);
        s.huyCell.push_back(c);
        s.huyAxis.push_back(axis);
        s.huySign.push_back(outSign);
        for (int a = 0; a < 3; ++a) s.huyPos.push_back(cc[a] - dom[a]);
    };
    const int x0 = o, x1 = nx - 1 - o, y0 = o, y1 = ny - 1 - o, z0 = o, z1 = nz - 1 - o;
    for (int k = z0; k <= z1; ++k)
        for (int j = y0; j <= y1; ++j)
        {
            add(x0, j, k, 0, -1);
            add(x1, j, k, 0, +1);
        }
    for (int k = z0; k <= z1; ++k)
        for (int i = x0; i <= x1; ++i)
        {
            add(i, y0, k, 1, -1);
            add(i, y1, k, 1, +1);
        }
    for (int j = y0; j <= y1; ++j)
        for (int i = x0; i <= x1; ++i)
        {
            add(i, j, z0, 2, -1);
            add(i, j, z1, 2, +1);
        }
}

void buildSurfaceLists(tlm_solver *h)
{
    buildFaceLists(h->nx, h->ny, h->nz, h->g.origin, h->g.dl, h->mat.data(), h->cfg.surface_monitors != 0,
                   h->cfg.huy_offset, h->surf);
}

bool surfaceActive(const tlm_solver *h)
{
    const SurfaceState &s = h->surf;
    return !s.jsCell.empty() || !s.huyCell.empty() || s.planeAxis >= 0 || h->cfg.record_every > 0;
}

void freeSurface(tlm_solver *h)
{
    SurfaceState &s = h->surf;
    devFree(h, s.dJsNode);
    devFree(h, s.dHuyNode);
    devFree(h, s.dJsInst);
    devFree(h, s.dJsAcc);
    devFree(h, s.dHuyAcc);
    devFree(h, s.dPlane);
    devFree(h, s.dFrames);
    s.planeCap = 0;
    s.planeValid = false;
    s.framesCap = s.framesUsed = 0;
    s.frames.clear();
}

// Upload the face lists and zero the accumulators (before the first step).
tlm_status prepareSurface(tlm_solver *h)
{
    SurfaceState &s = h->surf;
    const size_t r = realSize(h);
    auto upload = [&](long long **dst, const std::vector<uint64_t> &cells, const std::vector<int> &axis,
                      const std::vector<int> *sign) -> tlm_status {
        if (cells.empty()) return TLM_OK;
        std::vector<long long> code(cells.size());
        for (size_t f = 0; f < cells.size(); ++f)
            code[f] = paddedNode(h, cells[f]) * 8 + axis[f] * 2 + ((sign && (*sign)[f] < 0) ? 1 : 0);
        TLM_TRY(devAlloc(h, dst, code.size() * sizeof(long long)));
        TLM_CU(h, cudaMemcpyAsync(*dst, code.data(), code.size() * sizeof(long long), cudaMemcpyHostToDevice,
                                  h->stream));
        TLM_CU(h, cudaStreamSynchronize(h->stream));
        return TLM_OK;
    };
    TLM_TRY(upload(&s.dJsNode, s.jsCell, s.jsAxis, nullptr));
    TLM_TRY(upload(&s.dHuyNode, s.huyCell, s.huyAxis, &s.huySign));
    const size_t nj = s.jsCell.size(), nh = s.huyCell.size();
    if (nj)
    {
        TLM_TRY(devAlloc(h, &s.dJsInst, nj * r));
        TLM_TRY(devAlloc(h, &s.dJsAcc, nj * 4 * r));
    }
    if (nh) TLM_TRY(devAlloc(h, &s.dHuyAcc, nh * 8 * r));
    return rewindSurface(h);
}

tlm_status rewindSurface(tlm_solver *h)
{
    SurfaceState &s = h->surf;
    const size_t r = realSize(h);
    const size_t nj = s.jsCell.size(), nh = s.huyCell.size();
    if (s.dJsInst) TLM_CU(h, cudaMemsetAsync(s.dJsInst, 0, nj * r, h->stream));
    if (s.dJsAcc) TLM_CU(h, cudaMemsetAsync(s.dJsAcc, 0, nj * 4 * r, h->stream));
    if (s.dHuyAcc) TLM_CU(h, cudaMemsetAsync(s.dHuyAcc, 0, nh * 8 * r, h->stream));
    s.planeValid = false;
    s.frames.clear();
    s.framesUsed = 0;
    return TLM_OK;
}

namespace {

template <class S> tlm_status launchSurfaceT(tlm_solver *h, int n)
{
    using R = typename tlmk::Traits<S>::R;
    SurfaceState &s = h->surf;
    const int nj = (int)s.jsCell.size(), nh = (int)s.huyCell.size();
    const bool doDft = n >= h->cfg.settle_steps;
    const bool doPlane = s.planeAxis >= 0 && (n % 2) == 0;
    int n1 = 0, n2 = 0;
    if (doPlane)
    {
        const int dims[3] = { h->nx, h->ny, h->nz };
        n1 = dims[s.planeAxis == 0 ? 1 : 0];
        n2 = dims[s.planeAxis == 2 ? 1 : 2];
        const size_t need = (size_t)n1 * n2;
        if (need > s.planeCap)
        {
            devFree(h, s.dPlane);
            TLM_TRY(devAlloc(h, &s.dPlane, need * sizeof(R)));
            s.planeCap = need;
        }
    }
    const long long items = (long long)nj + (doDft ? nh : 0) + (doPlane ? (long long)n1 * n2 : 0);
    if (items > 0)
    {
        tlmk::SurfaceArgs<S> a;
        a.in = static_cast<const S *>(h->dPulses[h->curBuf]);
        a.incident = h->stateIncident ? 1 : 0;
        a.mat = h->dMat;
        a.P = h->P;
        a.nx = h->nx;
        a.ny = h->ny;
        a.nz = h->nz;
        a.px = h->px;
        a.rho = (R)h->cfg.boundary_rho;
        a.scale = (R)h->scale;
        a.spec = h->dSpec;
        a.nspec = h->dSpec ? h->specCount : 0;
        a.injLo = h->injLo;
        a.injHi = h->injHi;
        a.sv = (R)sourceValue(h, n);
        a.jsNode = s.dJsNode;
        a.njs = nj;
        a.jsInst = static_cast<R *>(s.dJsInst);
        a.jsAcc = static_cast<R *>(s.dJsAcc);
        a.huyNode = s.dHuyNode;
        a.nhuy = nh;
        a.huyAcc = static_cast<R *>(s.dHuyAcc);
        a.doDft = doDft ? 1 : 0;
        a.cph = a.sph = R(0);
        if ((nj || nh) && doDft)
        {
            // the DFT phase of step n, computed on the host like the reference
            if (h->storage == TLM_STORE_F64)
            {
                double c, sn;
                tlmh::dft_phase_f64(h->cfg.f0, h->dt64, n, &c, &sn);
                a.cph = (R)c;
                a.sph = (R)sn;
            }
            else
            {
                float c, sn;
                tlmh::dft_phase_f32(h->cfg.f0, h->dt32, n, &c, &sn);
                a.cph = (R)c;
                a.sph = (R)sn;
            }
        }
        a.planeAxis = doPlane ? s.planeAxis : -1;
        a.planeIndex = doPlane ? std::min(std::max(s.planeIndex, 0), (s.planeAxis == 0 ? h->nx : s.planeAxis == 1 ? h->ny : h->nz) - 1) : 0;
        a.planeN1 = n1;
        a.planeN2 = n2;
        a.plane = static_cast<R *>(s.dPlane);
        const long long blocks = (items + tlmk::kSurfaceThreads - 1) / tlmk::kSurfaceThreads;
        tlmk::surfaceMonitorKernel<S><<<(unsigned)blocks, tlmk::kSurfaceThreads, 0, h->stream>>>(a);
        TLM_CU(h, cudaGetLastError());
        if (doPlane)
        {
            s.planeValid = true;
            s.planeAxisDone = s.planeAxis;
            s.planeIndexDone = a.planeIndex;
            s.planeN1 = n1;
            s.planeN2 = n2;
        }
    }
    // playback frame (TlmSolver.cpp:746-762): |Js| and the latest cut plane
    if (h->cfg.record_every > 0 && (n % h->cfg.record_every) == 0)
    {
        const bool withPlane = s.planeAxis >= 0 && s.planeValid;
        const size_t np = withPlane ? (size_t)s.planeN1 * s.planeN2 : 0;
        const size_t need = s.framesUsed + nj + np;
        if (need > s.framesCap)
        {
            const size_t cap = std::max(need, s.framesCap * 2 + 1024);
            void *d = nullptr;
            TLM_TRY(devAlloc(h, &d, cap * sizeof(R)));
            if (s.framesUsed)
                TLM_CU(h, cudaMemcpyAsync(d, s.dFrames, s.framesUsed * sizeof(R), cudaMemcpyDeviceToDevice,
                                          h->stream));
            devFree(h, s.dFrames);
            s.dFrames = d;
            s.framesCap = cap;
        }
        R *base = static_cast<R *>(s.dFrames) + s.framesUsed;
        if (nj) TLM_CU(h, cudaMemcpyAsync(base, s.dJsInst, nj * sizeof(R), cudaMemcpyDeviceToDevice, h->stream));
        if (np) TLM_CU(h, cudaMemcpyAsync(base + nj, s.dPlane, np * sizeof(R), cudaMemcpyDeviceToDevice, h->stream));
        SurfaceState::Frame fr;
        fr.step = n;
        fr.hasPlane = withPlane ? 1 : 0;
        fr.axis = withPlane ? s.planeAxisDone : -1;
        fr.index = withPlane ? s.planeIndexDone : 0;
        fr.n1 = withPlane ? s.planeN1 : 0;
        fr.n2 = withPlane ? s.planeN2 : 0;
        fr.off = s.framesUsed;
        s.frames.push_back(fr);
        s.framesUsed = need;
    }
    return TLM_OK;
}

} // namespace

tlm_status launchSurface(tlm_solver *h, int n)
{
    switch (h->storage)
    {
    case TLM_STORE_F64: return launchSurfaceT<double>(h, n);
    case TLM_STORE_BF16: return launchSurfaceT<__nv_bfloat16>(h, n);
    case TLM_STORE_F16: return launchSurfaceT<__half>(h, n);
    case TLM_STORE_BFP16: return launchSurfaceT<tlmk::Bfp4>(h, n);
    default: return launchSurfaceT<float>(h, n);
    }
}

} // namespace tlmi

namespace tlmi {

// Near-to-far-field transform of the Huygens phasors on the device (FP64 sums), then the reference's directivity and peak
// search on the host (TlmSolver.cpp:893-915). `f64`: the phasors are double.
tlm_status farFieldTransform(cudaStream_t stream, cudaMemPool_t pool, bool f64, const void *dAcc,
                             const long long *dCode, const float *hostPos, int nh, float f0, int n_theta,
                             int n_phi, float *U, FarField &out, std::string &err)
{
    const int nd = n_theta * n_phi;
    float *dPos = nullptr;
    void *dU = nullptr;
    const size_t r = f64 ? 8 : 4;
    cudaError_t e = cudaMallocFromPoolAsync((void **)&dPos, (size_t)nh * 3 * sizeof(float), pool, stream);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(&dU, (size_t)nd * r, pool, stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(dPos, hostPos, (size_t)nh * 3 * sizeof(float), cudaMemcpyHostToDevice, stream);
    // slices of the faces, for directions too few to fill the card evenly; a
    // slice keeps 32 faces per thread or more, and without memory for the
    // partial sums there is one
    const int groups = (nd + tlmk::kFarDirs - 1) / tlmk::kFarDirs;
    int slices = std::max(1, std::min({ 4096 / groups, nh / (32 * tlmk::kFarThreads), 64 }));
    double *dPart = nullptr;
    if (e == cudaSuccess && slices > 1 &&
        cudaMallocFromPoolAsync((void **)&dPart, (size_t)slices * nd * 12 * sizeof(double), pool, stream) != cudaSuccess)
    {
        cudaGetLastError();
        dPart = nullptr;
        slices = 1;
    }
    if (e == cudaSuccess)
    {
        auto launch = [&](auto k0) {
            using R = decltype(k0);
            tlmk::farFieldKernel<R><<<dim3(groups, slices), tlmk::kFarThreads, 0, stream>>>(
                static_cast<const R *>(dAcc), dCode, dPos, nh, k0, n_theta, n_phi, static_cast<R *>(dU), dPart);
            if (dPart)
                tlmk::farFieldFinish<R><<<(nd + 127) / 128, 128, 0, stream>>>(dPart, slices, n_theta, n_phi,
                                                                              static_cast<R *>(dU));
        };
        if (f64)
            launch(2.0 * 3.14159265358979323846 * (double)f0 / (double)299792458.0f);
        else
            launch(2.0f * (float)3.14159265358979323846 * f0 / 299792458.0f);
        e = cudaGetLastError();
    }
    if (dPart) cudaFreeAsync(dPart, stream);
    std::vector<float> u(nd);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e == cudaSuccess)
    {
        if (f64)
        {
            std::vector<double> t(nd);
            e = cudaMemcpy(t.data(), dU, (size_t)nd * 8, cudaMemcpyDeviceToHost);
            for (int i = 0; i < nd; ++i) u[i] = (float)t[i];
        }
        else
            e = cudaMemcpy(u.data(), dU, (size_t)nd * 4, cudaMemcpyDeviceToHost);
    }
    if (dPos) cudaFreeAsync(dPos, stream);
    if (dU) cudaFreeAsync(dU, stream);
    if (e != cudaSuccess)
    {
        cudaGetLastError();
        err = std::string("far-field transform: ") + cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? TLM_ENOMEM : TLM_ECUDA;
    }
    const float pi = (float)3.14159265358979323846;
    float um = 0.0f;
    int iMax = 0;
    double prad = 0.0;
    const float dTh = pi / (float)(n_theta - 1);
    const float dPh = 2.0f * pi / (float)(n_phi - 1);
    for (int ti = 0; ti < n_theta; ++ti)
    {
        const float th = pi * (float)ti / (float)(n_theta - 1);
        const float wTh = (ti == 0 || ti == n_theta - 1) ? 0.5f : 1.0f;
        for (int pj = 0; pj < n_phi; ++pj)
        {
            const float wPh = (pj == 0 || pj == n_phi - 1) ? 0.5f : 1.0f;
            const float v = u[(size_t)ti * n_phi + pj];
            if (v > um)
            {
                um = v;
                iMax = ti * n_phi + pj;
            }
            prad += (double)v * std::sin(th) * wTh * wPh * dTh * dPh;
        }
    }
    if (U) std::copy(u.begin(), u.end(), U);
    out.uMax = um;
    out.directivity = prad > 0 ? (float)(4.0 * 3.14159265358979323846 * um / prad) : 0.0f;
    out.peakTheta = 180.0f * (float)(iMax / n_phi) / (float)(n_theta - 1);
    out.peakPhi = 360.0f * (float)(iMax % n_phi) / (float)(n_phi - 1);
    return TLM_OK;
}

} // namespace tlmi

namespace {

// Device buffer of the storage's real type -> host floats.
tlm_status realsToHost(tlm_solver *h, const void *d, size_t count, float *out)
{
    if (!count) return TLM_OK;
    if (h->storage == TLM_STORE_F64)
    {
        std::vector<double> t(count);
        TLM_CU(h, cudaMemcpy(t.data(), d, count * 8, cudaMemcpyDeviceToHost));
        for (size_t i = 0; i < count; ++i) out[i] = (float)t[i];
    }
    else
        TLM_CU(h, cudaMemcpy(out, d, count * 4, cudaMemcpyDeviceToHost));
    return TLM_OK;
}

int samplesOf(const tlm_solver *h)
{
    const int settle = std::max(h->cfg.settle_steps, 0);
    return std::max(0, h->curStep - settle);
}

} // namespace

extern "C" {

tlm_status tlm_get_surface_faces(tlm_handle h, uint64_t *air_cells, int *axis, int *sign, float *centers,
                                 int cap, int *n_out)
{
    TLM_TRY(checkReady(h));
    const SurfaceState &s = h->surf;
    const int n = (int)s.jsCell.size();
    if (n_out) *n_out = n;
    for (int f = 0; f < n && f < cap; ++f)
    {
        if (air_cells) air_cells[f] = s.jsCell[f];
        if (axis) axis[f] = s.jsAxis[f];
        if (sign) sign[f] = s.jsSign[f];
        if (centers) std::memcpy(centers + 3 * f, &s.jsCenter[3 * f], 3 * sizeof(float));
    }
    return TLM_OK;
}

tlm_status tlm_get_js_instant(tlm_handle h, float *out, int cap, int *n_out)
{
    TLM_TRY(checkReady(h));
    DeviceGuard dg(h->device);
    TLM_TRY(syncState(h));
    const SurfaceState &s = h->surf;
    const int n = (int)s.jsCell.size();
    if (n_out) *n_out = n;
    if (!out || cap <= 0 || n == 0) return TLM_OK;
    if (!s.dJsInst)
    {
        std::fill(out, out + std::min(n, cap), 0.0f);
        return TLM_OK;
    }
    std::vector<float> t(n);
    TLM_TRY(realsToHost(h, s.dJsInst, n, t.data()));
    std::copy(t.begin(), t.begin() + std::min(n, cap), out);
    return TLM_OK;
}

tlm_status tlm_get_js_dft(tlm_handle h, float *magnitude, float *re, float *im, int cap, int *n_out,
                          int *samples)
{
    TLM_TRY(checkReady(h));
    DeviceGuard dg(h->device);
    TLM_TRY(syncState(h));
    const SurfaceState &s = h->surf;
    const int n = (int)s.jsCell.size();
    const int ns = s.jsCell.empty() ? 0 : samplesOf(h);
    if (n_out) *n_out = n;
    if (samples) *samples = ns;
    if (n == 0 || cap <= 0) return TLM_OK;
    std::vector<float> acc((size_t)n * 4, 0.0f);
    if (s.dJsAcc) TLM_TRY(realsToHost(h, s.dJsAcc, (size_t)n * 4, acc.data()));
    for (int f = 0; f < n && f < cap; ++f)
    {
        const float r1 = acc[4 * f], i1 = acc[4 * f + 1], r2 = acc[4 * f + 2], i2 = acc[4 * f + 3];
        if (re)
        {
            re[2 * f] = r1;
            re[2 * f + 1] = r2;
        }
        if (im)
        {
            im[2 * f] = i1;
            im[2 * f + 1] = i2;
        }
        if (magnitude)
        {
            // finalizeDft (TlmSolver.cpp:467-481)
            float m = 0.0f;
            if (ns > 0)
            {
                const float norm = 2.0f / (float)ns;
                m = norm * std::sqrt(r1 * r1 + i1 * i1 + r2 * r2 + i2 * i2);
            }
            magnitude[f] = m;
        }
    }
    return TLM_OK;
}

tlm_status tlm_get_huygens_faces(tlm_handle h, uint64_t *cells, int *axis, int *out_sign, float *pos, int cap,
                                 int *n_out)
{
    TLM_TRY(checkReady(h));
    const SurfaceState &s = h->surf;
    const int n = (int)s.huyCell.size();
    if (n_out) *n_out = n;
    for (int f = 0; f < n && f < cap; ++f)
    {
        if (cells) cells[f] = s.huyCell[f];
        if (axis) axis[f] = s.huyAxis[f];
        if (out_sign) out_sign[f] = s.huySign[f];
        if (pos) std::memcpy(pos + 3 * f, &s.huyPos[3 * f], 3 * sizeof(float));
    }
    return TLM_OK;
}

tlm_status tlm_get_huygens_dft(tlm_handle h, float *acc8, int cap, int *n_out, int *samples)
{
    TLM_TRY(checkReady(h));
    DeviceGuard dg(h->device);
    TLM_TRY(syncState(h));
    const SurfaceState &s = h->surf;
    const int n = (int)s.huyCell.size();
    if (n_out) *n_out = n;
    if (samples) *samples = n ? samplesOf(h) : 0;
    if (!acc8 || n == 0 || cap <= 0) return TLM_OK;
    const int m = std::min(n, cap);
    if (!s.dHuyAcc)
    {
        std::fill(acc8, acc8 + (size_t)m * 8, 0.0f);
        return TLM_OK;
    }
    return realsToHost(h, s.dHuyAcc, (size_t)m * 8, acc8);
}

tlm_status tlm_set_field_plane(tlm_handle h, int axis, int index)
{
    TLM_TRY(checkReady(h));
    if (h->batch) return h->fail(TLM_ESTATE, "the handle is attached to a batch");
    if (axis < -1 || axis > 2) return h->fail(TLM_EINVAL, "plane axis must be -1 (off), 0, 1 or 2");
    DeviceGuard dg(h->device);
    TLM_TRY(syncState(h));
    h->surf.planeAxis = axis;
    h->surf.planeIndex = index;
    return TLM_OK;
}

tlm_status tlm_get_field_plane(tlm_handle h, float *out, size_t cap, int *axis, int *index, int *n1, int *n2)
{
    TLM_TRY(checkReady(h));
    DeviceGuard dg(h->device);
    TLM_TRY(syncState(h));
    const SurfaceState &s = h->surf;
    if (s.planeAxis < 0 || !s.planeValid) return h->fail(TLM_ESTATE, "no field plane has been computed");
    const size_t n = (size_t)s.planeN1 * s.planeN2;
    if (axis) *axis = s.planeAxisDone;
    if (index) *index = s.planeIndexDone;
    if (n1) *n1 = s.planeN1;
    if (n2) *n2 = s.planeN2;
    if (!out) return TLM_OK;
    if (cap < n) return h->fail(TLM_EINVAL, "output holds fewer values than the plane");
    return realsToHost(h, s.dPlane, n, out);
}

tlm_status tlm_frame_count(tlm_handle h, int *n)
{
    TLM_TRY(checkReady(h));
    if (!n) return h->fail(TLM_EINVAL, "null output");
    *n = (int)h->surf.frames.size();
    return TLM_OK;
}

tlm_status tlm_get_frame(tlm_handle h, int idx, int *step, float *js, int js_cap, float *plane, size_t plane_cap,
                         int *axis, int *index, int *n1, int *n2)
{
    TLM_TRY(checkReady(h));
    const SurfaceState &s = h->surf;
    if (idx < 0 || idx >= (int)s.frames.size()) return h->fail(TLM_EINVAL, "no such frame");
    DeviceGuard dg(h->device);
    TLM_TRY(syncState(h));
    const SurfaceState::Frame &fr = s.frames[idx];
    const int nj = (int)s.jsCell.size();
    const size_t np = fr.hasPlane ? (size_t)fr.n1 * fr.n2 : 0;
    if (step) *step = fr.step;
    if (axis) *axis = fr.axis;
    if (index) *index = fr.index;
    if (n1) *n1 = fr.n1;
    if (n2) *n2 = fr.n2;
    const size_t r = realBytes(h->storage);
    const char *base = static_cast<const char *>(s.dFrames) + fr.off * r;
    if (js && nj)
    {
        std::vector<float> t(nj);
        TLM_TRY(realsToHost(h, base, nj, t.data()));
        std::copy(t.begin(), t.begin() + std::min(nj, std::max(js_cap, 0)), js);
    }
    if (plane && np)
    {
        if (plane_cap < np) return h->fail(TLM_EINVAL, "plane output holds fewer values than the frame's plane");
        TLM_TRY(realsToHost(h, base + (size_t)nj * r, np, plane));
    }
    return TLM_OK;
}

tlm_status tlm_compute_far_field(tlm_handle h, int n_theta, int n_phi, float *U, float *u_max,
                                 float *directivity, float *peak_theta_deg, float *peak_phi_deg)
{
    TLM_TRY(checkReady(h));
    if (n_theta < 2 || n_phi < 2) return h->fail(TLM_EINVAL, "need at least 2 theta and 2 phi samples");
    const SurfaceState &s = h->surf;
    const int nh = (int)s.huyCell.size();
    if (nh == 0 || samplesOf(h) == 0 || !s.dHuyAcc)
        return h->fail(TLM_ESTATE, "no Huygens phasors recorded (surface_monitors, huy_offset >= 2, "
                                   "steps past settle_steps)");
    DeviceGuard dg(h->device);
    TLM_TRY(syncState(h));
    FarField out;
    std::string err;
    const tlm_status st = farFieldTransform(h->stream, h->pool, h->storage == TLM_STORE_F64, s.dHuyAcc,
                                            s.dHuyNode, s.huyPos.data(), nh, h->cfg.f0, n_theta, n_phi, U,
                                            out, err);
    if (st != TLM_OK) return h->fail(st, err);
    if (u_max) *u_max = out.uMax;
    if (directivity) *directivity = out.directivity;
    if (peak_theta_deg) *peak_theta_deg = out.peakTheta;
    if (peak_phi_deg) *peak_phi_deg = out.peakPhi;
    return TLM_OK;
}

} // extern "C"
