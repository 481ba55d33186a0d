// fdtd_solver.cu -- Yee FDTD time step on sm_100a (the reference's second
// time-domain solver, FdtdSolver.cpp), behind the C ABI of fdtd_b200.h.
//
// One step (FdtdSolver::step, FdtdSolver.cpp:401-446):
//   1. soft sources on E edges (per-edge thread applying its contributions in
//      the reference's source order, so edges shared by several source cells
//      add up exactly as the sequential loop does);
//   2. monitors on the current fields (ports, probes, surface currents,
//      Huygens phasors, cut plane; energy every 16 steps);
//   3. H update over all H components;
//   4. Mur snapshot of the two outermost layers of every tangential E
//      component, E update of the interior edges (PEC masks, lossy
//      coefficients), then the first-order Mur boundary in two launches whose
//      order reproduces the reference's six face passes (edges shared by two
//      faces end with the later pass's value).
// Steps 3 and 4 are one pass over memory (fusedStepKernel) from one field
// buffer to another, then a tail kernel (stepTailKernel): Mur, which takes the
// old boundary values from the input buffer, the monitors, and the next step's
// sources; without room for a second field buffer they run in place,
// one sweep for H and one for E.
// Fields: one plane set per component, all six with the same pitch (cell
// (i, j, k) of every component at (k*(ny+1) + j)*px + i, rows padded for fused
// passes only; entries that a
// component does not have stay zero). All arithmetic is FP32 in the
// reference's operation order (the library is compiled with --fmad=false),
// hence bitwise results.
#include "fdtd_b200.h"
#include "tlm_b200.h"
#include "tlm_internal.h"

#include "tlm_host_math.h"
#include "tlm_step_kernel.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

using tlmi::SurfaceState;

namespace fdk {

struct Dims
{
    int nx, ny, nz;
    int px;  // row pitch: nx + 1, rounded up to 4 for fused passes
    __host__ __device__ long long at(int i, int j, int k) const { return ((long long)k * (ny + 1) + j) * px + i; }
    __host__ __device__ long long iEx(int i, int j, int k) const { return at(i, j, k); }
    __host__ __device__ long long iEy(int i, int j, int k) const { return at(i, j, k); }
    __host__ __device__ long long iEz(int i, int j, int k) const { return at(i, j, k); }
    __host__ __device__ long long iHx(int i, int j, int k) const { return at(i, j, k); }
    __host__ __device__ long long iHy(int i, int j, int k) const { return at(i, j, k); }
    __host__ __device__ long long iHz(int i, int j, int k) const { return at(i, j, k); }
    // 32-bit form for the in-place sweeps: setup refuses grids whose
    // (nx+1)(ny+1)(nz+1) index box reaches 2^31, and the pitch adds at most
    // three fifths (8 for 5).
    __device__ unsigned q(int i, int j, int k) const
    {
        return ((unsigned)k * (unsigned)(ny + 1) + (unsigned)j) * (unsigned)px + (unsigned)i;
    }
};

// Class of an E edge, ten bits per component (x, y, z from the low bits up) in
// a word per cell: kEdgePec, kEdgeAir (the four cells around it are air), the
// id of the dielectric that fills all four, from kEdgeFirst on a pair of
// coefficients that edges between materials have, or, where the table has no
// room for more of those, kEdgeMixed: coefficients in ca / cb. The table holds
// the coefficients of every class below kEdgeMixed.
enum : unsigned { kEdgePec = 0, kEdgeAir = 1, kEdgeFirst = 256, kEdgeMixed = 511, kEdgeClasses = 512 };
__host__ __device__ __forceinline__ constexpr unsigned edgeWord(unsigned c) { return c * 0x00100401u; }  // all three
__device__ __forceinline__ unsigned edgeClass(unsigned word, int comp) { return (word >> (10 * comp)) & 1023u; }

struct Fields
{
    float *E[3], *H[3];
    const unsigned *cls;         // edge classes
    const float2 *tab;           // (ca, cb) of every class but kEdgeMixed
    const float *ca[3], *cb[3];  // of mixed edges (nullptr: no dielectric)
};

// ---- cell-centred averages (FdtdSolver.cpp:42-79) -------------------------
__device__ __forceinline__ float ecAt(const Fields &f, const Dims &d, int i, int j, int k, int c)
{
    if (c == 0)
        return 0.25f * (((f.E[0][d.iEx(i, j, k)] + f.E[0][d.iEx(i, j + 1, k)]) + f.E[0][d.iEx(i, j, k + 1)]) +
                        f.E[0][d.iEx(i, j + 1, k + 1)]);
    if (c == 1)
        return 0.25f * (((f.E[1][d.iEy(i, j, k)] + f.E[1][d.iEy(i + 1, j, k)]) + f.E[1][d.iEy(i, j, k + 1)]) +
                        f.E[1][d.iEy(i + 1, j, k + 1)]);
    return 0.25f * (((f.E[2][d.iEz(i, j, k)] + f.E[2][d.iEz(i + 1, j, k)]) + f.E[2][d.iEz(i, j + 1, k)]) +
                    f.E[2][d.iEz(i + 1, j + 1, k)]);
}
__device__ __forceinline__ float hcAt(const Fields &f, const Dims &d, int i, int j, int k, int c)
{
    if (c == 0) return 0.5f * (f.H[0][d.iHx(i, j, k)] + f.H[0][d.iHx(i + 1, j, k)]);
    if (c == 1) return 0.5f * (f.H[1][d.iHy(i, j, k)] + f.H[1][d.iHy(i, j + 1, k)]);
    return 0.5f * (f.H[2][d.iHz(i, j, k)] + f.H[2][d.iHz(i, j, k + 1)]);
}

// ---- 1. soft sources ----------------------------------------------------
// Edge e (code: component * 2^60 + field index) receives amps[off[e]..off[e+1])
// in source order: E += (-0.25 amp) sv each (FdtdSolver.cpp:404-437).
struct InjectArgs
{
    float *E[3];
    const long long *edge;
    const int *off;
    const float *amps;
    int nedges;
    float sv;
};
__device__ __forceinline__ void injectItem(const InjectArgs &a, int e)
{
    if (e >= a.nedges) return;
    const long long code = a.edge[e];
    const int c = (int)(code >> 60);
    const long long idx = code & ((1LL << 60) - 1);
    const int t0 = a.off[e], t1 = a.off[e + 1];
    float *E = c == 0 ? a.E[0] : c == 1 ? a.E[1] : a.E[2];
    float v = E[idx];
    for (int t = t0; t < t1; ++t) v = v + (-0.25f * a.amps[t]) * a.sv;
    E[idx] = v;
}
__global__ void injectKernel(const InjectArgs a) { injectItem(a, blockIdx.x * blockDim.x + threadIdx.x); }

// ---- 2. monitors ----------------------------------------------------------
struct MonArgs
{
    Fields f;
    Dims d;
    float dl, eta0;
    int step;
    // ports: cells of port p at cells[poff[p] .. poff[p+1]), middle cell pmid[p]
    int nports;
    const int *poff;
    const long long *pcells;
    const int *ppol;
    float *vrec, *irec;  // [step][nports]
    // probes
    int nprobes;
    const long long *probeCell;
    float *prec;         // [step][nprobes][3]
    // surface faces: code = cell * 8 + axis * 2 + (sign < 0)
    int njs;
    const long long *jsCode;
    float *jsInst, *jsAcc;
    int nhuy;
    const long long *huyCode;
    float *huyAcc;
    int doDft;
    float cph, sph;
    int planeAxis, planeIndex, planeN1, planeN2;
    float *plane;
};

// (cells number below 2^31: 32-bit divisions)
__device__ __forceinline__ void cellCo(long long c, const Dims &d, int co[3])
{
    const unsigned u = (unsigned)c, r = u / (unsigned)d.nx, k = r / (unsigned)d.ny;
    co[0] = (int)(u - r * (unsigned)d.nx);
    co[1] = (int)(r - k * (unsigned)d.ny);
    co[2] = (int)k;
}

__device__ __forceinline__ void monitorItem(const MonArgs &a, long long t)
{
    const Fields &f = a.f;
    const Dims &d = a.d;
    if (t < a.nports)
    {
        // FdtdSolver.cpp:753-781
        const int p = (int)t;
        const int pol = a.ppol[p];
        float vSum = 0.0f;
        for (int q = a.poff[p]; q < a.poff[p + 1]; ++q)
        {
            int co[3];
            cellCo(a.pcells[q], d, co);
            vSum += -ecAt(f, d, co[0], co[1], co[2], pol) * a.dl;
        }
        float iVal = 0.0f;
        if (a.poff[p + 1] > a.poff[p])
        {
            const int mid = a.poff[p] + (a.poff[p + 1] - a.poff[p]) / 2;
            int co[3];
            cellCo(a.pcells[mid], d, co);
            const int t1 = (pol + 1) % 3, t2 = (pol + 2) % 3;
            int d1[3] = { 0, 0, 0 }, d2[3] = { 0, 0, 0 };
            d1[t1] = 1;
            d2[t2] = 1;
            iVal = 2.0f * a.dl *
                   (((hcAt(f, d, co[0] + d1[0], co[1] + d1[1], co[2] + d1[2], t2) -
                      hcAt(f, d, co[0] - d1[0], co[1] - d1[1], co[2] - d1[2], t2)) -
                     hcAt(f, d, co[0] + d2[0], co[1] + d2[1], co[2] + d2[2], t1)) +
                    hcAt(f, d, co[0] - d2[0], co[1] - d2[1], co[2] - d2[2], t1));
        }
        a.vrec[(long long)a.step * a.nports + p] = vSum;
        a.irec[(long long)a.step * a.nports + p] = iVal;
        return;
    }
    t -= a.nports;
    if (t < a.nprobes)
    {
        int co[3];
        cellCo(a.probeCell[t], d, co);
        float *o = a.prec + ((long long)a.step * a.nprobes + t) * 3;
        const float ex = ecAt(f, d, co[0], co[1], co[2], 0), ey = ecAt(f, d, co[0], co[1], co[2], 1);
        const float ez = ecAt(f, d, co[0], co[1], co[2], 2);
        o[0] = ex;
        o[1] = ey;
        o[2] = ez;
        return;
    }
    t -= a.nprobes;
    if (t < a.njs)
    {
        // FdtdSolver.cpp:703-721: eta0 H at the face cell
        const long long code = a.jsCode[t];
        int co[3];
        cellCo(code >> 3, d, co);
        const int ax = (int)((code >> 1) & 3);
        const int t1 = ax == 0 ? 1 : 0, t2 = ax == 2 ? 1 : 2;
        const float h1 = a.eta0 * hcAt(f, d, co[0], co[1], co[2], t1);
        const float h2 = a.eta0 * hcAt(f, d, co[0], co[1], co[2], t2);
        a.jsInst[t] = sqrtf(h1 * h1 + h2 * h2);
        if (a.doDft)
        {
            float *acc = a.jsAcc + t * 4;
            acc[0] = acc[0] + h1 * a.cph;
            acc[1] = acc[1] - h1 * a.sph;
            acc[2] = acc[2] + h2 * a.cph;
            acc[3] = acc[3] - h2 * a.sph;
        }
        return;
    }
    t -= a.njs;
    const int nh = a.doDft ? a.nhuy : 0;
    if (t < nh)
    {
        // FdtdSolver.cpp:729-748: cell-centred E and eta0 H
        const long long code = a.huyCode[t];
        int co[3];
        cellCo(code >> 3, d, co);
        const int ax = (int)((code >> 1) & 3);
        const int t1 = ax == 0 ? 1 : 0, t2 = ax == 2 ? 1 : 2;
        const float e1 = ecAt(f, d, co[0], co[1], co[2], t1), e2 = ecAt(f, d, co[0], co[1], co[2], t2);
        const float m1 = a.eta0 * hcAt(f, d, co[0], co[1], co[2], t1);
        const float m2 = a.eta0 * hcAt(f, d, co[0], co[1], co[2], t2);
        float *acc = a.huyAcc + t * 8;
        acc[0] = acc[0] + e1 * a.cph;
        acc[1] = acc[1] - e1 * a.sph;
        acc[2] = acc[2] + e2 * a.cph;
        acc[3] = acc[3] - e2 * a.sph;
        acc[4] = acc[4] + m1 * a.cph;
        acc[5] = acc[5] - m1 * a.sph;
        acc[6] = acc[6] + m2 * a.cph;
        acc[7] = acc[7] - m2 * a.sph;
        return;
    }
    t -= nh;
    const long long np = a.planeAxis >= 0 ? (long long)a.planeN1 * a.planeN2 : 0;
    if (t < np)
    {
        // FdtdSolver.cpp:790-813: |E| dl over the plane, PEC cells included
        const int q1 = (int)(t % a.planeN1), q2 = (int)(t / a.planeN1);
        const int pa = a.planeAxis, a1 = pa == 0 ? 1 : 0, a2 = pa == 2 ? 1 : 2;
        int co[3];
        co[pa] = a.planeIndex;
        co[a1] = q1;
        co[a2] = q2;
        const float ex = ecAt(f, d, co[0], co[1], co[2], 0);
        const float ey = ecAt(f, d, co[0], co[1], co[2], 1);
        const float ez = ecAt(f, d, co[0], co[1], co[2], 2);
        a.plane[t] = sqrtf(ex * ex + ey * ey + ez * ez) * a.dl;
    }
}

__global__ void __launch_bounds__(256) monitorKernel(const MonArgs a)
{
    monitorItem(a, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

// Energy (FdtdSolver.cpp:836-870): sum E^2 + eta0^2 sum H^2 in FP64, block
// partials in a fixed order. Every component is swept as 16-byte vectors
// (device allocations are 256-byte aligned), four in flight per thread.
__device__ __forceinline__ double sumSquares(const float *arr, long long n)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const float4 *a4 = reinterpret_cast<const float4 *>(arr);
    const long long n4 = n >> 2;
    double acc = 0.0;
#pragma unroll 4
    for (long long i = t0; i < n4; i += stride)
    {
        const float4 v = a4[i];
        const double x = v.x, y = v.y, z = v.z, w = v.w;
        acc += ((x * x + y * y) + z * z) + w * w;
    }
    const long long r = (n4 << 2) + t0;
    if (r < n)
    {
        const double x = arr[r];
        acc += x * x;
    }
    return acc;
}
__global__ void __launch_bounds__(256) energyPartialKernel(Fields f, long long P, double eta2, double *part)
{
    __shared__ double red[8];
    const double se = (sumSquares(f.E[0], P) + sumSquares(f.E[1], P)) + sumSquares(f.E[2], P);
    const double sh = (sumSquares(f.H[0], P) + sumSquares(f.H[1], P)) + sumSquares(f.H[2], P);
    double s = se + sh * eta2;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        part[blockIdx.x] = t;
    }
}
__global__ void __launch_bounds__(256) energyFinalKernel(const double *part, int n, double *out)
{
    __shared__ double red[8];
    double t = 0.0;
    for (int b = threadIdx.x; b < n; b += blockDim.x) t += part[b];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
        *out = s;
    }
}

// ---- Mur boundary state ----------------------------------------------------
// Face planes: 0 x-faces Ey, 1 x-faces Ez, 2 y-faces Ex, 3 y-faces Ez,
// 4 z-faces Ex, 5 z-faces Ey. Plane position (q1, q2) over the two other
// axes; layers 0, 1, N-1, N along the face normal (N = grid size on it).
struct Mur
{
    int n1[6], n2[6];
    long long off[6];  // start of each plane's 4 layers in `snap`
    float *snap;
    float cMur;
};
__device__ __forceinline__ long long murIndex(const Dims &d, int F, int L, int q1, int q2)
{
    switch (F)
    {
    case 0: return d.iEy(L, q1, q2);
    case 1: return d.iEz(L, q1, q2);
    case 2: return d.iEx(q1, L, q2);
    case 3: return d.iEz(q1, L, q2);
    case 4: return d.iEx(q1, q2, L);
    default: return d.iEy(q1, q2, L);
    }
}
__device__ __forceinline__ float *murField(const Fields &f, int F)
{
    return (F == 0 || F == 5) ? f.E[1] : (F == 1 || F == 3) ? f.E[2] : f.E[0];
}
__device__ __forceinline__ int murN(const Dims &d, int F) { return F < 2 ? d.nx : F < 4 ? d.ny : d.nz; }

// A flat item index over planes [F0, F0 + NP) resolved to its plane F, the
// position (q1, q2), and that position's first layer in `snap` (with the
// layer stride pl). Unrolled so that the plane tables stay in parameter space.
struct MurAt
{
    int F, q1, q2;
    long long pl;
    float *s;
};
template <int F0, int NP>
__device__ __forceinline__ bool murItem(const Mur &m, unsigned t, MurAt *a)
{
    bool found = false;
#pragma unroll
    for (int p = F0; p < F0 + NP; ++p)
    {
        const unsigned n = (unsigned)m.n1[p] * (unsigned)m.n2[p];
        if (!found)
        {
            if (t < n)
            {
                found = true;
                a->F = p;
                a->q2 = (int)(t / (unsigned)m.n1[p]);
                a->q1 = (int)(t - (unsigned)a->q2 * (unsigned)m.n1[p]);
                a->pl = n;
                a->s = m.snap + m.off[p] + (long long)a->q2 * m.n1[p] + a->q1;
            }
            else
                t -= n;
        }
    }
    return found;
}

// Copy of layers 0, 1, N-1, N of every face plane, taken before the E
// update (it runs as extra blocks of the H update, which leaves E unchanged).
__device__ __forceinline__ void murSnapItem(const Fields &f, const Dims &d, const Mur &m, unsigned t)
{
    MurAt a;
    if (!murItem<0, 6>(m, t, &a)) return;
    const int N = murN(d, a.F);
    const float *E = murField(f, a.F);
    const float e0 = E[murIndex(d, a.F, 0, a.q1, a.q2)], e1 = E[murIndex(d, a.F, 1, a.q1, a.q2)];
    const float e2 = E[murIndex(d, a.F, N - 1, a.q1, a.q2)], e3 = E[murIndex(d, a.F, N, a.q1, a.q2)];
    a.s[0] = e0;
    a.s[a.pl] = e1;
    a.s[2 * a.pl] = e2;
    a.s[3 * a.pl] = e3;
}

// ---- 3. H update (FdtdSolver.cpp:449-484) and the Mur snapshot ------------
// One thread per Yee cell (i, j, k) of the (nx+1) x (ny+1) x (nz+1) index
// box, flattened (x fastest) so that no block is padded per row.
struct Box
{
    unsigned total;
    tlmk::FastDiv divX, divY;  // by nx + 1 and ny + 1
};
__device__ __forceinline__ bool boxCell(const Box &b, const Dims &d, int *i, int *j, int *k)
{
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= b.total) return false;
    const unsigned r = tlmk::fastDiv(t, b.divX);
    *i = (int)(t - r * (unsigned)(d.nx + 1));
    const unsigned kk = tlmk::fastDiv(r, b.divY);
    *j = (int)(r - kk * (unsigned)(d.ny + 1));
    *k = (int)kk;
    return true;
}

// Every load of the thread is issued before its first store (the three H
// components share E operands: 9 distinct E loads and 3 H loads), so one
// memory round trip covers the cell. Operation order per component is the
// reference's.
__global__ void __launch_bounds__(256) updateHKernel(Fields f, Dims d, Box b, float ch, Mur m, unsigned hBlocks)
{
    if (blockIdx.x >= hBlocks)
    {
        murSnapItem(f, d, m, (blockIdx.x - hBlocks) * blockDim.x + threadIdx.x);
        return;
    }
    int i, j, k;
    if (!boxCell(b, d, &i, &j, &k)) return;
    const float *__restrict__ Ex = f.E[0];
    const float *__restrict__ Ey = f.E[1];
    const float *__restrict__ Ez = f.E[2];
    const bool ax = j < d.ny && k < d.nz, ay = i < d.nx && k < d.nz, az = i < d.nx && j < d.ny;
    float hx = 0.f, hy = 0.f, hz = 0.f;
    float ez0 = 0.f, ezj = 0.f, ezi = 0.f, ey0 = 0.f, eyk = 0.f, eyi = 0.f, ex0 = 0.f, exk = 0.f, exj = 0.f;
    const unsigned q = d.q(i, j, k), qj = q + (unsigned)d.px, qk = q + (unsigned)d.px * (unsigned)(d.ny + 1);
    if (ax)
    {
        hx = f.H[0][q];
        ezj = Ez[qj];
        eyk = Ey[qk];
    }
    if (ay)
    {
        hy = f.H[1][q];
        exk = Ex[qk];
        ezi = Ez[q + 1];
    }
    if (az)
    {
        hz = f.H[2][q];
        eyi = Ey[q + 1];
        exj = Ex[qj];
    }
    if (ax || ay) ez0 = Ez[q];
    if (ax || az) ey0 = Ey[q];
    if (ay || az) ex0 = Ex[q];
    if (ax) f.H[0][q] = hx - ch * ((ezj - ez0) - (eyk - ey0));
    if (ay) f.H[1][q] = hy - ch * ((exk - ex0) - (ezi - ez0));
    if (az) f.H[2][q] = hz - ch * ((eyi - ey0) - (exj - ex0));
}

// The coefficients of an edge of class c at index q.
__device__ __forceinline__ float2 edgeCoef(const Fields &f, const float2 *tab, int comp, unsigned c, long long q)
{
    return c == kEdgeMixed ? make_float2(f.ca[comp][q], f.cb[comp][q]) : tab[c];
}

// E update of the interior edges (FdtdSolver.cpp:487-555), in place. As for
// H, the loads (classes, 6 distinct H values shared by the three components,
// the edges' own E) come before the stores. The update ca*E + cb*curl with the
// air class's ca = 1 is the reference's E + cb0*curl.
__global__ void __launch_bounds__(256) updateEKernel(Fields f, Dims d, Box b)
{
    int i, j, k;
    if (!boxCell(b, d, &i, &j, &k)) return;
    const float *__restrict__ Hx = f.H[0];
    const float *__restrict__ Hy = f.H[1];
    const float *__restrict__ Hz = f.H[2];
    const bool ix = i >= 1 && i < d.nx, jy = j >= 1 && j < d.ny, kz = k >= 1 && k < d.nz;
    const bool ax = i < d.nx && jy && kz, ay = ix && j < d.ny && kz, az = ix && jy && k < d.nz;
    if (!ax && !ay && !az) return;
    const unsigned q = d.q(i, j, k), qj = q - (unsigned)d.px, qk = q - (unsigned)d.px * (unsigned)(d.ny + 1);
    const unsigned c = f.cls[q];
    float ex = 0.f, ey = 0.f, ez = 0.f;
    float hzj = 0.f, hzi = 0.f, hyk = 0.f, hyi = 0.f, hxk = 0.f, hxj = 0.f;
    if (ax)
    {
        ex = f.E[0][q];
        hzj = Hz[qj];
        hyk = Hy[qk];
    }
    if (ay)
    {
        ey = f.E[1][q];
        hxk = Hx[qk];
        hzi = Hz[q - 1];
    }
    if (az)
    {
        ez = f.E[2][q];
        hyi = Hy[q - 1];
        hxj = Hx[qj];
    }
    const float hx0 = Hx[q], hy0 = Hy[q], hz0 = Hz[q];
    if (ax)
    {
        const unsigned cl = edgeClass(c, 0);
        const float2 co = edgeCoef(f, f.tab, 0, cl, q);
        const float curl = (hz0 - hzj) - (hy0 - hyk);
        f.E[0][q] = cl == kEdgePec ? 0.0f : co.x * ex + co.y * curl;
    }
    if (ay)
    {
        const unsigned cl = edgeClass(c, 1);
        const float2 co = edgeCoef(f, f.tab, 1, cl, q);
        const float curl = (hx0 - hxk) - (hz0 - hzi);
        f.E[1][q] = cl == kEdgePec ? 0.0f : co.x * ey + co.y * curl;
    }
    if (az)
    {
        const unsigned cl = edgeClass(c, 2);
        const float2 co = edgeCoef(f, f.tab, 2, cl, q);
        const float curl = (hy0 - hyi) - (hx0 - hxj);
        f.E[2][q] = cl == kEdgePec ? 0.0f : co.x * ez + co.y * curl;
    }
}

// Mur on planes [F0, F0 + 3): per plane position the low face, then the high
// face (FdtdSolver.cpp:624-670): E_b = E_1(old) + cMur (E_1(new) - E_b(old)).
template <int F0>
__global__ void murApplyKernel(Fields f, Dims d, Mur m)
{
    MurAt a;
    if (!murItem<F0, 3>(m, blockIdx.x * blockDim.x + threadIdx.x, &a)) return;
    const int N = murN(d, a.F);
    float *E = murField(f, a.F);
    const long long b0 = murIndex(d, a.F, 0, a.q1, a.q2), b1 = murIndex(d, a.F, 1, a.q1, a.q2);
    const long long bN = murIndex(d, a.F, N, a.q1, a.q2), bN1 = murIndex(d, a.F, N - 1, a.q1, a.q2);
    const float s0 = a.s[0], s1 = a.s[a.pl], s2 = a.s[2 * a.pl], s3 = a.s[3 * a.pl];
    const float e1 = E[b1], eN1 = E[bN1];
    E[b0] = s1 + m.cMur * (e1 - s0);
    E[bN] = s2 + m.cMur * (eN1 - s3);
}

// ---- 3 and 4 in one pass ---------------------------------------------------
// A block owns a column of TX x TY cells and walks a range of z planes. On
// every plane it computes the new H of the column and of the ring below it in
// x and y (the ring is computed by the neighbouring blocks as well), hands it
// to the block through shared memory (two buffers, one barrier per plane), and
// computes the new E from it and from the H of the plane below, which each
// thread keeps in registers. A thread owns two x-neighbours (packed FP32x2
// arithmetic, bitwise the scalar operations).
// The input planes come in by tensor-map bulk copies, three boxes per plane:
// Ex and Ey one plane ahead, Ez, and H. A stage's Ex and Ey serve two planes
// (as the plane above, then as the plane itself), so a stage is refilled two
// planes after its own; with three stages the next plane is always in flight.
// Per cell and step this reads E, H and one class word and writes E and H: 52
// bytes, against 99 for two sweeps with per-edge coefficients. Planes whose
// edges are all air (a flag per column and plane) read no classes.
template <int W_, int H_> struct FusedLayout
{
    static constexpr int W = W_, H = H_;  // pairs x rows of threads: the column and its ring
    static constexpr int maxTX = 2 * (W - 1) / 4 * 4, maxTY = H - 1;
    static constexpr int kThreads = (W * H + 31) / 32 * 32, kStages = 3;
    // a stage row holds the W2 cells from x0-4 on (16-byte aligned box starts); floats
    static constexpr int W2 = (2 * W + 4 + 3) / 4 * 4;
    static constexpr int round32(int f) { return (f + 31) / 32 * 32; }  // boxes start on 128-byte boundaries
    static constexpr int sE = (H + 1) * W2, sH = H * W2;
    static constexpr int offEz = round32(2 * sE), offH = offEz + round32(sE), stage = offH + round32(3 * sH);
    static constexpr unsigned stageBytes = (unsigned)(3 * sE + 3 * sH) * 4u;
    static constexpr int WE = 2 * W, slot = H * WE;  // exchange row and slot
    static constexpr int offEx = kStages * stage, offTab = offEx + 2 * 3 * slot;
    static constexpr int smemBytes = (offTab + 2 * kEdgeClasses) * 4;
    static constexpr int kFit = 227 * 1024 / (smemBytes + 1280);
    static constexpr int kMinBlocks = 1024 / kThreads < kFit ? 1024 / kThreads : kFit;
    static_assert(kMinBlocks >= 1, "a block fits an SM");
};
struct FusedArgs
{
    CUtensorMap mapExy, mapEz, mapH;  // boxes of the input buffer
    Fields in;
    float *out;       // Ex Ey Ez Hx Hy Hz planes of P values each
    long long P;
    Dims d;
    int TX, TY, ntx, nty, nchunk;
    const unsigned char *flags;  // [column][nz + 1]: some edge is not air
    float ch, cb0, neg_zero;
    unsigned *fault;
};

using tlmk::add2;
using tlmk::ld2;
using tlmk::mul2;
using tlmk::splat2;
using tlmk::sub2;

template <class L> __global__ void __launch_bounds__(L::kThreads, L::kMinBlocks) fusedStepKernel(const __grid_constant__ FusedArgs a)
{
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(8) unsigned long long full[L::kStages];
    const Dims &d = a.d;
    const int tid = threadIdx.x;
    const int ncol = a.ntx * a.nty;
    const int col = blockIdx.x % ncol, chunk = blockIdx.x / ncol;
    const int planes = d.nz + 1;
    const int kc0 = (int)((long long)chunk * planes / a.nchunk), kc1 = (int)((long long)(chunk + 1) * planes / a.nchunk);
    const int kA = kc0 > 0 ? kc0 - 1 : 0;
    const int x0 = (col % a.ntx) * a.TX, y0 = (col / a.ntx) * a.TY;
    const unsigned full0 = tlmk::smemAddr(full), sm0 = tlmk::smemAddr(sm);
    if (tid == 0)
    {
        for (int s = 0; s < L::kStages; ++s)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" : : "r"(full0 + 8 * s) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" : : : "memory");
    }
    float2 *const tab = reinterpret_cast<float2 *>(sm + L::offTab);
    for (int t = tid; t < (int)kEdgeClasses; t += L::kThreads) tab[t] = a.in.tab[t];
    __syncthreads();
    // stage of plane k (k from kA-1: only its Ex and Ey, those of plane kA, are used)
    auto issue = [&](int k) {
        const int s = (k - kA + 1) % L::kStages;
        const unsigned st = sm0 + (unsigned)(s * L::stage) * 4u, bar = full0 + 8 * s;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" : : "r"(bar), "r"(L::stageBytes) : "memory");
        tlmk::tmaBox4(st, &a.mapExy, x0 - 4, y0 - 1, k + 1, 0, bar);
        tlmk::tmaBox4(st + L::offEz * 4u, &a.mapEz, x0 - 4, y0 - 1, k, 2, bar);
        tlmk::tmaBox4(st + L::offH * 4u, &a.mapH, x0 - 4, y0 - 1, k, 3, bar);
    };
    int lastIssued = kA - 2;  // thread 0's
    if (tid == 0)
        while (lastIssued < kc1 - 1 && lastIssued < kA - 2 + L::kStages) issue(++lastIssued);

    const int r = tid / L::W, p = tid - r * L::W;
    const bool inTile = r < L::H;
    const int i = x0 - 2 + 2 * p, j = y0 - 1 + r;
    const bool own = inTile && p >= 1 && p <= a.TX / 2 && r >= 1 && r <= a.TY && i <= d.nx && j <= d.ny;
    const unsigned off = own ? (unsigned)j * (unsigned)d.px + (unsigned)i : 0u;
    const long long sz = (long long)d.px * (d.ny + 1);
    const unsigned char *flags = a.flags + (long long)col * planes;
    const bool i0 = i < d.nx, i1 = i + 1 < d.nx, up = j < d.ny;
    const bool jy = j >= 1 && up;
    // which of the pair's edges the E update writes (z conditions apart): bit
    // 2*component + node
    const bool iy = i >= 1 && up;
    const unsigned eMask = (i0 && jy ? 1u : 0u) | (i1 && jy ? 2u : 0u) | (iy && i0 ? 4u : 0u) | (up && i1 ? 8u : 0u) |
                           (i >= 1 && i0 && jy ? 16u : 0u) | (i1 && jy ? 32u : 0u);
    const float2 z = splat2(a.neg_zero), ch = splat2(a.ch);
    const int o = inTile ? r * L::W2 + 2 * p + 2 : 2;       // in a stage
    const int e0 = L::offEx + (inTile ? r * L::WE + 2 * p : 0);  // in an exchange buffer
    const float2 zero = make_float2(0.f, 0.f);
    float2 hxP = zero, hyP = zero;  // new H of the plane below
    bool waitOk = true;
    int sPrev = 0, sCur = 0;
    unsigned phase = 0;
    auto wait = [&]() {  // for the stage sCur
        if (waitOk && !tlmk::mbarWaitBounded(full0 + 8 * sCur, phase))
        {
            waitOk = false;
            *reinterpret_cast<volatile unsigned *>(a.fault) = tlmk::kStageTimeout;
        }
    };
    wait();
    sCur = 1;
    uint2 cNext = make_uint2(0, 0);
    // classes one plane ahead, the flags that say whether there are any three
    auto flagAt = [&](int k) -> unsigned { return k < kc1 ? flags[k] : 0u; };
    auto classesAt = [&](int k, unsigned f) -> uint2 {
        return f && own ? *reinterpret_cast<const uint2 *>(reinterpret_cast<const char *>(a.in.cls + k * sz) + off * 4u)
                        : make_uint2(0, 0);
    };
    unsigned f0 = flagAt(kA), f1 = flagAt(kA + 1), f2 = flagAt(kA + 2);
    cNext = classesAt(kA, f0);
    // lanes with cells at the high x and y faces, where some entries do not exist
    const bool warpHigh = __any_sync(0xffffffffu, !i1 || !up);
    for (int k = kA; k < kc1; ++k)
    {
        const bool kz = k < d.nz;
        const unsigned f3 = flagAt(k + 3);
        const uint2 c = cNext;
        cNext = classesAt(k + 1, f1);
        wait();
        const float *prev = sm + sPrev * L::stage, *st = sm + sCur * L::stage;
        // ---- H (FdtdSolver.cpp:449-484) ----
        const float2 ex = ld2(prev + o), ey = ld2(prev + L::sE + o), ez = ld2(st + L::offEz + o);
        const float2 exj = ld2(prev + o + L::W2), ezj = ld2(st + L::offEz + o + L::W2);
        const float2 ey1 = make_float2(prev[L::sE + o + 1], prev[L::sE + o + 2]);
        const float2 ez1 = make_float2(st[L::offEz + o + 1], st[L::offEz + o + 2]);
        const float2 exk = ld2(st + o), eyk = ld2(st + L::sE + o);
        float2 hx = ld2(st + L::offH + o), hy = ld2(st + L::offH + L::sH + o), hz = ld2(st + L::offH + 2 * L::sH + o);
        hx = sub2(hx, mul2(ch, sub2(sub2(ezj, ez), sub2(eyk, ey)), z));
        hy = sub2(hy, mul2(ch, sub2(sub2(exk, ex), sub2(ez1, ez)), z));
        hz = sub2(hz, mul2(ch, sub2(sub2(ey1, ey), sub2(exj, ex)), z));
        // entries a component does not have stay zero
        if (warpHigh || !kz)
        {
            if (!up || !kz) hx = zero;
            if (!up) hz = zero;
            if (!kz) hy = zero;
            if (!i0) hy.x = hz.x = 0.f;
            if (!i1) hy.y = hz.y = 0.f;
            if (i >= d.nx) hx.y = 0.f;
        }
        float *const xb = sm + (k & 1) * 3 * L::slot + e0;
        if (inTile)
        {
            *reinterpret_cast<float2 *>(xb) = hx;
            *reinterpret_cast<float2 *>(xb + L::slot) = hy;
            *reinterpret_cast<float2 *>(xb + 2 * L::slot) = hz;
        }
        __syncthreads();
        // every thread is past its reads of the stage before this one's
        if (tid == 0 && waitOk && lastIssued < kc1 - 1 && lastIssued < k + L::kStages - 1) issue(++lastIssued);
        if (own && k >= kc0)
        {
            // uniform plane pointers and a 32-bit lane offset
            char *const out = reinterpret_cast<char *>(a.out + k * sz);
            auto store = [&](int comp, float2 v) { *reinterpret_cast<float2 *>(out + comp * a.P * 4 + off * 4u) = v; };
            store(3, hx);
            store(4, hy);
            store(5, hz);
            // ---- E of the interior edges (FdtdSolver.cpp:487-555) ----
            const float2 hxj = ld2(xb - L::WE), hzj = ld2(xb + 2 * L::slot - L::WE);
            const float2 hyi = make_float2(xb[L::slot - 1], xb[L::slot]);
            const float2 hzi = make_float2(xb[2 * L::slot - 1], xb[2 * L::slot]);
            const float2 cx = sub2(sub2(hz, hzj), sub2(hy, hyP));
            const float2 cy = sub2(sub2(hx, hxP), sub2(hz, hzi));
            const float2 cz = sub2(sub2(hy, hyi), sub2(hx, hxj));
            float2 nx, ny, nz;
            const unsigned l = edgeClass(c.x, 0);
            if (!f0)
            {
                const float2 cb = splat2(a.cb0);
                nx = add2(ex, mul2(cb, cx, z));
                ny = add2(ey, mul2(cb, cy, z));
                nz = add2(ez, mul2(cb, cz, z));
            }
            else if (c.x == c.y && c.x == edgeWord(l) && l - 1u < kEdgeMixed - 1u)
            {
                // all six edges inside one material
                const float2 co = tab[l], ca = splat2(co.x), cb = splat2(co.y);
                nx = add2(mul2(ca, ex, z), mul2(cb, cx, z));
                ny = add2(mul2(ca, ey, z), mul2(cb, cy, z));
                nz = add2(mul2(ca, ez, z), mul2(cb, cz, z));
            }
            else
            {
                auto update = [&](int comp, float2 e, float2 curl) -> float2 {
                    const unsigned l0 = edgeClass(c.x, comp), l1 = edgeClass(c.y, comp);
                    const long long q = k * sz + off;
                    const float2 k0 = edgeCoef(a.in, tab, comp, l0, q), k1 = edgeCoef(a.in, tab, comp, l1, q + 1);
                    float2 v = add2(mul2(make_float2(k0.x, k1.x), e, z), mul2(make_float2(k0.y, k1.y), curl, z));
                    if (l0 == kEdgePec) v.x = 0.f;
                    if (l1 == kEdgePec) v.y = 0.f;
                    return v;
                };
                nx = update(0, ex, cx);
                ny = update(1, ey, cy);
                nz = update(2, ez, cz);
            }
            // boundary edges are written by the Mur kernel
            const bool kin = k >= 1 && kz;
            if (eMask == 63u && kin)
            {
                store(0, nx);
                store(1, ny);
                store(2, nz);
            }
            else
            {
                auto masked = [&](int comp, float2 v) {
                    const unsigned m = (eMask >> (2 * comp)) & 3u;
                    if (m) store(comp, make_float2((m & 1u) ? v.x : 0.f, (m & 2u) ? v.y : 0.f));
                };
                if (kin)
                {
                    masked(0, nx);
                    masked(1, ny);
                }
                if (kz) masked(2, nz);
            }
        }
        f0 = f1;
        f1 = f2;
        f2 = f3;
        hxP = hx;
        hyP = hy;
        sPrev = sCur;
        if (++sCur == L::kStages)
        {
            sCur = 0;
            phase ^= 1u;
        }
    }
    // Thread 0 waited for every copy, unless a wait ran out: then let those
    // still in flight land before the block's memory goes.
    if (!waitOk && tid == 0)
        for (int k = max(kA - 1, lastIssued - L::kStages + 1); k <= lastIssued; ++k)
            tlmk::mbarWaitBounded(full0 + 8 * ((k - kA + 1) % L::kStages),
                                  (unsigned)((k - kA + 1) / L::kStages) & 1u);
}

// Mur on all faces at once, from the old values `o` (input buffer) and the
// fused pass's new interior edges `n` (FdtdSolver.cpp:624-670). The reference
// runs the face planes one after the other and a later one overwrites the edges
// it shares with an earlier one, from an inner neighbour that the earlier one
// may have set: an edge of two faces takes the later face's formula here, with
// the earlier face's where the inner neighbour lies on that.
__device__ __forceinline__ float murStep(const float *o, const float *n, long long b, long long inner, float c)
{
    return o[inner] + c * (n[inner] - o[b]);
}
__device__ __forceinline__ void murFaceItem(const float *oldE, float *newE, long long P, const Dims &d, const Mur &m,
                                            unsigned t)
{
    MurAt a;
    if (!murItem<0, 6>(m, t, &a)) return;
    const int comp = (a.F == 0 || a.F == 5) ? 1 : (a.F == 1 || a.F == 3) ? 2 : 0;
    const float *o = oldE + comp * P;
    float *n = newE + comp * P;
    // planes 0, 1, 2 leave the edges that a later plane of their component
    // sets: (q1, q2) is (j, k) on planes 0, 1 and (i, k) on plane 2
    if (a.F == 0 && (a.q2 == 0 || a.q2 == d.nz)) return;
    if (a.F == 1 && (a.q1 == 0 || a.q1 == d.ny)) return;
    if (a.F == 2 && (a.q2 == 0 || a.q2 == d.nz)) return;
    const int N = murN(d, a.F);
    for (int side = 0; side < 2; ++side)
    {
        const int b = side ? N : 0, q = side ? N - 1 : 1;
        const long long ib = murIndex(d, a.F, b, a.q1, a.q2), iq = murIndex(d, a.F, q, a.q1, a.q2);
        float v1;
        if (a.F == 3 && (a.q1 == 0 || a.q1 == d.nx))  // inner edge on an x face (plane 1)
            v1 = murStep(o, n, iq, d.iEz(a.q1 == 0 ? 1 : d.nx - 1, q, a.q2), m.cMur);
        else if (a.F == 4 && (a.q2 == 0 || a.q2 == d.ny))  // on a y face (plane 2)
            v1 = murStep(o, n, iq, d.iEx(a.q1, a.q2 == 0 ? 1 : d.ny - 1, q), m.cMur);
        else if (a.F == 5 && (a.q1 == 0 || a.q1 == d.nx))  // on an x face (plane 0)
            v1 = murStep(o, n, iq, d.iEy(a.q1 == 0 ? 1 : d.nx - 1, a.q2, q), m.cMur);
        else
            v1 = n[iq];
        n[ib] = o[iq] + m.cMur * (v1 - o[ib]);
    }
}

// What follows the fused pass of a step, in one launch: Mur on the new fields,
// the step's monitors, which read the old ones, and, where none of the source
// edges lies on an outer face or next to one (so that Mur does not read them),
// the next step's sources.
struct TailArgs
{
    const float *oldE;
    float *newE;
    long long P;
    Mur mur;
    MonArgs mon;
    InjectArgs inj;
    unsigned murBlocks, monBlocks;
};
__global__ void __launch_bounds__(256) stepTailKernel(const __grid_constant__ TailArgs a)
{
    if (blockIdx.x < a.murBlocks)
        murFaceItem(a.oldE, a.newE, a.P, a.mon.d, a.mur, blockIdx.x * blockDim.x + threadIdx.x);
    else if (blockIdx.x < a.murBlocks + a.monBlocks)
        monitorItem(a.mon, (long long)(blockIdx.x - a.murBlocks) * blockDim.x + threadIdx.x);
    else
        injectItem(a.inj, (int)((blockIdx.x - a.murBlocks - a.monBlocks) * blockDim.x + threadIdx.x));
}

// ---- edge classes (FdtdSolver.cpp:135-231) ---------------------------------
// A free table entry: (ca, cb) = (NaN, NaN), which no edge has.
constexpr unsigned long long kEdgeFree = ~0ull;

// One thread per cell of the index box: the classes of its three edges, and
// the coefficients of those between materials, from the four cells around each (summed
// in the reference's order). Edges on the outer boundary are not updated from
// their classes.
__global__ void __launch_bounds__(256) edgeClassKernel(const uint8_t *__restrict__ mat, const float2 *__restrict__ props,
                                                       Dims d, Box b, float dt, float dl, float eps0, unsigned *cls,
                                                       unsigned long long *tab,
                                                       float *ca0, float *ca1, float *ca2, float *cb0, float *cb1,
                                                       float *cb2)
{
    int i, j, k;
    if (!boxCell(b, d, &i, &j, &k)) return;
    unsigned word = 0;
#pragma unroll
    for (int axis = 0; axis < 3; ++axis)
    {
        unsigned c = kEdgeAir;
        const int co[3] = { i, j, k };
        const int n[3] = { d.nx, d.ny, d.nz };
        const int t1 = axis == 0 ? 1 : 0, t2 = axis == 2 ? 1 : 2;
        if (co[axis] < n[axis] && co[t1] >= 1 && co[t1] < n[t1] && co[t2] >= 1 && co[t2] < n[t2])
        {
            uint8_t m[4];
            bool pec = false, same = true;
#pragma unroll
            for (int t = 0; t < 4; ++t)
            {
                int q[3] = { i, j, k };
                q[t1] -= t < 2 ? 1 : 0;
                q[t2] -= (t & 1) ? 0 : 1;
                m[t] = mat[((size_t)q[2] * d.ny + q[1]) * d.nx + q[0]];
                pec = pec || m[t] == TLM_MAT_PEC;
                same = same && m[t] == m[0];
            }
            if (pec)
                c = kEdgePec;
            else if (same)
                c = m[0] == TLM_MAT_AIR ? kEdgeAir : m[0];
            else
            {
                float e = 0.0f, s = 0.0f;
#pragma unroll
                for (int t = 0; t < 4; ++t)
                {
                    const float2 pr = m[t] >= TLM_MAT_DIEL0 ? props[m[t] - TLM_MAT_DIEL0] : make_float2(1.0f, 0.0f);
                    e += m[t] >= TLM_MAT_DIEL0 ? 1.0f + (pr.x - 1.0f) : 1.0f;
                    s += pr.y;
                }
                const float er = e / 4.0f, sg = s / 4.0f;
                const float eps = eps0 * (1.0f < er ? er : 1.0f);
                const float lf = sg * dt / (2.0f * eps);
                const float ca = (1.0f - lf) / (1.0f + lf), cb = (dt / (eps * dl)) / (1.0f + lf);
                // this pair's entry in the table, a new one if there is room
                const unsigned long long key = (unsigned long long)__float_as_uint(cb) << 32 | __float_as_uint(ca);
                c = kEdgeMixed;
                constexpr unsigned kRoom = kEdgeMixed - kEdgeFirst;
                const unsigned start = tlmk::mix32((unsigned)(key ^ (key >> 32))) % kRoom;
                for (unsigned u = 0; u < kRoom; ++u)
                {
                    const unsigned t = kEdgeFirst + (start + u) % kRoom;
                    unsigned long long old = reinterpret_cast<volatile unsigned long long *>(tab)[t];
                    if (old == kEdgeFree) old = atomicCAS(tab + t, kEdgeFree, key);
                    if (old == kEdgeFree || old == key)
                    {
                        c = t;
                        break;
                    }
                }
                if (c == kEdgeMixed)
                {
                    const long long q = d.at(i, j, k);
                    (axis == 0 ? ca0 : axis == 1 ? ca1 : ca2)[q] = ca;
                    (axis == 0 ? cb0 : axis == 1 ? cb1 : cb2)[q] = cb;
                }
            }
        }
        word |= c << (10 * axis);
    }
    cls[d.at(i, j, k)] = word;
}
// Columns and planes that hold an edge that is not air.
__global__ void __launch_bounds__(128) edgeFlagKernel(const unsigned *__restrict__ cls, Dims d, int TX, int TY, int ntx,
                                                      unsigned char *flags)
{
    const int k = blockIdx.x % (d.nz + 1), col = blockIdx.x / (d.nz + 1);
    const int xa = (col % ntx) * TX, ya = (col / ntx) * TY;
    const int w = min(TX, d.nx + 1 - xa), hgt = min(TY, d.ny + 1 - ya);
    const unsigned air = edgeWord(kEdgeAir);
    bool other = false;
    for (int t = threadIdx.x; t < w * hgt; t += blockDim.x)
        other = other || cls[d.at(xa + t % w, ya + t / w, k)] != air;
    other = __syncthreads_or(other);
    if (threadIdx.x == 0) flags[blockIdx.x] = other ? 1 : 0;
}

// `count` values, from the one numbered `first` on, of a component of extents n
// in the reference's layout (x fastest, no padding).
__global__ void __launch_bounds__(256) packFieldKernel(const float *__restrict__ f, Dims d, int n0, int n1, long long first,
                                                       long long count, float *__restrict__ out)
{
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < count;
         t += (long long)gridDim.x * blockDim.x)
    {
        const int i = (int)((first + t) % n0);
        const long long r = (first + t) / n0;
        out[t] = f[d.at(i, (int)(r % n1), (int)(r / n1))];
    }
}

} // namespace fdk

// ---------------------------------------------------------------------------
struct FdtdMaps
{
    CUtensorMap map[2][3];  // per field buffer: Ex and Ey, Ez, H
};
struct fdtd_solver
{
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaMemPool_t pool = nullptr;
    std::string err;
    bool configured = false;
    tlm_grid g{};
    tlm_config cfg{};
    tlmh::HostMap mat;
    std::vector<tlm_matprops> table;
    fdk::Dims d{};
    float dt = 0, cMur = 0, cb0 = 0, ch = 0;
    bool haveDiel = false;
    long long len[6] = {};       // Ex Ey Ez Hx Hy Hz lengths in the reference's layout
    long long P = 0;             // entries of a component's plane set (padded pitch)
    float *dBuf[2] = {};         // field buffers of 6 P values; the second only for fused passes
    int cur = 0;                 // buffer holding the current state
    unsigned *dCls = nullptr;    // edge classes
    float2 *dTab = nullptr;      // their coefficients
    float *dCa[3] = {}, *dCb[3] = {};  // of mixed edges
    unsigned char *dFlags = nullptr;   // [column][plane] of the fused pass
    unsigned *fault = nullptr;         // a bulk copy's wait ran out (a FaultWord)
    std::unique_ptr<FdtdMaps> maps;    // boxes of the fused pass in either buffer
    int layout = 0, TX = 0, TY = 0, ntx = 0, nty = 0, nchunk = 0;
    fdk::Mur mur{};
    float *field(int c) const { return dBuf[cur] + c * P; }
    tlmi::Lender lender;    // the second field buffer
    bool planning = false;  // allocating it
    bool lent = false;      // given back since set-up
    // sources
    struct Src
    {
        uint64_t cell;
        int pol;
        float amp;
    };
    std::vector<Src> planeSources;
    struct Port
    {
        std::vector<uint64_t> cells;
        int pol;
        float amp;
    };
    std::vector<Port> ports;
    std::vector<uint64_t> probeCells;
    std::vector<float> svTable;
    bool prepared = false;
    long long *dEdge = nullptr;
    int *dEdgeOff = nullptr;
    float *dAmps = nullptr;
    int nEdges = 0;
    bool edgesInside = false;  // no source edge on an outer face or one cell from it
    bool injected = false;     // the current state holds the next step's sources already
    int *dPoff = nullptr, *dPpol = nullptr;
    long long *dPcells = nullptr, *dProbe = nullptr;
    float *dVrec = nullptr, *dIrec = nullptr, *dPrec = nullptr;
    double *dEhist = nullptr, *dEpart = nullptr;
    long long recCap = 0;
    int nEpart = 0;
    SurfaceState surf;
    int curStep = 0;
    std::vector<void *> allocs;

    // whether the edge of component c at (i, j, k) touches no PEC cell
    bool freeEdge(int c, int i, int j, int k) const
    {
        const int t1 = c == 0 ? 1 : 0, t2 = c == 2 ? 1 : 2;
        const int n[3] = { d.nx, d.ny, d.nz };
        for (int d1 = -1; d1 <= 0; ++d1)
            for (int d2 = -1; d2 <= 0; ++d2)
            {
                int co[3] = { i, j, k };
                co[t1] += d1;
                co[t2] += d2;
                bool in = true;
                for (int a = 0; a < 3; ++a) in = in && co[a] >= 0 && co[a] < n[a];
                if (in && mat[((size_t)co[2] * d.ny + co[1]) * d.nx + co[0]] == TLM_MAT_PEC) return false;
            }
        return true;
    }
    tlm_status fail(tlm_status s, const std::string &m)
    {
        err = m;
        return s;
    }
    tlm_status cuda(cudaError_t e, const char *what)
    {
        if (e == cudaSuccess) return TLM_OK;
        cudaGetLastError();
        err = std::string(what) + ": " + cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? TLM_ENOMEM : TLM_ECUDA;
    }
};

namespace {

thread_local std::string g_fdtdErr;

#define FD_TRY(x)                                                                                                      \
    do                                                                                                                 \
    {                                                                                                                  \
        tlm_status s_ = (x);                                                                                           \
        if (s_ != TLM_OK) return s_;                                                                                   \
    } while (0)
#define FD_CU(h, call) FD_TRY((h)->cuda((call), #call))

struct Guard
{
    int prev = -1;
    explicit Guard(int dev)
    {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev != dev) cudaSetDevice(dev);
    }
    ~Guard()
    {
        int cur = -1;
        if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
    }
};

template <class T> tlm_status alloc(fdtd_solver *h, T **p, size_t bytes)
{
    void *q = nullptr;
    cudaError_t e = tlmi::poolAlloc(h->device, h->pool, h->stream, h->planning, &q, std::max<size_t>(bytes, 1));
    if (e != cudaSuccess)
    {
        cudaGetLastError();
        return h->fail(TLM_ENOMEM, "device allocation of " + std::to_string(bytes) + " bytes failed");
    }
    *p = static_cast<T *>(q);
    return TLM_OK;
}
template <class T> void release(fdtd_solver *h, T *&p)
{
    if (p) cudaFreeAsync((void *)p, h->stream);
    p = nullptr;
}

void freeMonitors(fdtd_solver *h)
{
    release(h, h->dEdge);
    release(h, h->dEdgeOff);
    release(h, h->dAmps);
    release(h, h->dPoff);
    release(h, h->dPpol);
    release(h, h->dPcells);
    release(h, h->dProbe);
    release(h, h->dVrec);
    release(h, h->dIrec);
    release(h, h->dPrec);
    release(h, h->dEhist);
    release(h, h->dEpart);
    SurfaceState &s = h->surf;
    release(h, s.dJsNode);
    release(h, s.dHuyNode);
    release(h, s.dJsInst);
    release(h, s.dJsAcc);
    release(h, s.dHuyAcc);
    release(h, s.dPlane);
    release(h, s.dFrames);
    s.planeCap = 0;
    s.planeValid = false;
    s.framesCap = s.framesUsed = 0;
    s.frames.clear();
    h->recCap = 0;
    h->prepared = false;
}

// Words of pinned host memory that kernels report a fault in: the host reads one
// after the synchronisation that ends fdtd_step, where a copy of a device word
// cost 10 us per call. A page of them is allocated once for all devices and
// kept; handles beyond its words (null) step in place.
class FaultWords
{
  public:
    unsigned *take()
    {
        std::lock_guard<std::mutex> lk(mu_);
        if (!page_)
        {
            void *p = nullptr;
            if (cudaHostAlloc(&p, kWords * sizeof(unsigned), cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess)
                cudaGetLastError();
            page_ = static_cast<unsigned *>(p);
            if (page_)
                for (int w = 0; w < kWords; ++w) free_.push_back(page_ + w);
        }
        if (free_.empty()) return nullptr;
        unsigned *w = free_.back();
        free_.pop_back();
        *w = 0;
        return w;
    }
    void give(unsigned *w)
    {
        std::lock_guard<std::mutex> lk(mu_);
        free_.push_back(w);
    }

  private:
    static constexpr int kWords = 4096;
    std::mutex mu_;
    unsigned *page_ = nullptr;
    std::vector<unsigned *> free_;
};
FaultWords &faultWords()
{
    static FaultWords *words = new FaultWords;  // (handles may outlive static objects)
    return *words;
}

// The second field buffer and what else only fused passes need.
void dropFused(fdtd_solver *h)
{
    release(h, h->dBuf[1]);
    release(h, h->dFlags);
    if (h->fault)
    {
        cudaStreamSynchronize(h->stream);  // no kernel writes to it any more
        faultWords().give(h->fault);
    }
    h->fault = nullptr;
    h->maps.reset();
}

void freeAll(fdtd_solver *h)
{
    freeMonitors(h);
    dropFused(h);
    release(h, h->dBuf[0]);
    release(h, h->dCls);
    release(h, h->dTab);
    for (int c = 0; c < 3; ++c)
    {
        release(h, h->dCa[c]);
        release(h, h->dCb[c]);
    }
    release(h, h->mur.snap);
}

tlm_status ready(fdtd_solver *h)
{
    if (!h)
    {
        g_fdtdErr = "null handle";
        return TLM_EINVAL;
    }
    if (!h->configured) return h->fail(TLM_ESTATE, "fdtd_setup has not been called");
    return TLM_OK;
}

float sourceValue(const fdtd_solver *h, int n)
{
    if (h->cfg.waveform == TLM_WAVE_TABLE) return (n >= 0 && n < (int)h->svTable.size()) ? h->svTable[n] : 0.0f;
    return tlmh::waveform_f32(h->cfg.waveform, h->cfg.f0, h->dt, n);
}

tlm_status ensureRecords(fdtd_solver *h, long long need)
{
    if (need <= h->recCap) return TLM_OK;
    long long cap = std::max<long long>(need, std::max<long long>(h->cfg.total_steps, 64));
    cap = std::max(cap, h->recCap * 2);
    const int np = std::max<int>((int)h->ports.size(), 1), nr = std::max<int>((int)h->probeCells.size(), 1);
    float *v = nullptr, *i = nullptr, *p = nullptr;
    double *e = nullptr;
    FD_TRY(alloc(h, &v, (size_t)cap * np * 4));
    FD_TRY(alloc(h, &i, (size_t)cap * np * 4));
    FD_TRY(alloc(h, &p, (size_t)cap * nr * 3 * 4));
    FD_TRY(alloc(h, &e, (size_t)(cap / 16 + 2) * 8));
    if (h->recCap > 0)
    {
        FD_CU(h, cudaMemcpyAsync(v, h->dVrec, (size_t)h->recCap * np * 4, cudaMemcpyDeviceToDevice, h->stream));
        FD_CU(h, cudaMemcpyAsync(i, h->dIrec, (size_t)h->recCap * np * 4, cudaMemcpyDeviceToDevice, h->stream));
        FD_CU(h, cudaMemcpyAsync(p, h->dPrec, (size_t)h->recCap * nr * 12, cudaMemcpyDeviceToDevice, h->stream));
        FD_CU(h, cudaMemcpyAsync(e, h->dEhist, (size_t)(h->recCap / 16 + 2) * 8, cudaMemcpyDeviceToDevice,
                                 h->stream));
    }
    release(h, h->dVrec);
    release(h, h->dIrec);
    release(h, h->dPrec);
    release(h, h->dEhist);
    h->dVrec = v;
    h->dIrec = i;
    h->dPrec = p;
    h->dEhist = e;
    h->recCap = cap;
    return TLM_OK;
}

// Source edges in CSR form: every E edge a source cell drives, with its
// amplitudes in the reference's order (plane-wave cells, then port cells).
tlm_status prepare(fdtd_solver *h)
{
    if (h->prepared) return TLM_OK;
    freeMonitors(h);
    const fdk::Dims &d = h->d;
    std::map<long long, std::vector<float>> edges;  // per edge, amplitudes in source order
    auto add = [&](uint64_t cell, int pol, float amp) {
        const int i = (int)(cell % d.nx), j = (int)((cell / d.nx) % d.ny), k = (int)(cell / ((uint64_t)d.nx * d.ny));
        // the four edges along pol, by increasing second, then first transverse axis
        const int t1 = pol == 0 ? 1 : 0, t2 = pol == 2 ? 1 : 2;
        for (int e = 0; e < 4; ++e)
        {
            int co[3] = { i, j, k };
            co[t1] += e & 1;
            co[t2] += e >> 1;
            if (h->freeEdge(pol, co[0], co[1], co[2]))
                edges[((long long)pol << 60) | d.at(co[0], co[1], co[2])].push_back(amp);
        }
    };
    for (const auto &s : h->planeSources) add(s.cell, s.pol, s.amp);
    for (const auto &p : h->ports)
        for (uint64_t c : p.cells) add(c, p.pol, p.amp);
    std::vector<long long> code;
    std::vector<int> off(1, 0);
    std::vector<float> amps;
    for (const auto &kv : edges)
    {
        code.push_back(kv.first);
        amps.insert(amps.end(), kv.second.begin(), kv.second.end());
        off.push_back((int)amps.size());
    }
    h->nEdges = (int)code.size();
    h->edgesInside = true;
    for (long long c : code)
    {
        const long long idx = c & ((1LL << 60) - 1);
        const int co[3] = { (int)(idx % d.px), (int)(idx / d.px % (d.ny + 1)), (int)(idx / ((long long)d.px * (d.ny + 1))) };
        const int n[3] = { d.nx, d.ny, d.nz };
        for (int q = 0; q < 3; ++q) h->edgesInside = h->edgesInside && co[q] >= 2 && co[q] <= n[q] - 2;
    }
    if (h->nEdges)
    {
        FD_TRY(alloc(h, &h->dEdge, code.size() * 8));
        FD_TRY(alloc(h, &h->dEdgeOff, off.size() * 4));
        FD_TRY(alloc(h, &h->dAmps, amps.size() * 4));
        FD_CU(h, cudaMemcpyAsync(h->dEdge, code.data(), code.size() * 8, cudaMemcpyHostToDevice, h->stream));
        FD_CU(h, cudaMemcpyAsync(h->dEdgeOff, off.data(), off.size() * 4, cudaMemcpyHostToDevice, h->stream));
        FD_CU(h, cudaMemcpyAsync(h->dAmps, amps.data(), amps.size() * 4, cudaMemcpyHostToDevice, h->stream));
    }
    // ports and probes
    const int np = (int)h->ports.size();
    std::vector<int> poff(np + 1, 0), ppol(std::max(np, 1), 0);
    std::vector<long long> pcells;
    for (int p = 0; p < np; ++p)
    {
        for (uint64_t c : h->ports[p].cells) pcells.push_back((long long)c);
        poff[p + 1] = (int)pcells.size();
        ppol[p] = h->ports[p].pol;
    }
    if (pcells.empty()) pcells.push_back(0);
    std::vector<long long> probes(h->probeCells.begin(), h->probeCells.end());
    if (probes.empty()) probes.push_back(0);
    FD_TRY(alloc(h, &h->dPoff, poff.size() * 4));
    FD_TRY(alloc(h, &h->dPpol, ppol.size() * 4));
    FD_TRY(alloc(h, &h->dPcells, pcells.size() * 8));
    FD_TRY(alloc(h, &h->dProbe, probes.size() * 8));
    FD_CU(h, cudaMemcpyAsync(h->dPoff, poff.data(), poff.size() * 4, cudaMemcpyHostToDevice, h->stream));
    FD_CU(h, cudaMemcpyAsync(h->dPpol, ppol.data(), ppol.size() * 4, cudaMemcpyHostToDevice, h->stream));
    FD_CU(h, cudaMemcpyAsync(h->dPcells, pcells.data(), pcells.size() * 8, cudaMemcpyHostToDevice, h->stream));
    FD_CU(h, cudaMemcpyAsync(h->dProbe, probes.data(), probes.size() * 8, cudaMemcpyHostToDevice, h->stream));
    // surface faces
    SurfaceState &s = h->surf;
    auto upload = [&](long long **dst, const std::vector<uint64_t> &cells, const std::vector<int> &axis,
                      const std::vector<int> *sign) -> tlm_status {
        if (cells.empty()) return TLM_OK;
        std::vector<long long> c(cells.size());
        for (size_t f = 0; f < cells.size(); ++f)
            c[f] = (long long)cells[f] * 8 + axis[f] * 2 + ((sign && (*sign)[f] < 0) ? 1 : 0);
        FD_TRY(alloc(h, dst, c.size() * 8));
        FD_CU(h, cudaMemcpyAsync(*dst, c.data(), c.size() * 8, cudaMemcpyHostToDevice, h->stream));
        FD_CU(h, cudaStreamSynchronize(h->stream));
        return TLM_OK;
    };
    FD_TRY(upload(&s.dJsNode, s.jsCell, s.jsAxis, nullptr));
    FD_TRY(upload(&s.dHuyNode, s.huyCell, s.huyAxis, &s.huySign));
    const size_t nj = s.jsCell.size(), nh = s.huyCell.size();
    if (nj)
    {
        FD_TRY(alloc(h, (float **)&s.dJsInst, nj * 4));
        FD_TRY(alloc(h, (float **)&s.dJsAcc, nj * 16));
        FD_CU(h, cudaMemsetAsync(s.dJsInst, 0, nj * 4, h->stream));
        FD_CU(h, cudaMemsetAsync(s.dJsAcc, 0, nj * 16, h->stream));
    }
    if (nh)
    {
        FD_TRY(alloc(h, (float **)&s.dHuyAcc, nh * 32));
        FD_CU(h, cudaMemsetAsync(s.dHuyAcc, 0, nh * 32, h->stream));
    }
    h->nEpart = 148 * 4;
    FD_TRY(alloc(h, &h->dEpart, (size_t)h->nEpart * 8));
    FD_TRY(ensureRecords(h, std::max(h->cfg.total_steps, 1)));
    FD_CU(h, cudaStreamSynchronize(h->stream));
    h->prepared = true;
    return TLM_OK;
}

fdk::Box boxOf(const fdk::Dims &d)
{
    fdk::Box box;
    box.total = (unsigned)((long long)(d.nx + 1) * (d.ny + 1) * (d.nz + 1));
    box.divX = tlmk::makeFastDiv((unsigned)(d.nx + 1));
    box.divY = tlmk::makeFastDiv((unsigned)(d.ny + 1));
    return box;
}

using FusedLayouts = std::tuple<fdk::FusedLayout<51, 10>, fdk::FusedLayout<35, 14>, fdk::FusedLayout<17, 15>>;
template <int I = 0, class F> void withFusedLayout(int layout, F &&f)
{
    if constexpr (I < (int)std::tuple_size<FusedLayouts>::value)
    {
        if (layout == I)
            f(std::tuple_element_t<I, FusedLayouts>{});
        else
            withFusedLayout<I + 1>(layout, f);
    }
}

// The columns of fused passes with the least cost: waves of resident blocks
// times planes (one of them the ring's plane below) times the threads of an SM's
// blocks. Returns it.
long long chooseFused(fdtd_solver *h, int sms)
{
    const fdk::Dims &d = h->d;
    long long best = -1;
    for (int l = 0; l < (int)std::tuple_size<FusedLayouts>::value; ++l)
        withFusedLayout(l, [&](auto L) {
            using Layout = decltype(L);
            const int nx = d.nx + 1, ny = d.ny + 1, nz = d.nz + 1;
            const int ntx = (nx + Layout::maxTX - 1) / Layout::maxTX;
            const int TX = ((nx + ntx - 1) / ntx + 3) / 4 * 4;
            const int rows0 = (ny + Layout::maxTY - 1) / Layout::maxTY;
            for (int rows = rows0; rows < rows0 + 6 && rows <= ny; ++rows)
            {
                const int TY = (ny + rows - 1) / rows, nty = (ny + TY - 1) / TY;
                // (of the counts of ranges with the same planes per range the smallest)
                for (int c = 1, p = nz; c <= std::max(1, nz / 2); c = p > 1 ? (nz + p - 2) / (p - 1) : nz + 1)
                {
                    p = (nz + c - 1) / c;
                    const long long slots = (long long)sms * Layout::kMinBlocks;
                    const long long waves = ((long long)ntx * nty * c + slots - 1) / slots;
                    const long long cost = waves * (p + (c > 1 ? 1 : 0)) *
                                           (Layout::kThreads * Layout::kMinBlocks);
                    if (best >= 0 && cost >= best) continue;
                    best = cost;
                    h->layout = l;
                    h->TX = TX;
                    h->TY = TY;
                    h->ntx = ntx;
                    h->nty = nty;
                    h->nchunk = c;
                }
            }
        });
    return best;
}

// Whether a fused pass of that cost takes less time than the in-place sweeps.
// Microseconds on a B200, from 51 shapes of 27 to 8 M cells: a pass takes 13
// with its tail, 1.9 per 1024 of its cost (2.2 with dielectrics), and 5 per
// million edges of the x faces, whose values lie a row apart (30 where the fields
// exceed L2); the sweeps take 27 and 10 per million cells, from about 1.3 M on 18
// and 17. Columns that leave most of a block idle lose: 4x500x500 air 83 us
// fused, 47 in place, 2x2x8000 32 and 21, 8x600x600 with dielectrics 141 and 91.
bool fusedPays(const fdk::Dims &d, long long cost, bool diel)
{
    const double m = (double)(d.nx + 1) * (d.ny + 1) * (d.nz + 1) * 1e-6, faces = 4.0 * d.ny * d.nz * 1e-6;
    const double pass = 13.0 + (diel ? 2.2 : 1.9) * (double)cost / 1024.0 + (m > 2.5 ? 30.0 : 5.0) * faces;
    return pass <= std::max(27.0 + 10.0 * m, 18.0 + 17.0 * m);
}

// Tensor maps of the fused pass's boxes and the kernel's shared memory.
tlm_status fusedMaps(fdtd_solver *h)
{
    const fdk::Dims &d = h->d;
    auto encode = tlmi::tensorMapEncoder();
    h->maps = std::make_unique<FdtdMaps>();
    tlm_status st = TLM_OK;
    withFusedLayout(h->layout, [&](auto L) {
        using Layout = decltype(L);
        for (int b = 0; b < 2; ++b)
            for (int m = 0; m < 3; ++m)
            {
                const cuuint64_t dims[4] = { (cuuint64_t)d.px, (cuuint64_t)d.ny + 1, (cuuint64_t)d.nz + 1, 6 };
                const cuuint64_t strides[3] = { (cuuint64_t)d.px * 4, (cuuint64_t)d.px * (d.ny + 1) * 4,
                                                (cuuint64_t)h->P * 4 };
                const cuuint32_t box[4] = { (cuuint32_t)Layout::W2, (cuuint32_t)(m == 2 ? Layout::H : Layout::H + 1), 1,
                                            m == 0 ? 2u : m == 1 ? 1u : 3u };
                const cuuint32_t es[4] = { 1, 1, 1, 1 };
                if (encode(&h->maps->map[b][m], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, h->dBuf[b], dims, strides, box, es,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                    st = h->fail(TLM_ECUDA, "tensor map of a field buffer");
            }
        if (st == TLM_OK)
            st = h->cuda(cudaFuncSetAttribute(fdk::fusedStepKernel<Layout>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              Layout::smemBytes),
                         "cudaFuncSetAttribute(fusedStepKernel)");
    });
    return st;
}

// For reclaim: the state moves to the first buffer's place, and the sweeps run
// in place from now on (or until there is room again).
bool giveBufferBack(fdtd_solver *h)
{
    if (!h->dBuf[1]) return false;
    if (h->cur == 1) std::swap(h->dBuf[0], h->dBuf[1]);
    h->cur = 0;
    dropFused(h);
    h->lent = true;
    cudaStreamSynchronize(h->stream);
    return true;
}

size_t fieldBytes(const fdtd_solver *h) { return 6 * (size_t)h->P * 4; }
bool roomForFused(const fdtd_solver *h)
{
    return fieldBytes(h) + ((size_t)256 << 20) <= tlmi::poolAvailable(h->device);
}

// Everything fused passes need beyond the in-place sweeps.
tlm_status allocFused(fdtd_solver *h)
{
    const fdk::Dims &d = h->d;
    const size_t field = fieldBytes(h);
    FD_TRY(alloc(h, &h->dBuf[1], field));
    if (reinterpret_cast<uintptr_t>(h->dBuf[1]) & 15) return h->fail(TLM_ECUDA, "field allocation not 16-byte aligned");
    FD_CU(h, cudaMemsetAsync(h->dBuf[1], 0, field, h->stream));
    h->fault = faultWords().take();
    if (!h->fault) return h->fail(TLM_ENOMEM, "no fault word");
    FD_TRY(fusedMaps(h));
    const size_t nf = (size_t)h->ntx * h->nty * (d.nz + 1);
    FD_TRY(alloc(h, &h->dFlags, nf));
    fdk::edgeFlagKernel<<<(unsigned)nf, 128, 0, h->stream>>>(h->dCls, d, h->TX, h->TY, h->ntx, h->dFlags);
    return h->cuda(cudaGetLastError(), "edge flags");
}
void planFused(fdtd_solver *h)
{
    const std::string err = h->err;
    h->planning = true;
    if (allocFused(h) != TLM_OK)
    {
        dropFused(h);
        h->err = err;
    }
    h->planning = false;
}

// more: another step follows at once (its sources may go in with this step's tail)
tlm_status launchStep(fdtd_solver *h, int n, bool more)
{
    const fdk::Dims &d = h->d;
    fdk::Fields f;
    for (int c = 0; c < 3; ++c)
    {
        f.E[c] = h->field(c);
        f.H[c] = h->field(3 + c);
        f.ca[c] = h->dCa[c];
        f.cb[c] = h->dCb[c];
    }
    f.cls = h->dCls;
    f.tab = h->dTab;
    // 1. soft sources
    auto injectArgs = [&](float *E, int step) {
        fdk::InjectArgs a;
        for (int c = 0; c < 3; ++c) a.E[c] = E + c * h->P;
        a.edge = h->dEdge;
        a.off = h->dEdgeOff;
        a.amps = h->dAmps;
        a.nedges = h->nEdges;
        a.sv = sourceValue(h, step);
        return a;
    };
    const unsigned injectBlocks = (unsigned)((h->nEdges + 255) / 256);
    if (h->nEdges && !h->injected)
        fdk::injectKernel<<<injectBlocks, 256, 0, h->stream>>>(injectArgs(h->dBuf[h->cur], n));
    h->injected = false;
    // 2. monitors
    SurfaceState &s = h->surf;
    const int nj = (int)s.jsCell.size(), nhuy = (int)s.huyCell.size();
    const bool doDft = n >= h->cfg.settle_steps;
    const bool doPlane = s.planeAxis >= 0 && (n % 2) == 0;
    int n1 = 0, n2 = 0;
    if (doPlane)
    {
        const int dims[3] = { d.nx, d.ny, d.nz };
        n1 = dims[s.planeAxis == 0 ? 1 : 0];
        n2 = dims[s.planeAxis == 2 ? 1 : 2];
        if ((size_t)n1 * n2 > s.planeCap)
        {
            release(h, s.dPlane);
            FD_TRY(alloc(h, (float **)&s.dPlane, (size_t)n1 * n2 * 4));
            s.planeCap = (size_t)n1 * n2;
        }
    }
    fdk::MonArgs a;
    a.f = f;
    a.d = d;
    a.dl = h->g.dl;
    a.eta0 = tlmh::eta0_f32();
    a.step = n;
    a.nports = (int)h->ports.size();
    a.poff = h->dPoff;
    a.pcells = h->dPcells;
    a.ppol = h->dPpol;
    a.vrec = h->dVrec;
    a.irec = h->dIrec;
    a.nprobes = (int)h->probeCells.size();
    a.probeCell = h->dProbe;
    a.prec = h->dPrec;
    a.njs = nj;
    a.jsCode = s.dJsNode;
    a.jsInst = static_cast<float *>(s.dJsInst);
    a.jsAcc = static_cast<float *>(s.dJsAcc);
    a.nhuy = nhuy;
    a.huyCode = s.dHuyNode;
    a.huyAcc = static_cast<float *>(s.dHuyAcc);
    a.doDft = doDft ? 1 : 0;
    a.cph = a.sph = 0.0f;
    if (doDft && (nj || nhuy)) tlmh::dft_phase_f32(h->cfg.f0, h->dt, n, &a.cph, &a.sph);
    a.planeAxis = doPlane ? s.planeAxis : -1;
    a.planeIndex = doPlane ? std::min(std::max(s.planeIndex, 0),
                                      (s.planeAxis == 0 ? d.nx : s.planeAxis == 1 ? d.ny : d.nz) - 1)
                           : 0;
    a.planeN1 = n1;
    a.planeN2 = n2;
    a.plane = static_cast<float *>(s.dPlane);
    const long long items = (long long)a.nports + a.nprobes + nj + (doDft ? nhuy : 0) + (doPlane ? (long long)n1 * n2 : 0);
    const bool fused = h->dBuf[1] != nullptr;
    if (items > 0 && !fused) fdk::monitorKernel<<<(unsigned)((items + 255) / 256), 256, 0, h->stream>>>(a);
    if (doPlane)
    {
        s.planeValid = true;
        s.planeAxisDone = s.planeAxis;
        s.planeIndexDone = a.planeIndex;
        s.planeN1 = n1;
        s.planeN2 = n2;
    }
    if ((n & 15) == 0)
    {
        const double eta = (double)tlmh::eta0_f32();
        fdk::energyPartialKernel<<<h->nEpart, 256, 0, h->stream>>>(f, h->P, eta * eta, h->dEpart);
        fdk::energyFinalKernel<<<1, 256, 0, h->stream>>>(h->dEpart, h->nEpart, h->dEhist + n / 16);
    }
    // 3. H, 4. E and Mur
    long long faceItems = 0;
    for (int F = 0; F < 6; ++F) faceItems += (long long)h->mur.n1[F] * h->mur.n2[F];
    const unsigned faceBlocks = (unsigned)((faceItems + 255) / 256);
    if (fused)
    {
        fdk::FusedArgs fa;
        fa.in = f;
        fa.mapExy = h->maps->map[h->cur][0];
        fa.mapEz = h->maps->map[h->cur][1];
        fa.mapH = h->maps->map[h->cur][2];
        fa.fault = h->fault;
        fa.out = h->dBuf[h->cur ^ 1];
        fa.P = h->P;
        fa.d = d;
        fa.TX = h->TX;
        fa.TY = h->TY;
        fa.ntx = h->ntx;
        fa.nty = h->nty;
        fa.nchunk = h->nchunk;
        fa.flags = h->dFlags;
        fa.ch = h->ch;
        fa.cb0 = h->cb0;
        fa.neg_zero = -0.0f;
        withFusedLayout(h->layout, [&](auto L) {
            using Layout = decltype(L);
            fdk::fusedStepKernel<Layout>
                <<<(unsigned)(h->ntx * h->nty * h->nchunk), Layout::kThreads, Layout::smemBytes, h->stream>>>(fa);
        });
        fdk::TailArgs ta;
        ta.oldE = h->dBuf[h->cur];
        ta.newE = fa.out;
        ta.P = h->P;
        ta.mur = h->mur;
        ta.mon = a;
        ta.inj = injectArgs(fa.out, n + 1);
        ta.murBlocks = faceBlocks;
        ta.monBlocks = (unsigned)((items + 255) / 256);
        h->injected = more && h->nEdges && h->edgesInside;
        fdk::stepTailKernel<<<faceBlocks + ta.monBlocks + (h->injected ? injectBlocks : 0), 256, 0, h->stream>>>(ta);
        h->cur ^= 1;
    }
    else
    {
        fdk::Box box = boxOf(d);
        const unsigned grid = (box.total + 255) / 256;
        fdk::updateHKernel<<<grid + faceBlocks, 256, 0, h->stream>>>(f, d, box, h->ch, h->mur, grid);
        fdk::updateEKernel<<<grid, 256, 0, h->stream>>>(f, d, box);
        long long aItems = 0, bItems = 0;
        for (int F = 0; F < 3; ++F) aItems += (long long)h->mur.n1[F] * h->mur.n2[F];
        for (int F = 3; F < 6; ++F) bItems += (long long)h->mur.n1[F] * h->mur.n2[F];
        fdk::murApplyKernel<0><<<(unsigned)((aItems + 255) / 256), 256, 0, h->stream>>>(f, d, h->mur);
        fdk::murApplyKernel<3><<<(unsigned)((bItems + 255) / 256), 256, 0, h->stream>>>(f, d, h->mur);
    }
    if (h->cfg.record_every > 0 && (n % h->cfg.record_every) == 0)
    {
        const bool withPlane = s.planeAxis >= 0 && s.planeValid;
        const size_t np = withPlane ? (size_t)s.planeN1 * s.planeN2 : 0;
        const size_t need = s.framesUsed + nj + np;
        if (need > s.framesCap)
        {
            const size_t cap = std::max(need, s.framesCap * 2 + 1024);
            float *dn = nullptr;
            FD_TRY(alloc(h, &dn, cap * 4));
            if (s.framesUsed)
                FD_CU(h, cudaMemcpyAsync(dn, s.dFrames, s.framesUsed * 4, cudaMemcpyDeviceToDevice, h->stream));
            release(h, s.dFrames);
            s.dFrames = dn;
            s.framesCap = cap;
        }
        float *base = static_cast<float *>(s.dFrames) + s.framesUsed;
        if (nj) FD_CU(h, cudaMemcpyAsync(base, s.dJsInst, nj * 4, cudaMemcpyDeviceToDevice, h->stream));
        if (np) FD_CU(h, cudaMemcpyAsync(base + nj, s.dPlane, np * 4, cudaMemcpyDeviceToDevice, h->stream));
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
    return h->cuda(cudaGetLastError(), "FDTD step launch");
}

} // namespace

extern "C" {

tlm_status fdtd_create(fdtd_handle *out, int device)
{
    if (!out)
    {
        g_fdtdErr = "null output";
        return TLM_EINVAL;
    }
    *out = nullptr;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0)
    {
        cudaGetLastError();
        g_fdtdErr = "no CUDA device";
        return TLM_ENODEV;
    }
    if (device < 0 || device >= count)
    {
        g_fdtdErr = "no such device";
        return TLM_EINVAL;
    }
    fdtd_solver *h = new fdtd_solver();
    h->device = device;
    Guard g(device);
    if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess)
    {
        cudaGetLastError();
        delete h;
        g_fdtdErr = "stream creation failed";
        return TLM_ECUDA;
    }
    h->pool = tlmi::devicePool(device);
    if (!h->pool)
    {
        cudaStreamDestroy(h->stream);
        delete h;
        g_fdtdErr = "memory pool unavailable";
        return TLM_ECUDA;
    }
    tlmi::enlist(h->lender, device, [h] { return giveBufferBack(h); });
    *out = h;
    return TLM_OK;
}

tlm_status fdtd_destroy(fdtd_handle h)
{
    if (!h) return TLM_OK;
    {
        Guard g(h->device);
        tlmi::delist(h->lender);
        cudaStreamSynchronize(h->stream);
        freeAll(h);
        cudaStreamSynchronize(h->stream);
        cudaStreamDestroy(h->stream);
    }
    delete h;
    return TLM_OK;
}

const char *fdtd_last_error(fdtd_handle h) { return h ? h->err.c_str() : g_fdtdErr.c_str(); }

tlm_status fdtd_setup(fdtd_handle h, const tlm_grid *grid, const uint8_t *mat, size_t n_cells,
                      const tlm_matprops *table, int n_table, const tlm_config *cfg)
{
    if (!h)
    {
        g_fdtdErr = "null handle";
        return TLM_EINVAL;
    }
    if (!grid || !mat || !cfg || (n_table > 0 && !table) || n_table < 0)
        return h->fail(TLM_EINVAL, "null grid, material map, table or config");
    if (grid->nx < 2 || grid->ny < 2 || grid->nz < 2) return h->fail(TLM_EINVAL, "grid must be at least 2 cells per axis");
    if ((long long)(grid->nx + 1) * (grid->ny + 1) * (grid->nz + 1) >= (1LL << 31))
        return h->fail(TLM_EINVAL, "grid too large");
    if (!(grid->dl > 0.0f)) return h->fail(TLM_EINVAL, "dl must be positive");
    const size_t n = (size_t)grid->nx * grid->ny * grid->nz;
    if (n_cells != n) return h->fail(TLM_EINVAL, "material map does not match the grid");
    // the host copy of the map and its largest id in one vectorised pass
    tlmh::HostMap hostMat;
    if (!hostMat.allocate(n)) return h->fail(TLM_ENOMEM, "no host memory for the material map");
    const uint8_t maxId = tlmh::copy_max_u8(mat, hostMat.data(), n);
    if (maxId >= TLM_MAT_DIEL0 && (int)(maxId - TLM_MAT_DIEL0) >= n_table)
        return h->fail(TLM_EINVAL, "material id without a table entry");
    if (cfg->waveform < 0 || cfg->waveform > TLM_WAVE_TABLE) return h->fail(TLM_EINVAL, "unknown waveform");
    if (cfg->record_every < 0 || cfg->huy_offset < 0) return h->fail(TLM_EINVAL, "negative record_every or huy_offset");
    Guard gd(h->device);
    std::lock_guard<std::recursive_timed_mutex> lk(h->lender.busy);
    cudaStreamSynchronize(h->stream);
    freeAll(h);
    h->configured = false;
    h->lent = false;
    h->g = *grid;
    h->cfg = *cfg;
    h->mat.swap(hostMat);
    h->table.assign(table, table + n_table);
    h->haveDiel = maxId >= TLM_MAT_DIEL0;
    h->d = fdk::Dims{ grid->nx, grid->ny, grid->nz, (grid->nx + 4) / 4 * 4 };
    const fdk::Dims &d = h->d;
    const int nx = d.nx, ny = d.ny, nz = d.nz;
    // fused passes where they pay (their lane offsets within a plane are 32-bit),
    // with rows padded for them; no_staging asks for the in-place sweeps on the
    // same rows
    int sms = 0;
    FD_CU(h, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device));
    bool fused = (long long)d.px * (ny + 1) < (1LL << 30) && tlmi::tensorMapEncoder() != nullptr &&
                 fusedPays(d, chooseFused(h, sms), h->haveDiel);
    if (!fused) h->d.px = nx + 1;
    fused = fused && !cfg->no_staging;
    h->dt = tlmh::fdtd_dt(grid->dl);
    h->cMur = tlmh::fdtd_cmur(h->dt, grid->dl);
    h->cb0 = tlmh::fdtd_cb0(h->dt, grid->dl);
    h->ch = tlmh::fdtd_ch(h->dt, grid->dl);
    h->len[0] = (long long)nx * (ny + 1) * (nz + 1);
    h->len[1] = (long long)(nx + 1) * ny * (nz + 1);
    h->len[2] = (long long)(nx + 1) * (ny + 1) * nz;
    h->len[3] = (long long)(nx + 1) * ny * nz;
    h->len[4] = (long long)nx * (ny + 1) * nz;
    h->len[5] = (long long)nx * ny * (nz + 1);
    // (components start on 16 bytes)
    auto planeSet = [&] { return ((long long)d.px * (ny + 1) * (nz + 1) + 3) / 4 * 4; };
    h->P = planeSet();
    h->cur = 0;
    // fields, edge classes, coefficients of mixed edges
    const size_t spare = (size_t)256 << 20;
    auto bytes = [&] { return (size_t)h->P * 4 * (h->haveDiel ? 13 : 7); };
    size_t avail = tlmi::poolAvailable(h->device);
    // a second field buffer for fused passes where it fits
    if (fused && bytes() + fieldBytes(h) + spare > avail)
    {
        fused = false;
        h->d.px = nx + 1;
        h->P = planeSet();
    }
    const size_t need = bytes(), field = fieldBytes(h), classes = (size_t)h->P * 4;
    if (need + spare > avail && tlmi::reclaim(h->device)) avail = tlmi::poolAvailable(h->device);
    if (need + spare > avail) return h->fail(TLM_ENOMEM, "grid needs " + std::to_string(need >> 20) + " MiB of HBM");
    FD_TRY(alloc(h, &h->dBuf[0], field));
    if (reinterpret_cast<uintptr_t>(h->dBuf[0]) & 15)  // vector loads
        return h->fail(TLM_ECUDA, "field allocation not 16-byte aligned");
    FD_CU(h, cudaMemsetAsync(h->dBuf[0], 0, field, h->stream));
    FD_TRY(alloc(h, &h->dCls, classes));
    FD_CU(h, cudaMemsetAsync(h->dCls, 0, classes, h->stream));
    if (h->haveDiel)
        for (int c = 0; c < 3; ++c)
        {
            FD_TRY(alloc(h, &h->dCa[c], (size_t)h->P * 4));
            FD_TRY(alloc(h, &h->dCb[c], (size_t)h->P * 4));
        }
    // coefficients of the edges inside one material: the sums over four equal cells
    std::vector<float2> tab(fdk::kEdgeClasses, make_float2(0.0f, 0.0f)), props(std::max(n_table, 1), make_float2(1.0f, 0.0f));
    tab[fdk::kEdgeAir] = make_float2(1.0f, h->cb0);
    for (int t = 0; t < n_table; ++t) props[t] = make_float2(table[t].epsr, table[t].sigma);
    // (a byte names 254 dielectrics; no cell can have a later entry)
    for (int t = 0; t < std::min(n_table, (int)fdk::kEdgeFirst - TLM_MAT_DIEL0); ++t)
    {
        const int id = t + TLM_MAT_DIEL0;
        const float e1 = 1.0f + (table[t].epsr - 1.0f), s1 = table[t].sigma;
        float e = 0.0f, sg = 0.0f;
        for (int q = 0; q < 4; ++q)
        {
            e += e1;
            sg += s1;
        }
        tlmh::fdtd_edge_coef(e, sg, 4, h->dt, grid->dl, &tab[id].x, &tab[id].y);
    }
    std::memset(&tab[fdk::kEdgeFirst], 0xff, (fdk::kEdgeClasses - fdk::kEdgeFirst) * sizeof(float2));
    FD_TRY(alloc(h, &h->dTab, tab.size() * sizeof(float2)));
    FD_CU(h, cudaMemcpyAsync(h->dTab, tab.data(), tab.size() * sizeof(float2), cudaMemcpyHostToDevice, h->stream));
    {
        uint8_t *dMat = nullptr;
        float2 *dProps = nullptr;
        FD_TRY(alloc(h, &dMat, n));
        tlm_status st = alloc(h, &dProps, props.size() * sizeof(float2));
        if (st == TLM_OK)
        {
            cudaError_t e = cudaMemcpyAsync(dMat, mat, n, cudaMemcpyHostToDevice, h->stream);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(dProps, props.data(), props.size() * sizeof(float2), cudaMemcpyHostToDevice,
                                    h->stream);
            if (e == cudaSuccess)
            {
                const fdk::Box box = boxOf(d);
                fdk::edgeClassKernel<<<(box.total + 255) / 256, 256, 0, h->stream>>>(
                    dMat, dProps, d, box, h->dt, grid->dl, tlmh::fdtd_eps0(), h->dCls,
                    reinterpret_cast<unsigned long long *>(h->dTab), h->dCa[0], h->dCa[1], h->dCa[2],
                    h->dCb[0], h->dCb[1], h->dCb[2]);
                e = cudaGetLastError();
            }
            st = h->cuda(e, "edge classes");
        }
        release(h, dMat);
        release(h, dProps);
        FD_TRY(st);
    }
    // Mur planes: x faces (Ey, Ez), y faces (Ex, Ez), z faces (Ex, Ey)
    const int n1[6] = { ny, ny + 1, nx, nx + 1, nx, nx + 1 };
    const int n2[6] = { nz + 1, nz, nz + 1, nz, ny + 1, ny };
    long long total = 0;
    for (int F = 0; F < 6; ++F)
    {
        h->mur.n1[F] = n1[F];
        h->mur.n2[F] = n2[F];
        h->mur.off[F] = total;
        total += 4LL * n1[F] * n2[F];
    }
    h->mur.cMur = h->cMur;
    FD_TRY(alloc(h, &h->mur.snap, (size_t)total * 4));
    FD_CU(h, cudaMemsetAsync(h->mur.snap, 0, (size_t)total * 4, h->stream));
    if (fused) planFused(h);
    FD_CU(h, cudaStreamSynchronize(h->stream));
    h->planeSources.clear();
    h->ports.clear();
    h->probeCells.clear();
    h->svTable.clear();
    h->surf = SurfaceState();
    tlmi::buildFaceLists(nx, ny, nz, grid->origin, grid->dl, mat, cfg->surface_monitors != 0, cfg->huy_offset,
                         h->surf);
    h->curStep = 0;
    h->injected = false;
    h->prepared = false;
    h->configured = true;
    return TLM_OK;
}

tlm_status fdtd_add_port(fdtd_handle h, const uint64_t *cells, int n_cells, int pol_axis, float amp, int *idx)
{
    FD_TRY(ready(h));
    if (h->curStep > 0) return h->fail(TLM_ESTATE, "ports must be added before the first step");
    if (pol_axis < 0 || pol_axis > 2 || n_cells < 0 || (n_cells > 0 && !cells))
        return h->fail(TLM_EINVAL, "bad port");
    fdtd_solver::Port p;
    p.pol = pol_axis;
    p.amp = amp;
    for (int t = 0; t < n_cells; ++t)
        if (cells[t] < h->mat.size() && h->mat[cells[t]] == TLM_MAT_AIR) p.cells.push_back(cells[t]);
    if (!p.cells.empty())
    {
        const uint64_t c = p.cells[p.cells.size() / 2];
        int co[3] = { (int)(c % h->d.nx), (int)((c / h->d.nx) % h->d.ny), (int)(c / ((uint64_t)h->d.nx * h->d.ny)) };
        const int dims[3] = { h->d.nx, h->d.ny, h->d.nz };
        for (int a : { (pol_axis + 1) % 3, (pol_axis + 2) % 3 })
            if (co[a] < 1 || co[a] > dims[a] - 2)
                return h->fail(TLM_EINVAL, "the port's current loop leaves the grid");
    }
    h->ports.push_back(p);
    h->prepared = false;
    if (idx) *idx = (int)h->ports.size() - 1;
    return TLM_OK;
}

tlm_status fdtd_add_plane_wave(fdtd_handle h, int prop_axis, int plane_index, int pol_axis, float amp)
{
    FD_TRY(ready(h));
    if (h->curStep > 0) return h->fail(TLM_ESTATE, "sources must be added before the first step");
    if (prop_axis < 0 || prop_axis > 2 || pol_axis < 0 || pol_axis > 2) return h->fail(TLM_EINVAL, "bad axis");
    for (int k = 0; k < h->d.nz; ++k)
        for (int j = 0; j < h->d.ny; ++j)
            for (int i = 0; i < h->d.nx; ++i)
            {
                const int co[3] = { i, j, k };
                if (co[prop_axis] != plane_index) continue;
                const size_t c = ((size_t)k * h->d.ny + j) * h->d.nx + i;
                if (h->mat[c] == TLM_MAT_AIR) h->planeSources.push_back({ c, pol_axis, amp });
            }
    h->prepared = false;
    return TLM_OK;
}

tlm_status fdtd_add_probe(fdtd_handle h, float x, float y, float z, int *idx)
{
    FD_TRY(ready(h));
    if (h->curStep > 0) return h->fail(TLM_ESTATE, "probes must be added before the first step");
    int i, j, k;
    tlmh::cell_of(h->g.origin, h->g.dl, x, y, z, &i, &j, &k);
    if (i < 0 || j < 0 || k < 0 || i >= h->d.nx || j >= h->d.ny || k >= h->d.nz)
    {
        if (idx) *idx = -1;
        return TLM_OK;
    }
    h->probeCells.push_back(((uint64_t)k * h->d.ny + j) * h->d.nx + i);
    h->prepared = false;
    if (idx) *idx = (int)h->probeCells.size() - 1;
    return TLM_OK;
}

tlm_status fdtd_set_source_table(fdtd_handle h, const float *values, int n)
{
    FD_TRY(ready(h));
    if (n < 0 || (n > 0 && !values)) return h->fail(TLM_EINVAL, "bad source table");
    h->svTable.assign(values, values + n);
    h->cfg.waveform = TLM_WAVE_TABLE;
    return TLM_OK;
}

tlm_status fdtd_step(fdtd_handle h, int n_steps)
{
    FD_TRY(ready(h));
    if (n_steps < 0) return h->fail(TLM_EINVAL, "n_steps must be >= 0");
    Guard gd(h->device);
    std::lock_guard<std::recursive_timed_mutex> lk(h->lender.busy);
    FD_TRY(prepare(h));
    FD_TRY(ensureRecords(h, (long long)h->curStep + n_steps));
    // (looking for room takes as long as a few steps)
    if (h->lent && n_steps >= 64 && roomForFused(h)) planFused(h);
    if (h->dBuf[1]) h->lent = false;
    for (int t = 0; t < n_steps; ++t)
    {
        FD_TRY(launchStep(h, h->curStep, t + 1 < n_steps));
        ++h->curStep;
    }
    FD_CU(h, cudaStreamSynchronize(h->stream));
    if (h->fault && *static_cast<volatile unsigned *>(h->fault)) return h->fail(TLM_ECUDA, "a field plane's bulk copies never arrived");
    return TLM_OK;
}

tlm_status fdtd_run(fdtd_handle h)
{
    FD_TRY(ready(h));
    return fdtd_step(h, std::max(0, h->cfg.total_steps - h->curStep));
}

int fdtd_current_step(fdtd_handle h) { return h ? h->curStep : 0; }
tlm_status fdtd_get_stream(fdtd_handle h, void **stream)
{
    if (!h || !stream)
    {
        g_fdtdErr = "null handle or output";
        return TLM_EINVAL;
    }
    *stream = (void *)h->stream;
    return TLM_OK;
}
float fdtd_timestep(fdtd_handle h) { return h ? h->dt : 0.0f; }

tlm_status fdtd_get_grid(fdtd_handle h, tlm_grid *grid)
{
    FD_TRY(ready(h));
    if (!grid) return h->fail(TLM_EINVAL, "null output");
    *grid = h->g;
    return TLM_OK;
}

tlm_status fdtd_get_field(fdtd_handle h, int which, float *out, size_t cap, size_t *n)
{
    FD_TRY(ready(h));
    if (which < 0 || which > 5) return h->fail(TLM_EINVAL, "which must be 0..5 (Ex Ey Ez Hx Hy Hz)");
    if (n) *n = (size_t)h->len[which];
    if (!out) return TLM_OK;
    if (cap < (size_t)h->len[which]) return h->fail(TLM_EINVAL, "output smaller than the field");
    Guard gd(h->device);
    std::lock_guard<std::recursive_timed_mutex> lk(h->lender.busy);
    // packed in pieces of at most 64 MiB, smaller ones on a card that is full
    const long long total = h->len[which];
    long long piece = std::min<long long>(total, 1LL << 24);
    float *packed = nullptr;
    while (alloc(h, &packed, (size_t)piece * 4) != TLM_OK)
    {
        if (piece <= 1024) return TLM_ENOMEM;
        piece /= 2;
    }
    const int a = which % 3;  // E: one more entry on the axes other than a; H: one more on a
    const int n0 = h->d.nx + ((which < 3) == (a != 0) ? 1 : 0), n1 = h->d.ny + ((which < 3) == (a != 1) ? 1 : 0);
    cudaError_t e = cudaSuccess;
    for (long long first = 0; first < total && e == cudaSuccess; first += piece)
    {
        const long long count = std::min(piece, total - first);
        fdk::packFieldKernel<<<tlmi::gridBlocksFor(count), 256, 0, h->stream>>>(h->field(which), h->d, n0, n1, first,
                                                                              count, packed);
        e = cudaGetLastError();
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(out + first, packed, (size_t)count * 4, cudaMemcpyDeviceToHost, h->stream);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    release(h, packed);
    return h->cuda(e, "field read-back");
}

tlm_status fdtd_get_probe(fdtd_handle h, int idx, float *ex, float *ey, float *ez, int cap, int *n)
{
    FD_TRY(ready(h));
    const int nr = (int)h->probeCells.size();
    if (idx < 0 || idx >= nr) return h->fail(TLM_EINVAL, "no such probe");
    const int steps = h->curStep;
    if (n) *n = steps;
    const int m = std::min(steps, cap);
    if (m <= 0 || !h->dPrec) return TLM_OK;
    Guard gd(h->device);
    std::vector<float> all((size_t)m * nr * 3);
    FD_CU(h, cudaMemcpy(all.data(), h->dPrec, all.size() * 4, cudaMemcpyDeviceToHost));
    for (int t = 0; t < m; ++t)
    {
        if (ex) ex[t] = all[((size_t)t * nr + idx) * 3];
        if (ey) ey[t] = all[((size_t)t * nr + idx) * 3 + 1];
        if (ez) ez[t] = all[((size_t)t * nr + idx) * 3 + 2];
    }
    return TLM_OK;
}

tlm_status fdtd_get_port(fdtd_handle h, int idx, float *v, float *i, int cap, int *n)
{
    FD_TRY(ready(h));
    const int np = (int)h->ports.size();
    if (idx < 0 || idx >= np) return h->fail(TLM_EINVAL, "no such port");
    const int steps = h->curStep;
    if (n) *n = steps;
    const int m = std::min(steps, cap);
    if (m <= 0 || !h->dVrec) return TLM_OK;
    Guard gd(h->device);
    std::vector<float> vv((size_t)m * np), ii((size_t)m * np);
    FD_CU(h, cudaMemcpy(vv.data(), h->dVrec, vv.size() * 4, cudaMemcpyDeviceToHost));
    FD_CU(h, cudaMemcpy(ii.data(), h->dIrec, ii.size() * 4, cudaMemcpyDeviceToHost));
    for (int t = 0; t < m; ++t)
    {
        if (v) v[t] = vv[(size_t)t * np + idx];
        if (i) i[t] = ii[(size_t)t * np + idx];
    }
    return TLM_OK;
}

tlm_status fdtd_get_energy_history(fdtd_handle h, int *steps, float *vals, double *vals64, int cap, int *n)
{
    FD_TRY(ready(h));
    const int ne = h->curStep > 0 ? (h->curStep - 1) / 16 + 1 : 0;
    if (n) *n = ne;
    const int m = std::min(ne, cap);
    if (m <= 0 || !h->dEhist) return TLM_OK;
    Guard gd(h->device);
    std::vector<double> buf(m);
    FD_CU(h, cudaMemcpy(buf.data(), h->dEhist, (size_t)m * 8, cudaMemcpyDeviceToHost));
    for (int t = 0; t < m; ++t)
    {
        if (steps) steps[t] = 16 * t;
        if (vals) vals[t] = (float)buf[t];
        if (vals64) vals64[t] = buf[t];
    }
    return TLM_OK;
}

// ---- surface monitors, cut plane, frames, far field -----------------------
tlm_status fdtd_get_surface_faces(fdtd_handle h, uint64_t *air_cells, int *axis, int *sign, float *centers, int cap,
                                  int *n)
{
    FD_TRY(ready(h));
    const SurfaceState &s = h->surf;
    const int nf = (int)s.jsCell.size();
    if (n) *n = nf;
    for (int f = 0; f < nf && f < cap; ++f)
    {
        if (air_cells) air_cells[f] = s.jsCell[f];
        if (axis) axis[f] = s.jsAxis[f];
        if (sign) sign[f] = s.jsSign[f];
        if (centers) std::memcpy(centers + 3 * f, &s.jsCenter[3 * f], 12);
    }
    return TLM_OK;
}

static int fdtdSamples(const fdtd_solver *h) { return std::max(0, h->curStep - std::max(h->cfg.settle_steps, 0)); }

tlm_status fdtd_get_js_instant(fdtd_handle h, float *out, int cap, int *n)
{
    FD_TRY(ready(h));
    const SurfaceState &s = h->surf;
    const int nf = (int)s.jsCell.size();
    if (n) *n = nf;
    if (!out || cap <= 0 || nf == 0) return TLM_OK;
    if (!s.dJsInst)
    {
        std::fill(out, out + std::min(nf, cap), 0.0f);
        return TLM_OK;
    }
    Guard gd(h->device);
    FD_CU(h, cudaStreamSynchronize(h->stream));
    std::vector<float> t(nf);
    FD_CU(h, cudaMemcpy(t.data(), s.dJsInst, (size_t)nf * 4, cudaMemcpyDeviceToHost));
    std::copy(t.begin(), t.begin() + std::min(nf, cap), out);
    return TLM_OK;
}

tlm_status fdtd_get_js_dft(fdtd_handle h, float *magnitude, float *re, float *im, int cap, int *n, int *samples)
{
    FD_TRY(ready(h));
    const SurfaceState &s = h->surf;
    const int nf = (int)s.jsCell.size();
    const int ns = nf ? fdtdSamples(h) : 0;
    if (n) *n = nf;
    if (samples) *samples = ns;
    if (nf == 0 || cap <= 0) return TLM_OK;
    std::vector<float> acc((size_t)nf * 4, 0.0f);
    if (s.dJsAcc)
    {
        Guard gd(h->device);
        FD_CU(h, cudaStreamSynchronize(h->stream));
        FD_CU(h, cudaMemcpy(acc.data(), s.dJsAcc, acc.size() * 4, cudaMemcpyDeviceToHost));
    }
    for (int f = 0; f < nf && f < cap; ++f)
    {
        const float r1 = acc[4 * f], i1 = acc[4 * f + 1], r2 = acc[4 * f + 2], i2 = acc[4 * f + 3];
        if (re) { re[2 * f] = r1; re[2 * f + 1] = r2; }
        if (im) { im[2 * f] = i1; im[2 * f + 1] = i2; }
        if (magnitude)
        {
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

tlm_status fdtd_get_huygens_faces(fdtd_handle h, uint64_t *cells, int *axis, int *out_sign, float *pos, int cap,
                                  int *n)
{
    FD_TRY(ready(h));
    const SurfaceState &s = h->surf;
    const int nh = (int)s.huyCell.size();
    if (n) *n = nh;
    for (int f = 0; f < nh && f < cap; ++f)
    {
        if (cells) cells[f] = s.huyCell[f];
        if (axis) axis[f] = s.huyAxis[f];
        if (out_sign) out_sign[f] = s.huySign[f];
        if (pos) std::memcpy(pos + 3 * f, &s.huyPos[3 * f], 12);
    }
    return TLM_OK;
}

tlm_status fdtd_get_huygens_dft(fdtd_handle h, float *acc8, int cap, int *n, int *samples)
{
    FD_TRY(ready(h));
    const SurfaceState &s = h->surf;
    const int nh = (int)s.huyCell.size();
    if (n) *n = nh;
    if (samples) *samples = nh ? fdtdSamples(h) : 0;
    if (!acc8 || nh == 0 || cap <= 0) return TLM_OK;
    const int m = std::min(nh, cap);
    if (!s.dHuyAcc)
    {
        std::fill(acc8, acc8 + (size_t)m * 8, 0.0f);
        return TLM_OK;
    }
    Guard gd(h->device);
    FD_CU(h, cudaStreamSynchronize(h->stream));
    FD_CU(h, cudaMemcpy(acc8, s.dHuyAcc, (size_t)m * 32, cudaMemcpyDeviceToHost));
    return TLM_OK;
}

tlm_status fdtd_set_field_plane(fdtd_handle h, int axis, int index)
{
    FD_TRY(ready(h));
    if (axis < -1 || axis > 2) return h->fail(TLM_EINVAL, "plane axis must be -1 (off), 0, 1 or 2");
    h->surf.planeAxis = axis;
    h->surf.planeIndex = index;
    return TLM_OK;
}

tlm_status fdtd_get_field_plane(fdtd_handle h, float *out, size_t cap, int *axis, int *index, int *n1, int *n2)
{
    FD_TRY(ready(h));
    const SurfaceState &s = h->surf;
    if (s.planeAxis < 0 || !s.planeValid) return h->fail(TLM_ESTATE, "no field plane has been computed");
    const size_t np = (size_t)s.planeN1 * s.planeN2;
    if (axis) *axis = s.planeAxisDone;
    if (index) *index = s.planeIndexDone;
    if (n1) *n1 = s.planeN1;
    if (n2) *n2 = s.planeN2;
    if (!out) return TLM_OK;
    if (cap < np) return h->fail(TLM_EINVAL, "output holds fewer values than the plane");
    Guard gd(h->device);
    FD_CU(h, cudaStreamSynchronize(h->stream));
    FD_CU(h, cudaMemcpy(out, s.dPlane, np * 4, cudaMemcpyDeviceToHost));
    return TLM_OK;
}

tlm_status fdtd_frame_count(fdtd_handle h, int *n)
{
    FD_TRY(ready(h));
    if (!n) return h->fail(TLM_EINVAL, "null output");
    *n = (int)h->surf.frames.size();
    return TLM_OK;
}

tlm_status fdtd_get_frame(fdtd_handle h, int idx, int *step, float *js, int js_cap, float *plane, size_t plane_cap,
                          int *axis, int *index, int *n1, int *n2)
{
    FD_TRY(ready(h));
    const SurfaceState &s = h->surf;
    if (idx < 0 || idx >= (int)s.frames.size()) return h->fail(TLM_EINVAL, "no such frame");
    const SurfaceState::Frame &fr = s.frames[idx];
    const int nj = (int)s.jsCell.size();
    const size_t np = fr.hasPlane ? (size_t)fr.n1 * fr.n2 : 0;
    if (step) *step = fr.step;
    if (axis) *axis = fr.axis;
    if (index) *index = fr.index;
    if (n1) *n1 = fr.n1;
    if (n2) *n2 = fr.n2;
    Guard gd(h->device);
    FD_CU(h, cudaStreamSynchronize(h->stream));
    const float *base = static_cast<const float *>(s.dFrames) + fr.off;
    if (js && nj && js_cap > 0)
        FD_CU(h, cudaMemcpy(js, base, (size_t)std::min(nj, js_cap) * 4, cudaMemcpyDeviceToHost));
    if (plane && np)
    {
        if (plane_cap < np) return h->fail(TLM_EINVAL, "plane output holds fewer values than the frame's plane");
        FD_CU(h, cudaMemcpy(plane, base + nj, np * 4, cudaMemcpyDeviceToHost));
    }
    return TLM_OK;
}

tlm_status fdtd_compute_far_field(fdtd_handle h, int n_theta, int n_phi, float *U, float *u_max, float *directivity,
                                  float *peak_theta_deg, float *peak_phi_deg)
{
    FD_TRY(ready(h));
    if (n_theta < 2 || n_phi < 2) return h->fail(TLM_EINVAL, "need at least 2 theta and 2 phi samples");
    const SurfaceState &s = h->surf;
    const int nh = (int)s.huyCell.size();
    if (nh == 0 || fdtdSamples(h) == 0 || !s.dHuyAcc)
        return h->fail(TLM_ESTATE, "no Huygens phasors recorded (surface_monitors, huy_offset >= 2, "
                                   "steps past settle_steps)");
    Guard gd(h->device);
    FD_CU(h, cudaStreamSynchronize(h->stream));
    tlmi::FarField out;
    std::string err;
    const tlm_status st = tlmi::farFieldTransform(h->stream, h->pool, false, s.dHuyAcc, s.dHuyNode, s.huyPos.data(),
                                                  nh, h->cfg.f0, n_theta, n_phi, U, out, err);
    if (st != TLM_OK) return h->fail(st, err);
    if (u_max) *u_max = out.uMax;
    if (directivity) *directivity = out.directivity;
    if (peak_theta_deg) *peak_theta_deg = out.peakTheta;
    if (peak_phi_deg) *peak_phi_deg = out.peakPhi;
    return TLM_OK;
}

} // extern "C"
