// tlm_pair_kernel.cuh -- two SCN TLM steps in one pass over memory (FP32).
//
// The single-step kernels read 12 pulses and write 12 pulses per node and
// step, and run at 0.90 of the copy bandwidth: only fewer passes can make a
// step cheaper. Here a block owns a column of the grid, TX x TY nodes wide,
// and walks a range of z planes. For every plane it computes the first step on
// the column grown by one node on each side (the ring is computed by the
// neighbouring blocks as well) and then, one plane behind, the second step on
// the column itself. The first step's pulses never leave the block:
//   * its z pulses pass from plane to plane in the thread's registers (a
//     thread keeps its (x, y) for the whole walk);
//   * its x and y pulses cross threads through a shared-memory exchange buffer
//     of two planes, one barrier per plane;
//   * its stub voltages stay in registers.
// So two steps cost one read and one write of the state (plus the ring, which
// mostly hits L2). The arithmetic of a node is that of the interior and
// general tile bodies (tlm_step_kernel.cuh), in their order, so pulses, stubs
// and monitor samples are bitwise those of two single steps. An energy step
// leaves every pair's FP64 share in `epair`, and pairEnergySums adds those up in
// the order of the single-step kernels' tiles: the energies are bitwise too.
//
// The input planes come in by tensor-map bulk copies (TMA), five boxes per
// plane: x slots at the column, y slots with one more row on either side (the
// row next door holds the neighbour's pulse, the own row the pulse that an
// outer wall or a PEC neighbour reflects), z slots from the planes below and
// above. A box that reaches outside the grid reads zeros there. One thread
// issues a plane's boxes a few planes ahead, right after the barrier that ends
// the reads of the stage it refills.
//
// Stubs are read by the ring's owners while they are rewritten, so they are
// double-buffered like the pulses.
//
// Measured on a B200, one step: 192^3 air 111 -> 66 us, the 192^3 heterogeneous
// grid 127 -> 98 us, 128^3 heterogeneous 48 -> 36 us, a 384x384x256 dipole 566
// -> 340 us and beside a stub-loaded slab 645 -> 440 us. What bounds it: air
// columns move 0.64 GB a pass at 4.9 TB/s, 0.75 of the copy bandwidth, with 16
// warps per SM coupled by a barrier per plane; stub-loaded columns issue about
// 570 instructions per warp and plane instead of 330. Two blocks of 256 threads
// per SM (smaller columns, larger rings) measured 77 against 66 us in air, a
// 640-thread block 80 us (spills), a second walk without stub code for the
// blocks of a stub-loaded grid that hold none 125 against 98 us (spills).
#pragma once

#include "tlm_step_kernel.cuh"

#include <cmath>

namespace tlmk {


// Per (column, plane) flags: some node of the grown column or next to it is
// PEC / a source or monitor node lies in the grown column / it holds
// stub-loaded nodes / the plane is an outer z wall. The kernel adds the bits
// of the energy steps, so that one test sends a plane past all the rare work.
enum : unsigned { kPairPec = 1, kPairSpec = 2, kPairDiel = 4, kPairWallZ = 8, kPairEnergy0 = 16, kPairEnergy1 = 32 };

// A kernel shape: W pairs x H rows of threads cover the grown column (x0-2 ..
// x0+TX+1, y0-1 .. y0+TY), for TX <= 2W-4 and TY <= H-2; a stage row holds the
// W2 nodes from x0-4 on (16-byte aligned box starts). The strides are
// compile-time constants, so that shared-memory addresses are one register
// plus an immediate. Offsets in floats; boxes start on 128-byte boundaries.
template <int W_, int H_, int STAGES_, int MINB_> struct PairLayout
{
    static constexpr int W = W_, H = H_, W2 = 2 * W + 4;
    static constexpr int kStages = STAGES_, kMinBlocks = MINB_;
    static constexpr int kThreads = (W * H + 31) / 32 * 32;
    static constexpr int maxTX = 2 * W - 4, maxTY = H - 2;
    static constexpr int round32(int f) { return (f + 31) / 32 * 32; }
    static constexpr int sX = H * W2, sY = (H + 1) * W2;      // slot strides within a box
    static constexpr int offYL = round32(4 * sX);              // x slots first, then slots 6,7
    static constexpr int offYH = offYL + round32(2 * sY);      // slots 4,5
    static constexpr int offZL = offYH + round32(2 * sY);      // slots 10,11
    static constexpr int offZH = offZL + round32(2 * sX);      // slots 8,9
    static constexpr int stage = offZH + round32(2 * sX);
    static constexpr unsigned stageBytes = (unsigned)((8 * H + 4 * (H + 1)) * W2) * 4u;
    static constexpr int WE = 2 * W, exSlot = H * WE, exBuf = 8 * exSlot;  // exchange buffers of 8 slots
    static constexpr int offEx = kStages * stage;
    static constexpr int offTab = offEx + 2 * exBuf;           // material table: yhat, d = 4+yhat+ghat negated, 1/d
    static constexpr int smemBytes = (offTab + 3 * 256) * 4;
    static_assert(kMinBlocks * (smemBytes + 1024 + 512) <= 228 * 1024, "the blocks of an SM fit its shared memory");
};

struct PairArgs
{
    CUtensorMap mapX, mapY, mapZ;  // boxes of 4 x slots, 2 y slots (one more row), 2 z slots
    PairShape sh;
    const float *in;               // PEC planes read own z pulses directly
    float *out;
    const float *stubIn;
    float *stubOut;
    const float *yhat, *ghat;
    int ntable;
    float divLimit;                // stubDivLimit of the material table
    const unsigned *flags;         // [column][nz]
    long long P;
    int nx, ny, nz, px;
    float rho;
    const unsigned *words;         // material word of every pair, with its PEC faces
    const SpecEntry *spec;
    const int *specRow;            // first entry of every row of nodes, and their number after the last
    float sv[2];                   // source values of the two steps
    float *samples[2];             // [nsamp][6]
    double *epair[2];              // FP64 energy share of every pair (nullptr: no energy step)
    float neg_zero;
    unsigned long long stage_wait_ns;
    unsigned int *fault;
};

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    float2 r;
    asm("{\n\t.reg .b64 pa, pb, pc, pd;\n\tmov.b64 pa, {%2, %3};\n\tmov.b64 pb, {%4, %5};\n\t"
        "mov.b64 pc, {%6, %7};\n\tfma.rn.f32x2 pd, pa, pb, pc;\n\tmov.b64 {%0, %1}, pd;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}

// One source or monitor entry of a node of the pair (`second`: its second
// node), as in the general tile body: a soft source adds to the node's incident
// pulses, a monitor writes its node voltages and circulations to dst.
__device__ __forceinline__ void pairSpecEntry(const SpecEntry &se, bool second, float sv, float *dst, unsigned live,
                                              float2 (&inc)[12])
{
    if (se.kind == kInject)
    {
        const float qv = (0.5f * se.amp) * sv;
#pragma unroll
        for (int s = 0; s < 12; ++s)
            if ((s >> 2) != se.arg && fieldOfSlot(s) == se.arg)
            {
                if (second) inc[s].y = inc[s].y + qv;
                else inc[s].x = inc[s].x + qv;
            }
    }
    else if (dst != nullptr)
    {
        const bool on = (live >> (second ? 1 : 0)) & 1u;
        float v[12];
#pragma unroll
        for (int s = 0; s < 12; ++s) v[s] = on ? (second ? inc[s].y : inc[s].x) : 0.0f;
#pragma unroll
        for (int j = 0; j < 3; ++j) dst[j] = nodeVoltage(v, j);
#pragma unroll
        for (int k = 0; k < 3; ++k) dst[3 + k] = circulation(v, k);
    }
}
__device__ __forceinline__ void pairSpec(const PairArgs &a, int step, long long row, long long node0, bool own,
                                         unsigned live, float2 (&inc)[12])
{
    int lo = a.specRow[row];
    const int end = a.specRow[row + 1];
    for (int hi = end; hi - lo > 4;)  // rows that a plane wave fills
    {
        const int mid = (lo + hi) >> 1;
        if (a.spec[mid].node < node0) lo = mid; else hi = mid;
    }
    for (int e = lo; e < end; ++e)
    {
        const SpecEntry se = a.spec[e];
        if (se.node >= node0 + 2) break;
        if (se.node < node0) continue;
        pairSpecEntry(se, se.node != node0, a.sv[step], own ? a.samples[step] + (long long)se.arg * 6 : nullptr, live,
                      inc);
    }
}

// The material word of a pair: the two ids, which nodes are stub-loaded, and
// which are dead (PEC, row padding or outside the grid); the twelve bits above
// hold its PEC faces.
enum : unsigned { kMatDiel = 3u << 16, kMatDead = 3u << 18 };
__device__ __forceinline__ unsigned matWord(unsigned ids, unsigned dead)
{
    const unsigned i0 = ids & 255u, i1 = ids >> 8;
    dead |= (i0 == kPec ? 1u : 0u) | (i1 == kPec ? 2u : 0u);
    const unsigned diel = ((i0 >= kDiel0 ? 1u : 0u) | (i1 >= kDiel0 ? 2u : 0u)) & ~dead;
    return ids | (diel << 16) | (dead << 18);
}

// num / den for the three node voltages of a pair, rounded like the IEEE
// division, from the denominators' reciprocals y = RN(1/den) (nden = -den):
// q = RN(n y), then twice q <- RN(q + RN(n - den q) y). After the first
// correction q is within an ulp of the quotient, so the residual is exact and
// the second one rounds correctly (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990),
// as long as nothing under- or overflows: |n| < 2^120, and above the table's limit
// (stubDivLimit), so that the quotient is normal.
//
// The limit for a table whose denominators, 4 or more, reach denMax: 2^-100, for a
// denominator above 2^25 as much more as keeps the quotient above 2^-125, and
// infinity (every pair divides as IEEE does) above 2^40, where a quotient of
// scaled numerators may be subnormal as well, and for infinities and NaN.
__host__ __device__ __forceinline__ float stubDivLimit(float denMax)
{
    if (!(denMax <= 0x1p40f)) return HUGE_VALF;
    return denMax <= 0x1p25f ? 0x1p-100f : denMax * 0x1p-125f;
}
__device__ __forceinline__ void divByTable(const float2 (&num)[3], float2 nden, float2 rcp, float2 z, float2 (&q)[3])
{
#pragma unroll
    for (int j = 0; j < 3; ++j)
    {
        float2 t = mul2(num[j], rcp, z);
        t = fma2(fma2(t, nden, num[j]), rcp, t);
        q[j] = fma2(fma2(t, nden, num[j]), rcp, t);
    }
}

// Scatter of a pair that holds a stub-loaded node, both nodes through the stub
// formula: an air node is one with yhat = -0 and ghat = 0, whose (2 sum)/4 is
// its 0.5 sum (signed zeros and subnormals included). While a wave fills the
// grid many numerators are zero or tiny. Those lanes divide numerators scaled
// by 2^64 (exact) and scale the quotients q back: exact for a normal result;
// a subnormal one is rounded twice, which can only differ from rounding once
// where q is a tie of the subnormal grid but not the exact quotient: there q
// moves an ulp towards the exact quotient, on the side its residual tells. A
// zero quotient has the numerator's sign (den > 0). Lanes with numerators of
// 2^40 and more beside tiny ones take the IEEE division, and so do all where
// `limit` (stubDivLimit) is infinite.
__device__ __forceinline__ void pairScatterStub(const float *tab, const float2 (&in)[12], float2 (&vs)[3], unsigned m,
                                                float limit, float2 z, float2 (&out)[12])
{
    const unsigned diel = (m & kMatDiel) >> 16;
    const float *t0 = tab + (m & 255u), *t1 = tab + ((m >> 8) & 255u);
    const float2 yh = make_float2(t0[0], t1[0]), nden = make_float2(t0[256], t1[256]),
                 rcp = make_float2(t0[512], t1[512]);
    float2 Vn[3], ZI[3], num[3];
    float lo = 3e38f, hi = 0.0f;
#pragma unroll
    for (int j = 0; j < 3; ++j)
    {
        const int a = (j == 0) ? 1 : 0;
        const int b = (j == 2) ? 1 : 2;
        const float2 sum4 =
            add2(add2(add2(in[slotOf(a, 0, j)], in[slotOf(a, 1, j)]), in[slotOf(b, 0, j)]), in[slotOf(b, 1, j)]);
        num[j] = mul2(splat2(2.0f), add2(sum4, mul2(yh, vs[j], z)), z);
        lo = fminf(lo, fminf(fabsf(num[j].x), fabsf(num[j].y)));
        hi = fmaxf(hi, fmaxf(fabsf(num[j].x), fabsf(num[j].y)));
    }
    if (lo > limit && hi < 0x1p120f)
        divByTable(num, nden, rcp, z, Vn);
    else if (hi == 0.0f && limit < 1.0f)
    {
#pragma unroll
        for (int j = 0; j < 3; ++j) Vn[j] = num[j];
    }
    else if (hi < 0x1p40f && limit < 1.0f)
    {
        // distance of each scaled quotient from the value it scales back to
        auto off = [&](float2 q) { return sub2(q, mul2(mul2(q, splat2(0x1p-64f), z), splat2(0x1p64f), z)); };
        bool tie = false;
#pragma unroll
        for (int j = 0; j < 3; ++j) num[j] = mul2(num[j], splat2(0x1p64f), z);
        divByTable(num, nden, rcp, z, Vn);
#pragma unroll
        for (int j = 0; j < 3; ++j)
        {
            const float2 d = off(Vn[j]);
            tie = tie || fabsf(d.x) == 0x1p-86f || fabsf(d.y) == 0x1p-86f;
        }
        if (tie)
        {
#pragma unroll
            for (int j = 0; j < 3; ++j)
            {
                const float2 d = off(Vn[j]), r = fma2(Vn[j], nden, num[j]);
                auto nudge = [](float q, float dd, float rr) {
                    const int up = (rr > 0.0f) == (q > 0.0f) ? 1 : -1;
                    return fabsf(dd) == 0x1p-86f && rr != 0.0f ? __int_as_float(__float_as_int(q) + up) : q;
                };
                Vn[j] = make_float2(nudge(Vn[j].x, d.x, r.x), nudge(Vn[j].y, d.y, r.y));
            }
        }
#pragma unroll
        for (int j = 0; j < 3; ++j)
        {
            const float2 v = mul2(Vn[j], splat2(0x1p-64f), z);
            Vn[j] = make_float2(copysignf(v.x, num[j].x), copysignf(v.y, num[j].y));
        }
    }
    else
    {
#pragma unroll
        for (int j = 0; j < 3; ++j)
            Vn[j] = make_float2((diel & 1u) ? stubDiv(num[j].x, -nden.x) : nodeVoltage2(in, j, z).x,
                                (diel & 2u) ? stubDiv(num[j].y, -nden.y) : nodeVoltage2(in, j, z).y);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) ZI[k] = circulation2(in, k, z);
    reflectLinks2(in, Vn, ZI, out);
#pragma unroll
    for (int j = 0; j < 3; ++j)
    {
        const float2 v = sub2(Vn[j], vs[j]);
        if (diel & 1u) vs[j].x = v.x;
        if (diel & 2u) vs[j].y = v.y;
    }
}

__device__ __forceinline__ double pairEnergy(const float2 (&inc)[12], unsigned live)
{
    double e = 0.0;
    if (live & 1u)
    {
#pragma unroll
        for (int s = 0; s < 12; ++s) e += (double)inc[s].x * (double)inc[s].x;
    }
    if (live & 2u)
    {
#pragma unroll
        for (int s = 0; s < 12; ++s) e += (double)inc[s].y * (double)inc[s].y;
    }
    return e;
}

__device__ __forceinline__ unsigned pecPair(const uint8_t *m)
{
    const unsigned v = *reinterpret_cast<const unsigned short *>(m);
    return ((v & 255u) == kPec ? 1u : 0u) | ((v >> 8) == kPec ? 2u : 0u);
}
// Faces of the pair at (x, j, k) behind which a PEC node lies, two bits per face
// (one per node of the pair): -x +x -y +y -z +z. A neighbour outside the grid
// counts as none (the wall comes first, as in the general tile body).
__device__ __forceinline__ unsigned pairPecFaces(const uint8_t *mat, int nx, int ny, int nz, int px, int x, int j, int k,
                                                 long long node0)
{
    const long long sz = (long long)px * ny;
    const unsigned own = pecPair(mat + node0);
    unsigned xm = (own << 1) & 2u, xp = x + 1 < nx ? own >> 1 : 0u;
    if (x > 0 && mat[node0 - 1] == kPec) xm |= 1u;
    if (x + 2 < nx && mat[node0 + 2] == kPec) xp |= 2u;
    unsigned f = xm | xp << 2;
    if (j > 0) f |= pecPair(mat + node0 - px) << 4;
    if (j < ny - 1) f |= pecPair(mat + node0 + px) << 6;
    if (k > 0) f |= pecPair(mat + node0 - sz) << 8;
    if (k < nz - 1) f |= pecPair(mat + node0 + sz) << 10;
    return f;
}
__device__ __forceinline__ void negWhere(float2 &v, unsigned mask, float2 own)
{
    if (mask & 1u) v.x = -own.x;
    if (mask & 2u) v.y = -own.y;
}
// DIEL: the grid has stub-loaded nodes.
template <class L, bool DIEL>
__global__ void __launch_bounds__(L::kThreads, L::kMinBlocks) stepPairKernel(const __grid_constant__ PairArgs a)
{
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(8) unsigned long long full[L::kStages];
    const PairShape &g = a.sh;
    const int tid = threadIdx.x;
    const int ncol = g.ntx * g.nty;
    const int col = blockIdx.x % ncol, chunk = blockIdx.x / ncol;
    const int x0 = (col % g.ntx) * g.TX, y0 = (col / g.ntx) * g.TY;
    const int kc0 = (int)((long long)chunk * a.nz / g.nchunk), kc1 = (int)((long long)(chunk + 1) * a.nz / g.nchunk);
    const int kA = kc0 > 0 ? kc0 - 1 : 0;        // first plane of the first step
    const int kB = kc1 < a.nz ? kc1 : a.nz - 1;  // its last plane
    const unsigned *colFlags = a.flags + (long long)col * a.nz;
    const unsigned full0 = smemAddr(full), sm0 = smemAddr(sm);
    if (tid == 0)
    {
        for (int s = 0; s < L::kStages; ++s)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" : : "r"(full0 + 8 * s) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" : : : "memory");
    }
    float *tab = sm + L::offTab;
    if constexpr (DIEL)
        for (int m = tid; m < 256; m += L::kThreads)
        {
            const bool in = m >= kDiel0 && m - kDiel0 < a.ntable;
            const float yh = in ? a.yhat[m - kDiel0] : -0.0f, gh = in ? a.ghat[m - kDiel0] : 0.0f;
            const float den = (4.0f + yh) + gh;
            tab[m] = yh;
            tab[256 + m] = -den;
            tab[512 + m] = __frcp_rn(den);
        }
    __syncthreads();

    // one plane's boxes: x slots; y slots 6,7 from row y0-2, 4,5 from row
    // y0-1 (H+1 rows each); z slots 10,11 one plane below (on the lowest
    // plane the own 8,9), 8,9 one plane above (highest: the own 10,11)
    auto issue = [&](int k) {
        const int s = (k - kA) % L::kStages;
        const unsigned st = sm0 + (unsigned)(s * L::stage) * 4u, bar = full0 + 8 * s;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" : : "r"(bar), "r"(L::stageBytes) : "memory");
        const int xs = x0 - 4, ys = y0 - 1;
        tmaBox4(st, &a.mapX, xs, ys, k, 0, bar);
        tmaBox4(st + L::offYL * 4u, &a.mapY, xs, ys - 1, k, 6, bar);
        tmaBox4(st + L::offYH * 4u, &a.mapY, xs, ys, k, 4, bar);
        tmaBox4(st + L::offZL * 4u, &a.mapZ, xs, ys, k == 0 ? 0 : k - 1, k == 0 ? 8 : 10, bar);
        tmaBox4(st + L::offZH * 4u, &a.mapZ, xs, ys, k == a.nz - 1 ? k : k + 1, k == a.nz - 1 ? 10 : 8, bar);
    };
    int lastIssued = kA - 1;  // thread 0's
    if (tid == 0)
        while (lastIssued < kB && lastIssued + 1 < kA + L::kStages) issue(++lastIssued);

    // the thread's pair of nodes
    const bool inExt = tid < L::W * L::H;
    const int r = inExt ? tid / L::W : 0, p = inExt ? tid - r * L::W : 0;
    const int x = x0 - 2 + 2 * p, j = y0 - 1 + r;
    const bool valid = inExt && x >= 0 && x < a.px && j >= 0 && j < a.ny && p <= g.TX / 2 + 1 && r <= g.TY + 1;
    const bool own = valid && p >= 1 && p <= g.TX / 2 && r >= 1 && r <= g.TY;
    const unsigned dead = !valid ? 3u : (x + 1 < a.nx ? 0u : x < a.nx ? 2u : 3u);
    const unsigned ownLanes = __ballot_sync(0xffffffffu, own);
    const long long sz = (long long)a.px * a.ny;
    const unsigned colOff = valid ? (unsigned)j * (unsigned)a.px + (unsigned)x : 0u;  // node within a plane
    const bool atYlo = j == 0, atYhi = j == a.ny - 1, atXlo = x == 0;
    const int cHi = a.nx - 1 - x;  // 0 or 1: the pair's node on the high x wall
    // An outer wall reflects rho times the own pulse: its lanes read the own
    // pulse of the face (by offset) and scale it; every other lane reads the
    // neighbour's and scales by one, which changes nothing.
    const float cXm = atXlo ? a.rho : 1.0f, cXp0 = cHi == 0 ? a.rho : 1.0f, cXp1 = cHi == 1 ? a.rho : 1.0f;
    const float2 cYm = splat2(atYlo ? a.rho : 1.0f), cYp = splat2(atYhi ? a.rho : 1.0f);
    // stage offsets of the own pair, of slots 2,3 at x-1, of slots 0,1 at x+1
    // and x+2, of slots 6,7 one row below and 4,5 one row above
    const int oX = r * L::W2 + 2 * p + 2;
    const int oXm = atXlo ? oX : 2 * L::sX + oX - 1;
    const int oXp0 = cHi == 0 ? 2 * L::sX + oX : oX + 1, oXp1 = cHi == 1 ? 2 * L::sX + oX + 1 : oX + 2;
    const int oYm = atYlo ? L::offYH + oX : L::offYL + oX;
    const int oYp = atYhi ? L::offYL + oX + L::W2 : L::offYH + oX + L::W2;
    // the same in the exchange buffers
    const int e0 = L::offEx + r * L::WE + 2 * p;
    const int eXm = atXlo ? e0 : 2 * L::exSlot + e0 - 1;
    const int eXp0 = cHi == 0 ? 2 * L::exSlot + e0 : e0 + 1, eXp1 = cHi == 1 ? 2 * L::exSlot + e0 + 1 : e0 + 2;
    const int eYm = atYlo ? 4 * L::exSlot + e0 : 6 * L::exSlot + e0 - L::WE;
    const int eYp = atYhi ? 6 * L::exSlot + e0 : 4 * L::exSlot + e0 + L::WE;
    const float2 negZero = splat2(a.neg_zero);

    // `lanes`: the lanes of the warp that scatter here
    auto scatter = [&](unsigned lanes, unsigned f, const float2(&inc)[12], float2(&vs)[3], unsigned m,
                       float2(&out)[12]) {
        if (DIEL && (f & kPairDiel) && __any_sync(lanes, (m & kMatDiel) != 0))
            pairScatterStub(tab, inc, vs, m, a.divLimit, negZero, out);
        else
            scatterAir2(inc, out, negZero);
    };
    const unsigned energyBits = (a.epair[0] ? kPairEnergy0 : 0u) | (a.epair[1] ? kPairEnergy1 : 0u);
    auto flagsAt = [&](int k) -> unsigned { return k <= kB ? colFlags[k] | energyBits : 0u; };
    // material word of the pair (only its dead nodes where the plane's flags say
    // neither PEC nor dielectric), fetched two planes ahead, the flags three
    auto wordAt = [&](int k, unsigned f) -> unsigned {
        if (!(f & (kPairPec | kPairDiel)) || !valid) return dead << 18;
        return a.words[(k * sz + colOff) >> 1];
    };
    auto loadStub = [&](unsigned m, int k, float2(&v)[3]) {
#pragma unroll
        for (int t = 0; t < 3; ++t) v[t] = make_float2(0.f, 0.f);
        if (m & kMatDiel)
        {
#pragma unroll
            for (int t = 0; t < 3; ++t)
                v[t] = *reinterpret_cast<const float2 *>(reinterpret_cast<const char *>(a.stubIn + t * a.P + k * sz) +
                                                         colOff * 4u);
        }
    };

    // The first step's z slots and stubs of a plane, by plane parity
    // (relative to kA), so that the loop body, unrolled by two, moves nothing.
    float2 z89[2][2], z1011[2][2], vs[2][3];
#pragma unroll
    for (int b = 0; b < 2; ++b)
    {
#pragma unroll
        for (int t = 0; t < 2; ++t) z89[b][t] = z1011[b][t] = make_float2(0.f, 0.f);
#pragma unroll
        for (int t = 0; t < 3; ++t) vs[b][t] = make_float2(0.f, 0.f);
    }
    unsigned f0 = flagsAt(kA), f1 = flagsAt(kA + 1), f2 = flagsAt(kA + 2), fPrev = 0;
    unsigned m0 = wordAt(kA, f0), m1 = wordAt(kA + 1, f1), mPrev = 0;
    if constexpr (DIEL) loadStub(m0, kA, vs[0]);
    bool waitOk = true;
    int si = 0;
    unsigned phase = 0;

    // The second step at plane k-1, after the first step at plane k (B: parity
    // of plane k).
    auto second = [&](auto par, int k) {
        constexpr int B = decltype(par)::value;
        const int kk = k - 1;
        const float *ex = sm + (B ^ 1) * L::exBuf;
        float2 inc[12];
#pragma unroll
        for (int t = 0; t < 2; ++t)
        {
            inc[t] = make_float2(cXm * ex[eXm + t * L::exSlot], ex[e0 + (2 + t) * L::exSlot]);
            inc[2 + t] = make_float2(cXp0 * ex[eXp0 + t * L::exSlot], cXp1 * ex[eXp1 + t * L::exSlot]);
            inc[4 + t] = mul2(ld2(ex + eYm + t * L::exSlot), cYm, negZero);
            inc[6 + t] = mul2(ld2(ex + eYp + t * L::exSlot), cYp, negZero);
            inc[8 + t] = z1011[B][t];  // plane k-2
            inc[10 + t] = z89[B][t];   // plane k
        }
        if (fPrev & ~kPairDiel)
        {
#pragma unroll
            for (int t = 0; t < 2; ++t)
            {
                if (kk == 0) inc[8 + t] = mul2(z89[B ^ 1][t], splat2(a.rho), negZero);
                if (kk == a.nz - 1) inc[10 + t] = mul2(z1011[B ^ 1][t], splat2(a.rho), negZero);
            }
            if (fPrev & kPairPec)
            {
                const unsigned q = mPrev >> 20;
                if (q)
                {
#pragma unroll
                    for (int t = 0; t < 2; ++t)
                    {
                        negWhere(inc[t], q & 3u, ld2(ex + e0 + t * L::exSlot));
                        negWhere(inc[2 + t], (q >> 2) & 3u, ld2(ex + e0 + (2 + t) * L::exSlot));
                        negWhere(inc[4 + t], (q >> 4) & 3u, ld2(ex + e0 + (4 + t) * L::exSlot));
                        negWhere(inc[6 + t], (q >> 6) & 3u, ld2(ex + e0 + (6 + t) * L::exSlot));
                        negWhere(inc[8 + t], (q >> 8) & 3u, z89[B ^ 1][t]);
                        negWhere(inc[10 + t], (q >> 10) & 3u, z1011[B ^ 1][t]);
                    }
                }
            }
            const unsigned live = 3u & ~(mPrev >> 18);
            if (fPrev & kPairSpec) pairSpec(a, 1, (long long)kk * a.ny + j, kk * sz + colOff, true, live, inc);
            if (fPrev & kPairEnergy1) a.epair[1][(kk * sz + colOff) >> 1] = pairEnergy(inc, live);
        }
        float2 o[12];
        scatter(ownLanes, fPrev, inc, vs[B ^ 1], mPrev, o);
        if (__any_sync(ownLanes, (mPrev & kMatDead) != 0))
        {
#pragma unroll
            for (int s = 0; s < 12; ++s)
            {
                if (mPrev & (1u << 18)) o[s].x = 0.0f;
                if (mPrev & (2u << 18)) o[s].y = 0.0f;
            }
        }
        // uniform plane pointers and a 32-bit lane offset
        char *const base = reinterpret_cast<char *>(a.out + kk * sz);
        const unsigned off = colOff * 4u;
        if (TLM_GUARD(kk * sz + colOff, a.P - 1, 14))
        {
#pragma unroll
            for (int s = 0; s < 12; ++s) *reinterpret_cast<float2 *>(base + s * a.P * 4 + off) = o[s];
            if constexpr (DIEL)
                if (mPrev & kMatDiel)
                {
#pragma unroll
                    for (int t = 0; t < 3; ++t)
                        *reinterpret_cast<float2 *>(reinterpret_cast<char *>(a.stubOut + t * a.P + kk * sz) + off) =
                            vs[B ^ 1][t];
                }
        }
    };

    auto plane = [&](auto par, int k) {
        constexpr int B = decltype(par)::value;
        const unsigned m2 = wordAt(k + 2, f2), f3 = flagsAt(k + 3);
        float2 s1011[2], vsNext[3];
        if (k <= kB)
        {
            // ---- first step at plane k ----
            if constexpr (DIEL)
                if (k < kB) loadStub(m1, k + 1, vsNext);  // used from the next plane on
            if (waitOk && !mbarWaitBounded(full0 + 8 * si, phase, a.stage_wait_ns))
            {
                waitOk = false;
                if (a.fault) atomicOr(a.fault, kStageTimeout);
            }
            const float *st = sm + si * L::stage;
            float2 inc[12];
#pragma unroll
            for (int t = 0; t < 2; ++t)
            {
                inc[t] = make_float2(cXm * st[oXm + t * L::sX], st[oX + (2 + t) * L::sX]);
                inc[2 + t] = make_float2(cXp0 * st[oXp0 + t * L::sX], cXp1 * st[oXp1 + t * L::sX]);
                inc[4 + t] = mul2(ld2(st + oYm + t * L::sY), cYm, negZero);
                inc[6 + t] = mul2(ld2(st + oYp + t * L::sY), cYp, negZero);
                inc[8 + t] = ld2(st + L::offZL + t * L::sX + oX);
                inc[10 + t] = ld2(st + L::offZH + t * L::sX + oX);
            }
            if (f0 & ~kPairDiel)
            {
#pragma unroll
                for (int t = 0; t < 2; ++t)
                {
                    if (k == 0) inc[8 + t] = mul2(inc[8 + t], splat2(a.rho), negZero);
                    if (k == a.nz - 1) inc[10 + t] = mul2(inc[10 + t], splat2(a.rho), negZero);
                }
                const long long node0 = k * sz + colOff;
                const unsigned q = m0 >> 20;
                if (q)
                {
#pragma unroll
                    for (int t = 0; t < 2; ++t)
                    {
                        negWhere(inc[t], q & 3u, ld2(st + t * L::sX + oX));
                        negWhere(inc[2 + t], (q >> 2) & 3u, ld2(st + (2 + t) * L::sX + oX));
                        negWhere(inc[4 + t], (q >> 4) & 3u, ld2(st + L::offYH + t * L::sY + oX));
                        negWhere(inc[6 + t], (q >> 6) & 3u, ld2(st + L::offYL + t * L::sY + oX + L::W2));
                        if ((q >> 8) & 3u) negWhere(inc[8 + t], (q >> 8) & 3u, ld2(a.in + (8 + t) * a.P + node0));
                        if ((q >> 10) & 3u) negWhere(inc[10 + t], (q >> 10) & 3u, ld2(a.in + (10 + t) * a.P + node0));
                    }
                }
                const unsigned live = 3u & ~(m0 >> 18);
                const bool mine = own && k >= kc0 && k < kc1;
                if ((f0 & kPairSpec) && valid) pairSpec(a, 0, (long long)k * a.ny + j, node0, mine, live, inc);
                if ((f0 & kPairEnergy0) && mine) a.epair[0][node0 >> 1] = pairEnergy(inc, live);
            }
            // Pulses of dead nodes need not be zeroed here: their neighbours
            // reflect their own (PEC, walls) and the second step writes zeros.
            float2 s1[12];
            scatter(0xffffffffu, f0, inc, vs[B], m0, s1);
            // x and y slots go to the block, z slots stay with the thread
            if (inExt)
            {
                float *ex = sm + B * L::exBuf + e0;
#pragma unroll
                for (int s = 0; s < 8; ++s) *reinterpret_cast<float2 *>(ex + s * L::exSlot) = s1[s];
            }
#pragma unroll
            for (int t = 0; t < 2; ++t)
            {
                z89[B][t] = s1[8 + t];
                s1011[t] = s1[10 + t];
            }
        }
        if (own && k > kc0) second(par, k);
        if (k <= kB)
        {
#pragma unroll
            for (int t = 0; t < 2; ++t) z1011[B][t] = s1011[t];
            if constexpr (DIEL)
            {
#pragma unroll
                for (int t = 0; t < 3; ++t) vs[B ^ 1][t] = vsNext[t];
            }
        }
        __syncthreads();
        // (after a wait that ran out no stage is refilled: its copy may still
        // be landing, and the other threads give up in turn)
        if (tid == 0 && waitOk && lastIssued < kB) issue(++lastIssued);
        mPrev = m0;
        m0 = m1;
        m1 = m2;
        fPrev = f0;
        f0 = f1;
        f1 = f2;
        f2 = f3;
        if (++si == L::kStages)
        {
            si = 0;
            phase ^= 1u;
        }
    };
    for (int k = kA; k <= kc1; k += 2)  // the second step of plane kc1-1 runs in iteration kc1
    {
        plane(std::integral_constant<int, 0>{}, k);
        if (k + 1 <= kc1) plane(std::integral_constant<int, 1>{}, k + 1);
    }
    // Thread 0 waited for every copy, unless a wait ran out: then let those
    // still in flight land before the block's memory goes.
    if (!waitOk && tid == 0)
        for (int k = max(kA, lastIssued - L::kStages + 1); k <= lastIssued; ++k)
            mbarWaitBounded(full0 + 8 * ((k - kA) % L::kStages), (unsigned)((k - kA) / L::kStages) & 1u);
}

// Flags of every (column, plane): PEC and dielectric nodes from the padded
// material map (one block per column and plane; PEC within one node of the
// grown column, the planes below and above included).
static __global__ void __launch_bounds__(128) pairMaterialFlags(const uint8_t *__restrict__ mat, int nx, int ny, int nz, int px,
                                                         PairShape g, unsigned *__restrict__ flags)
{
    const int k = blockIdx.x % nz, col = blockIdx.x / nz;
    const int x0 = (col % g.ntx) * g.TX, y0 = (col / g.ntx) * g.TY;
    const int xa = max(x0 - 3, 0), xb = min(x0 + g.TX + 2, nx - 1);
    const int ya = max(y0 - 2, 0), yb = min(y0 + g.TY + 1, ny - 1);
    const int za = max(k - 1, 0), zb = min(k + 1, nz - 1);
    const int w = xb - xa + 1, hgt = yb - ya + 1;
    unsigned f = 0;
    for (int t = threadIdx.x; t < w * hgt * (zb - za + 1); t += blockDim.x)
    {
        const int i = t % w, jj = (t / w) % hgt, kk = za + t / (w * hgt);
        const uint8_t m = mat[((long long)kk * ny + ya + jj) * px + xa + i];
        if (m == kPec) f |= kPairPec;
        else if (m >= kDiel0 && kk == k) f |= kPairDiel;
    }
    f = __reduce_or_sync(0xffffffffu, f);
    if (k == 0 || k == nz - 1) f |= kPairWallZ;
    if ((threadIdx.x & 31) == 0 && f) atomicOr(flags + (long long)col * nz + k, f);
}

// The material word of every pair, and the first source or monitor entry of
// every row of nodes (entries are sorted by node).
static __global__ void __launch_bounds__(256) pairWordKernel(const uint8_t *__restrict__ mat, int nx, int ny, int nz, int px,
                                                             FastDiv divH, FastDiv divY, unsigned npairs,
                                                             unsigned *__restrict__ words)
{
    const unsigned q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= npairs) return;
    const unsigned row = fastDiv(q, divH), k = fastDiv(row, divY);
    const int x = 2 * (int)(q - row * (unsigned)(px / 2)), j = (int)(row - k * (unsigned)ny);
    words[q] = matWord(*reinterpret_cast<const unsigned short *>(mat + 2LL * q), x + 1 < nx ? 0u : x < nx ? 2u : 3u) |
               pairPecFaces(mat, nx, ny, nz, px, x, j, (int)k, 2LL * q) << 20;
}
static __global__ void __launch_bounds__(256) pairSpecRows(const SpecEntry *__restrict__ spec, int n, int rows, int px,
                                                           int *__restrict__ first)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r > rows) return;
    int lo = 0, hi = n;
    while (lo < hi)
    {
        const int mid = (lo + hi) >> 1;
        if (spec[mid].node < (long long)r * px) lo = mid + 1; else hi = mid;
    }
    first[r] = lo;
}

// ... and the columns whose grown area holds a source or monitor node.
static __global__ void __launch_bounds__(128) pairSpecFlags(const SpecEntry *__restrict__ spec, int n, int ny, int nz, int px,
                                                     PairShape g, unsigned *__restrict__ flags)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const long long node = spec[e].node;
    const int x = (int)(node % px), j = (int)((node / px) % ny), k = (int)(node / ((long long)px * ny));
    for (int ty = max(j / g.TY - 1, 0); ty <= min(j / g.TY + 1, g.nty - 1); ++ty)
        for (int tx = max(x / g.TX - 1, 0); tx <= min(x / g.TX + 1, g.ntx - 1); ++tx)
            if (x >= tx * g.TX - 2 && x < tx * g.TX + g.TX + 2 && j >= ty * g.TY - 1 && j <= ty * g.TY + g.TY)
                atomicOr(flags + (long long)(ty * g.ntx + tx) * nz + k, (unsigned)kPairSpec);
}

// The tiles' energy sums from the pairs' shares: block (tile, energy step), in
// the order of blockSumDouble as the single-step kernels use it.
static __global__ void __launch_bounds__(kBlock) pairEnergySums(const double *__restrict__ epair, long long npairs,
                                                         double *__restrict__ epart, int nblocks)
{
    __shared__ double red[kBlock / 32];
    const long long q = (long long)blockIdx.x * kBlock + threadIdx.x;
    const double tot = blockSumDouble(q < npairs ? epair[blockIdx.y * npairs + q] : 0.0, red);
    if (threadIdx.x == 0) epart[(long long)blockIdx.y * nblocks + blockIdx.x] = tot;
}

} // namespace tlmk
