// tlm_resident_kernel.cuh -- many SCN TLM steps of a small FP32 grid in one
// launch, the state held in shared memory.
//
// A grid of up to about 300,000 nodes fits the shared memory of the GPU, and
// its steps are bound by latency: a launch (or two) per step, and inside it a
// chain of dependent loads (flags, material, neighbours' materials, pulses,
// sources and monitors). Here every block owns a brick of whole x rows, by
// rows in y and bz planes, for a whole launch window:
//   * the pulses live in two shared-memory buffers (the state and the next
//     one), the stubs in one, and everything that does not change
//     between steps (materials, PEC neighbours, walls, source and monitor
//     entries of a node) is worked out once per launch;
//   * only the y and z pulses that leave the brick go through global memory, as
//     8-byte packets of a pulse and the number of its step, written and read
//     whole. A thread polls the packets of its own nodes and needs no counter,
//     no fence and no other thread for it: the chain of a step is one store,
//     one load and the node's arithmetic. A node and the one across the face
//     send each other a packet per step, so two sets of packets, by step
//     parity, suffice: a node overwrites a packet of two steps ago only after
//     it received the other's packet of the last step, which the other sent
//     after reading that one;
//   * one barrier of the block ends a step.
// The blocks wait on one another, so the launch is cooperative (all blocks
// resident); every wait is bounded by the global timer, and one that runs out
// sets kResidentTimeout in *fault and stops waiting.
//
// The arithmetic of a node is that of the interior and general tile bodies in
// their order: pulses, stubs and samples are bitwise the same. Energy steps
// leave every pair's FP64 share in `epair`; pairEnergySums adds those up in the
// order of the single-step kernels' tiles, so the energies are the same too.
#pragma once

#include "tlm_pair_kernel.cuh"

namespace tlmk {

constexpr int kResidentThreads = 512;
constexpr unsigned kResidentTimeout = 1u << 30;
constexpr int kResidentSteps = 64;      // steps per launch at most
constexpr int kResidentEntries = 64;    // source and monitor entries of a brick kept in shared memory

// The four packets (32 bytes) that a pair receives across one face: two nodes
// of two slots.
struct __align__(16) ResPacket
{
    unsigned long long p[4];
};

struct ResidentArgs
{
    float *buf[2];            // pulse buffers; the state is in buf[0]
    float *stub;              // 3 planes (nullptr without dielectrics)
    const uint8_t *mat;
    const float *yhat, *ghat;
    int ntable;
    float divLimit;           // stubDivLimit of the material table
    long long P;
    int nx, ny, nz, px;
    int by, bz, gy, gz;       // rows and planes per brick (2 or more, or all), bricks in y and z
    float rho, neg_zero;
    const SpecEntry *spec;
    int nspec;
    float *samples;           // [step of this launch][nsamp][6]
    int nsamp;
    int steps;
    int first;                // absolute index of the first step (energy every 16)
    double *epair;            // [energy step of this launch][P / 2]
    ResPacket *packY, *packZ; // [parity][from below / above][brick][plane or row][pair]
    unsigned base;            // number of the step before this launch's first
    unsigned *fault;
    float sv[kResidentSteps]; // source value of every step
};

// What a pair needs to know about its place, worked out once per launch.
// Bits 0-11: PEC neighbours (two bits per face: -x +x -y +y -z +z); then walls
// and halo faces (at most one in y and one in z).
enum : unsigned
{
    kResPec = 0xfffu,
    kResWallXlo = 1u << 12, kResWallX0 = 1u << 13, kResWallX1 = 1u << 14,  // the pair's first / second node at x = nx-1
    kResWallYlo = 1u << 15, kResWallYhi = 1u << 16, kResWallZlo = 1u << 17, kResWallZhi = 1u << 18,
    kResHaloYlo = 1u << 19, kResHaloYhi = 1u << 20, kResHaloZlo = 1u << 21, kResHaloZhi = 1u << 22,
    kResHaloY = 3u << 19, kResHaloZ = 3u << 21, kResHalo = 15u << 19, kResWall = 127u << 12,
    kResSpec = 1u << 23, kResDead = 1u << 24, kResUsed = 1u << 25,
    kResRare = kResPec | kResWall | kResSpec
};

struct ResEntry
{
    float amp;
    unsigned code;  // argument << 2 | kind << 1 | second node of the pair
};

// Shared-memory layout (floats): two buffers of 12 slots, the stub planes, the
// material table, the entries. A slot holds the block's pairs in thread order,
// so slot strides are constants.
template <int M, bool DIEL> struct ResidentLayout
{
    static constexpr int SS = 2 * kResidentThreads * M;
    static constexpr int buf = 12 * SS + 8;  // (a pair at the end of a slot reads past it)
    static constexpr int offStub = 2 * buf, offTab = offStub + (DIEL ? 3 * SS : 0), offEnt = offTab + (DIEL ? 768 : 0);
    static constexpr int smemBytes = (offEnt + 2 * kResidentEntries) * 4;
};

__device__ __forceinline__ unsigned long long packet(float v, unsigned step)
{
    return (unsigned long long)step << 32 | __float_as_uint(v);
}
__device__ __forceinline__ void sendPackets(ResPacket *d, float2 a, float2 b, unsigned step)
{
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};"
                 : : "l"(d->p), "l"(packet(a.x, step)), "l"(packet(a.y, step)) : "memory");
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};"
                 : : "l"(d->p + 2), "l"(packet(b.x, step)), "l"(packet(b.y, step)) : "memory");
}
struct ResPulses
{
    unsigned long long v[4];
    __device__ __forceinline__ void load(const ResPacket *d)
    {
        asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v[0]), "=l"(v[1]) : "l"(d->p) : "memory");
        asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v[2]), "=l"(v[3]) : "l"(d->p + 2) : "memory");
    }
    __device__ __forceinline__ unsigned off(unsigned step) const  // 0: all four packets are of `step`
    {
        return ((unsigned)(v[0] >> 32) ^ step) | ((unsigned)(v[1] >> 32) ^ step) | ((unsigned)(v[2] >> 32) ^ step) |
               ((unsigned)(v[3] >> 32) ^ step);
    }
    __device__ __forceinline__ float2 get(int t) const
    {
        return make_float2(__uint_as_float((unsigned)v[2 * t]), __uint_as_float((unsigned)v[2 * t + 1]));
    }
};

// M (1 or 2) pairs per thread; DIEL: the grid has stub-loaded nodes.
template <int M, bool DIEL>
__global__ void __launch_bounds__(kResidentThreads, 1) residentKernel(const __grid_constant__ ResidentArgs a)
{
    using L = ResidentLayout<M, DIEL>;
    extern __shared__ __align__(128) float sm[];
    __shared__ int entries;
    const int tid = threadIdx.x;
    const int bj = blockIdx.x % a.gy, bk = blockIdx.x / a.gy;
    const int ya = bj * a.by, za = bk * a.bz;
    const int ny = min(a.by, a.ny - ya), nz = min(a.bz, a.nz - za);
    const int hx = a.px / 2, rows = a.by * a.bz;
    float *const stubs = sm + L::offStub;  // updated in place by each pair's thread
    float *const tab = sm + L::offTab;
    ResEntry *const ent = reinterpret_cast<ResEntry *>(sm + L::offEnt);
    const long long sz = (long long)a.px * a.ny;
    if (tid == 0) entries = 0;
    if constexpr (DIEL)
        for (int m = tid; m < 256; m += kResidentThreads)
        {
            const bool in = m >= kDiel0 && m - kDiel0 < a.ntable;
            const float yh = in ? a.yhat[m - kDiel0] : -0.0f, gh = in ? a.ghat[m - kDiel0] : 0.0f;
            const float den = (4.0f + yh) + gh;
            tab[m] = yh;
            tab[256 + m] = -den;
            tab[512 + m] = __frcp_rn(den);
        }
    __syncthreads();

    unsigned info[M], word[M], spec[M];
    int at[M], oYm[M], oYp[M], oZm[M], oZp[M];  // offsets of the pair and of the rows it gathers from
    unsigned node[M], pkY[M], pkZ[M];           // node within the grid; packet places
#pragma unroll
    for (int m = 0; m < M; ++m)
    {
        const int q = tid + m * kResidentThreads;
        const int r = q / hx, x = 2 * (q - r * hx), kk = r / a.by, jj = r - kk * a.by;
        info[m] = word[m] = spec[m] = node[m] = pkY[m] = pkZ[m] = 0;
        at[m] = oYm[m] = oYp[m] = oZm[m] = oZp[m] = 0;
        if (r < rows && jj < ny && kk < nz)
        {
            const int j = ya + jj, k = za + kk;
            const long long n0 = k * sz + (long long)j * a.px + x;
            node[m] = (unsigned)n0;
            const int o = 2 * q;
            at[m] = o;
            unsigned f = kResUsed;
            f |= pairPecFaces(a.mat, a.nx, a.ny, a.nz, a.px, x, j, k, n0);
            if (x == 0) f |= kResWallXlo;
            if (x == a.nx - 1) f |= kResWallX0;
            if (x + 1 == a.nx - 1) f |= kResWallX1;
            if (j == 0) f |= kResWallYlo;
            else if (jj == 0) f |= kResHaloYlo;
            if (j == a.ny - 1) f |= kResWallYhi;
            else if (jj == ny - 1) f |= kResHaloYhi;
            if (k == 0) f |= kResWallZlo;
            else if (kk == 0) f |= kResHaloZlo;
            if (k == a.nz - 1) f |= kResWallZhi;
            else if (kk == nz - 1) f |= kResHaloZhi;
            // walls and halo faces gather from the own row (slots 4-11 in place)
            oYm[m] = (f & (kResWallYlo | kResHaloYlo)) ? o - 2 * L::SS : o - a.px;
            oYp[m] = (f & (kResWallYhi | kResHaloYhi)) ? o + 2 * L::SS : o + a.px;
            oZm[m] = (f & (kResWallZlo | kResHaloZlo)) ? o - 2 * L::SS : o - a.by * a.px;
            oZp[m] = (f & (kResWallZhi | kResHaloZhi)) ? o + 2 * L::SS : o + a.by * a.px;
            word[m] = matWord(*reinterpret_cast<const unsigned short *>(a.mat + n0),
                              x + 1 < a.nx ? 0u : x < a.nx ? 2u : 3u);
            if (word[m] & kMatDead) f |= kResDead;
            // sources and monitors of the pair: into the block's list while it
            // has room (else looked up every step)
            int lo = 0, hi = a.nspec;
            while (lo < hi)
            {
                const int mid = (lo + hi) >> 1;
                if (a.spec[mid].node < n0) lo = mid + 1; else hi = mid;
            }
            int n = 0;
            while (lo + n < a.nspec && a.spec[lo + n].node < n0 + 2) ++n;
            if (n)
            {
                f |= kResSpec;
                const int p = atomicAdd(&entries, n);
                spec[m] = p + n <= kResidentEntries ? (unsigned)(p << 16 | n) : 0x80000000u | (unsigned)n;
                if (p + n <= kResidentEntries)
                    for (int e = 0; e < n; ++e)
                    {
                        const SpecEntry se = a.spec[lo + e];
                        ent[p + e].amp = se.amp;
                        ent[p + e].code = (unsigned)se.arg << 2 | (unsigned)se.kind << 1 | (se.node != n0 ? 1u : 0u);
                    }
            }
            info[m] = f;
            // packets that this pair receives, in direction 0 (from below) or 1
            pkY[m] = ((f & kResHaloYhi) ? (unsigned)a.gy * a.nz * hx : 0u) + ((unsigned)bj * a.nz + k) * hx + x / 2;
            pkZ[m] = ((f & kResHaloZhi) ? (unsigned)a.gz * a.ny * hx : 0u) + ((unsigned)bk * a.ny + j) * hx + x / 2;
#pragma unroll
            for (int s = 0; s < 12; ++s) *reinterpret_cast<float2 *>(sm + s * L::SS + o) = ld2(a.buf[0] + s * a.P + n0);
            if constexpr (DIEL)
                if (word[m] & kMatDiel)
                {
#pragma unroll
                    for (int t = 0; t < 3; ++t)
                        *reinterpret_cast<float2 *>(stubs + t * L::SS + o) = ld2(a.stub + t * a.P + n0);
                }
        }
    }

    const float2 z = splat2(a.neg_zero), rho = splat2(a.rho);
    // packets per parity: direction 0, then 1; a packet goes to the other
    // direction's place in the next (or previous) brick
    const unsigned cntY = (unsigned)a.gy * a.nz * hx, cntZ = (unsigned)a.gz * a.ny * hx;
    const unsigned nextY = (unsigned)a.nz * hx, nextZ = (unsigned)a.ny * hx;
    bool ok = true;
    // one pair's step: gather, sources, samples, energy, scatter, store
    auto pair = [&](auto mc, int s, const float *cur, float *nxt, bool last) __attribute__((always_inline)) {
        constexpr int m = decltype(mc)::value;
        const unsigned f = info[m];
        // what the neighbouring bricks sent: ask for it first
        ResPulses fromY, fromZ;
        const ResPacket *py = a.packY + (s & 1) * 2 * cntY + pkY[m], *pz = a.packZ + (s & 1) * 2 * cntZ + pkZ[m];
        const unsigned step = a.base + (unsigned)s;
        if (s > 0)
        {
            if (f & kResHaloY) fromY.load(py);
            if (f & kResHaloZ) fromZ.load(pz);
        }
        const float *c = cur + at[m];
        float2 inc[12];
#pragma unroll
        for (int t = 0; t < 2; ++t)
        {
            inc[t] = make_float2(c[(2 + t) * L::SS - (at[m] ? 1 : 0)], c[(2 + t) * L::SS]);
            inc[2 + t] = make_float2(c[t * L::SS + 1], c[t * L::SS + 2]);
            inc[4 + t] = ld2(cur + oYm[m] + (6 + t) * L::SS);
            inc[6 + t] = ld2(cur + oYp[m] + (4 + t) * L::SS);
            inc[8 + t] = ld2(cur + oZm[m] + (10 + t) * L::SS);
            inc[10 + t] = ld2(cur + oZp[m] + (8 + t) * L::SS);
        }
        if (f & kResHalo)
        {
            if (s > 0)
            {
                unsigned long long t0 = 0;
                for (unsigned it = 1;; ++it)
                {
                    const bool wy = (f & kResHaloY) && fromY.off(step), wz = (f & kResHaloZ) && fromZ.off(step);
                    if (!(wy || wz) || !ok) break;
                    if (wy) fromY.load(py);
                    if (wz) fromZ.load(pz);
                    if ((it & 255u) == 0)
                    {
                        const unsigned long long t = globalTimerNs();
                        if (t0 == 0) t0 = t;
                        if (t - t0 > kStageWaitNs)
                        {
                            ok = false;
                            atomicOr(a.fault, kResidentTimeout);
                        }
                    }
                }
            }
            else
            {
                // the state before this launch is whole in global memory
                const long long n0 = node[m];
                const float *in = a.buf[0];
                const int dy = (f & kResHaloYlo) ? 6 : 4, dz = (f & kResHaloZlo) ? 10 : 8;
                const long long ny0 = (f & kResHaloYlo) ? n0 - a.px : n0 + a.px, nz0 = (f & kResHaloZlo) ? n0 - sz : n0 + sz;
                auto put = [&](ResPulses &d, int slot, long long n) {
#pragma unroll
                    for (int t = 0; t < 2; ++t)
                    {
                        const float2 v = ld2(in + (slot + t) * a.P + n);
                        d.v[2 * t] = __float_as_uint(v.x);
                        d.v[2 * t + 1] = __float_as_uint(v.y);
                    }
                };
                if (f & kResHaloY) put(fromY, dy, ny0);
                if (f & kResHaloZ) put(fromZ, dz, nz0);
            }
#pragma unroll
            for (int t = 0; t < 2; ++t)
            {
                if (f & kResHaloYlo) inc[4 + t] = fromY.get(t);
                if (f & kResHaloYhi) inc[6 + t] = fromY.get(t);
                if (f & kResHaloZlo) inc[8 + t] = fromZ.get(t);
                if (f & kResHaloZhi) inc[10 + t] = fromZ.get(t);
            }
        }
        if (f & kResRare)
        {
            auto own = [&](int slot) { return ld2(c + slot * L::SS); };
            if (f & kResPec)
            {
#pragma unroll
                for (int t = 0; t < 2; ++t)
                {
                    negWhere(inc[t], f & 3u, own(t));
                    negWhere(inc[2 + t], (f >> 2) & 3u, own(2 + t));
                    negWhere(inc[4 + t], (f >> 4) & 3u, own(4 + t));
                    negWhere(inc[6 + t], (f >> 6) & 3u, own(6 + t));
                    negWhere(inc[8 + t], (f >> 8) & 3u, own(8 + t));
                    negWhere(inc[10 + t], (f >> 10) & 3u, own(10 + t));
                }
            }
#pragma unroll
            for (int t = 0; t < 2; ++t)
            {
                if (f & kResWallXlo) inc[t].x = a.rho * c[t * L::SS];
                if (f & kResWallX0) inc[2 + t].x = a.rho * c[(2 + t) * L::SS];
                if (f & kResWallX1) inc[2 + t].y = a.rho * c[(2 + t) * L::SS + 1];
                if (f & kResWallYlo) inc[4 + t] = mul2(inc[4 + t], rho, z);
                if (f & kResWallYhi) inc[6 + t] = mul2(inc[6 + t], rho, z);
                if (f & kResWallZlo) inc[8 + t] = mul2(inc[8 + t], rho, z);
                if (f & kResWallZhi) inc[10 + t] = mul2(inc[10 + t], rho, z);
            }
            if (f & kResSpec)
            {
                const unsigned live = 3u & ~(word[m] >> 18);
                float *smp = a.samples + (long long)s * a.nsamp * 6;
                const bool listed = !(spec[m] >> 31);
                int lo = (int)((spec[m] >> 16) & 0x7fffu);
                if (!listed)
                {
                    lo = 0;
                    for (int hi = a.nspec; lo < hi;)
                    {
                        const int mid = (lo + hi) >> 1;
                        if (a.spec[mid].node < (long long)node[m]) lo = mid + 1; else hi = mid;
                    }
                }
                const int n = (int)(spec[m] & (listed ? 0xffffu : 0x7fffffffu));
                for (int e = 0; e < n; ++e)
                {
                    SpecEntry se;
                    bool sec;
                    if (listed)
                    {
                        const ResEntry r = ent[lo + e];
                        se.amp = r.amp;
                        se.kind = (int)((r.code >> 1) & 1u);
                        se.arg = (int)(r.code >> 2);
                        sec = r.code & 1u;
                    }
                    else
                    {
                        se = a.spec[lo + e];
                        sec = se.node != (long long)node[m];
                    }
                    pairSpecEntry(se, sec, a.sv[s], smp + (long long)se.arg * 6, live, inc);
                }
            }
        }
        if (((a.first + s) & 15) == 0)
            a.epair[(long long)((a.first + s + 15) / 16 - (a.first + 15) / 16) * (a.P / 2) + node[m] / 2] =
                pairEnergy(inc, 3u & ~(word[m] >> 18));
        float2 o[12];
        if (DIEL && (word[m] & kMatDiel))
        {
            float2 vs[3];
#pragma unroll
            for (int t = 0; t < 3; ++t) vs[t] = ld2(stubs + t * L::SS + at[m]);
            pairScatterStub(tab, inc, vs, word[m], a.divLimit, z, o);
#pragma unroll
            for (int t = 0; t < 3; ++t) *reinterpret_cast<float2 *>(stubs + t * L::SS + at[m]) = vs[t];
        }
        else
            scatterAir2(inc, o, z);
        if (f & kResDead)
        {
#pragma unroll
            for (int q = 0; q < 12; ++q)
            {
                if (word[m] & (1u << 18)) o[q].x = 0.0f;
                if (word[m] & (2u << 18)) o[q].y = 0.0f;
            }
        }
        // what the neighbouring bricks wait for
        if ((f & kResHalo) && !last)
        {
            ResPacket *qy = a.packY + ((s & 1) ^ 1) * 2 * cntY + pkY[m], *qz = a.packZ + ((s & 1) ^ 1) * 2 * cntZ + pkZ[m];
            if (f & kResHaloYlo) sendPackets(qy + cntY - nextY, o[4], o[5], step + 1u);
            if (f & kResHaloYhi) sendPackets(qy - cntY + nextY, o[6], o[7], step + 1u);
            if (f & kResHaloZlo) sendPackets(qz + cntZ - nextZ, o[8], o[9], step + 1u);
            if (f & kResHaloZhi) sendPackets(qz - cntZ + nextZ, o[10], o[11], step + 1u);
        }
        float *w = nxt + at[m];
#pragma unroll
        for (int q = 0; q < 12; ++q) *reinterpret_cast<float2 *>(w + q * L::SS) = o[q];
    };

    for (int s = 0; s < a.steps; ++s)
    {
        const float *cur = sm + (s & 1) * L::buf;
        float *nxt = sm + ((s & 1) ^ 1) * L::buf;
        const bool last = s + 1 == a.steps;
        __syncthreads();
        if (info[0] & kResUsed) pair(std::integral_constant<int, 0>{}, s, cur, nxt, last);
        if constexpr (M > 1)
            if (info[M - 1] & kResUsed) pair(std::integral_constant<int, M - 1>{}, s, cur, nxt, last);
    }
    // the state back to global memory, every thread its own pairs
    const float *end = sm + (a.steps & 1) * L::buf;
    float *out = a.buf[a.steps & 1];
#pragma unroll
    for (int m = 0; m < M; ++m)
        if (info[m] & kResUsed)
        {
#pragma unroll
            for (int q = 0; q < 12; ++q)
                *reinterpret_cast<float2 *>(out + q * a.P + node[m]) = ld2(end + at[m] + q * L::SS);
            if constexpr (DIEL)
                if (word[m] & kMatDiel)
                {
#pragma unroll
                    for (int t = 0; t < 3; ++t)
                        *reinterpret_cast<float2 *>(a.stub + t * a.P + node[m]) = ld2(stubs + t * L::SS + at[m]);
                }
        }
}

} // namespace tlmk
