// tlm_noalloc.cu -- one TLM step over caller-owned device memory that
// performs no device allocation of its own.
//
// Who needs it: callers that may not call cudaMalloc/cudaFree. Typical cases
// are a host application that reserves the GPU's memory in its own pool at
// start-up and hands plug-ins only buffers it owns, and a time-critical loop
// that must not pay the implicit device-wide synchronisation that
// cudaMalloc/cudaFree can cause. Such a caller keeps the pulse planes itself
// and asks this entry point to advance them one step.
//
// One launch does the whole step: blocks walk over tiles of node pairs, build
// the stub table of the caller's materials in shared memory (ids past the
// caller's n_diel entries read NaN there instead of reading past the caller's
// buffers), and the last block to finish adds up the blocks' energies in a
// fixed order. The only scratch, an FP64 partial per block and the count of
// finished blocks, 16 slots of them, lives in the file-scope arrays below, a fixed
// 296 KiB of device memory that every GPU which loads this library holds until the
// process exits. Host code must not pass an array's name to a kernel (on the
// host that name is a stand-in, not a device address); the device addresses
// are looked up once per device with cudaGetSymbolAddress.
#include "tlm_b200.h"

#include "tlm_pair_kernel.cuh"

#include <algorithm>
#include <atomic>
#include <mutex>
#include <string>

// Defined in tlm_solver.cu: the calling thread's message, read back by
// tlm_last_error(NULL).
void tlmSetThreadError(const std::string &m);

// The grid is limited to 67,108,864 padded nodes (2^25 pairs).
constexpr long long kNoAllocMaxNodes = 67108864;
constexpr unsigned kNoAllocWave = 148 * 4;  // resident blocks
constexpr int kNoAllocMaxBlocks = 4 * kNoAllocWave, kNoAllocSlots = 16;
static __device__ __align__(256) double g_noallocPartials[kNoAllocSlots * kNoAllocMaxBlocks];
static __device__ __align__(256) unsigned long long g_noallocDone[kNoAllocSlots];
constexpr int kNoAllocTable = 256 - tlmk::kDiel0;  // dielectric ids
// Bounds-check record of the checked library build (cleared before every
// step, read back after it there); the regular build never writes it.
static __device__ __align__(256) unsigned g_noallocFault;

namespace {

constexpr int kMaxDevices = 64;
std::mutex g_noallocMutex;
std::atomic<unsigned long long> g_noallocCalls{ 0 };

struct NoAllocScratch
{
    double *partials = nullptr;
    unsigned long long *done = nullptr;
    unsigned *fault = nullptr;
};
NoAllocScratch g_noallocAddr[kMaxDevices];

tlm_status noallocFail(tlm_status s, const std::string &m)
{
    tlmSetThreadError(m);
    return s;
}

struct PlanesArgs
{
    const float *in;
    float *out, *stub;
    const uint8_t *mat;
    const float *yhat, *ghat;
    int ntable;
    int nx, ny, nz, px, hx;  // hx: pairs per row
    long long P;
    unsigned npairs;
    tlmk::FastDiv divH, divY;  // by hx and by ny
    float rho, neg_zero;
    double *partials, *energy;
    unsigned long long *done, call;  // finished blocks of this call: call + their number
    unsigned *fault;
};

// One step, a pair of nodes per thread at a time, the arithmetic of the general
// tile body (DIEL: with the caller's stubs). Every load of a pair that does not depend on its material
// is issued before the first use; a pair next to PEC (rare) then loads the own
// pulses it reflects. What bounds it at a few hundred thousand nodes is that
// latency: 93x80x71 nodes with dielectrics and the caller's energy took three
// launches and 34.6 us with the general tile body, four nodes per thread, and
// take 20.6 with the planes in L2 (36 and 22.5 with planes that are not).
template <bool INCIDENT, bool DIEL> __global__ void __launch_bounds__(256, 4) planesStepKernel(const PlanesArgs a)
{
    using namespace tlmk;
    __shared__ float tab[768];
    __shared__ double red[8];
    __shared__ bool lastBlock;
    float divLimit = 0.0f;
    if constexpr (DIEL)
    {
        static_assert(kBlock == 256, "a thread per material id");
        const int m = threadIdx.x;
        const float nan = __int_as_float(0x7fc00000);
        const bool in = m >= kDiel0 && m - kDiel0 < a.ntable;
        const float yh = m < kDiel0 ? -0.0f : in ? a.yhat[m - kDiel0] : nan;
        const float gh = m < kDiel0 ? 0.0f : in ? a.ghat[m - kDiel0] : nan;
        const float den = (4.0f + yh) + gh;
        tab[m] = yh;
        tab[256 + m] = -den;
        tab[512 + m] = __frcp_rn(den);
        // the limit of the caller's denominators, which may be anything, in
        // steps: at most 2^25, at most 2^40, or out of range (also below 4)
        const bool low = den >= 4.0f;
        divLimit = stubDivLimit(4.0f);
        if (__syncthreads_or(in && !(low && den <= 0x1p25f)))
            divLimit = stubDivLimit(__syncthreads_or(in && !(low && den <= 0x1p40f)) ? nan : 0x1p40f);
    }
    const long long P = a.P, sz = (long long)a.px * a.ny;
    const float2 z = splat2(a.neg_zero), rho = splat2(a.rho);
    double en = 0.0;
    for (unsigned q = blockIdx.x * 256u + threadIdx.x; q < a.npairs; q += gridDim.x * 256u)
    {
        const unsigned row = fastDiv(q, a.divH);
        const int x = 2 * (int)(q - row * (unsigned)a.hx);
        const unsigned k = fastDiv(row, a.divY);
        const int j = (int)(row - k * (unsigned)a.ny);
        const long long n0 = 2LL * q;
        if (!TLM_GUARD(n0, P - 1, 1)) continue;
        const bool ylo = j == 0, yhi = j == a.ny - 1, zlo = k == 0, zhi = (int)k == a.nz - 1;
        float2 inc[12];
        unsigned pec = 0;  // two bits per face: -x +x -y +y -z +z
        unsigned ids = *reinterpret_cast<const unsigned short *>(a.mat + n0);
        if constexpr (INCIDENT)
        {
#pragma unroll
            for (int s = 0; s < 12; ++s) inc[s] = ld2(a.in + s * P + n0);
        }
        else
        {
            const unsigned own = ((ids & 255u) == kPec ? 1u : 0u) | ((ids >> 8) == kPec ? 2u : 0u);
            const bool prev = x > 0, next = x + 2 < a.nx;
            const unsigned mp = prev ? a.mat[n0 - 1] : 0u, mn = next ? a.mat[n0 + 2] : 0u;
            const unsigned mym = ylo ? 0u : pecPair(a.mat + n0 - a.px), myp = yhi ? 0u : pecPair(a.mat + n0 + a.px);
            const unsigned mzm = zlo ? 0u : pecPair(a.mat + n0 - sz), mzp = zhi ? 0u : pecPair(a.mat + n0 + sz);
            float2 ox[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) ox[s] = ld2(a.in + s * P + n0);
#pragma unroll
            for (int t = 0; t < 2; ++t)
            {
                const float p = prev ? a.in[(2 + t) * P + n0 - 1] : 0.0f, n = next ? a.in[t * P + n0 + 2] : 0.0f;
                inc[t] = make_float2(p, ox[2 + t].x);
                inc[2 + t] = make_float2(ox[t].y, n);
                inc[4 + t] = ld2(a.in + (ylo ? (4 + t) * P + n0 : (6 + t) * P + n0 - a.px));
                inc[6 + t] = ld2(a.in + (yhi ? (6 + t) * P + n0 : (4 + t) * P + n0 + a.px));
                inc[8 + t] = ld2(a.in + (zlo ? (8 + t) * P + n0 : (10 + t) * P + n0 - sz));
                inc[10 + t] = ld2(a.in + (zhi ? (10 + t) * P + n0 : (8 + t) * P + n0 + sz));
            }
            pec = ((own << 1) & 2u) | (mp == kPec ? 1u : 0u);
            pec |= ((x + 1 < a.nx ? own >> 1 : 0u) | (mn == kPec ? 2u : 0u)) << 2;
            pec |= mym << 4 | myp << 6 | mzm << 8 | mzp << 10;
            if (pec)
            {
#pragma unroll
                for (int t = 0; t < 2; ++t)
                {
                    negWhere(inc[t], pec & 3u, ox[t]);
                    negWhere(inc[2 + t], (pec >> 2) & 3u, ox[2 + t]);
                    if ((pec >> 4) & 3u) negWhere(inc[4 + t], (pec >> 4) & 3u, ld2(a.in + (4 + t) * P + n0));
                    if ((pec >> 6) & 3u) negWhere(inc[6 + t], (pec >> 6) & 3u, ld2(a.in + (6 + t) * P + n0));
                    if ((pec >> 8) & 3u) negWhere(inc[8 + t], (pec >> 8) & 3u, ld2(a.in + (8 + t) * P + n0));
                    if ((pec >> 10) & 3u) negWhere(inc[10 + t], (pec >> 10) & 3u, ld2(a.in + (10 + t) * P + n0));
                }
            }
#pragma unroll
            for (int t = 0; t < 2; ++t)
            {
                if (x == 0) inc[t].x = a.rho * ox[t].x;
                if (x == a.nx - 1) inc[2 + t].x = a.rho * ox[2 + t].x;
                if (x + 1 == a.nx - 1) inc[2 + t].y = a.rho * ox[2 + t].y;
                if (ylo) inc[4 + t] = mul2(inc[4 + t], rho, z);
                if (yhi) inc[6 + t] = mul2(inc[6 + t], rho, z);
                if (zlo) inc[8 + t] = mul2(inc[8 + t], rho, z);
                if (zhi) inc[10 + t] = mul2(inc[10 + t], rho, z);
            }
        }
        unsigned word = matWord(ids, x + 1 < a.nx ? 0u : x < a.nx ? 2u : 3u);
        if (a.energy != nullptr) en += pairEnergy(inc, 3u & ~(word >> 18));
        float2 o[12];
        if (DIEL && (word & kMatDiel))
        {
            // the caller's stubs count on dielectric nodes only: the other node
            // of a pair may hold anything there, and keeps it
            const bool d0 = word & (1u << 16), d1 = word & (2u << 16);
            float2 vs[3];
#pragma unroll
            for (int t = 0; t < 3; ++t)
            {
                vs[t] = ld2(a.stub + t * P + n0);
                if (!d0) vs[t].x = 0.0f;
                if (!d1) vs[t].y = 0.0f;
            }
            pairScatterStub(tab, inc, vs, word, divLimit, z, o);
#pragma unroll
            for (int t = 0; t < 3; ++t)
            {
                float *w = a.stub + t * P + n0;
                if (d0 && d1)
                    *reinterpret_cast<float2 *>(w) = vs[t];
                else
                    w[d1 ? 1 : 0] = d1 ? vs[t].y : vs[t].x;
            }
        }
        else
        {
            // (without any table an id of a dielectric steps to NaN)
            scatterAir2(inc, o, z);
            if (!DIEL && (word & kMatDiel))
            {
#pragma unroll
                for (int s = 0; s < 12; ++s)
                {
                    if (word & (1u << 16)) o[s].x = __int_as_float(0x7fc00000);
                    if (word & (2u << 16)) o[s].y = __int_as_float(0x7fc00000);
                }
            }
        }
        if (word & kMatDead)
        {
#pragma unroll
            for (int s = 0; s < 12; ++s)
            {
                if (word & (1u << 18)) o[s].x = 0.0f;
                if (word & (2u << 18)) o[s].y = 0.0f;
            }
        }
#pragma unroll
        for (int s = 0; s < 12; ++s) *reinterpret_cast<float2 *>(a.out + s * P + n0) = o[s];
    }
    if (a.energy == nullptr) return;
    const double tot = blockSumDouble(en, red);
    if (threadIdx.x == 0)
    {
        a.partials[blockIdx.x] = tot;
        __threadfence();
        // whatever an earlier call left in the count, this call's begins at
        // its own number, which is larger
        atomicMax(a.done, a.call);
        lastBlock = atomicAdd(a.done, 1ull) == a.call + gridDim.x - 1;
    }
    __syncthreads();
    if (!lastBlock) return;
    __threadfence();
    double s = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += 256) s += __ldcg(a.partials + b);
    __syncthreads();
    const double all = blockSumDouble(s, red);
    if (threadIdx.x == 0) *a.energy = all;
}

// Device addresses of the scratch arrays for the current device, looked up
// on the first call on that device (with that device current).
tlm_status scratchForCurrentDevice(NoAllocScratch *out)
{
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices)
    {
        cudaGetLastError();
        return noallocFail(TLM_ENODEV, std::string("no current CUDA device: ") +
                                           (e != cudaSuccess ? cudaGetErrorString(e) : "bad index"));
    }
    std::lock_guard<std::mutex> lk(g_noallocMutex);
    NoAllocScratch &sc = g_noallocAddr[dev];
    if (!sc.partials)
    {
        void *p = nullptr, *t = nullptr, *f = nullptr;
        e = cudaGetSymbolAddress(&p, g_noallocPartials);
        if (e == cudaSuccess) e = cudaGetSymbolAddress(&t, g_noallocDone);
        if (e == cudaSuccess) e = cudaGetSymbolAddress(&f, g_noallocFault);
        if (e != cudaSuccess || !p || !t || !f)
        {
            cudaGetLastError();
            return noallocFail(TLM_ECUDA, std::string("cudaGetSymbolAddress of the scratch arrays: ") +
                                              cudaGetErrorString(e));
        }
        sc.done = static_cast<unsigned long long *>(t);
        sc.fault = static_cast<unsigned *>(f);
        sc.partials = static_cast<double *>(p);
    }
    *out = sc;
    return TLM_OK;
}

bool aligned16(const void *p) { return ((uintptr_t)p & 15u) == 0; }

} // namespace

extern "C" {

tlm_status tlm_step_planes_noalloc(const float *in_planes, float *out_planes, float *stubs,
                                   const uint8_t *mat, const float *yhat, const float *ghat, int n_diel,
                                   int nx, int ny, int nz, float rho, int input_is_incident,
                                   double *energy_out, void *stream)
{
    if (!in_planes || !out_planes || !mat)
        return noallocFail(TLM_EINVAL, "null pulse planes or material map");
    if (in_planes == out_planes)
        return noallocFail(TLM_EINVAL, "input and output planes must be different buffers");
    if (nx <= 0 || ny <= 0 || nz <= 0)
        return noallocFail(TLM_EINVAL, "grid dimensions must be positive");
    if (n_diel < 0 || n_diel > kNoAllocTable)
        return noallocFail(TLM_EINVAL, "n_diel must be in 0.." + std::to_string(kNoAllocTable));
    if (n_diel > 0 && (!stubs || !yhat || !ghat))
        return noallocFail(TLM_EINVAL, "a dielectric table (n_diel > 0) needs stubs, yhat and ghat");
    if (!aligned16(in_planes) || !aligned16(out_planes) || (stubs && !aligned16(stubs)) ||
        ((uintptr_t)mat & 3u))
        return noallocFail(TLM_EINVAL, "planes must be 16-byte aligned, the material map 4-byte aligned");
    constexpr long long kMaxNodes = kNoAllocMaxNodes;
    // the plane size grows one factor at a time, each partial product
    // checked against the limit, so nothing overflows
    const long long px = ((long long)nx + tlmk::kPadX - 1) / tlmk::kPadX * tlmk::kPadX;
    const long long row = px <= kMaxNodes ? px * ny : kMaxNodes + 1;
    const long long P = row <= kMaxNodes ? row * nz : kMaxNodes + 1;
    if (P <= 0 || P > kMaxNodes)
        return noallocFail(TLM_EINVAL,
                           "grid has more than " + std::to_string(kMaxNodes) + " padded nodes; the no-allocation "
                           "step handles at most " + std::to_string(kMaxNodes));
    NoAllocScratch sc;
    tlm_status st = scratchForCurrentDevice(&sc);
    if (st != TLM_OK) return st;

    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaSuccess;
#ifdef TLM_CHECKED
    if (e == cudaSuccess) e = cudaMemsetAsync(sc.fault, 0, sizeof(unsigned), s);
#endif
    if (e != cudaSuccess)
        return noallocFail(TLM_ECUDA, std::string("no-allocation step set-up: ") + cudaGetErrorString(e));

    PlanesArgs a;
    a.in = in_planes;
    a.out = out_planes;
    a.stub = stubs;
    a.mat = mat;
    a.yhat = yhat;
    a.ghat = ghat;
    a.ntable = n_diel;
    a.nx = nx;
    a.ny = ny;
    a.nz = nz;
    a.px = (int)px;
    a.hx = (int)(px / 2);
    a.P = P;
    a.npairs = (unsigned)(P / 2);
    a.divH = tlmk::makeFastDiv((unsigned)a.hx);
    a.divY = tlmk::makeFastDiv((unsigned)ny);
    a.rho = rho;
    a.neg_zero = -0.0f;
    // calls take the slots in turn, so that a few which overlap on the GPU keep
    // apart; what a collision beyond that leaves in a count harms no later call,
    // whose number is larger (in a captured call's replays it is always the same
    // one: they clear the count first)
    const unsigned long long call = g_noallocCalls.fetch_add(1) + 1;
    const unsigned slot = (unsigned)(call % kNoAllocSlots);
    a.partials = sc.partials + slot * kNoAllocMaxBlocks;
    a.energy = energy_out;
    a.done = sc.done + slot;
    a.call = call << 16;  // room for the blocks of many overlapping calls
    if (energy_out)
    {
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s, &capture) != cudaSuccess)
            cudaGetLastError();
        else if (capture == cudaStreamCaptureStatusActive)
            e = cudaMemsetAsync(a.done, 0, sizeof(*a.done), s);
        if (e != cudaSuccess)
            return noallocFail(TLM_ECUDA, std::string("no-allocation step set-up: ") + cudaGetErrorString(e));
    }
    a.fault = sc.fault;
    // Blocks that walk over several tiles of 256 pairs leave fewer partials to
    // add up, but nothing of their next tile is in flight while they finish one:
    // with an energy the grid is a wave of blocks per 4096 tiles, at most four,
    // without one a block per tile beyond two waves. One wave for all sizes took
    // 576 us for incident planes of 320^3 nodes without an energy, 574 with one;
    // now 469 and 508 (128^3: 38 and 41, now 36 and 41).
    const unsigned tiles = (a.npairs + 255u) / 256u;
    const unsigned most = energy_out ? kNoAllocWave * std::min(std::max(tiles / 4096u, 1u), 4u)
                          : tiles <= 2 * kNoAllocWave ? kNoAllocWave : tiles;
    const unsigned blocks = std::min(tiles, most);
    if (input_is_incident)
    {
        if (stubs) planesStepKernel<true, true><<<blocks, 256, 0, s>>>(a);
        else planesStepKernel<true, false><<<blocks, 256, 0, s>>>(a);
    }
    else
    {
        if (stubs) planesStepKernel<false, true><<<blocks, 256, 0, s>>>(a);
        else planesStepKernel<false, false><<<blocks, 256, 0, s>>>(a);
    }
    e = cudaGetLastError();
    if (e != cudaSuccess)
        return noallocFail(TLM_ECUDA, std::string("no-allocation step launch: ") + cudaGetErrorString(e));
#ifdef TLM_CHECKED
    // the checked build reports an index outside a buffer (and skips that
    // access): wait for the step and read the record back
    unsigned f = 0;
    e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = cudaMemcpy(&f, sc.fault, sizeof(unsigned), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess)
        return noallocFail(TLM_ECUDA, std::string("no-allocation step: ") + cudaGetErrorString(e));
    if (f) return noallocFail(TLM_ECUDA, "bounds check tripped in the no-allocation step, code mask " + std::to_string(f));
#endif
    return TLM_OK;
}

} // extern "C"
