// tlm_host_math.h -- host scalar math that must match the reference bit for bit.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <utility>

#include <sys/mman.h>

namespace tlmh {
float eta0_f32();
float timestep_f32(float dl);
double timestep_f64(float dl);
float waveform_f32(int type, float f0, float dt, int n);
double waveform_f64(int type, float f0, double dt, int n);
void tables_f32(const float *epsr, const float *sigma, int n, float dl, float *yhat,
                float *ghat);
void tables_f64(const float *epsr, const float *sigma, int n, float dl, double *yhat,
                double *ghat);
float probe_scale_f32(float dl);
float fdtd_dt(float dl);
float fdtd_cmur(float dt, float dl);
float fdtd_cb0(float dt, float dl);
float fdtd_ch(float dt, float dl);
float fdtd_eps0();
void fdtd_edge_coef(float eAcc, float sAcc, int cnt, float dt, float dl, float *ca, float *cb);
void dft_phase_f32(float f0, float dt, int n, float *c, float *s);
void dft_phase_f64(float f0, double dt, int n, double *c, double *s);
double probe_scale_f64(float dl);
void cell_of(const float origin[3], float dl, float x, float y, float z, int *i, int *j, int *k);
// copy n bytes and return the largest
uint8_t copy_max_u8(const uint8_t *src, uint8_t *dst, size_t n);

// A solver's host copy of its material map. Unlike a vector's, its bytes are not
// cleared before they are copied over, and a large one asks for huge pages: on
// 37.7 M cells the clearing and 9,216 page faults cost three times as much as
// the copy (set-up of a 384x384x256 grid on a B200 host: 22.4 -> 10.0 ms, of a
// 192^3 one 2.3 -> 1.4).
class HostMap
{
  public:
    HostMap() = default;
    HostMap(const HostMap &) = delete;
    HostMap &operator=(const HostMap &) = delete;
    ~HostMap() { std::free(p_); }
    // Uninitialised room for n bytes; false without memory.
    bool allocate(size_t n)
    {
        constexpr size_t kHuge = size_t(2) << 20;
        std::free(p_);
        const bool large = n >= 2 * kHuge;
        const size_t bytes = large ? (n + kHuge - 1) / kHuge * kHuge : n ? n : 1;
        p_ = static_cast<uint8_t *>(large ? std::aligned_alloc(kHuge, bytes) : std::malloc(bytes));
        n_ = p_ ? n : 0;
        if (p_ && large) madvise(p_, bytes, MADV_HUGEPAGE);
        return p_ != nullptr;
    }
    void swap(HostMap &o)
    {
        std::swap(p_, o.p_);
        std::swap(n_, o.n_);
    }
    uint8_t *data() { return p_; }
    const uint8_t *data() const { return p_; }
    size_t size() const { return n_; }
    uint8_t operator[](size_t i) const { return p_[i]; }

  private:
    uint8_t *p_ = nullptr;
    size_t n_ = 0;
};
} // namespace tlmh
