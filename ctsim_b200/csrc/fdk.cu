// FDK reconstruction (fbp/reconFDK.m) on the device:
//   1. cosine weight per detector pixel and, for short scans, Parker weight per
//      (view, detector column)                                   reconFDK.m:38-60
//   2. ramp x window filter along every detector row, by FFT with the zero padding
//      of filterFreq.m (length max(64, 2^nextpow2(2 nu - 1)))     reconFDK.m:62-71
//   3. back,hpd backprojection, times dbeta, times 10             reconFDK.m:78-84
// The filter itself is built on the host by the reference's design
// (fbp/filter/designFilter2.m flat, designEquiangularFilter2.m curved).
#include <cmath>
#include <complex>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/ctsim_b200.h"
#include "kernels.cuh"

using namespace ctsim;

extern ctsim_status ctsim_set_last_error(ctsim_status s, const char *msg);
// plan internals shared with capi.cu
extern const double *ctsim_plan_betas(const ctsim_plan *p);
extern const ctsim_geom *ctsim_plan_geom(const ctsim_plan *p);
extern ctsim_status ctsim_plan_back_hpd(ctsim_plan *p, const void *d_proj, int proj_dtype, float *d_image, float scale,
                                        float scale2, cudaStream_t st);
extern cudaError_t ctsim_plan_alloc(const ctsim_plan *p, void **ptr, size_t n);
extern void ctsim_plan_release(const ctsim_plan *p, void *ptr);
extern cudaError_t ctsim_plan_upload(const ctsim_plan *p, void *dst, const void *src, size_t n);

namespace {

constexpr int kFiltRows = 8;  // detector rows per block (4 complex FFTs)

int fft_order(int nu) {
    // order = max(64, 2^nextpow2(2*len-1)), designFilter2.m:18
    int L = 1;
    while (L < 2 * nu - 1) L <<= 1;
    return L < 64 ? 64 : L;
}

bool window_known(const std::string &w) {
    static const char *names[] = {"ram-lak", "shepp-logan", "cosine", "hamming", "hann", "hann50", "hann75",
                                  "hann80", "B50", "B75", "B80", "C50", "C75", "C80"};
    for (auto n : names)
        if (w == n) return true;
    return false;
}

// |DFT(h)|[0..count) by an iterative radix-2 FFT in double (size a power of two);
// every twiddle is evaluated directly (no recurrence).
std::vector<double> dft_magnitude(const std::vector<double> &h, int count) {
    const int n = (int)h.size();
    int lg = 0;
    while ((1 << lg) < n) lg++;
    std::vector<std::complex<double>> a(n);
    for (int i = 0; i < n; i++) {
        int r = 0;
        for (int b = 0; b < lg; b++) r |= ((i >> b) & 1) << (lg - 1 - b);
        a[r] = h[i];
    }
    for (int len = 2; len <= n; len <<= 1) {
        const int hl = len / 2;
        for (int j = 0; j < hl; j++) {
            const double ang = -2.0 * M_PI * j / len;
            const std::complex<double> w(std::cos(ang), std::sin(ang));
            for (int i = 0; i < n; i += len) {
                const std::complex<double> u = a[i + j], v = a[i + j + hl] * w;
                a[i + j] = u + v;
                a[i + j + hl] = u - v;
            }
        }
    }
    std::vector<double> m(count);
    for (int k = 0; k < count; k++) m[k] = std::sqrt(a[k].real() * a[k].real() + a[k].imag() * a[k].imag());
    return m;
}

// designFilter2.m:18-78 (flat) / designEquiangularFilter2.m:19-78 (curved), in double.
// gamma = du; SDD used by the equiangular kernel.  Returns H[order].
std::vector<double> design_filter(int nu, double du, double sdd, bool flat, const std::string &window, double crop) {
    const int order = fft_order(nu);
    // h over index = -order/2+1 .. order/2-1, then h(order) = 0 (zero padding)
    std::vector<double> h(order, 0.0);
    for (int n = 0; n < order - 1; n++) {
        const int index = -order / 2 + 1 + n;
        if (index == 0) {
            h[n] = 1.0 / (4.0 * du * du);
        } else if (((index % 2) + 2) % 2 == 1) {  // MATLAB mod(index,2)==1 (odd, either sign)
            const double d = flat ? (index * M_PI * du) : (sdd * M_PI * std::sin(index * du / sdd));
            h[n] = -1.0 / (d * d);
        }
    }
    // filt = abs(fft(h)), first order/2+1 bins
    const int half = order / 2 + 1;
    std::vector<double> filt = dft_magnitude(h, half);
    std::string win = window;
    if (win == "hann50" || win == "B50" || win == "C50") crop = 0.5;
    if (win == "hann75" || win == "B75" || win == "C75") crop = 0.75;
    if (win == "hann80" || win == "B80" || win == "C80") crop = 0.80;
    for (int k = 1; k < half; k++) {
        const double w = 2.0 * M_PI * k / order;
        if (win == "shepp-logan") filt[k] *= std::sin(w / (2 * crop)) / (w / (2 * crop));
        else if (win == "cosine" || win == "C50" || win == "C75" || win == "C80") filt[k] *= std::cos(w / (2 * crop));
        else if (win == "hamming") filt[k] *= 0.54 + 0.46 * std::cos(w / crop);
        else if (win == "hann" || win == "hann50" || win == "hann75" || win == "hann80")
            filt[k] *= (1.0 + std::cos(w / crop)) / 2.0;
    }
    for (int k = 0; k < half; k++)
        if (2.0 * M_PI * k / order > M_PI * crop) filt[k] = 0.0;  // crop, designFilter2.m:77
    // symmetric extension [filt ; filt(end-1:-1:2)]
    std::vector<double> H(order);
    for (int k = 0; k < half; k++) H[k] = filt[k];
    for (int k = half; k < order; k++) H[k] = filt[order - k];
    return H;
}

// MATLAB S-function of fbp/weights/shortScanParkerWeight.m:243-252
double parker_s(double b) {
    if (b <= -0.5) return 0.0;
    if (std::fabs(b) < 0.5) return 0.5 * (1.0 + std::sin(M_PI * b));
    return 1.0;
}

// ---------------------------------------------------------------------------
// Row filter: block = (group of 8 detector rows, view).  Rows 2p and 2p+1 are the
// real and imaginary parts of complex signal p (the filter is real and even, so the
// two filtered rows come back as the real and imaginary parts).
//
// In-place mixed-radix FFT of length L = 8^a 4^b (L a power of two, 64 at least): forward by
// decimation in frequency (natural order in, digit-reversed out), the filter applied in that
// order, inverse by decimation in time (natural order out).  The first forward pass reads the
// sinogram, the last inverse one writes it, and the passes around the filter stay in
// registers, so a signal crosses shared memory 2 (passes - 1) times.  Bound by instruction
// issue and those crossings: 1024 columns x 384 rows x 720 views take 3.6 ms (625 GB/s of
// sinogram), 10.8 ms in the 22 radix-2 passes of before; 256 x 96 x 360 0.10 ms, before 0.28.
// ---------------------------------------------------------------------------
constexpr int kFiltThreads = 256;
constexpr int kFiltSignals = kFiltRows / 2;

// Shared-memory position of element i of a signal (one float2 of padding per 32, so that
// strided passes spread over the banks), and a signal's length there.
__host__ __device__ __forceinline__ int filt_pos(int i) { return i + (i >> 5); }

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 w) {
    return make_float2(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
}
__device__ __forceinline__ float2 cmul_conj(float2 a, float2 w) {
    return make_float2(a.x * w.x + a.y * w.y, a.y * w.x - a.x * w.y);
}
// a * -i (forward) or a * i (inverse)
template <bool INV>
__device__ __forceinline__ float2 crot(float2 a) {
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

template <bool INV>
__device__ __forceinline__ void dft(float2 (&x)[4]) {
    const float2 s = cadd(x[0], x[2]), d = csub(x[0], x[2]), t = cadd(x[1], x[3]), r = crot<INV>(csub(x[1], x[3]));
    x[0] = cadd(s, t);
    x[1] = cadd(d, r);
    x[2] = csub(s, t);
    x[3] = csub(d, r);
}
template <bool INV>
__device__ __forceinline__ void dft(float2 (&x)[8]) {
    float2 e[4] = {x[0], x[2], x[4], x[6]}, o[4] = {x[1], x[3], x[5], x[7]};
    dft<INV>(e);
    dft<INV>(o);
    constexpr float h = 0.70710678118654752440f;  // sqrt(1/2): e^(-i pi/4) = h (1 - i)
    const float2 r1 = crot<INV>(o[1]), r3 = crot<INV>(o[3]);
    o[1] = make_float2(h * (o[1].x + r1.x), h * (o[1].y + r1.y));
    o[2] = crot<INV>(o[2]);
    o[3] = make_float2(h * (r3.x - o[3].x), h * (r3.y - o[3].y));
#pragma unroll
    for (int k = 0; k < 4; k++) {
        x[k] = cadd(e[k], o[k]);
        x[k + 4] = csub(e[k], o[k]);
    }
}

// One pass of radix R over sub-transforms of N = R << lm elements (lm: log2 N / R) in shared
// memory; tw its twiddles, e^(-2 pi i j k / N) at [(k - 1) N/R + j].  MID: the last forward pass (N = R), the
// filter and the first inverse pass.
template <int R, bool INV, bool MID>
__device__ __forceinline__ void filt_pass(float2 *buf, int L, int ls, int lm, const float2 *__restrict__ tw,
                                          const float *__restrict__ H) {
    const int per = L / R, m = 1 << lm;
    for (int b = threadIdx.x; b < kFiltSignals * per; b += kFiltThreads) {
        const int u = b & (per - 1);
        float2 *a = buf + (size_t)(b / per) * ls;
        const int j = u & (m - 1), base = ((u >> lm) * R << lm) + j;
        float2 x[R];
#pragma unroll
        for (int k = 0; k < R; k++) x[k] = a[filt_pos(base + (k << lm))];
        if (MID) {
            dft<false>(x);
#pragma unroll
            for (int k = 0; k < R; k++) {
                const float h = __ldg(H + base + k);
                x[k] = make_float2(x[k].x * h, x[k].y * h);
            }
            dft<true>(x);
        } else if (INV) {
#pragma unroll
            for (int k = 1; k < R; k++) x[k] = cmul_conj(x[k], __ldg(tw + ((k - 1) << lm) + j));
            dft<true>(x);
        } else {
            dft<false>(x);
#pragma unroll
            for (int k = 1; k < R; k++) x[k] = cmul(x[k], __ldg(tw + ((k - 1) << lm) + j));
        }
#pragma unroll
        for (int k = 0; k < R; k++) a[filt_pos(base + (k << lm))] = x[k];
    }
    __syncthreads();
}

// H: the filter over L, in the order of the forward transform's output.  tw: the passes' twiddles
// (filt_pass), those of the pass over sub-transforms of N elements from L - N on, so that a warp's
// loads are consecutive (strided out of one table of L they made the filter 1.4x slower).
__global__ void __launch_bounds__(kFiltThreads) fdk_filter_kernel(const void *__restrict__ sino, int in_dtype,
                                                                  void *__restrict__ out, int out_dtype,
                                                                  const float *__restrict__ wcos,
                                                                  const float *__restrict__ parker,
                                                                  const float *__restrict__ H,
                                                                  const float2 *__restrict__ tw, int nu, int nv, int L,
                                                                  int n8, int n4) {
    extern __shared__ float2 buf[];  // [kFiltSignals][filt_pos(L)]
    const int k = blockIdx.y;
    const int iv0 = blockIdx.x * kFiltRows;
    const size_t vbase = (size_t)k * nu * nv;
    const int ls = filt_pos(L);
    const int m8 = L / 8;
    // first pass: element i = j + q L/8 of signal `sig` (consecutive threads: the signals of one j)
    for (int b = threadIdx.x; b < kFiltSignals * m8; b += kFiltThreads) {
        const int sig = b & (kFiltSignals - 1), j = b / kFiltSignals;
        const int iv = iv0 + 2 * sig;
        float2 x[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int iu = j + q * m8;
            x[q] = make_float2(0.f, 0.f);  // zero padding beyond nu and past the last row
            if (iu < nu && iv < nv) {
                const size_t o = (size_t)iu * nv + iv;
                x[q].x = load_as_float(sino, vbase + o, in_dtype) * __ldg(wcos + o);  // reconFDK.m:54
                if (iv + 1 < nv) x[q].y = load_as_float(sino, vbase + o + 1, in_dtype) * __ldg(wcos + o + 1);
                if (parker) {  // reconFDK.m:66-68
                    const float p = __ldg(parker + (size_t)k * nu + iu);
                    x[q].x = x[q].x * p;
                    x[q].y = x[q].y * p;
                }
            }
        }
        dft<false>(x);
        float2 *a = buf + (size_t)sig * ls;
        a[filt_pos(j)] = x[0];
#pragma unroll
        for (int q = 1; q < 8; q++) a[filt_pos(j + q * m8)] = cmul(x[q], __ldg(tw + (q - 1) * m8 + j));
    }
    __syncthreads();
    int log2n = 31 - __clz(L) - 3;  // log2 of the sub-transforms left
    const int passes = n8 + n4;
    auto twiddles = [&](int lg) { return tw + (L - (1 << lg)); };
    for (int p = 1; p < passes - 1; p++) {
        if (p < n8) {
            filt_pass<8, false, false>(buf, L, ls, log2n - 3, twiddles(log2n), H);
            log2n -= 3;
        } else {
            filt_pass<4, false, false>(buf, L, ls, log2n - 2, twiddles(log2n), H);
            log2n -= 2;
        }
    }
    if (n4) filt_pass<4, false, true>(buf, L, ls, 0, nullptr, H);
    else filt_pass<8, false, true>(buf, L, ls, 0, nullptr, H);
    for (int p = passes - 2; p >= 1; p--) {
        if (p < n8) {
            log2n += 3;
            filt_pass<8, true, false>(buf, L, ls, log2n - 3, twiddles(log2n), H);
        } else {
            log2n += 2;
            filt_pass<4, true, false>(buf, L, ls, log2n - 2, twiddles(log2n), H);
        }
    }
    // last pass: the filtered rows, the first nu columns
    for (int b = threadIdx.x; b < kFiltSignals * m8; b += kFiltThreads) {
        const int sig = b & (kFiltSignals - 1), j = b / kFiltSignals;
        const int iv = iv0 + 2 * sig;
        const float2 *a = buf + (size_t)sig * ls;
        float2 x[8];
        x[0] = a[filt_pos(j)];
#pragma unroll
        for (int q = 1; q < 8; q++) x[q] = cmul_conj(a[filt_pos(j + q * m8)], __ldg(tw + (q - 1) * m8 + j));
        dft<true>(x);
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int iu = j + q * m8;
            if (iu < nu && iv < nv) {
                const size_t o = vbase + (size_t)iu * nv + iv;
                store_from_float(out, o, x[q].x, out_dtype);
                if (iv + 1 < nv) store_from_float(out, o + 1, x[q].y, out_dtype);
            }
        }
    }
}

}  // namespace

struct ctsim_fdk {
    ctsim_plan *plan = nullptr;
    int nu = 0, nv = 0, nviews = 0, L = 0, n8 = 0, n4 = 0;  // L = 8^n8 4^n4
    float dbeta = 0.f;
    float *d_H = nullptr, *d_wcos = nullptr, *d_parker = nullptr;
    void *d_filtered = nullptr;  // the filtered sinogram of ctsim_fdk_run_ex, in the input's storage type
    size_t filtered_bytes = 0;
    float2 *d_tw = nullptr;
};

extern "C" ctsim_status ctsim_fdk_design_filter(int nu, float du, float sdd, int detector_type, const char *window,
                                                float crop, double *H, int *order) {
    if (!window || !window_known(window)) return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "Invalid window selected.");
    if (nu < 1 || !(du > 0) || !(sdd > 0)) return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "invalid detector");
    const int L = fft_order(nu);
    if (order) *order = L;
    if (H) {
        std::vector<double> h = design_filter(nu, du, sdd, detector_type == 1, window, crop);
        std::memcpy(H, h.data(), sizeof(double) * L);
    }
    return CTSIM_OK;
}

// Device memory follows the plan's allocation mode (stream-ordered plans: on the
// plan's stream), so an FDK object is destroyed before its plan.
static void free_fdk(ctsim_fdk *f) {
    if (!f) return;
    ctsim_plan_release(f->plan, f->d_H);
    ctsim_plan_release(f->plan, f->d_wcos);
    ctsim_plan_release(f->plan, f->d_parker);
    ctsim_plan_release(f->plan, f->d_filtered);
    ctsim_plan_release(f->plan, f->d_tw);
    delete f;
}

extern "C" ctsim_status ctsim_fdk_create(ctsim_plan *plan, const char *window, float crop, int short_scan,
                                         ctsim_fdk **out) {
    if (!plan || !out) return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "null argument");
    if (!window || !window_known(window)) return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "Invalid window selected.");
    const ctsim_geom &G = *ctsim_plan_geom(plan);
    if (G.detector_type != 0 && G.detector_type != 1)
        return ctsim_set_last_error(CTSIM_ERR_UNSUPPORTED, "FDK needs a flat (1) or curved (0) detector");
    const double *betas = ctsim_plan_betas(plan);
    const bool flat = G.detector_type == 1;
    ctsim_fdk *f = new ctsim_fdk();
    f->plan = plan;
    f->nu = G.nu;
    f->nv = G.nv;
    f->nviews = G.noviews;
    f->L = fft_order(G.nu);
    int log2L = 0;
    while ((1 << log2L) < f->L) log2L++;
    f->n4 = log2L % 3 == 0 ? 0 : log2L % 3 == 2 ? 1 : 2;
    f->n8 = (log2L - 2 * f->n4) / 3;
    const double SAD = G.sad, SDD = G.sdd, du = G.du, dv = G.dv;
    // detector coordinates u, v in mm (reconFDK.m:33-34)
    std::vector<double> u(G.nu), v(G.nv);
    for (int i = 0; i < G.nu; i++) u[i] = ((-(G.nu - 1) / 2.0 + i) + G.offset_u) * du;
    for (int i = 0; i < G.nv; i++) v[i] = ((-(G.nv - 1) / 2.0 + i) + G.offset_v) * dv;
    // cosine weight (reconFDK.m:39 flat, :44 curved), stored [iu][iv] like the sinogram
    std::vector<float> wcos((size_t)G.nu * G.nv);
    for (int iu = 0; iu < G.nu; iu++)
        for (int iv = 0; iv < G.nv; iv++) {
            double w;
            if (flat) w = SAD * std::sqrt(1.0 + u[iu] * u[iu] / (SDD * SDD)) / std::sqrt(u[iu] * u[iu] + v[iv] * v[iv] + SDD * SDD);
            else w = SAD / SDD * std::cos(u[iu] / std::sqrt(SDD * SDD + v[iv] * v[iv]));
            wcos[(size_t)iu * G.nv + iv] = (float)w;
        }
    std::vector<double> Hd = design_filter(G.nu, du, SDD, flat, window, crop);
    // H = du * designFilter2(...), reconFDK.m:40, at the position that the forward transform leaves
    // the frequency (its digits, least significant first, from the slowest position down), with the
    // inverse transform's 1/L (a power of two: exact)
    std::vector<float> H(f->L);
    for (int i = 0; i < f->L; i++) {
        int rest = i, n = f->L, pos = 0;
        for (int p = 0; p < f->n8 + f->n4; p++) {
            const int r = p < f->n8 ? 8 : 4;
            n /= r;
            pos += rest % r * n;
            rest /= r;
        }
        H[pos] = (float)(du * Hd[i]) / (float)f->L;
    }
    std::vector<float2> tw(f->L);
    for (int p = 0, n = f->L; p < f->n8 + f->n4; p++) {
        const int r = p < f->n8 ? 8 : 4, m = n / r;
        for (int k = 1; k < r; k++)
            for (int j = 0; j < m; j++) {
                const double a = -2.0 * M_PI * j * k / n;
                tw[f->L - n + (k - 1) * m + j] = make_float2((float)std::cos(a), (float)std::sin(a));
            }
        n = m;
    }
    // Parker short-scan weights (reconFDK.m:41-42, :56-60; shortScanParkerWeight.m)
    std::vector<float> parker;
    double bmin = betas[0], bmax = betas[0];
    for (int k = 0; k < G.noviews; k++) {
        bmin = std::min(bmin, betas[k]);
        bmax = std::max(bmax, betas[k]);
    }
    if (short_scan) {
        const double Tau = flat ? std::fabs(betas[G.noviews - 1] - betas[0]) - M_PI : std::fabs(bmax - bmin) - M_PI;
        parker.resize((size_t)G.noviews * G.nu);
        for (int k = 0; k < G.noviews; k++) {
            const double beta = betas[k] - bmin;
            for (int iu = 0; iu < G.nu; iu++) {
                const double gammas = flat ? std::atan(-u[iu] / SDD) : -u[iu] / SDD;
                const double gamma = -gammas;
                const double w = parker_s(beta / (Tau - 2 * gamma) - 0.5) -
                                 parker_s((beta - M_PI + 2 * gamma) / (Tau + 2 * gamma) - 0.5);
                parker[(size_t)k * G.nu + iu] = (float)w;
            }
        }
    }
    // dbeta (reconFDK.m:78-81)
    double dbeta = G.noviews > 1 ? std::fabs(betas[G.noviews - 1] - betas[0]) / (G.noviews - 1) : 0.0;
    if (!short_scan) dbeta /= 2.0;
    f->dbeta = (float)dbeta;

    cudaError_t e;
    const ctsim_plan *p = plan;
    if ((e = ctsim_plan_alloc(p, (void **)&f->d_H, sizeof(float) * f->L)) != cudaSuccess ||
        (e = ctsim_plan_alloc(p, (void **)&f->d_wcos, sizeof(float) * wcos.size())) != cudaSuccess ||
        (e = ctsim_plan_alloc(p, (void **)&f->d_tw, sizeof(float2) * tw.size())) != cudaSuccess ||
        (short_scan && (e = ctsim_plan_alloc(p, (void **)&f->d_parker, sizeof(float) * parker.size())) != cudaSuccess)) {
        free_fdk(f);
        return ctsim_set_last_error(CTSIM_ERR_ALLOC, cudaGetErrorString(e));
    }
    if ((e = ctsim_plan_upload(p, f->d_H, H.data(), sizeof(float) * f->L)) != cudaSuccess ||
        (e = ctsim_plan_upload(p, f->d_wcos, wcos.data(), sizeof(float) * wcos.size())) != cudaSuccess ||
        (e = ctsim_plan_upload(p, f->d_tw, tw.data(), sizeof(float2) * tw.size())) != cudaSuccess ||
        (short_scan && (e = ctsim_plan_upload(p, f->d_parker, parker.data(), sizeof(float) * parker.size())) != cudaSuccess)) {
        free_fdk(f);
        return ctsim_set_last_error(CTSIM_ERR_CUDA, cudaGetErrorString(e));
    }
    *out = f;
    return CTSIM_OK;
}

extern "C" ctsim_status ctsim_fdk_destroy(ctsim_fdk *f) {
    free_fdk(f);
    return CTSIM_OK;
}

// The row filter of sino (sino_dtype) into out (out_dtype); FP32 arithmetic.
static ctsim_status fdk_filter(ctsim_fdk *f, const void *d_sino, int sino_dtype, void *out, int out_dtype,
                               void *stream) {
    const size_t sm = sizeof(float2) * kFiltSignals * filt_pos(f->L);
    if (sm > 200 * 1024) return ctsim_set_last_error(CTSIM_ERR_UNSUPPORTED, "detector too wide for the row filter");
    cudaError_t e = allow_dynamic_smem((const void *)fdk_filter_kernel, sm);
    if (e != cudaSuccess) return ctsim_set_last_error(CTSIM_ERR_CUDA, cudaGetErrorString(e));
    dim3 grid((f->nv + kFiltRows - 1) / kFiltRows, f->nviews);
    fdk_filter_kernel<<<grid, kFiltThreads, sm, (cudaStream_t)stream>>>(d_sino, sino_dtype, out, out_dtype, f->d_wcos,
                                                                f->d_parker, f->d_H, f->d_tw, f->nu, f->nv, f->L,
                                                                f->n8, f->n4);
    if ((e = cudaGetLastError()) != cudaSuccess) return ctsim_set_last_error(CTSIM_ERR_CUDA, cudaGetErrorString(e));
    return CTSIM_OK;
}

extern "C" ctsim_status ctsim_fdk_filter_ex(ctsim_fdk *f, const void *d_sino, int sino_dtype, float *d_filtered,
                                            void *stream) {
    if (!f || !d_sino || !d_filtered) return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "null argument");
    if (sino_dtype < kF32 || sino_dtype > kF16) return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "unknown storage type");
    return fdk_filter(f, d_sino, sino_dtype, d_filtered, kF32, stream);
}

extern "C" ctsim_status ctsim_fdk_filter(ctsim_fdk *f, const float *d_sino, float *d_filtered, void *stream) {
    return ctsim_fdk_filter_ex(f, d_sino, kF32, d_filtered, stream);
}

extern "C" ctsim_status ctsim_fdk_run_ex(ctsim_fdk *f, const void *d_sino, int sino_dtype, float *d_image,
                                         void *stream) {
    if (!f || !d_sino || !d_image) return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "null argument");
    if (sino_dtype < kF32 || sino_dtype > kF16) return ctsim_set_last_error(CTSIM_ERR_ARGUMENT, "unknown storage type");
    // the filtered sinogram is kept in the input's storage type (a BF16/FP16 request holds
    // no FP32 sinogram-sized buffer), allocated at the first run that needs its size
    const size_t need = (size_t)f->nu * f->nv * f->nviews * (sino_dtype == kF32 ? 4 : 2);
    if (f->filtered_bytes < need) {
        ctsim_plan_release(f->plan, f->d_filtered);
        f->d_filtered = nullptr;
        f->filtered_bytes = 0;
        cudaError_t e = ctsim_plan_alloc(f->plan, &f->d_filtered, need);
        if (e != cudaSuccess) return ctsim_set_last_error(CTSIM_ERR_ALLOC, cudaGetErrorString(e));
        f->filtered_bytes = need;
    }
    ctsim_status s = fdk_filter(f, d_sino, sino_dtype, f->d_filtered, sino_dtype, stream);
    if (s != CTSIM_OK) return s;
    // img = backProjectMex(sino, geom, 1, 0, 'back,hpd') * dbeta * 10  (reconFDK.m:84)
    return ctsim_plan_back_hpd(f->plan, f->d_filtered, sino_dtype, d_image, f->dbeta, 10.0f, (cudaStream_t)stream);
}

extern "C" ctsim_status ctsim_fdk_run(ctsim_fdk *f, const float *d_sino, float *d_image, void *stream) {
    return ctsim_fdk_run_ex(f, d_sino, kF32, d_image, stream);
}

extern "C" float ctsim_fdk_dbeta(const ctsim_fdk *f) { return f ? f->dbeta : 0.0f; }
