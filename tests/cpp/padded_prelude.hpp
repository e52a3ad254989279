// Host stand-ins for what launch_smooth_y_padded and launch_smooth
// (libapr_b200/csrc/pipeline.cu) call, so that tests/test_padded_lines_host.py
// can compile those functions with g++: device buffers only keep the sizes they
// were asked for, and the passes record what they were given.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

struct HostDim3 {
    unsigned x, y, z;
};
static HostDim3 blockIdx, threadIdx, blockDim;

#define __global__
#define __restrict__

struct uint4 {
    uint32_t x, y, z, w;
};
inline uint4 make_uint4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) { return {a, b, c, d}; }
struct float2 {
    float x, y;
};

typedef void *cudaStream_t;
enum { APRB_ERR_CUDA = 6 };
struct Error {
    int status;
};
inline void set_error(const std::string &) {}
inline void count_launch() {}
#define APRB_PROF(name, s)
#define APRB_CHECK_LAUNCH()
inline unsigned blocks_for(uint64_t n, unsigned threads) { return (unsigned)((n + threads - 1) / threads); }

// holds memory only up to kHeld bytes: the large cases look at sizes alone
constexpr size_t kHeld = size_t(1) << 20;
struct DevBuf {
    std::vector<uint64_t> mem;
    size_t cap = 0;
    template <typename T>
    T *as_on(size_t n, cudaStream_t) {
        cap = std::max(cap, n * sizeof(T));
        mem.resize(std::min(cap, kHeld) / 8 + 2);
        return (T *)mem.data();
    }
};

struct IIRDev {};
struct IIRCoef {};
inline IIRCoef iir_coefficients(float, int) { return {}; }
inline IIRDev dev_coef(const IIRCoef &) { return {}; }
constexpr int kAY = 64;

struct Run {
    const uint16_t *buf;
    uint64_t first, lines;  // of the working image
    size_t bytes;           // held by the padded copy
};
static std::vector<Run> g_runs;
static float *g_work;
static DevBuf *g_pad;
static int g_accept;  // TMA y passes that are taken before one is refused
static std::string g_passes;

inline bool launch_iir_y_tma(const uint16_t *img, float *work, int, int pitch, uint64_t nlines, const IIRDev &,
                             unsigned *, float2 *, uint64_t, cudaStream_t) {
    if (g_accept-- <= 0) return false;
    g_runs.push_back({img, (uint64_t)(work - g_work) / pitch, nlines, g_pad->cap});
    return true;
}
template <typename IT>
void launch_smooth_x(IT *, int yn, int, int, float, unsigned *, DevBuf &, cudaStream_t) {
    g_passes += "x" + std::to_string(yn) + " ";
}
template <typename IT>
void launch_smooth_yx(const uint16_t *, IT *, int yn, int, int, float, const float *, unsigned *, DevBuf &,
                      cudaStream_t) {
    g_passes += "yx" + std::to_string(yn) + " ";
}
template <typename IT>
void launch_smooth_z(IT *, int yn, int, int, float, unsigned *, DevBuf &, cudaStream_t) {
    g_passes += "z" + std::to_string(yn) + " ";
}

// the padded copy's launch: its lines must fit what the buffer holds
static bool g_fits = true, g_copy = false;
void pad_lines_kernel(const uint16_t *src, int yn, int pitch, uint64_t nlines, uint16_t *dst);
inline void run_pad(const uint16_t *src, int yn, int pitch, uint64_t nlines, uint16_t *dst) {
    g_fits = g_fits && nlines * (uint64_t)pitch * 2 <= g_pad->cap;
    if (!g_copy) return;
    blockDim = {256, 1, 1};
    for (uint64_t t = 0; t < nlines * (uint64_t)(pitch / 8) + 256; ++t) {
        blockIdx = {(unsigned)(t / 256), 0, 0};
        threadIdx = {(unsigned)(t % 256), 0, 0};
        pad_lines_kernel(src, yn, pitch, nlines, dst);
    }
}
