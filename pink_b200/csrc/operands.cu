// SOM operand quantiser, key fill, and the rotation-set entry point that never allocates (the rotation kernel itself:
// rotate.cu).
#include "../../include/pink_b200.h"
#include "kernels.cuh"
#include "quant.cuh"

#include <atomic>

#include <cmath>

namespace pinkb {

namespace {

template <typename Acc>
__device__ __forceinline__ Acc block_sum(Acc v, Acc* scratch)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    Acc r = 0;
    if (warp == 0) {
        r = lane < nw ? scratch[lane] : Acc(0);
        for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    }
    return r;   // valid in thread 0
}

// One CTA per neuron: centre crop of every channel, convert, row sum of squares.
// Replaces the per-image copy_and_transform_kernel pass over the whole SOM
// (src/CudaLib/generate_euclidean_distance_matrix.h:64-84); here it runs once
// when a SOM is loaded, afterwards the update kernel refreshes the rows it changes.
template <int MODE>
__global__ void __launch_bounds__(256)
quantize_som_kernel(Geometry g, const float* __restrict__ som, void* __restrict__ a0, void* __restrict__ a1,
                    void* __restrict__ anorm, uint2* __restrict__ wrange)
{
    __shared__ unsigned long long red[8];
    __shared__ uint32_t lo_s[8], hi_s[8];
    const size_t n = blockIdx.x;
    const float* src = som + n * g.Pp;
    const uint32_t K1 = g.ed * g.ed;
    const uint32_t groups = (g.K + 3) / 4;
    unsigned long long acc = 0;
    for (uint32_t k4 = threadIdx.x; k4 < groups; k4 += blockDim.x) {
        float val[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            uint32_t k = k4 * 4 + e;
            val[e] = 0.0f;
            if (k < g.K) {
                uint32_t c = k / K1, r = k - c * K1;
                uint32_t i = r / g.ed, jj = r - i * g.ed;
                if (in_region(g, i, jj)) val[e] = src[c * g.Pc + (g.off + i) * g.nd + g.off + jj];
            }
        }
        if (MODE == kModeU8) {
            uint32_t q0 = quant_u8(val[0]), q1 = quant_u8(val[1]), q2 = quant_u8(val[2]), q3 = quant_u8(val[3]);
            acc += q0 * q0 + q1 * q1 + q2 * q2 + q3 * q3;
            reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(a0) + n * g.Kp)[k4] = q0 | (q1 << 8) | (q2 << 16) | (q3 << 24);
        } else if (MODE == kModeU16) {
            uint32_t q0 = quant_u16(val[0]), q1 = quant_u16(val[1]), q2 = quant_u16(val[2]), q3 = quant_u16(val[3]);
            acc += (unsigned long long)q0 * q0 + (unsigned long long)q1 * q1
                 + (unsigned long long)q2 * q2 + (unsigned long long)q3 * q3;
            reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(a0) + n * g.Kp)[k4] =
                (q0 >> 8) | ((q1 >> 8) << 8) | ((q2 >> 8) << 16) | ((q3 >> 8) << 24);
            reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(a1) + n * g.Kp)[k4] =
                (q0 & 255) | ((q1 & 255) << 8) | ((q2 & 255) << 16) | ((q3 & 255) << 24);
        } else {
            reinterpret_cast<float4*>(static_cast<float*>(a0) + n * g.Kp)[k4] = make_float4(val[0], val[1], val[2], val[3]);
        }
    }
    if (MODE != kModeF32) {
        unsigned long long s = block_sum<unsigned long long>(acc, red);
        if (threadIdx.x == 0) {
            if (MODE == kModeU8) static_cast<uint32_t*>(anorm)[n] = (uint32_t)s;
            else static_cast<unsigned long long*>(anorm)[n] = s;
        }
    }
    if (wrange) {
        // bit patterns of min |w| and max |w| over the whole neuron (integer order = float order for
        // non-negative values; NaN patterns compare highest)
        uint32_t lo = 0xFFFFFFFFu, hi = 0;
        for (uint32_t c = 0; c < g.C; ++c) {
            for (uint32_t i = threadIdx.x; i < g.nd * g.nd; i += blockDim.x) {
                const uint32_t b = __float_as_uint(src[c * g.Pc + i]) & 0x7FFFFFFFu;
                lo = min(lo, b); hi = max(hi, b);
            }
        }
        lo = __reduce_min_sync(0xffffffffu, lo); hi = __reduce_max_sync(0xffffffffu, hi);
        if ((threadIdx.x & 31) == 0) { lo_s[threadIdx.x >> 5] = lo; hi_s[threadIdx.x >> 5] = hi; }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (uint32_t wv = 1; wv < blockDim.x / 32; ++wv) { lo = min(lo, lo_s[wv]); hi = max(hi, hi_s[wv]); }
            wrange[n] = make_uint2(lo, hi);
        }
    }
}

__global__ void fill_keys_kernel(unsigned long long* keys, size_t count)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x)
        keys[i] = kKeyEmpty;
}

constexpr size_t kRotateSmemLimit = 200 * 1024;

} // namespace

cudaError_t launch_quantize_som(const Geometry& g, const float* som, uint32_t n, void* a0, void* a1, void* anorm,
                                cudaStream_t st, uint2* wrange)
{
    if (n == 0) return cudaSuccess;
    if (g.mode == kModeU8) quantize_som_kernel<kModeU8><<<n, 256, 0, st>>>(g, som, a0, a1, anorm, wrange);
    else if (g.mode == kModeU16) quantize_som_kernel<kModeU16><<<n, 256, 0, st>>>(g, som, a0, a1, anorm, wrange);
    else quantize_som_kernel<kModeF32><<<n, 256, 0, st>>>(g, som, a0, a1, anorm, wrange);
    return cudaGetLastError();
}

cudaError_t launch_fill_keys(unsigned long long* keys, size_t count, cudaStream_t st)
{
    if (count == 0) return cudaSuccess;
    unsigned blocks = (unsigned)((count + 255) / 256);
    if (blocks > 1184) blocks = 1184;
    fill_keys_kernel<<<blocks, 256, 0, st>>>(keys, count);
    return cudaGetLastError();
}

} // namespace pinkb

// ---------------------------------------------------------------------------
// Rotation-set entry point that never allocates.
//
// pink_b200_op_rotate stages the cos/sin table of the rotation angles in device
// memory it obtains with cudaMalloc on every call.  Some callers must not do
// that: code running while the CUDA allocator is locked or forbidden (inside a
// memory-pool or caching-allocator callback, in a process whose device memory
// is fully pre-reserved by its own arena, or in a latency-critical loop where an
// implicit device synchronisation of cudaMalloc/cudaFree is unacceptable).
// For them the table lives in the fixed device array below, which every GPU
// that loads this library holds until the process exits.
namespace pinkb {
namespace {

constexpr uint32_t kStaticMaxQuadrant = 4096;     // rotations per quadrant, i.e. number_of_rotations <= 16384
static __device__ __align__(256) float g_rotate_scratch[2 * kStaticMaxQuadrant];   // [cos | sin], 32 KB

// Device address of the scratch array on the current device (looked up once per device).
cudaError_t rotate_scratch_address(float** out)
{
    constexpr int kMaxDevices = 64;
    static std::atomic<float*> addr[kMaxDevices];        // first calls may come from several host threads
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    float* known = addr[dev].load(std::memory_order_acquire);
    if (!known) {
        // In host code the array's name is only a handle; the kernels need its device address.
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_rotate_scratch);
        if (e != cudaSuccess) return e;
        known = static_cast<float*>(p);
        addr[dev].store(known, std::memory_order_release);   // every thread looks up the same address
    }
    *out = known;
    return cudaSuccess;
}

} // namespace
} // namespace pinkb

extern "C" int pink_b200_op_rotate_static(const pink_b200_config* cfg, const float* dev_images, uint32_t n_img,
                                          float* dev_base, void* dev_b0, void* dev_b1, void* dev_bnorm, void* stream)
{
    using namespace pinkb;
    if (!cfg || !dev_images || !dev_b0) return report_error(PINK_B200_EINVAL, "null argument");
    Geometry g{};
    int rc = geometry_from_config(cfg, &g);
    if (rc) return rc;
    const uint32_t nq = g.q ? g.q : 1;
    if (nq > kStaticMaxQuadrant)
        return report_error(PINK_B200_EINVAL,
                            "pink_b200_op_rotate_static supports at most 16384 rotations (4096 per quadrant); "
                            "use pink_b200_op_rotate for more");
    if (!dev_base && (size_t)g.P * sizeof(float) > kRotateSmemLimit)
        return report_error(PINK_B200_EINVAL, "dev_base is required when a base rotation does not fit shared memory");
    float* scratch = nullptr;
    cudaError_t e = rotate_scratch_address(&scratch);
    if (e != cudaSuccess) return report_error(PINK_B200_ECUDA, cudaGetErrorString(e));

    // cos/sin of t * (float(2*pi)/R), t < R/4, with the reference's expressions
    // (src/SelfOrganizingMapLib/generate_rotated_images.h:70, src/ImageProcessingLib/rotate.h:20-21).
    static thread_local float table[2 * kStaticMaxQuadrant];
    const float step = static_cast<float>(2 * M_PI) / g.R;
    for (uint32_t t = 0; t < nq; ++t) {
        const float angle = t * step;
        table[t] = std::cos(angle);
        table[nq + t] = std::sin(angle);
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // The shared array still holds the previous call's table; the part this call uses is overwritten in full.
    e = cudaMemcpyAsync(scratch, table, 2 * nq * sizeof(float), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = clear_operand_padding(g, (size_t)n_img * g.T, dev_b0, dev_b1, st);
    if (e == cudaSuccess) e = launch_rotate(g, dev_images, n_img, scratch, scratch + nq, dev_base, g.nd * g.nd, dev_b0, dev_b1, dev_bnorm, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);      // `table` is reused by this thread's next call
    if (e != cudaSuccess) return report_error(PINK_B200_ECUDA, cudaGetErrorString(e));
    return PINK_B200_OK;
}
