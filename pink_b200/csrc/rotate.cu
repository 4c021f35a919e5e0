// Rotation-set generator: base rotations and distance operand rows of a batch of images.
//
// rotate_kernel replaces the reference's seven-launch sequence
//   thrust::fill + resize_kernel + rotate_bilinear_kernel + 3 x rotate_90_degrees_list
//   + flip_kernel              (src/CudaLib/generate_rotated_images.h:56-167, :170-294)
// followed by the per-image crop/convert of every transform
//   copy_and_transform_kernel  (src/CudaLib/copy_and_transform_kernel.h:15-29,
//                               src/CudaLib/generate_euclidean_distance_matrix.h:86-112)
// with ONE launch that never materialises the T x P float set: a block computes
// interpolated base rotations, stores them once as float for the update step (training), and emits the
// distance operand rows of all eight transforms that are exact index permutations of a base (four
// quarter turns x optional flip), plus each row's sum of squares.
//
// Arithmetic: every product and sum of the interpolation is rounded
// separately (explicitly rounded operations are never contracted to FMA), in the order
// of the reference's CPU code (src/ImageProcessingLib/rotate.h:31-63), so the
// float pixels are bit-identical to the CPU reference built without FMA.
//
// What bounds it and why it is split this way.  The kernel issues instructions; the bytes are few.  So:
//   * a block keeps the image (one channel) in shared memory and works through a group of base rotations: the
//     four taps of a pixel are shared-memory reads.  A warp computes an 8 x 4 (twice: 16 x 4) tile of pixels,
//     whose taps lie in a compact patch of the image, and the row pitch of the staged image is chosen so that
//     such a patch maps to different banks (bank_pitch).
//   * the row and column terms of the rotation come from a small table per base rotation.
//   * without base rotations to store (mapping) only the distance region is interpolated.
//   * the converted region is staged once, in rows of odd pitch; each thread then gathers four operand elements
//     per transform with conflict-free one-element reads, for all eight transforms from one set of offsets, and
//     stores them as one word.
#include "kernels.cuh"
#include "ptx.cuh"
#include "quant.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace pinkb {

constexpr uint32_t kRotMaxThreads = 1024;
constexpr uint32_t kRotMaxGroup = 32;         // base rotations a block works through at most
constexpr uint32_t kRotSmemBudget = 216 * 1024;
constexpr uint32_t kRotHalfSm = 114 * 1024 - 1024 - 4096 - 256;   // dynamic shared memory of one of two blocks that share an SM

template <int MODE> struct StageType;
template <> struct StageType<kModeU8>  { using type = uint8_t; };
template <> struct StageType<kModeU16> { using type = uint16_t; };
template <> struct StageType<kModeF32> { using type = float; };

// Launch shape and shared-memory layout.
struct RotPlan
{
    uint32_t group, groups;          // base rotations per block, blocks per image
    uint32_t x0, nx;                 // window of the neuron that is interpolated (rows and columns alike): [x0, x0 + nx)
    uint32_t r0, side, pitch;        // staged part of the image: rows and columns [r0, r0 + side), one more of each repeated
    uint32_t win, sp;                // staged region: side (ed, or ed + 1 where the crop is off centre) and row pitch
    uint32_t off_image, off_region, off_plane;   // byte offsets in shared memory (row and column terms first): image, region or operand rows, float plane
    uint32_t use_image, use_region, use_plane;   // staged in shared memory
    uint32_t row_bufs, row_pitch, row_size;   // kPlanes: sets of operand rows (1 or 2), bytes from region row to region row, bytes of an operand row
    uint32_t base_plane;             // floats from one channel plane of base_out to the next
    uint32_t nband, ntile, magic_nband, magic_ed;      // bands of four rows, tiles of 4 x 16 pixels
};

// How a block finds its inputs: kFast -- image and region staged in shared memory, square region; kCircle -- the same with
// a circular region; kLarge -- images or regions that do not fit shared memory are read through the cache.
// kPlanes (uint8, one channel) -- as kFast, but the pixels are scattered straight into the eight operand rows, which leave
// shared memory as whole rows by bulk copies.
enum : int { kFast = 0, kCircle = 1, kLarge = 2, kPlanes = 3 };

// Launches rotate_kernel<MODE, ., KIND, .>; fills in rp.group and rp.groups.
template <int MODE, int KIND>
cudaError_t rotate_run(const Geometry& g, RotPlan& rp, bool inside, uint32_t n_img, size_t smem, const float* images, const float* cs, const float* sn,
                       float* base_out, void* b0, void* b1, void* b2, void* bnorm, uint32_t* rmax, cudaStream_t st);

// The file is compiled once for each (MODE, KIND) -- the kernels -- and once without the macros -- the choice between them.
// The CUDA runtime loads a module whole when its first kernel is launched: with all 32 variants in one the first call of a
// process took 2.4 ms longer than with a few.
#ifdef PINK_ROTATE_MODE

namespace {

// v / d for v * d < 2^32 with magic = floor(2^32 / d) + 1 (checked on the host).
// magic == 0 encodes the divisor 1.
__device__ __forceinline__ uint32_t fast_div(uint32_t v, uint32_t magic) { return magic ? __umulhi(v, magic) : v; }

template <int MODE>
__device__ __forceinline__ typename StageType<MODE>::type to_stage(float v)
{
    if (MODE == kModeU8) return (typename StageType<MODE>::type)quant_u8(v);
    if (MODE == kModeU16) return (typename StageType<MODE>::type)quant_u16(v);
    return (typename StageType<MODE>::type)v;
}

// Shared-memory accesses by 32-bit shared-window address (one add per access instead of a generic pointer's arithmetic).
__device__ __forceinline__ float lds_f32(uint32_t a) { float v; asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a)); return v; }
__device__ __forceinline__ float2 lds_f32x2(uint32_t a) { float2 v; asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a)); return v; }
__device__ __forceinline__ uint32_t lds_u8(uint32_t a) { uint32_t v; asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint32_t lds_u16(uint32_t a) { uint32_t v; asm volatile("{ .reg .u16 t; ld.shared.u16 t, [%1]; cvt.u32.u16 %0, t; }" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint4 lds_u32x4(uint32_t a) { uint4 v; asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a)); return v; }
__device__ __forceinline__ void sts_f32(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" :: "r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ void sts_u8(uint32_t a, uint32_t v) { asm volatile("st.shared.u8 [%0], %1;" :: "r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void sts_u16(uint32_t a, uint32_t v) { asm volatile("{ .reg .u16 t; cvt.u16.u32 t, %1; st.shared.u16 [%0], t; }" :: "r"(a), "r"(v) : "memory"); }

// INSIDE: the rotated window cannot leave the image at any angle -- half its diagonal, plus a margin far above the
// rounding of the positions, lies within half the image -- so every source position s satisfies 0 <= s < id - 1:
// the range test and the clamps are identities and are left out.
// FLAGS: bit 0 base rotations are stored, bit 1 the region is centred in the neuron; -1: decided at run time.
template <int MODE, bool INSIDE, int KIND, int FLAGS>
__global__ void __launch_bounds__(kRotMaxThreads, 1)
rotate_kernel(const __grid_constant__ Geometry g, const __grid_constant__ RotPlan rp, const float* __restrict__ images,
              const float* __restrict__ cs, const float* __restrict__ sn, float* __restrict__ base_out,
              void* __restrict__ b0, void* __restrict__ b1, void* __restrict__ b2, void* __restrict__ bnorm,
              uint32_t* __restrict__ rmax)
{
    using stage_t = typename StageType<MODE>::type;
    using sum_t = typename std::conditional<MODE == kModeF32, float,
                  typename std::conditional<MODE == kModeU8, uint32_t, unsigned long long>::type>::type;
    using total_t = typename std::conditional<MODE == kModeF32, double, unsigned long long>::type;
    extern __shared__ __align__(128) uint8_t rot_dyn[];
    __shared__ sum_t sum_s[kRotMaxThreads / 32][8];             // per warp: sums of squares of the current base rotation
    __shared__ total_t norm_s[kRotMaxGroup][8];                 // per base rotation of the group and transform: over the channels so far

    constexpr uint32_t esz = sizeof(stage_t);
    const bool staged = KIND != kLarge || rp.use_image, in_smem = KIND != kLarge || rp.use_region;
    const bool circle = KIND == kCircle || (KIND == kLarge && g.circle != nullptr);
    const uint32_t img_i = blockIdx.y;
    const uint32_t nbase = g.q ? g.q : 1;
    const uint32_t b_lo = blockIdx.x * rp.group, b_n = min(rp.group, nbase - b_lo);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const uint32_t nd = g.nd, ed = g.ed, P1 = nd * nd, K1 = ed * ed, idm1 = g.id - 1, Kp = g.Kp, goff = g.off;
    const uint32_t nq = g.q ? 4 : 1, nv = nq * (g.flip ? 2 : 1);
    const float sc = (g.id - 1) * 0.5f, dc = (nd - 1) * 0.5f, lim = (float)(g.id - 1);
    const bool with_norm = MODE != kModeF32 || b1 != nullptr;
    const uint32_t x0 = rp.x0, nx = rp.nx, win = rp.win, pitch = rp.pitch;
    const uint32_t smem = smem_u32(rot_dyn);
    const uint32_t img_a = smem + rp.off_image, region_a = smem + rp.off_region, plane_a = smem + rp.off_plane, table_a = smem;
    const uint32_t rpitch = rp.row_pitch, rsize = rp.row_size;      // kPlanes
    const bool padded = KIND == kPlanes && rpitch != ed;
    const bool with_base = FLAGS < 0 ? base_out != nullptr : (FLAGS & 1) != 0, centred = FLAGS < 0 ? win == ed : (FLAGS & 2) != 0;
    const bool use_plane = with_base && rp.use_plane;
    uint32_t vmax = 0;                    // bit pattern of max |pixel| (NaN patterns compare highest)

    for (uint32_t i = threadIdx.x; i < kRotMaxGroup * 8; i += blockDim.x) (&norm_s[0][0])[i] = total_t(0);
    if (KIND == kPlanes && !padded)       // the rows' padding beyond K is zero
        for (uint32_t r = warp; r < 8 * rp.row_bufs; r += nwarps)
            for (uint32_t k = g.K + lane; k < Kp; k += 32) sts_u8(region_a + r * rsize + k, 0);
    // Row and column terms of base rotation tq: {p * cos, p * sin} of every window position's distance p from the centre.
    auto make_table = [&](uint32_t tq) {
        const float ca = tq ? cs[tq] : 1.0f, sa = tq ? sn[tq] : 0.0f;
        for (uint32_t i = threadIdx.x; i < nx; i += blockDim.x) {
            const float p = __fsub_rn((float)(x0 + i), dc);
            sts_f32(table_a + 8 * i, __fmul_rn(p, ca));
            sts_f32(table_a + 8 * i + 4, __fmul_rn(p, sa));
        }
    };

    for (uint32_t c = 0; c < g.C; ++c) {
        const float* img = images + ((size_t)img_i * g.C + c) * g.id * g.id;
        if (staged) {
            // the last row and column are repeated: taps there carry weight 0 (INSIDE: they are not reached)
            const uint32_t full = rp.side + 1;
            for (uint32_t r = warp; r < full; r += nwarps) {
                const float* src = img + (size_t)min(rp.r0 + r, idm1) * g.id;
                for (uint32_t y = lane; y < full; y += 32) {
                    const float v = __ldg(src + min(rp.r0 + y, idm1));
                    sts_f32(img_a + 4 * (r * pitch + y), v);
                    vmax = max(vmax, __float_as_uint(v) & 0x7FFFFFFFu);
                }
            }
        }
        make_table(b_lo);
        __syncthreads();

        for (uint32_t b = 0; b < b_n; ++b) {
            const uint32_t tq = b_lo + b;
            float* gplane = with_base ? base_out + (((size_t)img_i * nbase + tq) * g.C + c) * rp.base_plane : nullptr;
            const uint32_t rows_a = region_a + (KIND == kPlanes && (b & (rp.row_bufs - 1)) ? 8 * rsize : 0u);
            sum_t sum[4] = { sum_t(0), sum_t(0), sum_t(0), sum_t(0) };   // [mirrored rows][mirrored columns]
            // Where the pixel at window row xi and column yi goes: its place in the float plane, and in the staged region or, kPlanes, in
            // the eight operand rows -- rows and columns as they are / mirrored, row-major or (quarter turns) column-major.
            struct Places { uint32_t plane, at[8]; };
            const uint32_t shift = goff - x0;                              // window position of the region's first row and column
            const uint32_t m1 = win - 1, rp_step = esz * rp.sp;
            auto places = [&](uint32_t xi, uint32_t yi) {
                Places p;
                p.plane = use_plane ? plane_a + 4 * (xi * nd + yi) : (x0 + xi) * nd + x0 + yi;
                const uint32_t wx = xi - shift, wy = yi - shift;
                if (KIND == kPlanes) {
                    p.at[0] = rows_a + wx * rpitch + wy;                  p.at[4] = rows_a + 4 * rsize + (m1 - wx) * rpitch + wy;
                    p.at[6] = rows_a + 6 * rsize + wx * rpitch + (m1 - wy);  p.at[2] = rows_a + 2 * rsize + (m1 - wx) * rpitch + (m1 - wy);
                    p.at[7] = rows_a + 7 * rsize + wy * rpitch + wx;      p.at[1] = rows_a + rsize + wy * rpitch + (m1 - wx);
                    p.at[3] = rows_a + 3 * rsize + (m1 - wy) * rpitch + wx;  p.at[5] = rows_a + 5 * rsize + (m1 - wy) * rpitch + (m1 - wx);
                } else {
                    p.at[0] = region_a + wx * rp_step + esz * wy;
                }
                return p;
            };
            // four rows further down
            auto advance = [&](Places& p) {
                p.plane += use_plane ? 16 * nd : 4 * nd;
                if (KIND == kPlanes) {
                    p.at[0] += 4 * rpitch; p.at[6] += 4 * rpitch; p.at[4] -= 4 * rpitch; p.at[2] -= 4 * rpitch;
                    p.at[7] += 4; p.at[3] += 4; p.at[1] -= 4; p.at[5] -= 4;
                } else {
                    p.at[0] += 4 * rp_step;
                }
            };
            // Stores pixel v of window position (xi, yi); E is 1 for the second pixel of a thread, eight columns further right.
            auto put = [&](auto second, const Places& p, uint32_t xi, uint32_t yi, float v) {
                constexpr uint32_t E = decltype(second)::value ? 8 : 0;
                if (with_base) {
                    if (use_plane) sts_f32(p.plane + 4 * E, v);
                    else gplane[p.plane + E] = v;
                }
                const uint32_t wx = xi - shift, wy = yi - shift;           // position in the region; unsigned wrap rejects xi < shift
                if (!with_base || (wx < win && wy < win)) {
                    const stage_t s = to_stage<MODE>(v);
                    const uint32_t sb = MODE == kModeF32 ? 0u : (uint32_t)s;
                    if (KIND == kPlanes) {
                        // a mirrored index drops row (column) 0 of an off-centre window
                        const uint32_t e8 = E * rpitch;
                        if (centred) {
                            sts_u8(p.at[0] + E, sb); sts_u8(p.at[4] + E, sb); sts_u8(p.at[6] - E, sb); sts_u8(p.at[2] - E, sb);
                            sts_u8(p.at[7] + e8, sb); sts_u8(p.at[1] + e8, sb); sts_u8(p.at[3] - e8, sb); sts_u8(p.at[5] - e8, sb);
                        } else {
                            if (wx < ed && wy < ed) { sts_u8(p.at[0] + E, sb); sts_u8(p.at[7] + e8, sb); }
                            if (wx > 0 && wy < ed) { sts_u8(p.at[4] + E, sb); sts_u8(p.at[1] + e8, sb); }
                            if (wx < ed && wy > 0) { sts_u8(p.at[6] - E, sb); sts_u8(p.at[3] - e8, sb); }
                            if (wx > 0 && wy > 0) { sts_u8(p.at[2] - E, sb); sts_u8(p.at[5] - e8, sb); }
                        }
                    } else if (in_smem) {
                        if (MODE == kModeU8) sts_u8(p.at[0] + E, sb);
                        else if (MODE == kModeU16) sts_u16(p.at[0] + 2 * E, sb);
                        else sts_f32(p.at[0] + 4 * E, (float)s);
                    }
                    if (with_norm && !circle) {
                        const sum_t sq = MODE == kModeF32 ? (sum_t)s * (sum_t)s : (sum_t)(sb * sb);
                        if (centred) sum[0] += sq;
                        else {
                            if (wx < ed && wy < ed) sum[0] += sq;
                            if (wx < ed && wy > 0) sum[1] += sq;
                            if (wx > 0 && wy < ed) sum[2] += sq;
                            if (wx > 0 && wy > 0) sum[3] += sq;
                        }
                    }
                }
            };
            using First = std::integral_constant<bool, false>;
            using Second = std::integral_constant<bool, true>;
            if (tq == 0) {
                // centre crop / zero pad (src/CudaLib/resize_kernel.h:15-32, integer margins)
                for (uint32_t xi = warp; xi < nx; xi += nwarps) {
                    for (uint32_t yi = lane; yi < nx; yi += 32) {
                        const uint32_t x = x0 + xi, y = x0 + yi;
                        float v = 0.0f;
                        const uint32_t ix = g.id >= nd ? x + (g.id - nd) / 2 : x - (nd - g.id) / 2;      // unsigned wrap rejects x < margin
                        const uint32_t iy = g.id >= nd ? y + (g.id - nd) / 2 : y - (nd - g.id) / 2;
                        if (ix < g.id && iy < g.id) v = staged ? lds_f32(img_a + 4 * ((ix - rp.r0) * pitch + (iy - rp.r0))) : __ldg(img + (size_t)ix * g.id + iy);
                        if (!staged) vmax = max(vmax, __float_as_uint(v) & 0x7FFFFFFFu);
                        put(First(), places(xi, yi), xi, yi, v);
                    }
                }
            } else {
                // ---- the base rotation, tile by tile: lane = 8 columns x 4 rows, each thread the columns ya and ya + 8.
                // Inverse rotation and bilinear taps; every product and sum rounded
                // separately, in the order of src/ImageProcessingLib/rotate.h:37-63.
                // The biases 0x4B000000 of both bit patterns below and the origin of the staged part, modulo 2^32:
                const uint32_t tap_a = img_a - 4 * ((0x4B000000u + rp.r0) * (pitch + 1)), pitch4 = 4 * pitch;
                auto pixel = [&](float2 tx, float2 ty) -> float {
                    float sx = __fadd_rn(__fsub_rn(tx.x, ty.y), sc);                 // px * cos - py * sin
                    float sy = __fadd_rn(__fadd_rn(tx.y, ty.x), sc);                 // px * sin + py * cos
                    bool in = true;
                    if (!INSIDE) {
                        // positions outside the image are clamped for the (then unused) taps and the result is zeroed
                        in = fminf(sx, sy) >= 0.0f && fmaxf(sx, sy) <= lim;
                        sx = fminf(fmaxf(sx, 0.0f), lim); sy = fminf(fmaxf(sy, 0.0f), lim);
                    }
                    // floor by adding 2^23 with truncation: exact for 0 <= s < 2^23, and it keeps
                    // the conversions off the (slow) conversion pipe
                    const float fx = __fadd_rz(sx, 8388608.0f), fy = __fadd_rz(sy, 8388608.0f);
                    const float rx = __fsub_rn(sx, __fsub_rn(fx, 8388608.0f)), ry = __fsub_rn(sy, __fsub_rn(fy, 8388608.0f));
                    const float cx = __fsub_rn(1.0f, rx), cy = __fsub_rn(1.0f, ry);
                    float p00, p01, p10, p11;
                    if (staged) {
                        const uint32_t t = tap_a + 4 * (__float_as_uint(fx) * pitch + __float_as_uint(fy)), u = t + pitch4;
                        p00 = lds_f32(t); p01 = lds_f32(t + 4); p10 = lds_f32(u); p11 = lds_f32(u + 4);
                    } else {
                        const uint32_t ix = __float_as_uint(fx) & 0x7FFFFFu, iy = __float_as_uint(fy) & 0x7FFFFFu;
                        // the +1 taps carry weight 0 when they would fall outside; clamp the index
                        const uint32_t dx = INSIDE || ix < idm1 ? g.id : 0u, dy = INSIDE || iy < idm1 ? 1u : 0u;
                        const float* t = img + (size_t)ix * g.id + iy;
                        p00 = __ldg(t); p01 = __ldg(t + dy); p10 = __ldg(t + dx); p11 = __ldg(t + dx + dy);
                    }
                    const float t00 = __fmul_rn(__fmul_rn(cx, cy), p00);
                    const float t01 = __fmul_rn(__fmul_rn(cx, ry), p01);
                    const float t10 = __fmul_rn(__fmul_rn(rx, cy), p10);
                    const float t11 = __fmul_rn(__fmul_rn(rx, ry), p11);
                    float v = __fadd_rn(__fadd_rn(__fadd_rn(t00, t01), t10), t11);
                    if (!INSIDE) v = in ? v : 0.0f;
                    if (!staged) vmax = max(vmax, __float_as_uint(v) & 0x7FFFFFFFu);
                    return v;
                };
                // A warp walks a contiguous range of the tiles, numbered down the columns: what depends on the column alone
                // stays in registers.
                const uint32_t nband = rp.nband;
                uint32_t t = rp.ntile * warp / nwarps;
                const uint32_t t_end = rp.ntile * (warp + 1) / nwarps;
                while (t < t_end) {
                    const uint32_t col = fast_div(t, rp.magic_nband), band = t - col * nband;
                    const uint32_t stop = min(t_end, (col + 1) * nband);
                    uint32_t xi = band * 4 + (lane >> 3);
                    const uint32_t ya = col * 16 + (lane & 7), yb = ya + 8;
                    const float2 ta = lds_f32x2(table_a + 8 * min(ya, nx - 1)), tb = lds_f32x2(table_a + 8 * min(yb, nx - 1));
                    Places at = places(xi, ya);
                    for (; t < stop; ++t, xi += 4) {
                        const float2 tx = lds_f32x2(table_a + 8 * min(xi, nx - 1));      // lanes beyond the window compute, but do not store
                        const float va = pixel(tx, ta), vb = pixel(tx, tb);
                        if (xi < nx && ya < nx) put(First(), at, xi, ya, va);
                        if (xi < nx && yb < nx) put(Second(), at, xi, yb, vb);
                        advance(at);
                    }
                }
            }
            if (with_norm && !circle) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (k == 0 || !centred) {
                        for (int o = 16; o > 0; o >>= 1) sum[k] += __shfl_down_sync(0xffffffffu, sum[k], o);
                        if (lane == 0) sum_s[warp][k] = sum[k];
                    }
                }
            }
            if (use_plane || (KIND == kPlanes && !padded)) fence_async_smem();   // this thread's part of the plane (rows) before the bulk stores
            __syncthreads();   // (also orders this block's global writes before its own reads below)
            if (use_plane && threadIdx.x == 0) {
                bulk_store(gplane, rot_dyn + rp.off_plane, ((P1 + 3) & ~3u) * 4);
                bulk_commit();
            }
            if (padded) {
                // rows of ed bytes (a multiple of 32) at a padded pitch: 16 bytes per thread and step
                const uint32_t per_row = ed / 16, per_variant = per_row * ed;
                for (uint32_t i = threadIdx.x; i < nv * per_variant; i += blockDim.x) {
                    const uint32_t v = i / per_variant, k = i - v * per_variant, r = k / per_row, ch = k - r * per_row;
                    const uint32_t f = v / nq, j = v - f * nq;
                    reinterpret_cast<uint4*>(static_cast<uint8_t*>(b0) + ((size_t)img_i * g.T + f * g.R + j * g.q + tq) * Kp)[k]
                        = lds_u32x4(rows_a + (4 * f + j) * rsize + r * rpitch + 16 * ch);
                }
            } else if (KIND == kPlanes && threadIdx.x >= 32 && threadIdx.x < 32 + nv) {
                const uint32_t v = threadIdx.x - 32, f = v / nq, j = v - f * nq;
                bulk_store(static_cast<uint8_t*>(b0) + ((size_t)img_i * g.T + f * g.R + j * g.q + tq) * g.Kp, rot_dyn + (rows_a - smem) + (4 * f + j) * rsize, Kp);
                bulk_commit();
            }
            if (with_norm && !circle && threadIdx.x < nv) {
                // transform (flip f, quadrant j): 0 reads rows mirrored by f; 1 mirrored rows, columns mirrored by f; 2 mirrored columns,
                // rows mirrored by not f; 3 rows as they are, columns mirrored by not f
                const uint32_t f = threadIdx.x / nq, j = threadIdx.x - f * nq;
                const uint32_t mr = j == 0 ? f : j == 1 ? 1u : j == 2 ? 1u - f : 0u, mc = j == 0 ? 0u : j == 1 ? f : j == 2 ? 1u : 1u - f;
                const uint32_t k = centred ? 0u : 2 * mr + mc;
                total_t tot = 0;
                for (uint32_t wv = 0; wv < nwarps; ++wv) tot += (total_t)sum_s[wv][k];
                norm_s[b][threadIdx.x] += tot;
            }

            // ---- operand rows of every transform derived from this base: four elements per thread and step
            const uint32_t k_lo = c * K1, w_lo = MODE == kModeF32 ? 0u : k_lo / 4;
            const uint32_t n_step = KIND == kPlanes ? 0u : MODE == kModeF32 ? (K1 + 127) / 128 * 32 : (k_lo + K1 + 3) / 4 - w_lo;
            const int32_t sp = in_smem ? (int32_t)rp.sp : (int32_t)nd;
            const int32_t cc = (int32_t)win - 1, cr = cc * sp;         // offsets of the region's last column and row
            const float* greg = gplane + (g.off * nd + g.off);         // kLarge: the region inside the float plane
            const size_t row0 = ((size_t)img_i * g.T + tq) * g.Kp;     // operand row of transform (0, 0), in elements
            sum_t vsum[8];
#pragma unroll
            for (int v = 0; v < 8; ++v) vsum[v] = sum_t(0);
            for (uint32_t st = threadIdx.x; st < n_step; st += blockDim.x) {
                // elements of this channel's K1, first, first + 1, ..; float: 32 apart, so that a warp's reads and stores are consecutive
                int32_t p[4], m[4], qq[4], rr[4];
                uint32_t mask = 0, have = 0;                           // byte e: element inside the circle; bit e: element exists
                const int32_t first = MODE == kModeF32 ? (int32_t)((st / 32) * 128 + (st & 31)) : (int32_t)(4 * (w_lo + st)) - (int32_t)k_lo;
                uint32_t i = fast_div((uint32_t)max(first, 0), rp.magic_ed), jj = (uint32_t)max(first, 0) - i * ed;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int32_t r = first + e * (MODE == kModeF32 ? 32 : 1);
                    const bool ok = r >= 0 && r < (int32_t)K1;
                    if (MODE == kModeF32 && e > 0) { i = fast_div((uint32_t)r, rp.magic_ed); jj = (uint32_t)r - i * ed; }
                    const int32_t ie = ok ? (int32_t)i : 0, je = ok ? (int32_t)jj : 0;
                    p[e] = ie * sp + je; m[e] = ie * sp - je; qq[e] = je * sp + ie; rr[e] = je * sp - ie;
                    if (ok) {
                        have |= 1u << e;
                        if (!circle || in_region(g, ie, je)) mask |= 0xFFu << (8 * e);
                        if (MODE != kModeF32 && ++jj == ed) { jj = 0; ++i; }
                    }
                }
                // a word that reaches beyond the last channel ends in padding, which stays zero; one that other channels share is written by bytes
                const bool whole = MODE == kModeF32 || (first >= 0 && (first + 4 <= (int32_t)K1 || c + 1 == g.C));
                const uint32_t at = MODE == kModeF32 ? k_lo + (uint32_t)first : 4 * (w_lo + st);
                auto emit = [&](int v, size_t row, const int32_t (&a)[4]) {
                    stage_t el[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if (!in_smem) el[e] = to_stage<MODE>(greg[a[e]]);
                        else if (MODE == kModeU8) el[e] = (stage_t)lds_u8(region_a + (uint32_t)a[e]);
                        else if (MODE == kModeU16) el[e] = (stage_t)lds_u16(region_a + 2 * (uint32_t)a[e]);
                        else el[e] = (stage_t)lds_f32(region_a + 4 * (uint32_t)a[e]);
                    }
                    if (MODE == kModeU8) {
                        const uint32_t w = __byte_perm(__byte_perm((uint32_t)el[0], (uint32_t)el[1], 0x0040),
                                                       __byte_perm((uint32_t)el[2], (uint32_t)el[3], 0x0040), 0x5410) & mask;
                        if (circle) vsum[v] = (sum_t)__dp4a(w, w, (uint32_t)vsum[v]);
                        uint8_t* dst = static_cast<uint8_t*>(b0) + row + at;
                        if (whole) *reinterpret_cast<uint32_t*>(dst) = w;
                        else for (int e = 0; e < 4; ++e) if (have >> e & 1u) dst[e] = (uint8_t)(w >> (8 * e));
                    } else if (MODE == kModeU16) {
                        const uint32_t e01 = __byte_perm((uint32_t)el[0], (uint32_t)el[1], 0x5410), e23 = __byte_perm((uint32_t)el[2], (uint32_t)el[3], 0x5410);
                        const uint32_t hi = __byte_perm(e01, e23, 0x7531) & mask, lo = __byte_perm(e01, e23, 0x6420) & mask;
                        if (circle) {
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const uint32_t qv = (mask >> (8 * e) & 1u) ? (uint32_t)el[e] : 0u;
                                vsum[v] += (sum_t)(qv * qv);
                            }
                        }
                        uint8_t* d0 = static_cast<uint8_t*>(b0) + row + at;
                        uint8_t* d1 = static_cast<uint8_t*>(b1) + row + at;
                        if (whole) { *reinterpret_cast<uint32_t*>(d0) = hi; *reinterpret_cast<uint32_t*>(d1) = lo; }
                        else for (int e = 0; e < 4; ++e) if (have >> e & 1u) { d0[e] = (uint8_t)(hi >> (8 * e)); d1[e] = (uint8_t)(lo >> (8 * e)); }
                    } else {
                        float* d0 = static_cast<float*>(b0) + row + at;
                        float* d1 = static_cast<float*>(b1) + row + at;
                        float* d2 = static_cast<float*>(b2) + row + at;
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            if (have >> e & 1u) {
                                const float x = (mask >> (8 * e) & 1u) ? (float)el[e] : 0.0f;
                                d0[32 * e] = x;
                                if (b1) {
                                    // planes of the tensor-core estimate: the top 19 bits of every value and the (exact) rest
                                    const float h = __uint_as_float(__float_as_uint(x) & 0xFFFFE000u);
                                    d1[32 * e] = h;
                                    d2[32 * e] = __fsub_rn(x, h);
                                    if (circle) vsum[v] += (sum_t)(x * x);
                                }
                            }
                        }
                    }
                };
                // flip is a row reversal applied last (src/CudaLib/flip_kernel.h:28); one quarter turn maps
                // (x, y) <- (nd-1-y, x) (src/CudaLib/rotate_90_degrees_list.h:28)
                int32_t a[4];
                auto emit_at = [&](int v, size_t row, int32_t base, const int32_t (&o)[4], bool minus) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) a[e] = minus ? base - o[e] : base + o[e];
                    emit(v, row, a);
                };
                const size_t sq = (size_t)g.q * g.Kp, sf = (size_t)g.R * g.Kp;       // operand elements per quadrant and per flip
                emit_at(0, row0, 0, p, false);
                if (nq > 1) {
                    emit_at(1, row0 + sq, cr, rr, true);
                    emit_at(2, row0 + 2 * sq, cr + cc, p, true);
                    emit_at(3, row0 + 3 * sq, cc, rr, false);
                }
                if (g.flip) {
                    emit_at(4, row0 + sf, cr, m, true);
                    if (nq > 1) {
                        emit_at(5, row0 + sf + sq, cr + cc, qq, true);
                        emit_at(6, row0 + sf + 2 * sq, cc, m, false);
                        emit_at(7, row0 + sf + 3 * sq, 0, qq, false);
                    }
                }
            }
            if (b + 1 < b_n) make_table(tq + 1);                       // (every warp is past this base rotation's tiles)
            if (with_norm && circle) {
                __syncthreads();
#pragma unroll
                for (int v = 0; v < 8; ++v) {
                    for (int o = 16; o > 0; o >>= 1) vsum[v] += __shfl_down_sync(0xffffffffu, vsum[v], o);
                    if (lane == 0) sum_s[warp][v] = vsum[v];
                }
                __syncthreads();
                if (threadIdx.x < nv) {
                    const uint32_t f = threadIdx.x / nq, j = threadIdx.x - f * nq;
                    total_t tot = 0;
                    for (uint32_t wv = 0; wv < nwarps; ++wv) tot += (total_t)sum_s[wv][4 * f + j];
                    norm_s[b][threadIdx.x] += tot;
                }
            }
            if (use_plane && threadIdx.x == 0) bulk_wait_read_all();      // the plane may be overwritten
            if (KIND == kPlanes && !padded && threadIdx.x >= 32 && threadIdx.x < 32 + nv) {      // and so may the set of rows filled next
                if (rp.row_bufs == 2) bulk_wait_read_one(); else bulk_wait_read_all();
            }
            __syncthreads();
        }
    }
    if (with_norm) {
        for (uint32_t i = threadIdx.x; i < b_n * nv; i += blockDim.x) {
            const uint32_t b = i / nv, v = i - b * nv, f = v / nq, j = v - f * nq;
            const size_t orow = (size_t)img_i * g.T + f * g.R + j * g.q + b_lo + b;
            if (MODE == kModeF32) static_cast<float*>(bnorm)[orow] = (float)norm_s[b][v];
            else if (MODE == kModeU8) static_cast<uint32_t*>(bnorm)[orow] = (uint32_t)norm_s[b][v];
            else static_cast<unsigned long long*>(bnorm)[orow] = (unsigned long long)norm_s[b][v];
        }
    }
    if (rmax) {
        vmax = __reduce_max_sync(0xffffffffu, vmax);
        // a rounded bilinear mean of pixels exceeds the largest of them by a few units in the last place at most
        if (staged) vmax = vmax < 0x7F000000u ? __float_as_uint(__fmul_ru(__uint_as_float(vmax), 1.00000095f)) : max(vmax, 0x7F800000u);
        if (lane == 0) atomicMax(rmax + img_i, vmax);
    }
    if (rp.use_plane && threadIdx.x == 0) bulk_wait_all();
    if (KIND == kPlanes && !padded && threadIdx.x >= 32 && threadIdx.x < 32 + nv) bulk_wait_all();
}

template <int MODE, bool INSIDE, int KIND, int FLAGS>
cudaError_t rotate_launch(const Geometry& g, RotPlan& rp, uint32_t n_img, size_t smem, const float* images, const float* cs, const float* sn,
                          float* base_out, void* b0, void* b1, void* b2, void* bnorm, uint32_t* rmax, cudaStream_t st)
{
    auto kernel = rotate_kernel<MODE, INSIDE, KIND, FLAGS>;
    // Dynamic shared memory above 48 KB is an opt-in, per-device function attribute.
    static thread_local int attr_dev = -1, sms = 0;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev != attr_dev) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRotSmemBudget);
        if (e != cudaSuccess) return e;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        attr_dev = dev;
    }
    // Two blocks of 512 threads share an SM where their shared memory allows it (one block's barriers then hide behind
    // the other's work); otherwise one block of 1024.
    const uint32_t per_sm = smem <= kRotHalfSm ? 2 : 1, threads = per_sm == 2 ? 512 : 1024;
    // Groups: the split of an image's base rotations over blocks that finishes first -- waves of resident blocks times
    // the base rotations of a block plus its fixed cost (staging the image, about one base rotation's time).
    const uint32_t nbase = g.q ? g.q : 1;
    const uint64_t resident = (uint64_t)per_sm * (sms > 0 ? sms : 148);
    uint64_t best = ~0ull;
    for (uint32_t per = 1; per <= std::min(nbase, kRotMaxGroup); ++per) {
        const uint32_t groups = (nbase + per - 1) / per;
        const uint64_t cost = ((uint64_t)groups * n_img + resident - 1) / resident * (per + 1);
        if (cost < best) { best = cost; rp.group = per; rp.groups = groups; }
    }
    kernel<<<dim3(rp.groups, n_img), threads, smem, st>>>(g, rp, images, cs, sn, base_out, b0, b1, b2, bnorm, rmax);
    return cudaGetLastError();
}

} // namespace

template <int MODE, int KIND>
cudaError_t rotate_run(const Geometry& g, RotPlan& rp, bool inside, uint32_t n_img, size_t smem, const float* images, const float* cs, const float* sn,
                       float* base_out, void* b0, void* b1, void* b2, void* bnorm, uint32_t* rmax, cudaStream_t st)
{
#define PINK_ROTATE(I, FLAGS) rotate_launch<MODE, I, KIND, FLAGS>(g, rp, n_img, smem, images, cs, sn, base_out, b0, b1, b2, bnorm, rmax, st)
    if constexpr (KIND == kFast || KIND == kPlanes) {
        // the common case -- a neuron that fits the image -- has its flags compiled in
        if (!inside) return PINK_ROTATE(false, -1);
        if (base_out) return rp.win == g.ed ? PINK_ROTATE(true, 3) : PINK_ROTATE(true, 1);
        return rp.win == g.ed ? PINK_ROTATE(true, 2) : PINK_ROTATE(true, 0);
    } else {
        return inside ? PINK_ROTATE(true, -1) : PINK_ROTATE(false, -1);
    }
#undef PINK_ROTATE
}

template cudaError_t rotate_run<PINK_ROTATE_MODE, PINK_ROTATE_KIND>(const Geometry&, RotPlan&, bool, uint32_t, size_t, const float*, const float*,
    const float*, float*, void*, void*, void*, void*, uint32_t*, cudaStream_t);

#else

namespace {

inline uint32_t div_magic(uint32_t d) { return d == 1 ? 0u : (uint32_t)((1ull << 32) / d) + 1; }


// Row pitch (floats) of the staged image, at least `width`: the banks of an 8 x 4 tile of taps at any angle are the
// points of the lattice {(dx, dy): dx * pitch + dy = 0 mod 32} away from one another; these residues keep the
// lattice's shortest vector at 5.4 to 5.7 pixels (the densest possible packing has 6.1), so that a tile meets at most
// two points of it and a read takes one to two passes.
uint32_t bank_pitch(uint32_t width)
{
    for (uint32_t p = width;; ++p) {
        const uint32_t r = p & 31u;
        if (r == 6 || r == 7 || r == 9 || r == 23 || r == 25 || r == 26) return p;
    }
}

// Shared memory of the row and column terms of a window, and of the converted region (its rows one odd pitch apart).
size_t table_bytes(uint32_t nx) { return (8 * (size_t)nx + 127) & ~size_t(127); }
size_t staged_region_bytes(const Geometry& g)
{
    const uint32_t win = g.nd - 2 * g.off;
    return ((size_t)win * (win | 1u) * (g.mode == kModeF32 ? 4 : g.mode == kModeU16 ? 2 : 1) + 127) & ~size_t(127);
}

template <int MODE>
cudaError_t rotate_dispatch(const Geometry& g, const float* images, uint32_t n_img, const float* cs, const float* sn, float* base_out,
                            uint32_t base_plane, void* b0, void* b1, void* b2, void* bnorm, uint32_t* rmax, cudaStream_t st)
{
    if ((uint64_t)g.nd * g.nd * g.nd >= (1ull << 32) || (uint64_t)g.ed * g.ed * g.ed >= (1ull << 32) || n_img > 65535u) return cudaErrorInvalidValue;
    const uint32_t P1 = g.nd * g.nd;
    RotPlan rp{};
    rp.base_plane = base_plane;
    rp.win = g.nd - 2 * g.off;                       // ed or ed + 1
    rp.sp = rp.win | 1u;                             // odd pitch: reads along rows and along columns are free of bank conflicts
    rp.x0 = base_out ? 0 : g.off;
    rp.nx = base_out ? g.nd : rp.win;
    rp.nband = (rp.nx + 3) / 4;
    rp.ntile = rp.nband * ((rp.nx + 15) / 16);
    if ((uint64_t)rp.ntile * rp.nband >= (1ull << 32)) return cudaErrorInvalidValue;
    rp.magic_nband = div_magic(rp.nband);
    rp.magic_ed = div_magic(g.ed);
    // the part of the image the window reaches at any angle
    const double sc = (g.id - 1) * 0.5, dc = (g.nd - 1) * 0.5;
    const double half = std::max(dc - rp.x0, rp.x0 + rp.nx - 1 - dc), reach = half * 1.4142136;
    const bool inside = reach + 0.01 <= sc;
    const double lo = std::floor(sc - reach) - 1, hi = std::ceil(sc + reach) + 2;
    rp.r0 = lo > 0 ? (uint32_t)lo : 0u;
    rp.side = std::min<uint32_t>(g.id, hi < g.id ? (uint32_t)hi + 1 : g.id) - rp.r0;
    rp.pitch = bank_pitch(rp.side + 1);
    const size_t region = staged_region_bytes(g);
    const size_t image = ((size_t)(rp.side + 1) * rp.pitch * 4 + 127) & ~size_t(127);
    const size_t plane = ((size_t)P1 * 4 + 127) & ~size_t(127);
    size_t smem = table_bytes(rp.nx);
    if (smem > 64 * 1024) return cudaErrorInvalidValue;
    const size_t table = smem;
    // uint8, one channel: scatter into whole operand rows, in two sets (one filled while the other is copied out) as long
    // as the block stays within half an SM's shared memory
    // rows of a multiple of 32 bytes would put the quarter turns' stores into few banks: they are padded by 16 bytes and copied out by the threads
    rp.row_pitch = g.ed % 32 == 0 ? g.ed + 16 : g.ed;
    rp.row_size = g.ed % 32 == 0 ? g.ed * rp.row_pitch : g.Kp;
    const size_t rows = (size_t)8 * rp.row_size;
    bool planes = MODE == kModeU8 && g.C == 1 && !g.circle && table + image + rows <= kRotSmemBudget;
    rp.row_bufs = planes && table + image + 2 * rows <= kRotHalfSm ? 2 : 1;
    rp.use_region = table + region <= kRotSmemBudget;
    if (!rp.use_region && !base_out) return cudaErrorInvalidValue;      // (rotate_needs_base)
    if (planes) smem += rp.row_bufs * rows;
    else if (rp.use_region) smem += region;
    const bool staged = smem + image <= kRotSmemBudget;
    rp.use_image = staged;
    if (staged) smem += image;
    rp.off_image = (uint32_t)table;
    rp.off_region = (uint32_t)(table + (staged ? image : 0));
    rp.off_plane = (uint32_t)smem;
    // the float plane goes to global memory by one bulk copy where whole 16-byte groups may be written
    rp.use_plane = base_out && base_plane % 4 == 0 && (reinterpret_cast<uintptr_t>(base_out) & 15u) == 0 && (planes || rp.use_region)
                   && smem + plane <= kRotSmemBudget;
    // -- unless it is what keeps a second block off the SM: then the threads store the pixels themselves
    if (smem <= kRotHalfSm && smem + plane > kRotHalfSm) rp.use_plane = 0;
    if (rp.use_plane) smem += plane;
#define PINK_ROTATE(KIND) rotate_run<MODE, KIND>(g, rp, inside, n_img, smem, images, cs, sn, base_out, b0, b1, b2, bnorm, rmax, st)
    if (planes) {
        if constexpr (MODE == kModeU8) return PINK_ROTATE(kPlanes);
    }
    if (!staged || !rp.use_region) return PINK_ROTATE(kLarge);
    return g.circle ? PINK_ROTATE(kCircle) : PINK_ROTATE(kFast);
#undef PINK_ROTATE
}

} // namespace

cudaError_t launch_rotate(const Geometry& g, const float* images, uint32_t n_img, const float* cs, const float* sn, float* base_out,
                          uint32_t base_plane, void* b0, void* b1, void* bnorm, cudaStream_t st, uint32_t* rmax, void* b2)
{
    if (n_img == 0) return cudaSuccess;
    if (g.mode == kModeU8) return rotate_dispatch<kModeU8>(g, images, n_img, cs, sn, base_out, base_plane, b0, b1, nullptr, bnorm, rmax, st);
    if (g.mode == kModeU16) return rotate_dispatch<kModeU16>(g, images, n_img, cs, sn, base_out, base_plane, b0, b1, nullptr, bnorm, rmax, st);
    // float: the planes are written only when both are given (b1 alone has no meaning in this mode)
    return rotate_dispatch<kModeF32>(g, images, n_img, cs, sn, base_out, base_plane, b0, b2 ? b1 : nullptr, b2, bnorm, rmax, st);
}

bool rotate_needs_base(const Geometry& g) { return table_bytes(g.nd - 2 * g.off) + staged_region_bytes(g) > kRotSmemBudget; }

cudaError_t clear_operand_padding(const Geometry& g, size_t rows, void* b0, void* b1, cudaStream_t st)
{
    const size_t esz = g.mode == kModeF32 ? 4 : 1, used = g.K * esz, pitch = g.Kp * esz;
    if (rows == 0 || used == pitch) return cudaSuccess;
    cudaError_t e = cudaMemset2DAsync(static_cast<uint8_t*>(b0) + used, pitch, 0, pitch - used, rows, st);
    if (e == cudaSuccess && g.mode == kModeU16) e = cudaMemset2DAsync(static_cast<uint8_t*>(b1) + used, pitch, 0, pitch - used, rows, st);
    return e;
}

#endif // PINK_ROTATE_MODE

} // namespace pinkb
