// Integral images on the GPU (kernel a) and the device-resident dataset.
//
// The reference integrates each channel sequentially in double with a Kahan carry and stores
// float (colour) / int (depth) (image.cpp:236-277, 531-556). For integer-valued input the
// double scan is exact, so an exact 32-bit integer scan followed by one round-to-nearest
// conversion (__uint2float_rn) gives bit-identical colour integrals. Depth sums are kept as
// wrapping 32-bit integers: box differences stay exact even where the reference's int
// integral overflows (1280x960 frames at up to 5 m).
//
// Two passes: a warp-per-row inclusive scan of the five channels, then running sums down the columns in
// segments. Traffic: 5 B/px read raw, 20 B/px written, then 20 B/px read and written again.
#include <algorithm>
#include <cstring>

#include "features.h"

namespace cf {

namespace {

constexpr int kRowWarps = 4;
constexpr int kColLanes = 32, kColSegments = 16, kColRun = 8;   // columns x row segments of a CTA, rows of a segment

// Row prefix sums, a warp per row, 128 pixels a step with the next step's reads under way. A lane takes four
// pixels; red and green, and blue and the valid count, share a word (sums of 128 pixels stay below 2^16), so a
// step scans three words. kQuad: rows start on whole quads and the pointers are aligned (whole-word reads,
// 16-byte writes); otherwise pixel by pixel.
template <bool kQuad>
__global__ void __launch_bounds__(kRowWarps * 32)
integral_rows_kernel(const uint8_t* __restrict__ rgb, const uint16_t* __restrict__ depth, int count, int W, int H,
                     uint32_t* __restrict__ color_out, int2* __restrict__ depth_out) {
    const int lane = threadIdx.x & 31;
    const long long row = static_cast<long long>(blockIdx.x) * kRowWarps + (threadIdx.x >> 5);
    if (row >= static_cast<long long>(count) * H) return;
    const long long img = row / H;
    const int y = static_cast<int>(row - img * H);
    const long long plane = static_cast<long long>(W) * H;
    const uint8_t* src_rgb = rgb + (img * plane + static_cast<long long>(y) * W) * 3;
    const uint16_t* src_d = depth + img * plane + static_cast<long long>(y) * W;
    uint32_t* dst_c = color_out + img * 3 * plane + static_cast<long long>(y) * W;
    int2* dst_d = depth_out + img * plane + static_cast<long long>(y) * W;
    struct Quad {
        uint32_t c[3];   // twelve colour bytes
        uint32_t d[2];   // four depths
    };
    auto read = [&](int x) {
        Quad q = {};
        if (kQuad) {
            if (x < W) {
                const uint32_t* c = reinterpret_cast<const uint32_t*>(src_rgb + 3 * x);
                q.c[0] = __ldg(c);
                q.c[1] = __ldg(c + 1);
                q.c[2] = __ldg(c + 2);
                const uint2 d = __ldg(reinterpret_cast<const uint2*>(src_d + x));
                q.d[0] = d.x;
                q.d[1] = d.y;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 12; k++)
                if (x + k / 3 < W) q.c[k >> 2] |= static_cast<uint32_t>(src_rgb[3 * x + k]) << (8 * (k & 3));
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (x + k < W) q.d[k >> 1] |= static_cast<uint32_t>(src_d[x + k]) << (16 * (k & 1));
        }
        return q;
    };
    uint32_t cr = 0, cg = 0, cb = 0, cd = 0, cn = 0;   // sums of the steps before
    Quad next = read(4 * lane);
    for (int x0 = 0; x0 < W; x0 += 128) {
        const Quad q = next;
        const int x = x0 + 4 * lane;
        if (x0 + 128 < W) next = read(x + 128);
        uint32_t rg[4], bn[4], d[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            auto byte = [&](int b) { return q.c[b >> 2] >> (8 * (b & 3)) & 255u; };
            d[k] = q.d[k >> 1] >> (16 * (k & 1)) & 0xFFFFu;
            rg[k] = byte(3 * k) | byte(3 * k + 1) << 16;
            bn[k] = byte(3 * k + 2) | (d[k] > 0 ? 1u << 16 : 0u);
            if (k > 0) {
                rg[k] += rg[k - 1];
                bn[k] += bn[k - 1];
                d[k] += d[k - 1];
            }
        }
        uint32_t srg = rg[3], sbn = bn[3], sd = d[3];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t a = __shfl_up_sync(0xffffffffu, srg, off), b = __shfl_up_sync(0xffffffffu, sbn, off);
            const uint32_t c = __shfl_up_sync(0xffffffffu, sd, off);
            if (lane >= off) {
                srg += a;
                sbn += b;
                sd += c;
            }
        }
        uint32_t r4[4], g4[4], b4[4];
        int2 d4[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t prg = srg - rg[3] + rg[k], pbn = sbn - bn[3] + bn[k];
            r4[k] = cr + (prg & 0xFFFFu);
            g4[k] = cg + (prg >> 16);
            b4[k] = cb + (pbn & 0xFFFFu);
            d4[k] = make_int2(static_cast<int>(cd + sd - d[3] + d[k]), static_cast<int>(cn + (pbn >> 16)));
        }
        if (kQuad) {
            if (x < W) {
                *reinterpret_cast<uint4*>(dst_c + x) = make_uint4(r4[0], r4[1], r4[2], r4[3]);
                *reinterpret_cast<uint4*>(dst_c + plane + x) = make_uint4(g4[0], g4[1], g4[2], g4[3]);
                *reinterpret_cast<uint4*>(dst_c + 2 * plane + x) = make_uint4(b4[0], b4[1], b4[2], b4[3]);
                int4* o = reinterpret_cast<int4*>(dst_d + x);
                o[0] = make_int4(d4[0].x, d4[0].y, d4[1].x, d4[1].y);
                o[1] = make_int4(d4[2].x, d4[2].y, d4[3].x, d4[3].y);
            }
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (x + k < W) {
                    dst_c[x + k] = r4[k];
                    dst_c[plane + x + k] = g4[k];
                    dst_c[2 * plane + x + k] = b4[k];
                    dst_d[x + k] = d4[k];
                }
        }
        srg = __shfl_sync(0xffffffffu, srg, 31);
        sbn = __shfl_sync(0xffffffffu, sbn, 31);
        cr += srg & 0xFFFFu;
        cg += srg >> 16;
        cb += sbn & 0xFFFFu;
        cn += sbn >> 16;
        cd += __shfl_sync(0xffffffffu, sd, 31);
    }
}

// Column sums of one plane (three colours, then depth) in place: a CTA takes 32 columns, a thread 8 rows of one
// of them at a time (all its reads under way together), the 16 segments of 128 rows are joined through shared
// memory. A thread per column keeps too few reads in flight on one frame (66 us a frame of 640x480; 64 frames
// 197 us).
template <bool kDepth>
__device__ __forceinline__ void sum_columns(void* column, bool ok, int W, int H) {
    __shared__ uint32_t s_a[kColSegments][kColLanes], s_b[kColSegments][kColLanes];
    uint32_t* c = static_cast<uint32_t*>(column);
    int2* d = static_cast<int2*>(column);
    const int seg = threadIdx.y;
    uint32_t carry_a = 0, carry_b = 0;
    for (int y0 = 0; y0 < H; y0 += kColSegments * kColRun) {
        const int ya = y0 + seg * kColRun;
        uint32_t va[kColRun], vb[kDepth ? kColRun : 1];
#pragma unroll
        for (int k = 0; k < kColRun; k++) {
            va[k] = 0;
            if constexpr (kDepth) vb[k] = 0;
            if (ok && ya + k < H) {
                const long long o = static_cast<long long>(ya + k) * W;
                if constexpr (kDepth) {
                    const int2 v = d[o];
                    va[k] = static_cast<uint32_t>(v.x);
                    vb[k] = static_cast<uint32_t>(v.y);
                } else {
                    va[k] = c[o];
                }
            }
        }
#pragma unroll
        for (int k = 1; k < kColRun; k++) {
            va[k] += va[k - 1];
            if constexpr (kDepth) vb[k] += vb[k - 1];
        }
        __syncthreads();   // the previous step's sums are read
        s_a[seg][threadIdx.x] = va[kColRun - 1];
        if constexpr (kDepth) s_b[seg][threadIdx.x] = vb[kColRun - 1];
        __syncthreads();
        uint32_t before_a = carry_a, before_b = carry_b;
#pragma unroll
        for (int g = 0; g < kColSegments; g++) {
            const uint32_t a = s_a[g][threadIdx.x];
            before_a += g < seg ? a : 0u;
            carry_a += a;
            if constexpr (kDepth) {
                const uint32_t b = s_b[g][threadIdx.x];
                before_b += g < seg ? b : 0u;
                carry_b += b;
            }
        }
#pragma unroll
        for (int k = 0; k < kColRun; k++)
            if (ok && ya + k < H) {
                const long long o = static_cast<long long>(ya + k) * W;
                if constexpr (kDepth) d[o] = make_int2(static_cast<int>(before_a + va[k]), static_cast<int>(before_b + vb[k]));
                else reinterpret_cast<float*>(c)[o] = __uint2float_rn(before_a + va[k]);
            }
    }
}

__global__ void __launch_bounds__(kColLanes * kColSegments, 2)
integral_cols_kernel(int W, int H, uint32_t* __restrict__ color, int2* __restrict__ depth) {
    const int strips = (W + kColLanes - 1) / kColLanes;
    long long b = blockIdx.x;
    const int x = static_cast<int>(b % strips) * kColLanes + threadIdx.x;
    b /= strips;
    const int p = static_cast<int>(b & 3);
    const long long img = b >> 2, plane = static_cast<long long>(W) * H;
    if (p < 3) sum_columns<false>(color + (img * 3 + p) * plane + x, x < W, W, H);
    else sum_columns<true>(depth + img * plane + x, x < W, W, H);
}

// RGBDImage::resizeImage (image.cpp:450-475) applied to integral images: the w x h integrals go to the
// top-left corner of the W x H frames, colour NaN and depth {0, 0} everywhere else.
__global__ void pad_integral_kernel(const float* __restrict__ color_in, const int2* __restrict__ depth_in, int count,
                                    int w, int h, int W, int H, float* __restrict__ color_out,
                                    int2* __restrict__ depth_out) {
    const long long plane = static_cast<long long>(W) * H, small = static_cast<long long>(w) * h;
    const long long total = plane * count;
    const float nan = __int_as_float(0x7fc00000);
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long img = i / plane;
        const long long p = i - img * plane;
        const int y = static_cast<int>(p / W), x = static_cast<int>(p - static_cast<long long>(y) * W);
        float* c = color_out + img * 3 * plane + p;
        if (x < w && y < h) {
            const long long q = img * small + static_cast<long long>(y) * w + x;
            const float* s = color_in + img * 3 * small + static_cast<long long>(y) * w + x;
            c[0] = s[0];
            c[plane] = s[small];
            c[2 * plane] = s[2 * small];
            depth_out[i] = depth_in[q];
        } else {
            c[0] = nan;
            c[plane] = nan;
            c[2 * plane] = nan;
            depth_out[i] = make_int2(0, 0);
        }
    }
}

}  // namespace

// Integrates `count` raw frames (device pointers) into the given integral buffers.
void integrate_frames(cf_context* ctx, const uint8_t* rgb_dev, uint16_t* depth_dev, int count, int W, int H,
                      float* color_out, int2* depth_out, cudaStream_t stream, int preprocess) {
    if (stream == nullptr) stream = ctx->stream;
    if (preprocess & kPreFillDepth) fill_depth_frames(ctx, depth_dev, count, W, H, stream);
    const long long rows = static_cast<long long>(count) * H;
    auto aligned = [](const void* p, size_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; };
    const bool quad = W % 4 == 0 && aligned(rgb_dev, 4) && aligned(depth_dev, 8) && aligned(color_out, 16) && aligned(depth_out, 16);
    launch_on(ctx, stream, "integral_rows", dim3(static_cast<unsigned>((rows + kRowWarps - 1) / kRowWarps)),
              dim3(kRowWarps * 32), 0, quad ? integral_rows_kernel<true> : integral_rows_kernel<false>, rgb_dev,
              static_cast<const uint16_t*>(depth_dev), count, W, H, reinterpret_cast<uint32_t*>(color_out), depth_out);
    const long long strips = (W + kColLanes - 1) / kColLanes;
    launch_on(ctx, stream, "integral_cols", dim3(static_cast<unsigned>(strips * 4 * count)),
              dim3(kColLanes, kColSegments), 0, integral_cols_kernel, W, H, reinterpret_cast<uint32_t*>(color_out),
              depth_out);
    if (preprocess & kPreCieLab) lab_color_integral(ctx, rgb_dev, count, W, H, color_out, stream);
}

DsView view_of(const cf_dataset* ds) {
    DsView v;
    v.color = ds->color.get();
    v.depth = ds->depth.get();
    v.n = ds->n;
    v.width = ds->width;
    v.height = ds->height;
    v.plane = static_cast<long long>(ds->width) * ds->height;
    return v;
}

}  // namespace cf

extern "C" {

cf_status cf_dataset_create(cf_context* ctx, int num_images, int width, int height, cf_dataset** out) {
    return cf::guard([&] {
        CF_REQUIRE(ctx && out, "cf_dataset_create: NULL argument");
        CF_REQUIRE(num_images > 0 && width > 0 && height > 0, "cf_dataset_create: empty dataset");
        CF_REQUIRE(width <= 65535 && height <= 65535, "cf_dataset_create: frames wider or higher than 65535 px");
        cf::make_current(ctx);
        auto* ds = new cf_dataset();
        ds->ctx = ctx;
        ds->n = num_images;
        ds->width = width;
        ds->height = height;
        const size_t plane = static_cast<size_t>(width) * height;
        try {
            ds->color.reserve(plane * 3 * num_images);
            ds->depth.reserve(plane * num_images);
        } catch (...) {
            delete ds;
            throw;
        }
        cf::context_retain(ctx);
        *out = ds;
    });
}

cf_status cf_dataset_destroy(cf_dataset* ds) {
    return cf::guard([&] {
        if (!ds) return;
        cf_context* ctx = ds->ctx;
        cudaSetDevice(ctx->device);
        cudaStreamSynchronize(ctx->stream);
        {
            // the dataset's training buffers stay with the context for the next dataset
            std::lock_guard<std::mutex> lock(ctx->mu);
            if (ds->trainer && ctx->spare_trainer == nullptr) {
                ctx->spare_trainer = ds->trainer;
                ctx->spare_trainer_free = ds->trainer_free;
                ds->trainer = nullptr;
            }
        }
        delete ds;
        cf::context_release(ctx);
    });
}

cf_status cf_dataset_info(cf_dataset* ds, int* num_images, int* width, int* height) {
    return cf::guard([&] {
        CF_REQUIRE(ds, "cf_dataset_info: ds is NULL");
        if (num_images) *num_images = ds->n;
        if (width) *width = ds->width;
        if (height) *height = ds->height;
    });
}

cf_status cf_dataset_upload_raw(cf_dataset* ds, int first, int count, const uint8_t* rgb, const uint16_t* depth_mm,
                                int device_pointers) {
    return cf_dataset_upload_raw_ex(ds, first, count, rgb, depth_mm, device_pointers, 0, 0);
}

cf_status cf_dataset_upload_raw_ex(cf_dataset* ds, int first, int count, const uint8_t* rgb, const uint16_t* depth_mm,
                                   int device_pointers, int fill_depth, int cie_lab) {
    return cf::guard([&] {
        CF_REQUIRE(ds && rgb && depth_mm, "cf_dataset_upload_raw: NULL argument");
        CF_REQUIRE(first >= 0 && count >= 0 && first + count <= ds->n, "cf_dataset_upload_raw: image range");
        if (count == 0) return;
        cf_context* ctx = ds->ctx;
        cf::make_current(ctx);
        const size_t plane = static_cast<size_t>(ds->width) * ds->height;
        const int pre = (fill_depth ? cf::kPreFillDepth : 0) | (cie_lab ? cf::kPreCieLab : 0);
        if (!device_pointers || fill_depth) {
            // bounded staging (the depth frames are filled in place there); chunks keep the extra
            // memory small for large datasets
            const cudaMemcpyKind kind = device_pointers ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
            const int chunk = static_cast<int>(std::max<size_t>(1, std::min<size_t>(count, (256u << 20) / (plane * 5))));
            ds->raw_rgb.reserve(plane * 3 * chunk);
            ds->raw_depth.reserve(plane * chunk);
            for (int i = 0; i < count; i += chunk) {
                const int c = std::min(chunk, count - i);
                CF_CUDA_CHECK(cudaMemcpyAsync(ds->raw_rgb.get(), rgb + plane * 3 * i, plane * 3 * c, kind, ctx->stream));
                CF_CUDA_CHECK(cudaMemcpyAsync(ds->raw_depth.get(), depth_mm + plane * i, plane * 2 * c, kind, ctx->stream));
                cf::integrate_frames(ctx, ds->raw_rgb.get(), ds->raw_depth.get(), c, ds->width, ds->height,
                                     ds->color.get() + plane * 3 * (first + i), ds->depth.get() + plane * (first + i),
                                     ctx->stream, pre);
            }
            CF_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
        } else {
            // without depth filling the frames are only read
            cf::integrate_frames(ctx, rgb, const_cast<uint16_t*>(depth_mm), count, ds->width, ds->height,
                                 ds->color.get() + plane * 3 * first, ds->depth.get() + plane * first, ctx->stream,
                                 pre);
        }
    });
}

cf_status cf_dataset_upload_raw_padded(cf_dataset* ds, int first, int count, int width, int height, const uint8_t* rgb,
                                       const uint16_t* depth_mm, int device_pointers, int fill_depth, int cie_lab) {
    return cf::guard([&] {
        CF_REQUIRE(ds && rgb && depth_mm, "cf_dataset_upload_raw_padded: NULL argument");
        CF_REQUIRE(first >= 0 && count >= 0 && first + count <= ds->n, "cf_dataset_upload_raw_padded: image range");
        CF_REQUIRE(width >= 1 && height >= 1 && width <= ds->width && height <= ds->height,
                   "cf_dataset_upload_raw_padded: frames must be at most as large as the dataset's");
        if (count == 0) return;
        cf_context* ctx = ds->ctx;
        cf::make_current(ctx);
        const size_t small = static_cast<size_t>(width) * height;
        const size_t plane = static_cast<size_t>(ds->width) * ds->height;
        const int pre = (fill_depth ? cf::kPreFillDepth : 0) | (cie_lab ? cf::kPreCieLab : 0);
        const cudaMemcpyKind kind = device_pointers ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
        const int chunk = static_cast<int>(std::max<size_t>(1, std::min<size_t>(count, (256u << 20) / (small * 25))));
        cf::DevArray<uint8_t> raw_rgb;
        cf::DevArray<uint16_t> raw_depth;
        cf::DevArray<float> color;
        cf::DevArray<int2> depth;
        raw_rgb.reserve(small * 3 * chunk);
        raw_depth.reserve(small * chunk);
        color.reserve(small * 3 * chunk);
        depth.reserve(small * chunk);
        for (int i = 0; i < count; i += chunk) {
            const int c = std::min(chunk, count - i);
            CF_CUDA_CHECK(cudaMemcpyAsync(raw_rgb.get(), rgb + small * 3 * i, small * 3 * c, kind, ctx->stream));
            CF_CUDA_CHECK(cudaMemcpyAsync(raw_depth.get(), depth_mm + small * i, small * 2 * c, kind, ctx->stream));
            cf::integrate_frames(ctx, raw_rgb.get(), raw_depth.get(), c, width, height, color.get(), depth.get(),
                                 ctx->stream, pre);
            const long long total = static_cast<long long>(plane) * c;
            const int grid = static_cast<int>(std::min<long long>(ctx->num_sms * 8LL, (total + 255) / 256));
            cf::launch(ctx, "pad_integral", dim3(grid), dim3(256), 0, cf::pad_integral_kernel, color.get(), depth.get(),
                       c, width, height, ds->width, ds->height, ds->color.get() + plane * 3 * (first + i),
                       ds->depth.get() + plane * (first + i));
        }
        CF_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
    });
}

cf_status cf_dataset_upload_integral(cf_dataset* ds, int first, int count, const float* color, const int32_t* depth) {
    return cf::guard([&] {
        CF_REQUIRE(ds && color && depth, "cf_dataset_upload_integral: NULL argument");
        CF_REQUIRE(first >= 0 && count >= 0 && first + count <= ds->n, "cf_dataset_upload_integral: image range");
        cf_context* ctx = ds->ctx;
        cf::make_current(ctx);
        const size_t plane = static_cast<size_t>(ds->width) * ds->height;
        CF_CUDA_CHECK(cudaMemcpyAsync(ds->color.get() + plane * 3 * first, color, plane * 3 * count * sizeof(float),
                                      cudaMemcpyHostToDevice, ctx->stream));
        std::vector<int2> inter(plane);
        for (int i = 0; i < count; i++) {
            const int32_t* src = depth + plane * 2 * i;
            for (size_t p = 0; p < plane; p++) inter[p] = make_int2(src[p], src[plane + p]);
            CF_CUDA_CHECK(cudaMemcpyAsync(ds->depth.get() + plane * (first + i), inter.data(), plane * sizeof(int2),
                                          cudaMemcpyHostToDevice, ctx->stream));
            CF_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
        }
        CF_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
    });
}

cf_status cf_dataset_download_integral(cf_dataset* ds, int first, int count, float* color, int32_t* depth) {
    return cf::guard([&] {
        CF_REQUIRE(ds, "cf_dataset_download_integral: ds is NULL");
        CF_REQUIRE(first >= 0 && count >= 0 && first + count <= ds->n, "cf_dataset_download_integral: image range");
        cf_context* ctx = ds->ctx;
        cf::make_current(ctx);
        const size_t plane = static_cast<size_t>(ds->width) * ds->height;
        if (color)
            CF_CUDA_CHECK(cudaMemcpyAsync(color, ds->color.get() + plane * 3 * first, plane * 3 * count * sizeof(float),
                                          cudaMemcpyDeviceToHost, ctx->stream));
        if (depth) {
            std::vector<int2> inter(plane);
            for (int i = 0; i < count; i++) {
                CF_CUDA_CHECK(cudaMemcpyAsync(inter.data(), ds->depth.get() + plane * (first + i), plane * sizeof(int2),
                                              cudaMemcpyDeviceToHost, ctx->stream));
                CF_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
                int32_t* dst = depth + plane * 2 * i;
                for (size_t p = 0; p < plane; p++) {
                    dst[p] = inter[p].x;
                    dst[plane + p] = inter[p].y;
                }
            }
        }
        CF_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
    });
}

}  // extern "C"
