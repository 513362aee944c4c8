// Rotational flow and Lax-Wendroff image propagation: the reference's
// RotationalFlowImagePredictor (src/gpu/rotation.cu:55-96; flow kernel
// src/gpu/device/rotation_k.cu:17-43; camera src/gpu/camera.cu:15-31) and
// LaxWendroffPropagator (src/gpu/propagation.cu:506-716; kernels
// include/flowfilter/gpu/device/propagation_k.h:49-132).
//
// The reference runs 2N launches (a Y pass then an X pass per iteration, each a full-image
// round trip through HBM or L2).  Here one CTA computes a band of rows of a 64-column window: it
// loads the image over them plus a halo of P pixels (P = iterations in this launch) into shared
// memory with the flow, then runs all P iterations there, each over a region one pixel smaller
// (clamped at the image edges as the reference's texture reads are), and writes only its own
// pixels.  More than kMaxFused iterations take several launches through a
// caller workspace.  The rotational flow is computed in the same kernel from the camera and
// the angular velocity (and written once), so the predictor is one launch.
//
// Arithmetic follows the reference operation for operation, with the contraction nvcc
// applies to it made explicit (pinned against the reference on a B200):
//   flow: c = w x p with p.z = 1 folded, c.x = fma(-wz, py, wy), c.y = fma(wz, px, -wx),
//         c.z = fma(wx, py, -(wy px)); flow = (fma(ax, c.x, (cx - x) c.z), fma(ay, c.y, (cy - y) c.z)).
//   depth 1: the update is evaluated in double (the source's 0.5, and the Y pass's 2.0, are
//         double literals) and rounded once: fma(R^2/2, d2, I - R/2 d0).
//   depth 4: float through the float4 operators: t1 = fma(-d0, R/2, I), I' = fma(d2, R^2/2, t1).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <string>

#include "ffb200.h"
#include "launch.cuh"

ff_status ffb_fail(ff_status s, const std::string& msg);  // capi.cu: last error + log

namespace ffb {
namespace {

constexpr int kMaxFused = 16;  // iterations per launch (halo = iterations)

struct LWArgs {
    const float* flow;  // input flow (ROT = false)
    size_t flow_pitch;
    float* flow_out;  // rotational flow written for the tile (ROT = true)
    size_t flow_out_pitch;
    float ax, ay, cx, cy, wx, wy, wz;
    const float* src;
    size_t src_pitch;
    float* dst;
    size_t dst_pitch;
    int H, W, passes;
    float dt;
};

// px, py: the pixel on the unit image plane
__device__ __forceinline__ float2 rotational_flow(const LWArgs& a, int x, int y, float px, float py) {
    const float c_x = __fmaf_rn(-a.wz, py, a.wy);
    const float c_y = __fmaf_rn(a.wz, px, -a.wx);
    const float c_z = __fmaf_rn(a.wx, py, -__fmul_rn(a.wy, px));
    return make_float2(__fmaf_rn(a.ax, c_x, __fmul_rn(__fsub_rn(a.cx, (float)x), c_z)),
                       __fmaf_rn(a.ay, c_y, __fmul_rn(__fsub_rn(a.cy, (float)y), c_z)));
}

// one Lax-Wendroff update along AXIS (0 = X, 1 = Y) of a depth-1 value
template <int AXIS>
__device__ __forceinline__ float lw1(float m, float i0, float p, float R) {
    const float d0 = __fsub_rn(p, m);
    float d2;
    if (AXIS == 0)
        d2 = __fadd_rn(__fsub_rn(m, __fmul_rn(2.0f, i0)), p);
    else
        d2 = __double2float_rn(__dadd_rn(__dsub_rn((double)m, __dmul_rn(2.0, (double)i0)), (double)p));
    const double h = __dmul_rn(0.5, (double)R);
    const double t1 = __dsub_rn((double)i0, __dmul_rn(h, (double)d0));
    return __double2float_rn(__fma_rn(__dmul_rn(h, (double)R), (double)d2, t1));
}

// the same for one channel of a depth-4 value (float4 operator arithmetic)
__device__ __forceinline__ float lw4(float m, float i0, float p, float b, float b2) {
    const float d0 = __fsub_rn(p, m);
    const float d2 = __fadd_rn(__fsub_rn(m, __fmul_rn(2.0f, i0)), p);
    return __fmaf_rn(d2, b2, __fmaf_rn(-d0, b, i0));
}

// two adjacent pixels of D channels
template <int D>
struct Pix2 {
    float a[D], b[D];
};

// rows of 64 columns in shared memory, two pixels per lane: the image, then dt times the flow
constexpr int kCols = 64, kWarps = 8;
__host__ __device__ constexpr int row_bytes(int D) { return kCols * 4 * D + kCols * 8; }
// halo columns of a window (lanes hold even pairs) and the columns from a window to the next
__host__ __device__ constexpr int halo_of(int passes) { return (passes + 1) & ~1; }
__host__ __device__ constexpr int step_of(int passes) { return kCols - 2 * halo_of(passes); }

template <int D>
__device__ __forceinline__ Pix2<D> lds(const char* row, int lane) {
    Pix2<D> v;
    if constexpr (D == 1) {
        const float2 q = reinterpret_cast<const float2*>(row)[lane];
        v.a[0] = q.x, v.b[0] = q.y;
    } else {
        const float4 q = reinterpret_cast<const float4*>(row)[2 * lane], r = reinterpret_cast<const float4*>(row)[2 * lane + 1];
        v.a[0] = q.x, v.a[1] = q.y, v.a[2] = q.z, v.a[3] = q.w;
        v.b[0] = r.x, v.b[1] = r.y, v.b[2] = r.z, v.b[3] = r.w;
    }
    return v;
}
template <int D>
__device__ __forceinline__ void sts(char* row, int lane, const Pix2<D>& v) {
    if constexpr (D == 1) {
        reinterpret_cast<float2*>(row)[lane] = make_float2(v.a[0], v.b[0]);
    } else {
        reinterpret_cast<float4*>(row)[2 * lane] = make_float4(v.a[0], v.a[1], v.a[2], v.a[3]);
        reinterpret_cast<float4*>(row)[2 * lane + 1] = make_float4(v.b[0], v.b[1], v.b[2], v.b[3]);
    }
}
// one update of a pixel from its neighbours along AXIS
template <int D, int AXIS>
__device__ __forceinline__ void update(const float (&m)[D], const float (&i0)[D], const float (&p)[D], float R,
                                       float (&o)[D]) {
    if constexpr (D == 1) {
        o[0] = lw1<AXIS>(m[0], i0[0], p[0], R);
    } else {
        // R / 2 and R^2 / 2 as the reference rounds them from double: the halving is exact, so
        // the float products round the same values (where R / 2 underflows, R^2 / 2 is zero)
        const float b = __fmul_rn(0.5f, R), b2 = __fmul_rn(b, R);
#pragma unroll
        for (int ch = 0; ch < D; ++ch) o[ch] = lw4(m[ch], i0[ch], p[ch], b, b2);
    }
}

// One CTA: a window of 64 columns (two per lane) and `rows` output rows.  The image and dt times
// the flow over the rows and P more on each side go to shared memory once; a pass then gives
// every warp a run of rows, of which it makes the Y update from a three-row register window and,
// from the lanes beside it, the X update, and stores the row in place: one pass over shared
// memory and two barriers per iteration.  The outer P columns of a window belong to its
// neighbours.  Bound by the latency of the depth-1 update's conversions and FP64 chain.
// Measured (us, launches back to back, with the rotational flow), against 32x32 tiles whose X and
// Y updates were passes of their own over 32-lane steps of a 40-column region: 640x480 depth 1,
// 4 iterations 8.2 against 19.8; depth 4 9.8 against 24.9; 1920x1080 depth 1 36.5 against 75.5;
// 2048x2048 depth 4, 16 iterations 616 against 1668.
template <int D, bool ROT>
__global__ void __launch_bounds__(32 * kWarps) lw_rows_k(LWArgs a, int nwx, int rows) {
    grid_dep_wait();
    extern __shared__ __align__(16) char smem[];
    constexpr int ROWB = row_bytes(D), IMG = kCols * 4 * D;
    const int P = a.passes, H = a.H, W = a.W;
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int wx = blockIdx.x % nwx, ys = blockIdx.x / nwx * rows, ye = min(ys + rows, H);
    const int x0 = wx * step_of(P), c0 = x0 + 2 * lane;
    const int xo = wx == 0 ? 0 : x0 + halo_of(P), xe = wx == nwx - 1 ? W : x0 + kCols - halo_of(P);
    const int nout = c0 >= xo && c0 < xe ? min(2, W - c0) : 0;  // pixels this lane stores
    const int ca = min(c0, W - 1), cb = min(c0 + 1, W - 1);
    const bool e_l = c0 == 0, e_ra = c0 == W - 1, e_rb = c0 + 1 == W - 1;
    const int sy0 = max(ys - P, 0), sy1 = min(ye + P, H);
    // image and dt * flow of the rows
    float pxa = 0.f, pxb = 0.f;
    if (ROT) {
        pxa = __fdiv_rn(__fsub_rn((float)ca, a.cx), a.ax);
        pxb = __fdiv_rn(__fsub_rn((float)cb, a.cx), a.ax);
    }
    // a row ahead of its use (plain loads: the kernel before may have written image and flow)
    Pix2<D> v;
    float2 fa = make_float2(0.f, 0.f), fb = fa;
    auto fetch = [&](int y) {
        y = min(y, sy1 - 1);
        const float* srow = reinterpret_cast<const float*>(reinterpret_cast<const char*>(a.src) + y * a.src_pitch);
        if constexpr (D == 4) {
            const float4 q = reinterpret_cast<const float4*>(srow)[ca], r = reinterpret_cast<const float4*>(srow)[cb];
            v.a[0] = q.x, v.a[1] = q.y, v.a[2] = q.z, v.a[3] = q.w;
            v.b[0] = r.x, v.b[1] = r.y, v.b[2] = r.z, v.b[3] = r.w;
        } else {
            v.a[0] = srow[ca];
            v.b[0] = srow[cb];
        }
        if (!ROT) {
            const float2* frow = reinterpret_cast<const float2*>(reinterpret_cast<const char*>(a.flow) + y * a.flow_pitch);
            fa = frow[ca];
            fb = frow[cb];
        }
    };
    fetch(sy0 + warp);
    for (int y = sy0 + warp; y < sy1; y += kWarps) {
        char* row = smem + (y - sy0) * ROWB;
        const Pix2<D> w = v;
        float2 wa = fa, wb = fb;
        fetch(y + kWarps);
        if (ROT) {
            const float py = __fdiv_rn(__fsub_rn((float)y, a.cy), a.ay);
            wa = rotational_flow(a, ca, y, pxa, py);
            wb = rotational_flow(a, cb, y, pxb, py);
            if (y >= ys && y < ye) {
                float2* frow = reinterpret_cast<float2*>(reinterpret_cast<char*>(a.flow_out) + y * a.flow_out_pitch);
                if (nout > 0) frow[c0] = wa;
                if (nout > 1) frow[c0 + 1] = wb;
            }
        }
        sts<D>(row, lane, w);
        reinterpret_cast<float4*>(row + IMG)[lane] = make_float4(__fmul_rn(a.dt, wa.x), __fmul_rn(a.dt, wa.y),
                                                                 __fmul_rn(a.dt, wb.x), __fmul_rn(a.dt, wb.y));
    }
    grid_dep_launch();
    __syncthreads();
    for (int it = 1; it <= P; ++it) {
        // rows the later iterations need, a run of them per warp
        const int r = P - it, ya = max(ys - r, 0), n = min(ye + r, H) - ya;
        const int y0 = ya + n * warp / kWarps, y1 = ya + n * (warp + 1) / kWarps;
        // the rows around the run belong to other warps, which overwrite them: read first (at an
        // image edge the row itself is its neighbour)
        Pix2<D> prev, last;
        if (y0 < y1) {
            prev = lds<D>(smem + (max(y0 - 1, 0) - sy0) * ROWB, lane);
            last = lds<D>(smem + (min(y1, H - 1) - sy0) * ROWB, lane);
        }
        __syncthreads();
        if (y0 < y1) {
            Pix2<D> cur = lds<D>(smem + (y0 - sy0) * ROWB, lane);
#pragma unroll 2
            for (int y = y0; y < y1; ++y) {
                char* row = smem + (y - sy0) * ROWB;
                const Pix2<D> next = y + 1 < y1 ? lds<D>(row + ROWB, lane) : last;
                const float4 R = reinterpret_cast<const float4*>(row + IMG)[lane];  // (x, y) of both pixels
                Pix2<D> t, o;
                update<D, 1>(prev.a, cur.a, next.a, R.y, t.a);
                update<D, 1>(prev.b, cur.b, next.b, R.w, t.b);
                float ma[D], pa[D], pb[D];
#pragma unroll
                for (int ch = 0; ch < D; ++ch) {
                    const float l = __shfl_up_sync(0xffffffffu, t.b[ch], 1), rr = __shfl_down_sync(0xffffffffu, t.a[ch], 1);
                    ma[ch] = e_l ? t.a[ch] : l;
                    pa[ch] = e_ra ? t.a[ch] : t.b[ch];
                    pb[ch] = e_rb ? t.b[ch] : rr;
                }
                update<D, 0>(ma, t.a, pa, R.x, o.a);
                update<D, 0>(t.a, t.b, pb, R.z, o.b);
                if (it < P) {
                    sts<D>(row, lane, o);
                } else {
                    float* drow = reinterpret_cast<float*>(reinterpret_cast<char*>(a.dst) + y * a.dst_pitch);
                    if constexpr (D == 4) {
                        if (nout > 0) reinterpret_cast<float4*>(drow)[c0] = make_float4(o.a[0], o.a[1], o.a[2], o.a[3]);
                        if (nout > 1) reinterpret_cast<float4*>(drow)[c0 + 1] = make_float4(o.b[0], o.b[1], o.b[2], o.b[3]);
                    } else {
                        if (nout > 0) drow[c0] = o.a[0];
                        if (nout > 1) drow[c0 + 1] = o.b[0];
                    }
                }
                prev = cur;
                cur = next;
            }
        }
        __syncthreads();
    }
}

__global__ void rotational_flow_k(LWArgs a) {
    grid_dep_wait();
    grid_dep_launch();
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= a.W || y >= a.H) return;
    reinterpret_cast<float2*>(reinterpret_cast<char*>(a.flow_out) + y * a.flow_out_pitch)[x] =
        rotational_flow(a, x, y, __fdiv_rn(__fsub_rn((float)x, a.cx), a.ax), __fdiv_rn(__fsub_rn((float)y, a.cy), a.ay));
}

template <int D, bool ROT>
cudaError_t launch_lw(LWArgs a, cudaStream_t s) {
    const int step = step_of(a.passes);
    const int nwx = 1 + (std::max(a.W - kCols, 0) + step - 1) / step;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // Bands of as few rows as give two windows per SM (16 rows at the least, against halo rows;
    // at the most what two blocks' shared memory holds)
    const int most = 108 * 1024 / row_bytes(D) - 2 * a.passes;
    const int bands = std::max(1, 2 * std::max(sms, 1) / nwx);
    const int rows = std::min(std::min(std::max((a.H + bands - 1) / bands, 16), most), a.H);
    const size_t smem = (size_t)(rows + 2 * a.passes) * row_bytes(D);
    // once per device: room for the largest launch; no static smem
    static std::atomic<unsigned long long> prepared{0};
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(prepared.load() & bit)) {
        e = cudaFuncSetAttribute(lw_rows_k<D, ROT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 108 * 1024);
        if (e != cudaSuccess) return e;
        prepared.fetch_or(bit);
    }
    const long blocks = (long)nwx * ((a.H + rows - 1) / rows);
    return launch_k(lw_rows_k<D, ROT>, dim3((unsigned)blocks), dim3(32 * kWarps), smem, s, a, nwx, rows);
}

// Full propagation: ceil(n / kMaxFused) launches ending in `out`; earlier ones alternate
// with the workspace.  rot: the first launch computes (and writes) the rotational flow.
cudaError_t propagate(LWArgs a, int depth, int iterations, bool rot, float* out, size_t out_pitch, float* ws,
                      size_t ws_pitch, cudaStream_t s) {
    const int n = std::max(iterations, 1);
    a.dt = iterations > 0 ? 1.0f / (float)iterations : 0.0f;  // setIterations, propagation.cu:647-656
    const int launches = (n + kMaxFused - 1) / kMaxFused;
    int done = 0;
    for (int i = 0; i < launches; ++i) {
        const int p = std::min(kMaxFused, n - done);
        const bool to_out = ((launches - 1 - i) % 2) == 0;
        a.dst = to_out ? out : ws;
        a.dst_pitch = to_out ? out_pitch : ws_pitch;
        a.passes = p;
        const bool r = rot && i == 0;
        cudaError_t e;
        if (depth == 1)
            e = r ? launch_lw<1, true>(a, s) : launch_lw<1, false>(a, s);
        else
            e = r ? launch_lw<4, true>(a, s) : launch_lw<4, false>(a, s);
        if (e != cudaSuccess) return e;
        if (r) {  // later launches read the flow just written
            a.flow = a.flow_out;
            a.flow_pitch = a.flow_out_pitch;
        }
        a.src = a.dst;
        a.src_pitch = a.dst_pitch;
        done += p;
    }
    return cudaSuccess;
}

bool aligned(const void* p, size_t pitch, size_t row_bytes, size_t align) {
    return p && pitch >= row_bytes && (((uintptr_t)p | pitch) % align) == 0;
}

ff_status fail(ff_status st, const std::string& msg) { return ffb_fail(st, msg); }

ff_status check_common(int depth, int h, int w, int iterations, const float* image, size_t image_pitch, float* out,
                       size_t out_pitch, float* ws, size_t ws_pitch) {
    if (h < 1 || w < 1 || h > 65535 * 32) return fail(FF_ERR_SHAPE, "lax_wendroff: bad height or width");
    if (depth != 1 && depth != 4) return fail(FF_ERR_INVALID_ARGUMENT, "lax_wendroff: image depth should be 1 or 4");
    if (iterations < 0) return fail(FF_ERR_INVALID_ARGUMENT, "lax_wendroff: iterations less than zero");
    const size_t row = (size_t)w * depth * 4, al = depth == 4 ? 16 : 4;
    if (!aligned(image, image_pitch, row, al) || !aligned(out, out_pitch, row, al))
        return fail(FF_ERR_INVALID_ARGUMENT, "lax_wendroff: image and output need aligned rows of width pixels");
    if (image == out) return fail(FF_ERR_INVALID_ARGUMENT, "lax_wendroff: the output must not be the input image");
    if (std::max(iterations, 1) > kMaxFused && (!aligned(ws, ws_pitch, row, al) || ws == image || ws == out))
        return fail(FF_ERR_INVALID_ARGUMENT,
                    "lax_wendroff: more than " + std::to_string(kMaxFused) + " iterations need a workspace image");
    return FF_OK;
}

ff_status cuda_status(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return FF_OK;
    return fail(FF_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

}  // namespace
}  // namespace ffb

extern "C" {

int ff_lax_wendroff_max_fused(void) { return ffb::kMaxFused; }

ff_status ff_camera_perspective(float focal, int height, int width, float sensor_height, float sensor_width,
                                ff_camera* cam) {
    if (!cam) return ffb::fail(FF_ERR_INVALID_ARGUMENT, "camera_perspective: cam must not be NULL");
    const int imgX = width - 1, imgY = height - 1;
    cam->alphaX = focal * (float)imgX / sensor_width;
    cam->alphaY = focal * (float)imgY / sensor_height;
    cam->centerX = 0.5f * (float)imgX;
    cam->centerY = 0.5f * (float)imgY;
    return FF_OK;
}

ff_status ff_rotational_flow(const ff_camera* cam, float wx, float wy, float wz, float* flow, size_t flow_pitch,
                             int height, int width, void* stream) {
    if (!cam) return ffb::fail(FF_ERR_INVALID_ARGUMENT, "rotational_flow: cam must not be NULL");
    if (height < 1 || width < 1 || height > 65535 * 8) return ffb::fail(FF_ERR_SHAPE, "rotational_flow: bad size");
    if (!ffb::aligned(flow, flow_pitch, (size_t)width * 8, 8))
        return ffb::fail(FF_ERR_INVALID_ARGUMENT, "rotational_flow: flow needs 8-byte aligned rows of width float2");
    ffb::LWArgs a{};
    a.flow_out = flow;
    a.flow_out_pitch = flow_pitch;
    a.ax = cam->alphaX, a.ay = cam->alphaY, a.cx = cam->centerX, a.cy = cam->centerY;
    a.wx = wx, a.wy = wy, a.wz = wz;
    a.H = height, a.W = width;
    return ffb::cuda_status(ffb::launch_k(ffb::rotational_flow_k, dim3((width + 31) / 32, (height + 7) / 8),
                                          dim3(32, 8), 0, (cudaStream_t)stream, a),
                            "rotational_flow");
}

ff_status ff_lax_wendroff(const float* flow, size_t flow_pitch, const float* image, size_t image_pitch, int depth,
                          int height, int width, int iterations, float* out, size_t out_pitch, float* workspace,
                          size_t workspace_pitch, void* stream) {
    ff_status st = ffb::check_common(depth, height, width, iterations, image, image_pitch, out, out_pitch, workspace,
                                     workspace_pitch);
    if (st != FF_OK) return st;
    if (!ffb::aligned(flow, flow_pitch, (size_t)width * 8, 8))
        return ffb::fail(FF_ERR_INVALID_ARGUMENT, "lax_wendroff: flow needs 8-byte aligned rows of width float2");
    ffb::LWArgs a{};
    a.flow = flow;
    a.flow_pitch = flow_pitch;
    a.src = image;
    a.src_pitch = image_pitch;
    a.H = height, a.W = width;
    return ffb::cuda_status(ffb::propagate(a, depth, iterations, false, out, out_pitch, workspace, workspace_pitch,
                                           (cudaStream_t)stream),
                            "lax_wendroff");
}

ff_status ff_rotational_predict(const ff_camera* cam, float wx, float wy, float wz, const float* image,
                                size_t image_pitch, int depth, int height, int width, int iterations, float* flow,
                                size_t flow_pitch, float* out, size_t out_pitch, float* workspace,
                                size_t workspace_pitch, void* stream) {
    if (!cam) return ffb::fail(FF_ERR_INVALID_ARGUMENT, "rotational_predict: cam must not be NULL");
    ff_status st = ffb::check_common(depth, height, width, iterations, image, image_pitch, out, out_pitch, workspace,
                                     workspace_pitch);
    if (st != FF_OK) return st;
    if (!ffb::aligned(flow, flow_pitch, (size_t)width * 8, 8))
        return ffb::fail(FF_ERR_INVALID_ARGUMENT, "rotational_predict: flow needs 8-byte aligned rows of width float2");
    ffb::LWArgs a{};
    a.flow_out = flow;
    a.flow_out_pitch = flow_pitch;
    a.ax = cam->alphaX, a.ay = cam->alphaY, a.cx = cam->centerX, a.cy = cam->centerY;
    a.wx = wx, a.wy = wy, a.wz = wz;
    a.src = image;
    a.src_pitch = image_pitch;
    a.H = height, a.W = width;
    return ffb::cuda_status(ffb::propagate(a, depth, iterations, true, out, out_pitch, workspace, workspace_pitch,
                                           (cudaStream_t)stream),
                            "rotational_predict");
}

}  // extern "C"
