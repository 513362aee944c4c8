// Launch side of the slab level step (slab.cuh).
#include "slab.cuh"

#include <atomic>
#include <cmath>

namespace ffb {
namespace slab {

template <bool DELTA, typename P>
__global__ void __launch_bounds__(32 * kWarps, 1) slab_k(LevelArgs a, Geom g) {
    level_slab<DELTA, P>(a, g, blockIdx.x);
}

// level steps of many streams and levels in one launch; a block finds its job by binary search
__global__ void __launch_bounds__(32 * kWarps, 1) slab_jobs_k(const SlabJob* __restrict__ jobs, int n) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].first_block <= (int)blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const SlabJob& j = jobs[lo];
    const Geom g{j.N, j.S, j.nwx, j.rows, j.rows_e, j.nby_e, j.ne};
    const int i = (int)blockIdx.x - j.first_block;
    if (j.delta) level_slab<true, uint8_t>(j.a, g, i);
    else level_slab<false, uint8_t>(j.a, g, i);
}

// the same over a batch of float images (every field dense, image after image); TAPE: with the
// intermediates kept
template <bool DELTA, bool TAPE>
__global__ void __launch_bounds__(32 * kWarps, 1) slab_images_k(LevelArgs a, Geom g, int slabs, int images, Tape tape) {
    const size_t b = blockIdx.x / slabs, n = (size_t)a.H * a.W;
    auto at = [&](auto*& p, size_t elements) {
        if (p) p += b * elements;
    };
    at(a.fs_in, 2 * n);
    at(a.io_in, n);
    at(a.d_in, 2 * n);
    at(a.fs_out, 2 * n);
    at(a.io_out, n);
    at(a.d_out, 2 * n);
    at(a.fu_out, 2 * n);
    at(a.y_out, 2 * n);
    at(a.coarse, 2 * (size_t)a.Hc * a.Wc);
    a.img = reinterpret_cast<const float*>(a.img) + b * n;
    at(tape.f, 2 * n);
    at(tape.s, n);
    at(tape.v, 2 * n);
    at(tape.grad, 2 * n);
    at(tape.sm, 2 * n);
    level_slab<DELTA, float, TAPE>(a, g, blockIdx.x % slabs, tape);
}

// The propagation stage alone (FlowPropagator, FlowPropagatorPayload): all N sub-step pairs of a
// slab in one launch, where the per-pass kernels make 2N round trips through HBM or L2
template <bool DELTA>
__global__ void __launch_bounds__(32 * kWarps, 1) propagate_slab_k(LevelArgs a, Geom g) {
    grid_dep_wait();
    Ctx c;
    int sy1;
    make_ctx<DELTA>(a, g, blockIdx.x, c, sy1);
    load_state<DELTA>(a, c, sy1);
    propagate<DELTA, false, true>(c, g.N, g.N, Tape{});
    grid_dep_launch();
    if (c.nout <= 0) return;
    for (int y = c.ys + c.warp; y < c.ye; y += kWarps) {
        typename Prop<DELTA>::Row r;
        Prop<DELTA>::load(c.l16 + (unsigned)((y - c.sy0) * Prop<DELTA>::ROWB), r);
        store_f2(c.vec, c.nout, rowp(reinterpret_cast<float2*>(a.fs_out) + c.c0, (unsigned)a.fs_out_pitch, y), r.q[0], r.q[1]);
        if constexpr (DELTA) {
            store_f1(c.vec, c.nout, rowp(a.io_out + c.c0, (unsigned)a.io_out_pitch, y), r.q[2]);
            store_f2(c.vec, c.nout, rowp(reinterpret_cast<float2*>(a.d_out) + c.c0, (unsigned)a.d_out_pitch, y), r.q[3], r.q[4]);
        }
    }
}

// The smoothing stage alone (FlowSmoother)
__global__ void __launch_bounds__(32 * kWarps, 1) smooth_slab_k(LevelArgs a, Geom g) {
    grid_dep_wait();
    Ctx c;
    int sy1;
    make_ctx<false>(a, g, blockIdx.x, c, sy1);
    load_state<false>(a, c, sy1);
    grid_dep_launch();
    smooth<false, false>(c, a, g.S, Tape{});
}

// The image model stage alone (ImageModel): a warp takes a 128-column window of `rows` rows, the
// vertical windows in registers; only 4-column halos and 4 rows per run are computed twice.
template <typename P>
__global__ void __launch_bounds__(32 * kWarps) image_model_rows_k(const P* img, size_t pitch, int H, int W,
                                                                 float* __restrict__ a0, size_t a0_pitch,
                                                                 float2* __restrict__ grad, size_t grad_pitch, int nwx,
                                                                 int rows) {
    grid_dep_wait();
    grid_dep_launch();
    constexpr int HX = 4, STEP = kCols - 2 * HX;
    const int w = blockIdx.x * kWarps + (threadIdx.x >> 5);
    Ctx c;
    c.W = W;
    c.H = H;
    c.lane = threadIdx.x & 31;
    const int wx = w % nwx, x0 = wx * STEP;
    c.c0 = x0 + 4 * c.lane;
    c.ys = w / nwx * rows;
    c.ye = min(c.ys + rows, H);
    if (c.ys >= H) return;  // whole warps leave together
    c.e_l = c.c0 == 0;
    const bool edge = wx == 0 || wx == nwx - 1;
    const int xo = wx == 0 ? 0 : x0 + HX, xe = wx == nwx - 1 ? W : x0 + kCols - HX;
    const int nout = c.c0 >= xo && c.c0 < xe ? min(4, W - c.c0) : 0;
    const bool vec = nout == 4 && (((uintptr_t)a0 | a0_pitch) % 16) == 0 && (((uintptr_t)grad | grad_pitch) % 32) == 0;
    // four pixels at once where they are inside and aligned, else one by one at clamped columns
    const bool word = c.c0 + 3 < W && (((uintptr_t)img | pitch) % (4 * sizeof(P))) == 0;
    int o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] = min(c.c0 + j, W - 1);
    auto load = [&](int y) {
        const P* r = rowp(img, (unsigned)pitch, min(max(y, 0), H - 1));
        float v[4];
        if constexpr (sizeof(P) == 1) {
            uint32_t q;
            if (word) q = ld_waited(reinterpret_cast<const uint32_t*>(r + c.c0));
            else q = r[o[0]] | r[o[1]] << 8 | r[o[2]] << 16 | (uint32_t)r[o[3]] << 24;
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = u8_to_unit((q >> (8 * j)) & 0xffu);
        } else if (word) {
            const float4 q = ld_waited(reinterpret_cast<const float4*>(r + c.c0));
            v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = ld_waited(r + o[j]);
        }
        return Q{make_float2(v[0], v[1]), make_float2(v[2], v[3])};
    };
    auto around = [&](const Q& v) {
        Ext e = extend(v);
        if (edge) clamp_ext(c, e);  // warp-uniform
        return e;
    };
    Q im[4], bx[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) im[k] = load(c.ys - 2 + k);
    Q nxt = load(c.ys + 2);
#pragma unroll
    for (int k = 0; k < 4; ++k) bx[k] = smooth_x(around(im[k]));
#pragma unroll 2
    for (int y = c.ys; y < c.ye; ++y) {
        const Q i4 = nxt;
        nxt = load(y + 3);
        const Q b4 = smooth_x(around(i4));
        const Ext e = around(smooth_y(im[0], im[1], im[2], im[3], i4));
        const Q ay = diff_y(bx[0], bx[1], bx[2], bx[3], b4);
        if (nout > 0) {
            store_f1(vec, nout, rowp(a0 + c.c0, (unsigned)a0_pitch, y), smooth_x(e));
            store_f2(vec, nout, rowp(grad + c.c0, (unsigned)grad_pitch, y), diff_x(e), ay);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            im[k] = im[k + 1];
            bx[k] = bx[k + 1];
        }
        im[3] = i4;
        bx[3] = b4;
    }
}

constexpr int kSmem = 227 * 1024;  // shared memory a block may use on B200

int max_rows(bool delta, int N, int S) {
    return kSmem / (planes(delta) * kPlane) - 2 * (N + 2 * S) - kWarps;
}

int sm_count() {
    static std::atomic<int> cache[64] = {};  // several threads may ask first
    int dev = 0;
    cudaGetDevice(&dev);
    int n = cache[dev & 63].load(std::memory_order_relaxed);
    if (n == 0) {
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 148;
        cache[dev & 63].store(n, std::memory_order_relaxed);
    }
    return n;
}

// Slabs of `rows` output rows (edge windows: a row costs about 1.3 times an inner one's, so
// they get 3/4 of the rows and all slabs of a wave end together; measured with 0.5 to 1.0 of
// them, 640x480 N 4 S 2: 28.0 us at 0.5, 26.0 at 0.7, 28.1 at 1.0).
Geom geom_of(int N, int S, int W, int H, int rows) {
    Geom g;
    g.N = N;
    g.S = S;
    const int step = slab_cols(N, S);
    g.nwx = 1 + (std::max(W - kCols, 0) + step - 1) / step;
    g.ne = std::min(g.nwx, 2);
    g.rows = std::max(1, std::min(rows, H));
    g.rows_e = std::max(1, std::min((3 * g.rows + 2) / 4, H));
    g.nby_e = (H + g.rows_e - 1) / g.rows_e;
    return g;
}

// The fewest rows per slab that still take the number of waves (one slab per SM) the tallest
// slabs need: equal slabs over full waves.
Geom auto_geom(bool delta, int N, int S, int W, int H, int images) {
    const int sms = sm_count(), top = max_rows(delta, N, S);
    auto waves = [&](int rows) { return ((long)geom_of(N, S, W, H, rows).slabs(H) * images + sms - 1) / sms; };
    const long w = waves(top);
    int lo = 1, hi = std::min(top, H);  // waves(hi) == w
    while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if (waves(mid) <= w) hi = mid;
        else lo = mid + 1;
    }
    return geom_of(N, S, W, H, hi);
}

// rows of W pixels that may be accessed four pixels (4 * bytes) at a time, up to the next
// multiple of four columns
bool rows4(const void* p, size_t pitch, int W, int bytes) {
    return ((uintptr_t)p | pitch) % (4 * bytes) == 0 && pitch >= (size_t)((W + 3) & ~3) * bytes;
}

// checks and access widths of a launch
cudaError_t set_access(bool delta, LevelArgs& a) {
    // row offsets are computed as 32 x 32-bit products (rowp)
    for (size_t p : {a.img_pitch, a.fs_in_pitch, a.io_in_pitch, a.d_in_pitch, a.fs_out_pitch, a.io_out_pitch,
                     a.d_out_pitch, a.fu_out_pitch, a.coarse_pitch})
        if (p >> 32) return cudaErrorInvalidPitchValue;
    a.vec = rows4(a.fs_in, a.fs_in_pitch, a.W, 8) && rows4(a.fs_out, a.fs_out_pitch, a.W, 8) &&
            (!a.io_in || rows4(a.io_in, a.io_in_pitch, a.W, 4)) && (!a.io_out || rows4(a.io_out, a.io_out_pitch, a.W, 4)) &&
            (delta ? rows4(a.d_in, a.d_in_pitch, a.W, 8) && rows4(a.d_out, a.d_out_pitch, a.W, 8)
                   : !a.fu_out || rows4(a.fu_out, a.fu_out_pitch, a.W, 8)) &&
            (!a.y_out || rows4(a.y_out, a.fs_out_pitch, a.W, 8));
    a.img_vec = ((uintptr_t)a.img | a.img_pitch) % 16 == 0;
    return cudaSuccess;
}

// The same for fields of a caller: rows4 counts on the padding after a row's last pixel, which
// after the last row is not the caller's to read
cudaError_t set_access_of_caller(bool delta, LevelArgs& a) {
    const cudaError_t e = set_access(delta, a);
    a.vec = a.vec && a.W % 4 == 0;
    return e;
}

// once per kernel and device: the shared-memory limit, and the full shared carve-out as for the
// tile kernels (SMs running small slabs can then also host the other levels' kernels)
template <auto* K>
cudaError_t prepare() {
    static std::atomic<unsigned long long> prepared{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (prepared.load() & bit) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(K, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess) prepared.fetch_or(bit);
    return e;
}

size_t smem_of(bool delta, const Geom& g) { return (size_t)slab_smem(delta, g.N, g.S, std::max(g.rows, g.rows_e)); }

template <bool DELTA, typename P>
cudaError_t launch(LevelArgs a, int N, int S, cudaStream_t s) {
    cudaError_t e = set_access(DELTA, a);
    if (e == cudaSuccess) e = prepare<slab_k<DELTA, P>>();
    if (e != cudaSuccess) return e;
    const Geom g = a.band > 0 ? geom_of(N, S, a.W, a.H, std::min(a.band, max_rows(DELTA, N, S)))
                              : auto_geom(DELTA, N, S, a.W, a.H, 1);
    return launch_k(slab_k<DELTA, P>, dim3(g.slabs(a.H)), dim3(32 * kWarps), smem_of(DELTA, g), s, a, g);
}

template <bool DELTA>
cudaError_t launch_propagate_slab(LevelArgs a, int N, cudaStream_t s) {
    cudaError_t e = set_access_of_caller(DELTA, a);
    if (e == cudaSuccess) e = prepare<propagate_slab_k<DELTA>>();
    if (e != cudaSuccess) return e;
    const Geom g = auto_geom(DELTA, N, 0, a.W, a.H, 1);
    return launch_k(propagate_slab_k<DELTA>, dim3(g.slabs(a.H)), dim3(32 * kWarps), smem_of(DELTA, g), s, a, g);
}

// the H rows of a field of `row` bytes each, from the first byte of the first to the last of the
// last (rows may lie closer than their length, or all be one row: pitch 0)
struct Rows {
    const void* p;
    size_t pitch, row;
    uintptr_t begin() const { return (uintptr_t)p; }
    uintptr_t end(int H) const { return begin() + (size_t)(H - 1) * pitch + row; }
};
bool overlap(const Rows& a, const Rows& b, int H) { return a.begin() < b.end(H) && b.begin() < a.end(H); }

// the most sub-step pairs or smoothing iterations of one slab launch
constexpr int kMaxFused = 8;

// A single sub-step pair on rows that do not allow four pixels at a time: the slab saves one
// launch and loads and stores pixel by pixel.  Measured (us, slab / two passes) 321x241 payload
// 6.6 / 8.2, 641x481 9.3 / 8.2, flow 6.2 / 6.8, 1001x701 17.7 / 12.4 and 9.1 / 7.9, 2049x1089
// 46.8 / 36.1 and 22.6 / 20.5; two pairs 0.6 to 0.85 of the passes' time, one of smoothing 0.97
// to 1.08.  The passes from this many pixels on.
constexpr long kSinglePixels = 500000, kSinglePixelsPayload = 200000;
bool rows_of_caller4(bool delta, LevelArgs a) { return set_access_of_caller(delta, a) == cudaSuccess && a.vec; }

template <bool DELTA, bool TAPE>
cudaError_t launch_images(LevelArgs a, int N, int S, int images, const Tape& tape, cudaStream_t s) {
    cudaError_t e = set_access(DELTA, a);
    if (e == cudaSuccess) e = prepare<slab_images_k<DELTA, TAPE>>();
    if (e != cudaSuccess) return e;
    // (an image's fields start a multiple of four pixels after the one before where rows may be
    // accessed by four pixels, so the first image's alignment is every image's)
    if (TAPE) {
        auto at = [](const void* p, int bytes) { return (uintptr_t)p % bytes == 0; };
        a.vec = a.vec && at(tape.f, 32) && at(tape.grad, 32) && at(tape.sm, 32) &&
                (!DELTA || (at(tape.s, 16) && at(tape.v, 32))) && (tape.step | tape.sm_step) % 8 == 0;
    }
    const Geom g = auto_geom(DELTA, N, S, a.W, a.H, images);
    const int slabs = g.slabs(a.H);
    return launch_k(slab_images_k<DELTA, TAPE>, dim3((unsigned)slabs * images), dim3(32 * kWarps), smem_of(DELTA, g), s,
                    a, g, slabs, images, tape);
}

}  // namespace slab

int slab_max_rows(bool delta, int N, int S) { return slab::max_rows(delta, N, S); }

int slab_job(SlabJob& j, bool delta, int N, int S, const LevelArgs& a, int rows, size_t* smem) {
    j.a = a;
    j.delta = delta ? 1 : 0;
    if (slab::set_access(delta, j.a) != cudaSuccess) return 0;
    const slab::Geom g = slab::geom_of(N, S, a.W, a.H, std::min(rows, slab::max_rows(delta, N, S)));
    j.N = N;
    j.S = S;
    j.nwx = g.nwx;
    j.rows = g.rows;
    j.rows_e = g.rows_e;
    j.nby_e = g.nby_e;
    j.ne = g.ne;
    if (smem) *smem = slab::smem_of(delta, g);
    return g.slabs(a.H);
}

cudaError_t launch_slab_jobs(const SlabJob* jobs, int n, int blocks, size_t smem, cudaStream_t s) {
    const cudaError_t e = slab::prepare<slab::slab_jobs_k>();
    if (e != cudaSuccess) return e;
    return launch_k(slab::slab_jobs_k, dim3(blocks), dim3(32 * slab::kWarps), smem, s, jobs, n);
}

bool slab_available(bool delta, int N, int S) { return N >= 1 && S >= 1 && slab::max_rows(delta, N, S) >= 1; }

// A slab works on N + 2S more rows on each side than it has, and the most rows it can have fall
// with them: at N 10, S 15 two of 82.  Estimated times (us) of its stages over the rows of each,
// and of the 2 + 2N + 2S per-stage launches, which go through memory but work on no pixel twice;
// fitted on a B200 to 200 levels of 120x160 to 1088x2048, N 1..36, S 1..20 (beyond 20 halo rows
// the medians are 6% and 5% off, and the worst choice takes 1.15 times the other one).  Measured,
// us, slab / per-stage: delta levels of 720x1280 N 8 S 8 186 / 218, N 10 S 8 221 / 246, N 10 S 12
// 579 / 282, N 10 S 15 4354 / 310; top levels N 4 S 12 106 / 166, N 10 S 12 243 / 216, N 28 S 12
// 19906 / 368.  Halos of up to 20 rows always pay (0.86 of the per-stage time at the most).
bool slab_pays(bool delta, int N, int S, int W, int H, int images) {
    const int R = N + 2 * S;
    if (R <= 20) return true;
    const slab::Geom g = slab::auto_geom(delta, N, S, W, H, images);
    const double sms = slab::sm_count(), waves = std::ceil((double)g.slabs(H) * images / sms);
    auto rows = [&](int r) { return (double)std::min(g.rows + 2 * r, H); };
    // instructions of a 128-column row: a sub-step pair, model and update, a smoothing iteration
    double work = 330.0 * rows(2 * S);
    for (int k = 1; k <= N; ++k) work += (delta ? 185.0 : 80.0) * rows(R - k);
    for (int s = 1; s <= S; ++s) work += 110.0 * rows(2 * (S - s) + 1);
    const double slab_us = 14.5 + waves * (3.23e-4 * work + 0.88 * N + 0.24 * S - 5.6);
    const double mpx = 1e-6 * W * H * images, pass = 1.0 + 3.5 * mpx;
    const double stage_us = 7.7 + (delta ? 33.4 : 27.0) * mpx + 2 * N * (delta ? 1.76 + 6.13 * mpx : pass) + 2 * S * pass;
    return slab_us <= stage_us;
}

cudaError_t launch_slab_level(bool delta, int N, int S, const LevelArgs& a, cudaStream_t s) {
    if (!slab_available(delta, N, S)) return cudaErrorInvalidConfiguration;
    if (delta) return a.item == 1 ? slab::launch<true, uint8_t>(a, N, S, s) : slab::launch<true, float>(a, N, S, s);
    return a.item == 1 ? slab::launch<false, uint8_t>(a, N, S, s) : slab::launch<false, float>(a, N, S, s);
}

cudaError_t launch_slab_images(bool delta, int N, int S, int images, const LevelArgs& a, const SlabTape* tape,
                               cudaStream_t s) {
    if (!slab_available(delta, N, S) || a.item != 4) return cudaErrorInvalidConfiguration;
    slab::Tape t{};
    if (tape) {
        const size_t n = (size_t)a.H * a.W * images;
        t.f = tape->prop;
        t.s = tape->prop + 2 * n;
        t.v = tape->prop + 3 * n;
        t.step = tape->prop_step;
        t.grad = tape->grad;
        t.sm = tape->sm;
        t.sm_step = tape->sm_step;
        return delta ? slab::launch_images<true, true>(a, N, S, images, t, s)
                     : slab::launch_images<false, true>(a, N, S, images, t, s);
    }
    return delta ? slab::launch_images<true, false>(a, N, S, images, t, s)
                 : slab::launch_images<false, false>(a, N, S, images, t, s);
}

// Stage API.  One slab launch instead of 2N (2S) passes, where the outputs share no memory with
// the inputs (a slab reads its neighbours' rows while they may already be written) and one
// launch covers the iterations; the per-pass kernels otherwise.  Measured at 1280x720 (device us,
// against the launches replaced): payload propagation, 4 iterations, 31.1 against 66 (8 launches);
// smoothing, 2 iterations, 11.7 against 25.8 (4); image model of uint8 8.9 against 23.6, whose
// one-thread-per-pixel form reads 50 pixels for each
cudaError_t launch_propagate_stage(const float* flow, size_t fp, int H, int W, int N, int border, float* out, size_t op,
                                   float* tmp, size_t tp, cudaStream_t s) {
    if (N > slab::kMaxFused || ((fp | op) >> 32) || slab::overlap({flow, fp, 8 * (size_t)W}, {out, op, 8 * (size_t)W}, H))
        return launch_propagate(flow, fp, H, W, N, border, out, op, tmp, tp, s);
    LevelArgs a{};
    a.H = H;
    a.W = W;
    a.fs_in = flow, a.fs_in_pitch = fp;
    a.fs_out = out, a.fs_out_pitch = op;
    a.border = border;
    if (N == 1 && (long)H * W >= slab::kSinglePixels && !slab::rows_of_caller4(false, a))
        return launch_propagate(flow, fp, H, W, N, border, out, op, tmp, tp, s);
    return slab::launch_propagate_slab<false>(a, N, s);
}

cudaError_t launch_propagate_payload_stage(const float* flow, size_t fp, const float* sc, size_t sp, const float* ve,
                                           size_t vp, int H, int W, int N, int border, float* of, size_t ofp, float* os,
                                           size_t osp, float* ov, size_t ovp, float* tf, size_t tfp, float* ts, size_t tsp,
                                           float* tv, size_t tvp, cudaStream_t s) {
    const size_t w = (size_t)W;
    const slab::Rows in[3] = {{flow, fp, 8 * w}, {sc, sp, 4 * w}, {ve, vp, 8 * w}};
    const slab::Rows out[3] = {{of, ofp, 8 * w}, {os, osp, 4 * w}, {ov, ovp, 8 * w}};
    bool plain = N > slab::kMaxFused || ((fp | sp | vp | ofp | osp | ovp) >> 32);
    for (const slab::Rows& i : in)
        for (const slab::Rows& o : out) plain |= slab::overlap(i, o, H);
    if (plain)
        return launch_propagate_payload(flow, fp, sc, sp, ve, vp, H, W, N, border, of, ofp, os, osp, ov, ovp, tf, tfp, ts,
                                        tsp, tv, tvp, s);
    LevelArgs a{};
    a.H = H;
    a.W = W;
    a.fs_in = flow, a.fs_in_pitch = fp;
    a.io_in = sc, a.io_in_pitch = sp;
    a.d_in = ve, a.d_in_pitch = vp;
    a.fs_out = of, a.fs_out_pitch = ofp;
    a.io_out = os, a.io_out_pitch = osp;
    a.d_out = ov, a.d_out_pitch = ovp;
    a.border = border;
    if (N == 1 && (long)H * W >= slab::kSinglePixelsPayload && !slab::rows_of_caller4(true, a))
        return launch_propagate_payload(flow, fp, sc, sp, ve, vp, H, W, N, border, of, ofp, os, osp, ov, ovp, tf, tfp, ts,
                                        tsp, tv, tvp, s);
    return slab::launch_propagate_slab<true>(a, N, s);
}

cudaError_t launch_smooth_stage(const float* flow, size_t fp, int H, int W, int S, float* out, size_t op, float* tmp,
                                size_t tp, cudaStream_t s) {
    if (S > slab::kMaxFused || ((fp | op) >> 32) || slab::overlap({flow, fp, 8 * (size_t)W}, {out, op, 8 * (size_t)W}, H))
        return launch_smooth(flow, fp, H, W, S, out, op, tmp, tp, s);
    LevelArgs a{};
    a.H = H;
    a.W = W;
    a.fs_in = flow, a.fs_in_pitch = fp;
    a.fs_out = out, a.fs_out_pitch = op;
    cudaError_t e = slab::set_access_of_caller(false, a);
    if (e == cudaSuccess) e = slab::prepare<slab::smooth_slab_k>();
    if (e != cudaSuccess) return e;
    const slab::Geom g = slab::auto_geom(false, 0, S, W, H, 1);
    return launch_k(slab::smooth_slab_k, dim3(g.slabs(H)), dim3(32 * slab::kWarps), slab::smem_of(false, g), s, a, g);
}

cudaError_t launch_image_model_stage(const void* img, size_t pitch, int item, int H, int W, float* a0, size_t a0p,
                                     float* grad, size_t gp, cudaStream_t s) {
    if ((pitch | a0p | gp) >> 32) return launch_image_model(img, pitch, item, H, W, a0, a0p, grad, gp, s);
    constexpr int step = slab::kCols - 8;
    const int nwx = 1 + (std::max(W - slab::kCols, 0) + step - 1) / step;
    // runs of 8 rows (half the vertical windows' work again for their first rows) unless a level
    // has too few of them to give every SM a block
    const int rows = (long)nwx * ((H + 7) / 8) >= (long)slab::sm_count() * slab::kWarps ? 8 : 4;
    const int blocks = (nwx * ((H + rows - 1) / rows) + slab::kWarps - 1) / slab::kWarps;
    if (item == 1)
        return launch_k(slab::image_model_rows_k<uint8_t>, dim3(blocks), dim3(32 * slab::kWarps), 0, s, (const uint8_t*)img,
                        pitch, H, W, a0, a0p, (float2*)grad, gp, nwx, rows);
    return launch_k(slab::image_model_rows_k<float>, dim3(blocks), dim3(32 * slab::kWarps), 0, s, (const float*)img, pitch, H,
                    W, a0, a0p, (float2*)grad, gp, nwx, rows);
}

}  // namespace ffb
