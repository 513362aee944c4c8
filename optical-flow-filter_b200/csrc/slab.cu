// Launch side of the slab level step (slab.cuh).
#include "slab.cuh"

#include <atomic>

namespace ffb {
namespace slab {

template <bool DELTA, typename P>
__global__ void __launch_bounds__(32 * kWarps, 1) slab_k(LevelArgs a, Geom g) {
    level_slab<DELTA, P>(a, g, blockIdx.x);
}

constexpr int kSmem = 227 * 1024;  // shared memory a block may use on B200

int max_rows(bool delta, int N, int S) {
    return kSmem / (planes(delta) * kPlane) - 2 * (N + 2 * S) - kWarps;
}

int sm_count() {
    static int cache[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    int& n = cache[dev & 63];
    if (n == 0) {
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 148;
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
    const int ox = slab_cols(N, S);
    g.nwx = (W + ox - 1) / ox;
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

bool rows16(const void* p, size_t pitch, int W, int bytes) {
    return ((uintptr_t)p | pitch) % 16 == 0 && pitch >= (size_t)((W + 3) & ~3) * bytes;
}

template <bool DELTA, typename P>
cudaError_t launch(LevelArgs a, int N, int S, cudaStream_t s) {
    // row offsets are computed as 32 x 32-bit products (rowp)
    for (size_t p : {a.img_pitch, a.fs_in_pitch, a.io_in_pitch, a.d_in_pitch, a.fs_out_pitch, a.io_out_pitch,
                     a.d_out_pitch, a.fu_out_pitch, a.coarse_pitch})
        if (p >> 32) return cudaErrorInvalidPitchValue;
    a.vec = rows16(a.fs_in, a.fs_in_pitch, a.W, 8) && rows16(a.io_in, a.io_in_pitch, a.W, 4) &&
            rows16(a.fs_out, a.fs_out_pitch, a.W, 8) && rows16(a.io_out, a.io_out_pitch, a.W, 4) &&
            (DELTA ? rows16(a.d_in, a.d_in_pitch, a.W, 8) && rows16(a.d_out, a.d_out_pitch, a.W, 8)
                   : !a.fu_out || rows16(a.fu_out, a.fu_out_pitch, a.W, 8)) &&
            (!a.y_out || rows16(a.y_out, a.fs_out_pitch, a.W, 8));
    a.img_vec = ((uintptr_t)a.img | a.img_pitch) % 16 == 0;
    static std::atomic<unsigned long long> prepared{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(prepared.load() & bit)) {
        cudaError_t e = cudaFuncSetAttribute(slab_k<DELTA, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
        if (e != cudaSuccess) return e;
        // full shared carve-out, as for the tile kernels: SMs running small slabs can then also
        // host the other levels' kernels
        e = cudaFuncSetAttribute(slab_k<DELTA, P>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        prepared.fetch_or(bit);
    }
    const Geom g = a.band > 0 ? geom_of(N, S, a.W, a.H, std::min(a.band, max_rows(DELTA, N, S)))
                              : auto_geom(DELTA, N, S, a.W, a.H, 1);
    return launch_k(slab_k<DELTA, P>, dim3(g.slabs(a.H)), dim3(32 * kWarps), (size_t)slab_smem(DELTA, N, S, std::max(g.rows, g.rows_e)),
                    s, a, g);
}

}  // namespace slab

bool slab_available(bool delta, int N, int S) { return N >= 1 && S >= 1 && slab::max_rows(delta, N, S) >= 1; }

cudaError_t launch_slab_level(bool delta, int N, int S, const LevelArgs& a, cudaStream_t s) {
    if (!slab_available(delta, N, S)) return cudaErrorInvalidConfiguration;
    if (delta) return a.item == 1 ? slab::launch<true, uint8_t>(a, N, S, s) : slab::launch<true, float>(a, N, S, s);
    return a.item == 1 ? slab::launch<false, uint8_t>(a, N, S, s) : slab::launch<false, float>(a, N, S, s);
}

}  // namespace ffb
