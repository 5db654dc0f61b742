// batch_layout.h -- where a target's buffers lie in the pool of a batched IBR_gradient call (host.cpp's render_views).
#pragma once
#include <cstddef>
#include <cstdint>

namespace lfrv {

// Float offsets from a target's first float, N pixels: the image U (3 planes), the gradients gx and gy, CG's
// exchanged borders dA and dB (3 planes each), 8 doubles of solver state, and for a target seeded by the learned warm
// start the seed (3 planes) and the network input (N x channels BF16 values). The kernels read and write these in pieces
// of up to 16 bytes (k_cg_strip's borders as float2, the convolutions' input by TMA and 16-byte copies) whatever N is, so
// every section, and with `size` every target, starts on kBatchAlign floats.
constexpr size_t kBatchAlign = 64;  // 256 bytes, as cudaMalloc aligns the pool

struct BatchLayout {
    size_t U, gx, gy, dA, dB, state, seed, input, size;
};

inline BatchLayout batch_layout(size_t N, bool seeded, size_t channels) {
    BatchLayout L{};
    auto place = [&](size_t floats) {
        const size_t off = L.size;
        L.size += (floats + kBatchAlign - 1) / kBatchAlign * kBatchAlign;
        return off;
    };
    L.U = place(3 * N);
    L.gx = place(N);
    L.gy = place(N);
    L.dA = place(3 * N);
    L.dB = place(3 * N);
    L.state = place(16);
    if (seeded) {
        L.seed = place(3 * N);
        L.input = place((N * channels + 1) / 2);
    }
    return L;
}

// Whether k_cg_strip may use dA and dB for its borders.
inline bool cg_borders_aligned(const float *dA, const float *dB) {
    return ((reinterpret_cast<uintptr_t>(dA) | reinterpret_cast<uintptr_t>(dB)) & 7u) == 0;
}

}  // namespace lfrv
