// Random numbers of the FP32 electron step in shared memory: the next numbers
// of a thread's stream wait in a column of its own.
#pragma once
#include "omc_rng.cuh"

namespace omc {

// A particle's stream in the electron kernel (FP32).  A condensed-history
// step draws some eighteen numbers at two dozen places; with a block of four
// in registers (Philox) every draw picks one of four and may be the one
// where a lane's block runs out, so a warp executed the generator at nearly
// every draw, for a quarter of its lanes.  Here the next numbers wait in
// shared memory (slot = stream position modulo RING, a column per thread: no
// bank conflicts), filled for all lanes together at the top of a step and
// of each multiple-scattering pass (rng_ensure); a draw is one load, and
// rejection loops ask for their next turn.  The numbers are the same.  16 KB
// a block, four blocks an SM.  Measured on the slab beam (1e7 histories):
// 136.5 -> 105.1 ms, code of the kernel 78 -> 63 KB; a fill to 12 at the top
// of a step and 10 a pass beat 3 / 10 (111.8), 8 / 8 (108.4), 3 / 13 (108.6).
// COLS: threads of the block.  ROWS: numbers a thread holds; ensure() takes
// up to ROWS - 3.
constexpr int RING = 16;
template <int COLS, int ROWS>
struct RingStore {
    float v[ROWS][COLS];
    uint32_t k0[COLS], k1[COLS];
};
template <int COLS, int ROWS>
__device__ __forceinline__ RingStore<COLS, ROWS> &ring() {
    if constexpr (sizeof(RingStore<COLS, ROWS>) > 48 * 1024) {
        extern __shared__ float ring_shared[];
        return *reinterpret_cast<RingStore<COLS, ROWS> *>(ring_shared);
    } else {
        __shared__ RingStore<COLS, ROWS> r;
        return r;
    }
}
// Block `block` of the stream of column t.
template <int COLS, int ROWS>
__device__ __forceinline__ void ring_block(uint32_t block, uint32_t seedw, int t) {
    RingStore<COLS, ROWS> &r = ring<COLS, ROWS>();
    const U4 b = philox4x32_10(U4{block, seedw, 0x6f6d6321u, 0u}, r.k0[t], r.k1[t]);
    const int row = (block & (ROWS / 4 - 1)) * 4;
    r.v[row][t] = u01f(b.x);
    r.v[row + 1][t] = u01f(b.y);
    r.v[row + 2][t] = u01f(b.z);
    r.v[row + 3][t] = u01f(b.w);
}
template <int COLS, int ROWS>
__device__ __noinline__ void ring_fill(uint32_t block, uint32_t seedw) {
    ring_block<COLS, ROWS>(block, seedw, threadIdx.x);
}
template <int COLS, int ROWS = RING>
struct RingStream {
    uint32_t seedw, pos, filled;
    __device__ __forceinline__ void init(uint64_t key, uint32_t seed_word, uint32_t position = 0) {
        ring<COLS, ROWS>().k0[threadIdx.x] = (uint32_t)key;
        ring<COLS, ROWS>().k1[threadIdx.x] = (uint32_t)(key >> 32);
        seedw = seed_word;
        pos = position;
        filled = position & ~3u;
    }
    __device__ __forceinline__ uint32_t position() const { return pos; }
    __device__ __forceinline__ uint64_t key() const {
        return ((uint64_t)ring<COLS, ROWS>().k1[threadIdx.x] << 32) | ring<COLS, ROWS>().k0[threadIdx.x];
    }
    __device__ __forceinline__ void ensure(int n) {
        while ((int)(filled - pos) < n) {
            ring_fill<COLS, ROWS>(filled >> 2, seedw);
            filled += 4;
        }
    }
    // The whole warp fills the rings of the lanes of `lanes`: ROWS / 4 lanes
    // a ring and pass.  Keys that lanes have just written (init) are read by
    // others here, and neither a vote nor a shuffle orders shared memory: the
    // barrier before the fill does, the one after it orders the numbers.
    __device__ __forceinline__ void assist(unsigned lanes) {
        __syncwarp();
        constexpr int PER = ROWS / 4 > 32 ? 32 : ROWS / 4;
        const int lane = threadIdx.x & 31;
        for (unsigned m = lanes; m;) {
            unsigned t = m;
#pragma unroll
            for (int q = 0; q < 32 / PER; q++) {
                if (q < lane / PER) t &= t - 1;
                m &= m - 1;
            }
            const int src = t ? __ffs(t) - 1 : 0;
            const uint32_t f = __shfl_sync(0xffffffffu, filled, src), at = __shfl_sync(0xffffffffu, pos, src);
            const uint32_t block = (f >> 2) + lane % PER;
            if (t && (int)(block * 4 + 4 - at) <= ROWS) ring_block<COLS, ROWS>(block, seedw, (threadIdx.x & ~31) + src);
        }
        if (lanes >> lane & 1) filled = (pos + ROWS) & ~3u;
        __syncwarp();
    }
    // continue at a later position (numbers drawn elsewhere)
    __device__ __forceinline__ void seek(uint32_t p) {
        pos = p;
        if ((int)(filled - p) < 0) filled = p & ~3u;
    }
    // the caller has asked for it (ensure)
    __device__ __forceinline__ float uni() {
        const float v = ring<COLS, ROWS>().v[pos & (ROWS - 1)][threadIdx.x];
        pos++;
        return v;
    }
};
template <typename Rng>
struct IsRing {
    static constexpr bool value = false;
};
template <int COLS, int ROWS>
struct IsRing<RingStream<COLS, ROWS>> {
    static constexpr bool value = true;
};

}  // namespace omc
