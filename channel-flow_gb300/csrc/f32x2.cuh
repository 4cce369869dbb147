// f32x2.cuh -- packed FP32x2 arithmetic and the asynchronous tile copies of
// the split path's marching stencil kernels (k_dsm32.cu, k_rhs32.cu).
#pragma once

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 sp(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, sp(-1.f), a); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

template <int B>
__device__ __forceinline__ void copy_async(float *sm, const float *gm) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(sm);
    if constexpr (B == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gm) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(gm), "n"(B) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
// all but the N groups committed last are complete
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// columns i-1, i, i+1, i+2 of one row as two pairs
struct Quad {
    float2 p, q;
    __device__ __forceinline__ float2 c() const { return f2(p.y, q.x); }  // columns i, i+1
};
__device__ __forceinline__ Quad quad(const float *s) {
    Quad r;
    r.p = *(const float2 *)s;
    r.q = *(const float2 *)(s + 2);
    return r;
}

// tile of a kernel that reads one halo cell: R rows of 2 LS columns, T threads
template <int LS, int T>
struct HaloTile {
    static constexpr int WS = 2 * LS, R = T / LS, SX = WS + 2, SY = R + 2, NP = SX * SY, NL = (NP + T - 1) / T;
    // the thread's row: with LS = 8 the two rows that half a warp reads at
    // once are 8 apart, 8 SX = 144 words or 16 banks
    static __device__ __forceinline__ int row() {
        const int t = threadIdx.x / LS;
        return LS == 8 ? (t & 1) * 8 + (t >> 1) : t;
    }
};

// lanes per tile row: the width that leaves the fewest idle columns, the
// widest of them
inline int tile_lanes(int nxp) {
    int best = 32;
    for (int ls : {16, 8})
        if (cdiv(nxp, 2 * ls) * ls < cdiv(nxp, 2 * best) * best) best = ls;
    return best;
}

// z-chunk length of a marching kernel with `blocks` tiles and `per` resident
// blocks per SM: the one that minimises (waves of blocks) x (planes per chunk
// + 1.5, the planes below and above and the first copies) x (1 + 0.3 for each
// resident block of an SM past the first: where one wave is not full, fewer
// blocks run faster; 64^3 right-hand side: 256 blocks of 4 planes 8.6 us, 352
// of 3 planes 10.4).
inline int chunk_len(long blocks, int per, int sms, int nzp) {
    if (per < 1) per = 1;
    double best_cost = 1e300;
    int best = nzp;
    for (int n = 1; n <= nzp; n++) {
        const int len = cdiv(nzp, n);
        const long tot = blocks * cdiv(nzp, len);
        const int b = (int)(tot < (long)per * sms ? cdiv(tot, sms) : per);
        const double cost = (double)cdiv(tot, (long)per * sms) * (len + 1.5) * (1.0 + 0.3 * (b - 1));
        if (cost < best_cost - 1e-9) {
            best_cost = cost;
            best = len;
        }
    }
    return best;
}
