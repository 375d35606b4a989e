// Fused z pass of the Poisson solve on meshes of 128, 256, 512 and 1024 cells per side:
// forward DFT along z, the multiplier Kφ, inverse DFT along z, in place on the half
// spectrum.
//
// The 3-D R2C / C2R transforms of the force calculation are split into a batched 2-D
// transform of the z planes (cuFFT) and this kernel, which does both z transforms of
// one (ky, kx) pencil around the multiplication while the pencil is on chip. That
// replaces three passes over the spectrum (the z stage of the forward transform, the
// k-space multiplication and the z stage of the inverse transform) by one.
//
// Layout: spectrum f[kz][pencil], pencil = ky * nh + kx, nh = N/2 + 1 (the 2-D R2C halves
// x). A tile is 16 consecutive pencils of this flat plane: per kz one 128-byte line (the
// plane is a multiple of 16 pencils, so no line is split and no tile is partly empty).
// Lines of 64 bytes cost twice the time at N = 1024 (a plain read-modify-write of the
// spectrum in this order: 1.5 ms with 128-byte lines, 2.9 ms with 64): consecutive kz lie
// 4 MB apart there, so each line is an address translation of its own. A persistent CTA
// takes every gridDim-th tile; each thread copies its own points of the next tile to its
// private slots in shared memory (8-byte asynchronous copies, no barrier) while it
// transforms this one, which is what hides the load latency: with loads straight to
// registers the warps waited for them three quarters of the time (issue slots 42% used).
// N = 32 M (Cooley-Tukey with n = n2 + M n1 and k = k1 + 32 k2), 16 x M threads, thread
// (q, t) at threadIdx.x = q + 16 t holding 32 points of pencil q in registers:
//   A  loads x[t + M n1], DFT over n1 (radix-2 DIF), multiplies by W^(t k1)
//      (W = exp(-2 pi i / N)), exchanges through shared memory;
//   B  holds rows k1 = (32/M) t + j, DFT over n2 -> X[k1 + 32 k2]; X *= Kφ(kx, ky, kz);
//   B' inverse DFT over k2 (radix-2 DIT on the bit-reversed registers), multiplies by
//      W^-(n2 k1), exchanges back;
//   A' inverse DFT over k1 (DIT) -> x[t + M n1], stored where A loaded.
// Both transforms are unnormalised, as cuFFT's, so Kφ keeps its 1/N^3 factor. The
// twiddles of the small DFTs are compile-time constants (multiplications by 1, -i and
// the eighth roots cost nothing or two multiplications); W^(n2 k1) comes from a float
// table of the N roots computed in float64 on the host.
//
// Measured per mesh: 1024^3 4.79 ms (8 pencils per CTA on thread pairs) -> 4.19 (this split,
// loads to registers) -> 3.44 (prefetch) -> 3.21 (twiddles at constant distances, one
// reciprocal per mode); 512^3 0.45 -> 0.40 -> 0.36 ms, where the 3-D transforms with the
// multiplication took 0.85 + 0.24 + 0.86 ms and the 2-D ones take 0.53 + 0.54. About 85
// instructions per mode for 16 bytes moved: the issue slots are half busy (four warps per
// scheduler, all that 128 registers allow), memory would allow 1.5 ms at 1024^3.
#pragma once

#include <cstdint>

namespace djb {

constexpr int kZPencils = 16;   // pencils per tile
constexpr int kZPoints = 32;    // points per thread
__host__ __device__ constexpr bool zpass_size(int res) { return res == 128 || res == 256 || res == 512 || res == 1024; }

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {   // a conj(b)
    return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

// cos(2 pi m / 32) for m = 0 .. 8
__host__ __device__ constexpr float cos32(int m) {
    return m == 0 ? 1.0f : m == 1 ? 0.98078528040323044913f : m == 2 ? 0.92387953251128675613f
         : m == 3 ? 0.83146961230254523708f : m == 4 ? 0.70710678118654752440f : m == 5 ? 0.55557023301960222474f
         : m == 6 ? 0.38268343236508977173f : m == 7 ? 0.19509032201612826785f : 0.0f;
}

// d exp(-+2 pi i m / 32) for 0 <= m < 16, m a constant after unrolling (INV: + sign).
template <bool INV>
__device__ __forceinline__ float2 twiddle32(float2 d, int m) {
    if (m == 0) return d;
    if (m == 8) return INV ? make_float2(-d.y, d.x) : make_float2(d.y, -d.x);
    if (m == 4) {
        constexpr float c = cos32(4);
        return INV ? make_float2((d.x - d.y) * c, (d.x + d.y) * c) : make_float2((d.x + d.y) * c, (d.y - d.x) * c);
    }
    if (m == 12) {
        constexpr float c = cos32(4);
        return INV ? make_float2((d.x + d.y) * -c, (d.x - d.y) * c) : make_float2((d.y - d.x) * c, (d.x + d.y) * -c);
    }
    const float wr = m < 8 ? cos32(m) : -cos32(16 - m);
    const float wi = m < 8 ? cos32(8 - m) : cos32(m - 8);   // sin(2 pi m / 32)
    return INV ? make_float2(d.x * wr - d.y * wi, d.y * wr + d.x * wi)
               : make_float2(d.x * wr + d.y * wi, d.y * wr - d.x * wi);
}

// L-point DFTs on consecutive groups of L of the 32 registers. DIF: natural order in,
// bit-reversed out; DIT: bit-reversed in, natural out.
template <int LEN, bool INV>
__device__ __forceinline__ void dif_stage(float2 (&a)[kZPoints]) {
#pragma unroll
    for (int s = 0; s < kZPoints; s += LEN)
#pragma unroll
        for (int j = 0; j < LEN / 2; ++j) {
            const float2 u = a[s + j], v = a[s + j + LEN / 2];
            a[s + j] = make_float2(u.x + v.x, u.y + v.y);
            a[s + j + LEN / 2] = twiddle32<INV>(make_float2(u.x - v.x, u.y - v.y), j * (32 / LEN));
        }
}
template <int LEN, bool INV>
__device__ __forceinline__ void dit_stage(float2 (&a)[kZPoints]) {
#pragma unroll
    for (int s = 0; s < kZPoints; s += LEN)
#pragma unroll
        for (int j = 0; j < LEN / 2; ++j) {
            const float2 u = a[s + j];
            const float2 v = twiddle32<INV>(a[s + j + LEN / 2], j * (32 / LEN));
            a[s + j] = make_float2(u.x + v.x, u.y + v.y);
            a[s + j + LEN / 2] = make_float2(u.x - v.x, u.y - v.y);
        }
}
template <int L, bool INV>
__device__ __forceinline__ void dft_dif(float2 (&a)[kZPoints]) {
    if constexpr (L >= 32) dif_stage<32, INV>(a);
    if constexpr (L >= 16) dif_stage<16, INV>(a);
    if constexpr (L >= 8) dif_stage<8, INV>(a);
    if constexpr (L >= 4) dif_stage<4, INV>(a);
    dif_stage<2, INV>(a);
}
template <int L, bool INV>
__device__ __forceinline__ void dft_dit(float2 (&a)[kZPoints]) {
    dit_stage<2, INV>(a);
    if constexpr (L >= 4) dit_stage<4, INV>(a);
    if constexpr (L >= 8) dit_stage<8, INV>(a);
    if constexpr (L >= 16) dit_stage<16, INV>(a);
    if constexpr (L >= 32) dit_stage<32, INV>(a);
}

// Bit reversal of i < L (L a power of two).
template <int L>
__host__ __device__ constexpr int brev(int i) {
    int r = 0;
    for (int b = 1; b < L; b <<= 1) r = 2 * r + ((i & b) ? 1 : 0);
    return r;
}

// Shared memory: the tables (the N twiddles W^(k1 n2) at k1 M + n2, so that every thread
// reads its own at constant distances from one base; N terms of the inverse Laplacian, with
// deconvolution N window factors), the prefetch slots [n1][thread], and the exchange area
// [k1][n2][pencil] of one float per point (real and imaginary parts are exchanged one
// after the other), rows of k1 padded so that the two threads t of a warp read different
// banks. 128 registers per thread and about 200 KB of shared memory per SM.
template <int N>
struct ZGeom {
    static constexpr int M = N / kZPoints;              // threads per pencil
    static constexpr int kThreads = kZPencils * M;
    static constexpr int J = 32 / M;                    // rows per thread in stage B
    static constexpr int kRow = M * kZPencils + 16 / J; // words per k1: J rows = 16 modulo 32
    static constexpr size_t kStage = size_t(kZPoints) * kThreads * 8;
    static constexpr size_t kSmem = size_t(N) * 24 + kStage + size_t(32) * kRow * 4;
    static constexpr int kBlocks = 1024 / N;            // CTAs per SM
};

// Registers of stage A (a[i] = point k1 = brev(i) of column n2 = t) to stage B's rows
// (a[j M + n2], k1 = J t + j) or back. A thread starts an exchange by writing the slots that
// it alone read at the end of the one before, so no barrier stands between exchanges.
template <int N, bool TO_ROWS>
__device__ __forceinline__ void zexchange(float2 (&a)[kZPoints], float* e, int q, int t) {
    using G = ZGeom<N>;
    constexpr int M = G::M;
    float* const ca = e + t * kZPencils + q;               // + k1 * row
    float* const cb = e + G::J * t * G::kRow + q;          // + j * row + n2 * 16
#pragma unroll
    for (int part = 0; part < 2; ++part) {
        if (part) __syncthreads();   // the first component has been read
#pragma unroll
        for (int i = 0; i < kZPoints; ++i) {
            const float v = part ? a[i].y : a[i].x;
            if (TO_ROWS) ca[brev<32>(i) * G::kRow] = v;
            else cb[(i / M) * G::kRow + (i % M) * kZPencils] = v;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kZPoints; ++i) {
            const float v = TO_ROWS ? cb[(i / M) * G::kRow + (i % M) * kZPencils] : ca[brev<32>(i) * G::kRow];
            if (part) a[i].y = v;
            else a[i].x = v;
        }
    }
}

template <int N, class KPhi>
__global__ void __launch_bounds__(ZGeom<N>::kThreads, ZGeom<N>::kBlocks) k_zpass(
    float2* __restrict__ f, const float2* __restrict__ wN, KPhi kphi) {
    using G = ZGeom<N>;
    constexpr int M = G::M, J = G::J, nh = N / 2 + 1;
    constexpr int64_t plane = int64_t(N) * nh;
    constexpr int kTiles = int(plane / kZPencils);
    extern __shared__ __align__(16) unsigned char zs[];
    float2* const w = reinterpret_cast<float2*>(zs);
    double* const T = reinterpret_cast<double*>(zs + size_t(N) * 8);
    double* const D = T + N;
    float2* const stage = reinterpret_cast<float2*>(zs + size_t(N) * 24) + threadIdx.x;
    float* const area = reinterpret_cast<float*>(zs + size_t(N) * 24 + G::kStage);
    const int q = threadIdx.x % kZPencils, t = threadIdx.x / kZPencils;
    const auto fetch = [&](int tile) {   // this thread's points of the tile to its slots
        if (tile < kTiles) {
            const float2* src = f + int64_t(tile) * kZPencils + q + t * plane;
#pragma unroll
            for (int i = 0; i < kZPoints; ++i)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                                 unsigned(__cvta_generic_to_shared(stage + i * G::kThreads))),
                             "l"(src + int64_t(M * i) * plane)
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(blockIdx.x);
    for (int i = threadIdx.x; i < N; i += G::kThreads) {
        w[i] = wN[(i / M) * (i % M)];   // k1 n2 < N
        T[i] = kphi.T[i];
        if (kphi.M) D[i] = kphi.M[i];
    }
    __syncthreads();
    for (int tile = blockIdx.x; tile < kTiles; tile += gridDim.x) {
        float2 a[kZPoints];
        asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
        for (int i = 0; i < kZPoints; ++i) a[i] = stage[i * G::kThreads];
        dft_dif<32, false>(a);   // a[i] = Y[k1 = brev(i)] of n2 = t
        fetch(tile + gridDim.x); // the slots have been read: the transform above depends on them
#pragma unroll
        for (int i = 1; i < kZPoints; ++i) a[i] = cmul(a[i], w[brev<32>(i) * M + t]);
        zexchange<N, true>(a, area, q, t);
        dft_dif<M, false>(a);    // a[j M + i] = X[k1 + 32 brev(i)], k1 = J t + j
        const int pencil = tile * kZPencils + q, ky = pencil / nh, kx = pencil - ky * nh;
        const typename KPhi::Pencil kp = kphi.pencil(kx, ky, T, D);
#pragma unroll
        for (int i = 0; i < kZPoints; ++i) {
            const float K = kphi.at(kp, J * t + i / M + 32 * brev<M>(i % M), T, D);
            a[i] = make_float2(a[i].x * K, a[i].y * K);
        }
        dft_dit<M, true>(a);     // a[j M + n2]
#pragma unroll
        for (int i = 0; i < kZPoints; ++i)
            if (i % M != 0) a[i] = cmulc(a[i], w[J * t * M + i]);   // k1 M + n2
        zexchange<N, false>(a, area, q, t);
        dft_dit<32, true>(a);    // a[i] = x[t + M i]
        float2* const dst = f + int64_t(tile) * kZPencils + q + t * plane;
#pragma unroll
        for (int i = 0; i < kZPoints; ++i) __stcs(dst + int64_t(M * i) * plane, a[i]);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

}  // namespace djb
