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
// Layout: spectrum f[(kz * N + ky) * nh + kx], nh = N/2 + 1 (the 2-D R2C halves x).
// A CTA owns 16 consecutive kx of one ky: rows of 128 bytes. Rows of 64 bytes, half of
// that, cost twice the time at N = 1024 (a plain read-modify-write of the spectrum in
// this order: 1.5 ms with 128-byte rows, 2.9 ms with 64-byte rows): consecutive kz lie
// 4 MB apart there, so each row is an address translation of its own.
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
// Measured (force phases of a step, per mesh): 1024^3 4.79 -> 4.19 ms against the earlier
// form with 8 pencils per CTA on thread pairs; 512^3 0.85 + 0.24 + 0.86 ms (3-D transforms
// and the multiplication) -> 0.53 + 0.45 + 0.54 ms. The arithmetic of the two DFTs and of
// Kφ (about 100 lane instructions per mode) bounds it, not memory (1.5 ms at 1024^3).
#pragma once

#include <cstdint>

namespace djb {

constexpr int kZPencils = 16;   // kx per CTA
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

// Shared memory: the N twiddles, then the exchange area [k1][n2][pencil], rows of k1
// padded so that the two threads t of a warp read from different banks: float2 elements,
// or at N = 1024 one component at a time (float elements), which leaves two CTAs' worth
// of shared memory to the L1 cache.
template <int N>
struct ZGeom {
    static constexpr int M = N / kZPoints;              // threads per pencil
    static constexpr int kThreads = kZPencils * M;
    static constexpr int J = 32 / M;                    // rows per thread in stage B
    static constexpr bool kSplit = N == 1024;           // exchange one component at a time
    static constexpr int kPad = kSplit ? 16 : 0;        // J * row = 16 modulo 32 words
    static constexpr int kRow = M * kZPencils + kPad;   // elements per k1
    static constexpr size_t kSmem = size_t(N) * 8 + size_t(32) * kRow * (kSplit ? 4 : 8);
    static constexpr int kBlocks = N == 1024 ? 1 : (N == 512 ? 2 : (N == 256 ? 4 : 8));   // 128 registers per thread
};

// Registers a[R(c)] of stage A (c = k1) against stage B's rows through the exchange area.
// to_rows: thread (q, t) writes a[brev(k1)] at (k1, n2 = t) and reads (k1 = J t + j, n2)
// into a[j M + n2]; otherwise the reverse, into a[brev(k1)]. A thread starts the second
// exchange by writing the slots that it alone read last in the first: no barrier between.
template <int N, bool TO_ROWS>
__device__ __forceinline__ void zexchange(float2 (&a)[kZPoints], void* area, int q, int t) {
    using G = ZGeom<N>;
    constexpr int M = G::M, J = G::J;
    const int ca = t * kZPencils + q;          // + k1 * row
    const int cb = J * t * G::kRow + q;        // + j * row + n2 * 16
    if constexpr (G::kSplit) {
        float* e = static_cast<float*>(area);
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            if (part) __syncthreads();   // the first component has been read
#pragma unroll
            for (int i = 0; i < kZPoints; ++i) {
                const int at = TO_ROWS ? ca + brev<32>(i) * G::kRow : cb + (i / M) * G::kRow + (i % M) * kZPencils;
                e[at] = part ? a[i].y : a[i].x;
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < kZPoints; ++i) {
                const int at = TO_ROWS ? cb + (i / M) * G::kRow + (i % M) * kZPencils : ca + brev<32>(i) * G::kRow;
                (part ? a[i].y : a[i].x) = e[at];
            }
        }
    } else {
        float2* e = static_cast<float2*>(area);
#pragma unroll
        for (int i = 0; i < kZPoints; ++i)
            e[TO_ROWS ? ca + brev<32>(i) * G::kRow : cb + (i / M) * G::kRow + (i % M) * kZPencils] = a[i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kZPoints; ++i)
            a[i] = e[TO_ROWS ? cb + (i / M) * G::kRow + (i % M) * kZPencils : ca + brev<32>(i) * G::kRow];
    }
}

template <int N, class KPhi>
__global__ void __launch_bounds__(ZGeom<N>::kThreads, ZGeom<N>::kBlocks) k_zpass(
    float2* __restrict__ f, const float2* __restrict__ wN, KPhi kphi) {
    using G = ZGeom<N>;
    constexpr int M = G::M, J = G::J, nh = N / 2 + 1;
    extern __shared__ __align__(16) unsigned char zs[];
    float2* const w = reinterpret_cast<float2*>(zs);
    void* const area = zs + size_t(N) * 8;
    const int q = threadIdx.x % kZPencils, t = threadIdx.x / kZPencils;
    const int ky = blockIdx.y, kx = blockIdx.x * kZPencils + q;
    const bool active = kx < nh;
    constexpr int64_t zstride = int64_t(N) * nh;
    float2* __restrict__ const col = f + int64_t(ky) * nh + (active ? kx : 0) + t * zstride;
    float2 a[kZPoints];
#pragma unroll
    for (int i = 0; i < kZPoints; ++i)
        a[i] = active ? __ldcs(col + int64_t(M * i) * zstride) : make_float2(0.0f, 0.0f);
    for (int i = threadIdx.x; i < N; i += G::kThreads) w[i] = wN[i];
    __syncthreads();
    dft_dif<32, false>(a);   // a[i] = Y[k1 = brev(i)] of n2 = t
#pragma unroll
    for (int i = 1; i < kZPoints; ++i) a[i] = cmul(a[i], w[(t * brev<32>(i)) & (N - 1)]);
    zexchange<N, true>(a, area, q, t);
    dft_dif<M, false>(a);    // a[j M + i] = X[k1 + 32 brev(i)], k1 = J t + j
    const typename KPhi::Pencil kp = kphi.pencil(active ? kx : 0, ky);
#pragma unroll
    for (int i = 0; i < kZPoints; ++i) {
        const float K = kphi.at(kp, J * t + i / M + 32 * brev<M>(i % M));
        a[i] = make_float2(a[i].x * K, a[i].y * K);
    }
    dft_dit<M, true>(a);     // a[j M + n2]
#pragma unroll
    for (int i = 0; i < kZPoints; ++i)
        if (i % M != 0) a[i] = cmulc(a[i], w[((i % M) * (J * t + i / M)) & (N - 1)]);
    zexchange<N, false>(a, area, q, t);
    dft_dit<32, true>(a);    // a[i] = x[t + M i]
    if (active) {
#pragma unroll
        for (int i = 0; i < kZPoints; ++i) __stcs(col + int64_t(M * i) * zstride, a[i]);
    }
}

}  // namespace djb
