// rsf_kernels.cuh -- device code of one RSF iteration: four kernels per step.
//
//   x-pass   phi, I -> H, 1-H, I*H, I*(1-H) (kernel.cu:210-298) and their
//            valid correlation along x (kernel.cu:1000-1014)
//   y-pass   valid correlation along y (kernel.cu:1017-1031)
//   z-pass   valid correlation along z (kernel.cu:1035-1049), local fits
//            f = blur(I H)/blur(H) (kernel.cu:191-207), e = (I - f)^2
//            (kernel.cu:25-55) and the data factor lambda (e_out - e_in)
//   stencil  gradient, |gradient|, normalised gradient, curvature and the
//            "Laplacian" with the reference's boundary rules (kernel.cu:57-125,
//            173-189, 630-933), the border band f = 30/30 (kernel.cu:300-325),
//            delta (kernel.cu:265-280) and the explicit update
//            (kernel.cu:365-387); writes phi once.
//
// Every kernel takes the whole batch: a table of sub-volumes and, per kernel,
// a prefix sum of the blocks each sub-volume needs (block b finds its
// sub-volume by binary search).  A single volume is a batch of one.
//
// Summation order is the reference's: each blurred value is accumulated with
// fused multiply-adds from +0 over ascending taps, x first, then y, then z.
// Two values share one packed f32x2 multiply-add, which rounds each lane exactly
// like fmaf.  The fields lie interleaved, a float4 per voxel.  The y and z
// correlations stream along their axis with K rotating accumulators per column
// (the accumulator of output o is slot o mod K), so every input is loaded once:
// a y-pass thread owns one pair of fields of a column, a z-pass thread all four
// (its fits and data factor then need no exchange).  Tap counts that are not
// compiled in run in chunks over a register window.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "rsf_arith.cuh"
#include "rsf_internal.h"
#include "rsf_pair.cuh"

namespace rsf {

__device__ __forceinline__ int find_sv(const int *__restrict__ pre, int n, int b) {
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(pre + mid) <= b) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Programmatic dependent launch: the kernels of an iteration are launched so
// that the next one's blocks may start while the last blocks of this one still
// run.  A block reads its tables (which no kernel writes), waits for the previous
// kernel's results before it touches a field, and lets its dependents go when
// its work is done (at its start they crowd onto the SMs that are free first:
// 128^3 took 886 us per 10 iterations that way, 742 so and 857 without).
// Every thread of every block waits, also those without work: a grid that
// finished before its predecessor would let its own successor through.  The
// first kernel after a table upload is launched the ordinary way: its tables'
// writes are only visible behind a full dependency.  What a kernel of the chain
// writes (level set, blurred fields, data factor) is read with ordinary loads or
// cp.async: __ldg wants memory that nothing writes while the reading kernel is
// resident, which holds for the image and the tables alone.  (The x-pass lets its
// dependents go by ending: an explicit call after its row loop takes it from 56
// to 182 registers at 35 taps.)
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... Q>
cudaError_t launch_dependent(bool dependent, void (*kernel)(P...), unsigned blocks, int threads, size_t smem,
                             cudaStream_t st, const Q &...args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = dependent ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

__device__ __forceinline__ float load_img(const void *img, size_t i, int f32) {
    return f32 ? __ldg(static_cast<const float *>(img) + i)
               : (float)__ldg(static_cast<const unsigned char *>(img) + i);
}

// Valid correlation of XB consecutive outputs of both field pairs: src points at
// the lane's first input in the shared slab of float4 (H, 1-H, I H, I (1-H)) per
// element; one 128-bit load feeds both pairs.  With a run-time tap count the
// taps go in chunks of XB over a window of 2 XB inputs (which may read up to
// 2 XB elements past the slab; they lie in the next slab or the padding after the
// last, and no tap uses them).
template <int K, int XB>
__device__ __forceinline__ void xconv(const float4 *src, const StepConst &c, int k, unsigned long long (&u)[XB],
                                      unsigned long long (&v)[XB]) {
    const ulonglong2 *in = reinterpret_cast<const ulonglong2 *>(src);
    if constexpr (K > 0) {
#pragma unroll
        for (int q = 0; q < XB + K - 1; ++q) {
            const ulonglong2 w = in[q];
#pragma unroll
            for (int m = 0; m < XB; ++m) {
                const int tt = q - m;
                if (tt < 0 || tt >= K) continue;
                u[m] = fma2(w.x, c.tap2(tt), tt == 0 ? 0ull : u[m]);
                v[m] = fma2(w.y, c.tap2(tt), tt == 0 ? 0ull : v[m]);
            }
        }
    } else {
        // one pair after the other: the window of both at once takes 76
        // registers instead of 48 and measured 181 against 171 us
        auto pair = [&](const unsigned long long *in1, unsigned long long (&o)[XB]) {
            unsigned long long w[2 * XB];
#pragma unroll
            for (int m = 0; m < XB; ++m) {
                o[m] = 0ull;
                w[m] = in1[2 * m];
            }
            for (int t0 = 0; t0 < k; t0 += XB) {
#pragma unroll
                for (int m = 0; m < XB; ++m) w[XB + m] = in1[2 * (t0 + XB + m)];
#pragma unroll
                for (int j = 0; j < XB; ++j) {
                    if (t0 + j >= k) break;
                    const unsigned long long g = c.tap2(t0 + j);
#pragma unroll
                    for (int m = 0; m < XB; ++m) o[m] = fma2(w[m + j], g, o[m]);
                }
#pragma unroll
                for (int m = 0; m < XB; ++m) w[m] = w[XB + m];
            }
        };
        pair(reinterpret_cast<const unsigned long long *>(src), u);
        pair(reinterpret_cast<const unsigned long long *>(src) + 1, v);
    }
}

// ---------------------------------------------------------------------------
// x-pass.  One warp per row segment of 32*XB outputs.  The four fields of
// the segment's inputs sit in shared memory as float4 (H, 1-H, I H, I (1-H));
// a lane produces XB consecutive outputs of both pairs (XB odd, so the lanes'
// 128-bit loads fall in distinct banks).  Besides issue, the kernel is bound by
// shared-memory wavefronts (73 % of peak at 21 taps).
// Shared memory: XP_ROWS * span float4 inputs and 2 * XB float4 of padding.
// ---------------------------------------------------------------------------
template <int K, int XB, Arith A>
__global__ void __launch_bounds__(XP_ROWS * 32) xpass_kernel(const SubVolDev *__restrict__ svs,
                                                              const int *__restrict__ pre,
                                                              const __grid_constant__ StepConst c, int parity) {
    extern __shared__ float4 sm4[];
    constexpr int XT = 32 * XB;
    const int k = K > 0 ? K : c.k;
    const int span = XT + k - 1;
    const int b = blockIdx.x;
    const int sv = find_sv(pre, c.nsv, b);
    const SubVolDev s = svs[sv];
    int t = b - __ldg(pre + sv);
    const int ntx = (s.Wv + XT - 1) / XT, nty = (s.H + XP_ROWS * c.xrpw - 1) / (XP_ROWS * c.xrpw);
    const int tx = t % ntx;
    t /= ntx;
    const int ty = t % nty;
    const int z = t / nty;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float4 *in = sm4 + warp * span;
    const int x0 = tx * XT;
    pdl_wait();
    // The warp's next row into L2: lanes 0 .. 7 its phi lines, 8 and 9 its image
    // lines.  A row's loads are waited for at once, and from memory they took
    // most of its time: 5.30 ms per launch on the 48 sub-volumes without this,
    // 4.68 with it; two rows ahead 4.76.  Float images gained nothing (865
    // against 888 us on 195 M voxels, 29 taps) and go without.
    auto prefetch_next = [&](int j, int y, size_t row) {
        if (c.img_f32 || j + 1 >= c.xrpw || y + XP_ROWS >= s.H) return;
        const size_t next = row + (size_t)XP_ROWS * s.W;
        const int xp = x0 + 32 * lane, xi = x0 + 128 * (lane - 8);
        if (lane < 8) {
            if (xp < s.W && 32 * lane < span)
                asm volatile("prefetch.global.L2 [%0];" ::"l"((parity ? s.phi[1] : s.phi[0]) + next + xp));
        } else if (lane < 10 && xi < s.W) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const unsigned char *>(s.img) + next + xi));
        }
    };
    // c.xrpw rows per warp, XP_ROWS apart: the block setup above is paid
    // once per c.xrpw row segments
    for (int j = 0; j < c.xrpw; ++j) {
        const int y = (ty * c.xrpw + j) * XP_ROWS + warp;
        if (y >= s.H) break;
        if (j > 0) __syncwarp();  // the previous row's stores have read the slab
        const size_t row = ((size_t)z * s.H + y) * s.W;
        const float *phi = (parity ? s.phi[1] : s.phi[0]) + row;
        prefetch_next(j, y, row);
        if constexpr (K > 0) {
            // all of the lane's loads first, so that they are in flight together
            constexpr int NE = ((XT + K - 1 + 31) / 32 + 1) & ~1;
            float ph[NE], im[NE];
#pragma unroll
            for (int q = 0; q < NE; ++q) {
                const int e = lane + 32 * q, x = x0 + e;
                const bool ok = e < span && x < s.W;
                ph[q] = ok ? phi[x] : 0.0f;
                im[q] = ok ? load_img(s.img, row + x, c.img_f32) : 0.0f;
            }
            // (elements past the row feed only outputs past Wv)
#pragma unroll
            for (int q = 0; q < NE; q += 2) {
                const int e = lane + 32 * q;
                const float2 h = heaviside2<A>(make_float2(ph[q], ph[q + 1]), c.eps, c.pk);
                const float2 hi = sub2(dup2(1.0f), h);
                if (e < span) in[e] = make_float4(h.x, hi.x, __fmul_rn(im[q], h.x), __fmul_rn(im[q], hi.x));
                if (e + 32 < span)
                    in[e + 32] = make_float4(h.y, hi.y, __fmul_rn(im[q + 1], h.y), __fmul_rn(im[q + 1], hi.y));
            }
        } else {
            for (int e = lane; e < span; e += 64) {
                const int x = x0 + e;
                const bool ok0 = x < s.W, ok1 = e + 32 < span && x + 32 < s.W;
                const float p0 = ok0 ? phi[x] : 0.0f, p1 = ok1 ? phi[x + 32] : 0.0f;
                const float i0 = ok0 ? load_img(s.img, row + x, c.img_f32) : 0.0f;
                const float i1 = ok1 ? load_img(s.img, row + x + 32, c.img_f32) : 0.0f;
                const float2 h = heaviside2<A>(make_float2(p0, p1), c.eps, c.pk);
                const float2 hi = sub2(dup2(1.0f), h);
                in[e] = make_float4(h.x, hi.x, __fmul_rn(i0, h.x), __fmul_rn(i0, hi.x));
                if (e + 32 < span) in[e + 32] = make_float4(h.y, hi.y, __fmul_rn(i1, h.y), __fmul_rn(i1, hi.y));
            }
        }
        __syncwarp();
        unsigned long long u[XB], v[XB];
        xconv<K, XB>(in + XB * lane, c, k, u, v);
        // staged in the slab, once every lane has finished reading it, so that
        // the rows go out coalesced
        __syncwarp();
#pragma unroll
        for (int m = 0; m < XB; ++m) reinterpret_cast<ulonglong2 *>(in)[XB * lane + m] = make_ulonglong2(u[m], v[m]);
        __syncwarp();
        float4 *dst = reinterpret_cast<float4 *>(s.xb) + ((size_t)z * s.H + y) * s.Wp + x0;
#pragma unroll
        for (int q = 0; q < XB; ++q) {
            const int e = lane + 32 * q;
            if (x0 + e < s.Wv) dst[e] = in[e];
        }
    }
}

// ---------------------------------------------------------------------------
// Streaming valid correlation along a strided axis for a pair of columns:
// inputs src[i * stride] for i in [0, n), outputs o = i - K + 1 in [0, n-K+1)
// handed to emit(o, value) as soon as they complete.
// ---------------------------------------------------------------------------
// Inputs reach the thread through a private ring of RING float2 slots in
// shared memory filled by cp.async, so that RING loads per thread are in
// flight while the multiply-adds run.  Element i lives in slot i % RING and
// in commit group i; iteration i first refills the slot element i-1 used
// (with element i-1+RING, group RING+i-1), then waits until at most RING-1
// groups are pending, which completes group i.
constexpr int RING = 8;

__device__ __forceinline__ void cp_async8(float2 *smem_dst, const float *gsrc) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem_dst, const void *gsrc) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait_ring() { asm volatile("cp.async.wait_group %0;" ::"n"(RING - 1) : "memory"); }

struct Ring {
    float2 *base;     // this thread's slot 0; slot s at base + s * step
    int step;         // threads per block
    const float *src; // element i at src + i * stride
    size_t stride;
    int n;
    bool act;         // inactive threads load nothing (their results are discarded)
    __device__ __forceinline__ float2 *slot(int i) const { return base + (i & (RING - 1)) * step; }
    __device__ __forceinline__ void fill(int i) const {
        if (act && i < n) cp_async8(slot(i), src + (size_t)i * stride);
    }
};

template <int K, bool GUARD, typename Emit>
__device__ __forceinline__ void stream_block(const Ring &rg, int base, const StepConst &c,
                                             unsigned long long (&acc)[K], Emit &emit) {
#pragma unroll
    for (int j = 0; j < K; ++j) {
        const int i = base + j;
        if (GUARD && i >= rg.n) break;
        if (i > 0) {
            rg.fill(i - 1 + RING);
            cp_commit();
        }
        cp_wait_ring();
        const unsigned long long v = *reinterpret_cast<const unsigned long long *>(rg.slot(i));
#pragma unroll
        for (int tt = 0; tt < K; ++tt) {
            const int slot = (j - tt + K) % K;
            acc[slot] = fma2(v, c.tap2(tt), tt == 0 ? 0ull : acc[slot]);
        }
        const int o = i - (K - 1);
        if (o >= 0) emit(o, unpack2(acc[(j + 1) % K]), i);
    }
}

template <int K, typename Emit>
__device__ __forceinline__ void stream_axis(const Ring &rg, const StepConst &c, Emit &emit) {
#pragma unroll
    for (int q = 0; q < RING; ++q) {
        rg.fill(q);
        cp_commit();
    }
    unsigned long long acc[K];
#pragma unroll
    for (int j = 0; j < K; ++j) acc[j] = 0ull;
    int base = 0;
    for (; base + K <= rg.n; base += K) stream_block<K, false>(rg, base, c, acc, emit);
    if (base < rg.n) stream_block<K, true>(rg, base, c, acc, emit);
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// Register-blocked version for a tap count known only at run time: NB
// consecutive outputs per call, same accumulation order.
template <int NB>
__device__ __forceinline__ void conv_block_rt(const float *__restrict__ base, size_t stride, int start, int n,
                                              const float *taps_s, int k, float (&acc)[NB]) {
#pragma unroll
    for (int m = 0; m < NB; ++m) acc[m] = 0.0f;
    for (int q = 0; q < NB + k - 1; ++q) {
        const int p = start + q;
        const float v = (p >= 0 && p < n) ? __ldg(base + (size_t)p * stride) : 0.0f;
#pragma unroll
        for (int m = 0; m < NB; ++m) {
            const int tt = q - m;
            if (tt >= 0 && tt < k) acc[m] = __fmaf_rn(v, taps_s[tt], acc[m]);
        }
    }
}

// ---------------------------------------------------------------------------
// y-pass.  One thread streams one column of one pair (every other float2 of
// the interleaved fields): the 2 Wp float2 columns of a z plane, over all
// planes, are numbered consecutively, and each is cut into c.yout outputs.
// ---------------------------------------------------------------------------
template <int K>
__global__ void __launch_bounds__(YP_COLS) ypass_kernel(const SubVolDev *__restrict__ svs,
                                                        const int *__restrict__ pre,
                                                        const __grid_constant__ StepConst c) {
    const int b = blockIdx.x;
    const int sv = find_sv(pre, c.nsv, b);
    const SubVolDev s = svs[sv];
    const int row = 2 * s.Wp, t = b - __ldg(pre + sv);
    const int ntq = (int)(((long long)row * s.L + YP_COLS - 1) / YP_COLS);
    const long long q = (long long)(t % ntq) * YP_COLS + threadIdx.x;
    const int y0 = (t / ntq) * c.yout;
    const int z = (int)(q / row), x = (int)(q - (long long)z * row);
    __shared__ float2 ring[RING * YP_COLS];
    pdl_wait();
    if (z >= s.L || x >= 2 * s.Wv) return;
    const float *src = s.xb + 2 * (((size_t)z * s.H + y0) * row + x);
    float2 *dst = reinterpret_cast<float2 *>(s.yb) + ((size_t)z * s.Hv + y0) * row + x;
    // The y-pass is bound by HBM bandwidth: it keeps the deeper 8-slot ring
    // (more loads in flight) rather than the compile-time-slot ring.
    auto emit = [&](int o, float2 v, int) { dst[(size_t)o * row] = v; };
    const Ring rg = {ring + threadIdx.x, YP_COLS, src, 2 * (size_t)row, min(c.yout, s.Hv - y0) + K - 1, true};
    stream_axis<K>(rg, c, emit);
    pdl_launch();
}

// Run-time tap count: a thread forms YG_NB consecutive outputs of its column.
// The taps go in chunks of YG_NB over a window of 2 YG_NB inputs in registers,
// whose upper half is loaded a chunk ahead, so a tap costs YG_NB multiply-adds,
// one load and no index test.
template <int NB, class Const, class Load>
__device__ __forceinline__ void conv_chunks(const Const &c, Load load, unsigned long long (&u)[NB]) {
    unsigned long long w[2 * NB];
#pragma unroll
    for (int m = 0; m < NB; ++m) {
        u[m] = 0ull;
        w[m] = load(m);
    }
    for (int t0 = 0; t0 < c.k; t0 += NB) {
#pragma unroll
        for (int m = 0; m < NB; ++m) w[NB + m] = load(t0 + NB + m);
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            if (t0 + j >= c.k) break;
            const unsigned long long g = c.tap2(t0 + j);
#pragma unroll
            for (int m = 0; m < NB; ++m) u[m] = fma2(w[m + j], g, u[m]);
        }
#pragma unroll
        for (int m = 0; m < NB; ++m) w[m] = w[NB + m];
    }
}

template <int NB>
__global__ void __launch_bounds__(YP_COLS) ypass_chunk_kernel(const SubVolDev *__restrict__ svs,
                                                              const int *__restrict__ pre,
                                                              const __grid_constant__ StepConst c) {
    const int b = blockIdx.x;
    const int sv = find_sv(pre, c.nsv, b);
    const SubVolDev s = svs[sv];
    const int row = 2 * s.Wp;
    const int t = b - __ldg(pre + sv);
    pdl_wait();
    const int ntq = (int)(((long long)row * s.L + YP_COLS - 1) / YP_COLS);
    const long long q = (long long)(t % ntq) * YP_COLS + threadIdx.x;
    const int y0 = (t / ntq) * NB;
    const int z = (int)(q / row), x = (int)(q - (long long)z * row);
    if (z >= s.L || x >= 2 * s.Wv) return;
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(s.xb) +
                                    ((size_t)z * s.H + y0) * row + x;
    unsigned long long *dst = reinterpret_cast<unsigned long long *>(s.yb) + ((size_t)z * s.Hv + y0) * row + x;
    const int have = min(s.H - y0, NB + c.k - 1);
    unsigned long long u[NB];
    conv_chunks<NB>(c, [&](int i) { return i < have ? src[(size_t)i * row] : 0ull; }, u);
#pragma unroll
    for (int m = 0; m < NB; ++m)
        if (y0 + m < s.Hv) dst[(size_t)m * row] = u[m];
    pdl_launch();
}

// ---------------------------------------------------------------------------
// z-pass.  One thread streams one column of all four fields (float4 elements),
// so that it forms both local fits of its voxel by itself: 2 K rotating
// accumulator pairs, inputs through a per-thread ring of float4 slots filled by
// cp.async.  The kernel is bound by instruction issue, and everything but the
// multiply-adds is paid once per voxel this way (with the two pairs on
// different lanes it took 186 thread instructions per voxel, 21 taps, and
// 6.78 ms per launch on the 48 sub-volumes of 946 M voxels; now 3.72 ms).
// The ring's depth divides the taps (7 for 21 and 35; K for 11, 15 and 29), so every
// slot index of a K-element block is a constant; element i is commit group i,
// and iteration i refills the slot of element i-1 with element i-1+RD before it
// waits for group i.  A block takes ZP_COLS columns, numbered consecutively
// over the padded rows of a plane, and c.zout output planes.
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int ring_depth(int K) { return K % 7 == 0 ? 7 : K; }
__host__ __device__ constexpr size_t zpass_smem(int K) { return (size_t)ring_depth(K) * ZP_COLS * sizeof(float4); }

// One block of K elements.  The steady form has no branch, so that the fits of
// one element overlap the multiply-adds of the next (with the end tested inside
// it, and one copy of the body for start, middle and end, the 21-tap kernel
// took 6.4 ms per launch instead of 3.5).
template <int K, bool FIRST, bool GUARD, class Fill, class Emit>
__device__ __forceinline__ void zstream_block(const ulonglong2 *ring, int left, const StepConst &c,
                                              unsigned long long (&a)[K], unsigned long long (&b)[K], Fill &fill,
                                              Emit &emit) {
    constexpr int RD = ring_depth(K);
#pragma unroll
    for (int j = 0; j < K; ++j) {
        if (GUARD && j >= left) break;
        fill((j - 1 + RD) % RD);
        asm volatile("cp.async.wait_group %0;" ::"n"(RD - 1) : "memory");
        const ulonglong2 v = ring[(j % RD) * ZP_COLS];
#pragma unroll
        for (int tt = 0; tt < K; ++tt) {
            const int s = (j - tt + K) % K;
            if (FIRST && tt > j) continue;  // an output that starts before element 0
            a[s] = fma2(v.x, c.tap2(tt), tt == 0 ? 0ull : a[s]);
            b[s] = fma2(v.y, c.tap2(tt), tt == 0 ? 0ull : b[s]);
        }
        if (!FIRST || j == K - 1) emit(unpack2(a[(j + 1) % K]), unpack2(b[(j + 1) % K]));
    }
}

// Rotating accumulation of n inputs (n >= K) src[i * stride]: hands
// emit(pair 0, pair 1) the outputs 0 .. n - K in order.
template <int K, class Emit>
__device__ __forceinline__ void zstream(const float4 *src, size_t stride, int n, const StepConst &c, Emit emit) {
    constexpr int RD = ring_depth(K);
    extern __shared__ ulonglong2 zring_s[];
    ulonglong2 *ring = zring_s + threadIdx.x;
    const float4 *next = src;
    int unread = n;
    auto fill = [&](int slot) {
        if (unread > 0) {
            const unsigned d = (unsigned)__cvta_generic_to_shared(ring + slot * ZP_COLS);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(next) : "memory");
        }
        next += stride;  // addresses past the end are formed but never read
        --unread;
        cp_commit();
    };
#pragma unroll
    for (int q = 0; q + 1 < RD; ++q) fill(q);
    unsigned long long a[K], b[K];
    zstream_block<K, true, false>(ring, K, c, a, b, fill, emit);
    int left = n - K;
    for (; left >= K; left -= K) zstream_block<K, false, false>(ring, left, c, a, b, fill, emit);
    if (left > 0) zstream_block<K, false, true>(ring, left, c, a, b, fill, emit);
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// The column of this thread: offset p within a plane of the padded fields, valid
// x and y, outputs [o0, o0 + n).
struct ZCol {
    size_t p, plane;   // plane: Wp * Hv
    int x, y, o0, n;
    bool live;
};
__device__ __forceinline__ ZCol zcol_of(const SubVolDev &s, const StepConst &c, int t) {
    ZCol z;
    z.plane = (size_t)s.Wp * s.Hv;
    const int ntp = (int)((z.plane + ZP_COLS - 1) / ZP_COLS);
    z.p = (size_t)(t % ntp) * ZP_COLS + threadIdx.x;
    z.y = (int)(z.p / s.Wp);
    z.x = (int)(z.p - (size_t)z.y * s.Wp);
    z.o0 = (t / ntp) * c.zout;
    z.n = min(c.zout, s.Lv - z.o0);
    z.live = z.p < z.plane && z.x < s.Wv;
    return z;
}

// The image at an address, as the bits that image_value turns into a float
// once it is needed (loads run three outputs ahead).
__device__ __forceinline__ unsigned image_bits(const unsigned char *ip, int f32) {
    return f32 ? __ldg(reinterpret_cast<const unsigned *>(ip)) : (unsigned)__ldg(ip);
}
__device__ __forceinline__ float image_value(unsigned w, int f32) { return f32 ? __uint_as_float(w) : (float)w; }

template <int K>
__global__ void __launch_bounds__(ZP_COLS, zpass_blocks(K)) zpass_kernel(const SubVolDev *__restrict__ svs,
                                                                         const int *__restrict__ pre,
                                                                         const __grid_constant__ StepConst c) {
    const int blk = blockIdx.x;
    const int sv = find_sv(pre, c.nsv, blk);
    const SubVolDev s = svs[sv];
    const ZCol z = zcol_of(s, c, blk - __ldg(pre + sv));
    pdl_wait();
    if (!z.live) return;  // no barrier or shuffle below
    const size_t esz = c.img_f32 ? 4 : 1, istep = (size_t)s.W * s.H * esz;
    const unsigned char *ip = static_cast<const unsigned char *>(s.img) +
                              (((size_t)(z.o0 + c.r) * s.H + (z.y + c.r)) * s.W + (z.x + c.r)) * esz;
    float *db = s.db + (size_t)z.o0 * z.plane + z.p;
    int unread = z.n;  // image words not yet loaded
    auto image = [&] {
        const unsigned w = unread > 0 ? image_bits(ip, c.img_f32) : 0u;
        ip += istep;
        --unread;
        return w;
    };
    unsigned i0 = image(), i1 = image(), i2 = image();
    zstream<K>(reinterpret_cast<const float4 *>(s.yb) + (size_t)z.o0 * z.plane + z.p, z.plane, z.n + K - 1, c,
               [&](float2 h, float2 ih) {
                   const float I = image_value(i0, c.img_f32);
                   i0 = i1;
                   i1 = i2;
                   i2 = image();
                   const float2 f = div2(ih, h);  // f_out, f_in
                   const float d0 = __fsub_rn(I, f.x), d1 = __fsub_rn(I, f.y);
                   *db = data_factor(__fmul_rn(d0, d0), __fmul_rn(d1, d1), c.l1, c.l2, c.lam_equal != 0);
                   db += z.plane;
               });
    pdl_launch();
}

// Run-time tap count: ZG_NB outputs of one column of all four fields per thread,
// in chunks as the y-pass.  emit(m, h, ih) gets output m's pairs.
template <int NB, class Emit>
__device__ __forceinline__ void zchunk(const SubVolDev &s, const StepConst &c, const ZCol &z, Emit emit) {
    const ulonglong2 *src = reinterpret_cast<const ulonglong2 *>(s.yb) + (size_t)z.o0 * z.plane + z.p;
    const int have = min(s.L - z.o0, NB + c.k - 1);
    ulonglong2 w[2 * NB];
    unsigned long long a[NB], b[NB];
    auto load = [&](int i) { return i < have ? src[(size_t)i * z.plane] : make_ulonglong2(0ull, 0ull); };
#pragma unroll
    for (int m = 0; m < NB; ++m) {
        a[m] = b[m] = 0ull;
        w[m] = load(m);
    }
    for (int t0 = 0; t0 < c.k; t0 += NB) {
#pragma unroll
        for (int m = 0; m < NB; ++m) w[NB + m] = load(t0 + NB + m);
#pragma unroll
        for (int j = 0; j < NB; ++j) {
            if (t0 + j >= c.k) break;
            const unsigned long long g = c.tap2(t0 + j);
#pragma unroll
            for (int m = 0; m < NB; ++m) {
                a[m] = fma2(w[m + j].x, g, a[m]);
                b[m] = fma2(w[m + j].y, g, b[m]);
            }
        }
#pragma unroll
        for (int m = 0; m < NB; ++m) w[m] = w[NB + m];
    }
#pragma unroll
    for (int m = 0; m < NB; ++m)
        if (m < z.n) emit(m, unpack2(a[m]), unpack2(b[m]));
}

template <bool DEBUG>
__global__ void __launch_bounds__(ZP_COLS) zpass_chunk_kernel(const SubVolDev *__restrict__ svs,
                                                              const int *__restrict__ pre,
                                                              const __grid_constant__ StepConst c, DebugOut dbg) {
    const int blk = blockIdx.x;
    const int sv = find_sv(pre, c.nsv, blk);
    const SubVolDev s = svs[sv];
    const ZCol z = zcol_of(s, c, blk - __ldg(pre + sv));
    pdl_wait();
    if (!z.live) return;
    const size_t v0 = ((size_t)(z.o0 + c.r) * s.H + (z.y + c.r)) * s.W + (z.x + c.r), plane = (size_t)s.W * s.H;
    zchunk<ZG_NB>(s, c, z, [&](int m, float2 h, float2 ih) {
        const size_t vi = v0 + (size_t)m * plane, di = (size_t)(z.o0 + m) * z.plane + z.p;
        const float2 f = div2(ih, h);  // f_out, f_in
        if (DEBUG) {
            dbg.f[0 * dbg.n + vi] = f.x;
            dbg.f[1 * dbg.n + vi] = f.y;
        }
        if (c.full_data) {  // the box or expanded data-term kernels form e from the fits
            s.db[di] = f.x;
            s.db[z.plane * s.Lv + di] = f.y;
            return;
        }
        const float I = load_img(s.img, vi, c.img_f32);
        const float d_o = __fsub_rn(I, f.x), d_i = __fsub_rn(I, f.y);
        const float eo = __fmul_rn(d_o, d_o), ei = __fmul_rn(d_i, d_i);
        s.db[di] = data_factor(eo, ei, c.l1, c.l2, c.lam_equal != 0);
        if (DEBUG) {
            dbg.f[2 * dbg.n + vi] = eo;
            dbg.f[3 * dbg.n + vi] = ei;
        }
    });
    pdl_launch();
}

// The adjoint's recompute of the fits (rsf_adjoint.cu): the forward z-pass,
// emitting at each valid voxel, instead of the data factor,
//   e_out = (I - f_out)^2 and e_in at the full-volume index, and the pair
//   (B1_bar - B3_bar, B2_bar - B4_bar) as a float2 in the valid layout (row
//   stride Wv),
// with B1..B4 the blurs of I H, H, I (1-H), 1-H, f_out = B1 / B2,
// f_in = B3 / B4, and for data_bar = -u dt delta(phi)
//   f_out_bar = -2 (I - f_out) lambda1 data_bar, f_in_bar = 2 (I - f_in) lambda2 data_bar,
//   B1_bar = f_out_bar / B2, B2_bar = -f_out_bar f_out / B2 (B3, B4 alike).
// The pair goes to a.xs (2 Wv Hv Lv floats), e_out and e_in to a.xs + 2 N and
// a.xs + 3 N.
struct AdjFits {
    float eo, ei, p, q;
};
__device__ __forceinline__ AdjFits adjoint_fits(const StepConst &c, float I, float ph, float uo, float2 h, float2 ih) {
    const float delta = __fdividef(0.318309886183790672f * c.eps, fmaf(ph, ph, c.eps * c.eps));
    const float data_bar = -uo * c.dt * delta;
    auto side = [&](float num, float den, float weight, float &bn, float &bd) {
        const float rb = __frcp_rn(den);
        const float fv = num * rb;
        const float d = I - fv;
        const float fbar = -2.0f * d * (weight * data_bar);
        bn = fbar * rb;
        bd = -fbar * fv * rb;
        return d * d;
    };
    float bn0, bd0, bn1, bd1;
    const float eo = side(ih.x, h.x, c.l1, bn0, bd0), ei = side(ih.y, h.y, -c.l2, bn1, bd1);
    return {eo, ei, bn0 - bn1, bd0 - bd1};
}

// phi and u of the next three output planes ride in registers with the image.
template <int K>
__global__ void __launch_bounds__(ZP_COLS, zpass_blocks(K)) zpass_adjoint_kernel(const SubVolDev *__restrict__ svs,
                                                                                 const int *__restrict__ pre,
                                                                                 const __grid_constant__ StepConst c,
                                                                                 const AdjVol *__restrict__ vols) {
    const int blk = blockIdx.x;
    const int sv = find_sv(pre, c.nsv, blk);
    const SubVolDev s = svs[sv];
    const AdjVol a = vols[sv];
    const ZCol z = zcol_of(s, c, blk - __ldg(pre + sv));
    if (!z.live) return;
    const size_t esz = c.img_f32 ? 4 : 1, plane = (size_t)s.W * s.H;
    size_t v = ((size_t)(z.o0 + c.r) * s.H + (z.y + c.r)) * s.W + (z.x + c.r);  // the next load's voxel
    float *eo = a.xs + 2 * plane * s.L + v, *ei = eo + plane * s.L;
    const size_t vplane = (size_t)s.Wv * s.Hv;
    float2 *pq = reinterpret_cast<float2 *>(a.xs) + (size_t)z.o0 * vplane + (size_t)z.y * s.Wv + z.x;
    struct In {
        unsigned i;
        float phi, u;
    };
    int unread = z.n;
    auto load = [&] {
        In n = {0u, 0.0f, 0.0f};
        if (unread > 0)
            n = In{image_bits(static_cast<const unsigned char *>(s.img) + v * esz, c.img_f32), __ldg(a.phi + v),
                   __ldg(a.u + v)};
        v += plane;
        --unread;
        return n;
    };
    In n0 = load(), n1 = load(), n2 = load();
    zstream<K>(reinterpret_cast<const float4 *>(s.yb) + (size_t)z.o0 * z.plane + z.p, z.plane, z.n + K - 1, c,
               [&](float2 h, float2 ih) {
                   const float I = image_value(n0.i, c.img_f32), ph = n0.phi, uo = n0.u;
                   n0 = n1;
                   n1 = n2;
                   n2 = load();
                   const AdjFits f = adjoint_fits(c, I, ph, uo, h, ih);
                   *eo = f.eo;
                   *ei = f.ei;
                   *pq = make_float2(f.p, f.q);
                   eo += plane;
                   ei += plane;
                   pq += vplane;
               });
}

template <int NB>
__global__ void __launch_bounds__(ZP_COLS) zchunk_adjoint_kernel(const SubVolDev *__restrict__ svs,
                                                                 const int *__restrict__ pre,
                                                                 const __grid_constant__ StepConst c,
                                                                 const AdjVol *__restrict__ vols) {
    const int blk = blockIdx.x;
    const int sv = find_sv(pre, c.nsv, blk);
    const SubVolDev s = svs[sv];
    const AdjVol a = vols[sv];
    const ZCol z = zcol_of(s, c, blk - __ldg(pre + sv));
    if (!z.live) return;
    const size_t plane = (size_t)s.W * s.H, n = plane * s.L;
    const size_t v0 = ((size_t)(z.o0 + c.r) * s.H + (z.y + c.r)) * s.W + (z.x + c.r);
    const size_t vplane = (size_t)s.Wv * s.Hv;
    float2 *pq = reinterpret_cast<float2 *>(a.xs) + (size_t)z.o0 * vplane + (size_t)z.y * s.Wv + z.x;
    zchunk<NB>(s, c, z, [&](int m, float2 h, float2 ih) {
        const size_t v = v0 + (size_t)m * plane;
        const AdjFits f = adjoint_fits(c, load_img(s.img, v, c.img_f32), __ldg(a.phi + v), __ldg(a.u + v), h, ih);
        a.xs[2 * n + v] = f.eo;
        a.xs[3 * n + v] = f.ei;
        pq[(size_t)m * vplane] = make_float2(f.p, f.q);
    });
}

// ---------------------------------------------------------------------------
// Stencil / update.  A block is ST_WARPS warps, one image row each (rows
// y0-1 .. y0+ST_OY; the outer two are halo rows), 32 lanes wide (columns
// x0-1 .. x0+30; lanes 0 and 31 are halo columns), streaming c.zc planes.
// Each step computes the gradient / normalised gradient of plane s+1 once
// per thread, exchanges x neighbours by warp shuffles and y neighbours
// through triple-buffered shared rows (one barrier per plane), and writes the
// updated phi of plane s.
// ---------------------------------------------------------------------------
struct GN {
    float gx, gy, gz, nx, ny, nz;
};

template <Arith A>
__device__ __forceinline__ GN gn_from(float xl, float xr, float yl, float yr, float zl, float zr) {
    GN g;
    g.gx = half_diff(xr, xl);
    g.gy = half_diff(yr, yl);
    g.gz = half_diff(zr, zl);
    const NormDen d = norm_den<A>(grad_mag(g.gx, g.gy, g.gz));
    g.nx = normalise<A>(g.gx, d);
    g.ny = normalise<A>(g.gy, d);
    g.nz = normalise<A>(g.gz, d);
    return g;
}

// Gradient and normalised gradient at (x, y, z) straight from global memory
// with the boundary rules of kernel.cu:57-125; used for the previous-row
// neighbour that x = 0 reads in the reference boundary mode.
template <Arith A>
__device__ __forceinline__ GN gn_global(const float *__restrict__ phi, int x, int y, int z, int W, int H, int L,
                                     int boundary) {
    const size_t WH = (size_t)W * H;
    auto at = [&](int xx, int yy, int zz) { return __ldg(phi + (size_t)zz * WH + (size_t)yy * W + xx); };
    const float c0 = at(x, y, z);
    float xl;
    if (x > 0) xl = at(x - 1, y, z);
    else if (boundary == 0) {
        if (y > 0) xl = at(W - 1, y - 1, z);
        else if (z > 0) xl = at(W - 1, H - 1, z - 1);
        else xl = c0;
    } else xl = c0;
    const float xr = x < W - 1 ? at(x + 1, y, z) : c0;
    const float yl = y > 0 ? at(x, y - 1, z) : c0, yr = y < H - 1 ? at(x, y + 1, z) : c0;
    const float zl = z > 0 ? at(x, y, z - 1) : c0, zr = z < L - 1 ? at(x, y, z + 1) : c0;
    return gn_from<A>(xl, xr, yl, yr, zl, zr);
}

// Per-block state of the stencil kernel.  Planes are numbered relative to
// the block's first step; every ring below is indexed by (relative plane mod
// 3), which the 3-way unrolled step loop turns into compile-time register and
// shared-memory slots.
struct StencilCtx {
    const SubVolDev *s;
    const float *phi;       // this thread's column of phi (plane 0 at offset 0)
    float *phi_out;
    const float *dcol;      // this thread's column of the data factor (plane r)
    size_t WH, dplane;
    int W, H, L, r, x, y, w, lane, z0, z1, first;
    bool in, outp, ref, inside_xy, blk_inside;
    bool need_x, need_y;
    ptrdiff_t xoff, yoff;   // offsets of the extra neighbour loads
    size_t col;
};

// nx, gx, nz, gz of a plane (ny, gy live in the shared rows)
struct GN4 {
    float nx, gx, nz, gz;
};

struct StencilState {
    float P[3];     // phi of the planes
    float EX[3];    // extra x neighbour
    float EY[3];    // extra y neighbour
    float DT[3];    // data factor of the planes
    GN4 G[3];       // gradient / normalised gradient of the planes
};

__device__ __forceinline__ float st_ld(const StencilCtx &k, int p) {
    return (k.in && p >= 0 && p < k.L) ? __ldg(k.phi + (size_t)p * k.WH) : 0.0f;
}
__device__ __forceinline__ float st_ldx(const StencilCtx &k, int p) {
    if (!k.need_x || p < 0 || p >= k.L) return 0.0f;
    // previous linear element of voxel 0 is defined as voxel 0 itself
    if (k.xoff < 0 && p == 0 && k.col == 0) return __ldg(k.phi);
    return __ldg(k.phi + (ptrdiff_t)((size_t)p * k.WH) + k.xoff);
}
__device__ __forceinline__ float st_ldy(const StencilCtx &k, int p) {
    return (k.need_y && p >= 0 && p < k.L) ? __ldg(k.phi + (ptrdiff_t)((size_t)p * k.WH) + k.yoff) : 0.0f;
}
// data factor at plane p: from the z-pass inside the valid region, from
// f_out = f_in = 30/30 = 1 in the border band (kernel.cu:300-325).
__device__ __forceinline__ float st_data(const StencilCtx &k, const StepConst &c, int p) {
    if (!k.outp || p < k.z0 || p >= k.z1) return 0.0f;
    if (k.blk_inside || (k.inside_xy && p >= k.r && p < k.L - k.r))
        return __ldg(k.dcol + (ptrdiff_t)((size_t)p * k.dplane) - (ptrdiff_t)((size_t)k.r * k.dplane));
    const float I = load_img(k.s->img, (size_t)p * k.WH + k.col, c.img_f32);
    const float d = __fsub_rn(I, 1.0f);
    const float e = __fmul_rn(d, d);
    return data_factor(e, e, c.l1, c.l2, c.lam_equal != 0);
}

template <int C, Arith A>
__device__ __forceinline__ void stencil_step(const StencilCtx &k, const StepConst &c, StencilState &S, int rel,
                                             float (*Pb)[ST_WARPS + 2][32], float2 (*Gb)[ST_WARPS][32],
                                             unsigned *flag, const DebugOut &dbg) {
    constexpr int C1 = (C + 1) % 3, C2 = (C + 2) % 3;
    const int sc = k.first + rel;  // output plane of this step
    const int pn = sc + 1;         // plane whose gradient this step computes
    // prefetch for the next steps
    const float p3 = st_ld(k, sc + 3);
    const float exn = st_ldx(k, sc + 3), eyn = st_ldy(k, sc + 3);
    const float dn = st_data(k, c, sc + 1);
    Pb[C2][k.w + 1][k.lane] = S.P[C2];
    const float p0 = S.P[C], p1 = S.P[C1], p2 = S.P[C2];
    float L1 = __shfl_up_sync(0xffffffffu, p1, 1);
    float R1 = __shfl_down_sync(0xffffffffu, p1, 1);
    if (k.need_x && k.xoff < 0) L1 = S.EX[C1];
    if (k.need_x && k.xoff > 0) R1 = S.EX[C1];
    const float U1 = k.w > 0 ? Pb[C1][k.w][k.lane] : S.EY[C1];
    const float D1 = k.w < ST_WARPS - 1 ? Pb[C1][k.w + 2][k.lane] : S.EY[C1];
    GN gn = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (k.in && pn >= 0 && pn < k.L) {
        const float xl = (k.x > 0 || k.ref) ? L1 : p1;
        const float xr = k.x < k.W - 1 ? R1 : p1;
        const float yl = k.y > 0 ? U1 : p1, yr = k.y < k.H - 1 ? D1 : p1;
        const float zl = pn > 0 ? p0 : p1, zr = pn < k.L - 1 ? p2 : p1;
        gn = gn_from<A>(xl, xr, yl, yr, zl, zr);
    }
    S.G[C1] = GN4{gn.nx, gn.gx, gn.nz, gn.gz};
    Gb[C1][k.w][k.lane] = make_float2(gn.ny, gn.gy);
    __syncthreads();
    const GN4 &gc = S.G[C];
    const float nxL = __shfl_up_sync(0xffffffffu, gc.nx, 1), nxR = __shfl_down_sync(0xffffffffu, gc.nx, 1);
    const float gxL = __shfl_up_sync(0xffffffffu, gc.gx, 1), gxR = __shfl_down_sync(0xffffffffu, gc.gx, 1);
    if (sc >= k.z0 && k.outp) {
        float nxl = nxL, gxl = gxL;
        if (k.x == 0) {
            if (k.ref && (k.y > 0 || sc > 0)) {
                const float *phi0 = k.phi - k.col;  // plane 0, voxel 0
                const GN wg = k.y > 0 ? gn_global<A>(phi0, k.W - 1, k.y - 1, sc, k.W, k.H, k.L, c.boundary)
                                      : gn_global<A>(phi0, k.W - 1, k.H - 1, sc - 1, k.W, k.H, k.L, c.boundary);
                nxl = wg.nx;
                gxl = wg.gx;
            } else {
                nxl = gc.nx;
                gxl = gc.gx;
            }
        }
        const bool xr_in = k.x < k.W - 1;
        const float nxr = xr_in ? nxR : gc.nx, gxr = xr_in ? gxR : gc.gx;
        const int wl = k.y > 0 ? k.w - 1 : k.w, wr = k.y < k.H - 1 ? k.w + 1 : k.w;
        const float2 yl2 = Gb[C][wl][k.lane], yr2 = Gb[C][wr][k.lane];
        const float nyl = yl2.x, nyr = yr2.x, gyl = yl2.y, gyr = yr2.y;
        const GN4 &gp = S.G[C2];
        const float nzl = sc > 0 ? gp.nz : gc.nz, nzr = sc < k.L - 1 ? gn.nz : gc.nz;
        const float gzl = sc > 0 ? gp.gz : gc.gz, gzr = sc < k.L - 1 ? gn.gz : gc.gz;
        const float kap = __fadd_rn(__fadd_rn(half_diff(nxr, nxl), half_diff(nyr, nyl)), half_diff(nzr, nzl));
        const float lap = __fadd_rn(__fadd_rn(half_diff(gxr, gxl), half_diff(gyr, gyl)), half_diff(gzr, gzl));
        const float dh = dirac<A>(p0, c.eps);
        const float out = update_phi(p0, dh, S.DT[C], kap, lap, c.dt, c.nu, c.mu);
        const size_t vi = (size_t)sc * k.WH + k.col;
        k.phi_out[vi] = out;
        if (!isfinite(out)) atomicOr(flag, kFlagNonFinite);
        const bool inside = k.inside_xy && sc >= k.r && sc < k.L - k.r;
        if (!inside) {
            dbg.f[0 * dbg.n + vi] = 1.0f;
            dbg.f[1 * dbg.n + vi] = 1.0f;
            if (!c.full_data) {  // else the data-term kernels wrote e everywhere
                const float I = load_img(k.s->img, vi, c.img_f32);
                const float d = __fsub_rn(I, 1.0f);
                dbg.f[2 * dbg.n + vi] = __fmul_rn(d, d);
                dbg.f[3 * dbg.n + vi] = __fmul_rn(d, d);
            }
        }
        dbg.f[4 * dbg.n + vi] = dh;
        dbg.f[5 * dbg.n + vi] = kap;
        dbg.f[6 * dbg.n + vi] = lap;
        dbg.f[7 * dbg.n + vi] = grad_mag(gc.gx, Gb[C][k.w][k.lane].y, gc.gz);
    }
    S.P[C] = p3;    // plane rel+3
    S.EX[C] = exn;  // plane rel+3
    S.EY[C] = eyn;
    S.DT[C1] = dn;  // plane rel+1
}

// ---------------------------------------------------------------------------
// Box e-term, CUDA_RSF/kernel.cu:25-55 with s = (int)sigma2 >= 1: for every
// voxel c, e = sum over the neighbours n of the (2s+1)^3 box that lie inside
// the volume of w (I_n - f(c))^2, w = 1/(2s+1)^2, accumulated in the
// reference's order (y outer, then x, then z) with each term fused in double
// and rounded to float.  f(c) comes from the z-pass in the valid region and
// is 30/30 = 1 in the border band.  Writes the data factor of every voxel;
// runs on the stencil's tiling (lanes 1..30 x warps 1..14 x c.zc planes), a
// grid row per BOX_Z of the planes or fewer.
//
// Double precision is what bounds the sum in its own terms (four operations
// and six conversions per neighbour on a pipe with 1/64 of the FP32 rate), so
// the terms are formed in pairs of floats (d^2 and w d^2 by their exact residuals,
// the sum by Knuth's two-sum), e_out and e_in in the two lanes of packed
// instructions.  That gives the sum to within 2^-45 of its size, while the
// double sequence is within 2^-52; where the two ends of a 2^-43 margin round
// to the same float, that float is the reference's.  Elsewhere the z column is
// redone in double.  For s = 1 that is one column in 3000 to 4000 with fractional
// fits (random values, restated on the CPU), but one in 15 where f = 1 meets an integer
// image, in the border band: w d^2 is then whole for every third d, and most warps
// go there.  With equal weights and a byte image the border needs no sum.
// 72x100x131 voxels, half of them border, s = 1, a whole iteration: 1259 us with
// the sums in double, 118 for bytes and equal weights (box kernel 60; 67 with a grid
// row per plane), 377 with unequal weights or a float image of integers, 162 with a
// fractional one.
// ---------------------------------------------------------------------------
// One z column of the box in double, from the sums before it.
static __device__ __noinline__ float2 box_column_double(const void *img, size_t i, size_t step, int n, int f32,
                                                        double wt, float fo, float fi, float2 s) {
    for (int q = 0; q < n; ++q) {
        const float In = load_img(img, i + (size_t)q * step, f32);
        const float d1 = __fsub_rn(In, fo), d2 = __fsub_rn(In, fi);
        s.x = __double2float_rn(__fma_rn(__dmul_rn(wt, (double)d1), (double)d1, (double)s.x));
        s.y = __double2float_rn(__fma_rn(__dmul_rn(wt, (double)d2), (double)d2, (double)s.y));
    }
    return s;
}

template <bool DEBUG>
__global__ void __launch_bounds__(ST_WARPS * 32, 2) box_kernel(const SubVolDev *__restrict__ svs,
                                                            const int *__restrict__ pre, const StepConst c,
                                                            DebugOut dbg) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int b = blockIdx.x;
    const int sv = find_sv(pre, c.nsv, b);
    const SubVolDev &s = svs[sv];
    int t = b - __ldg(pre + sv);
    const int ntx = (s.W + ST_OX - 1) / ST_OX, nty = (s.H + ST_OY - 1) / ST_OY;
    const int tx = t % ntx;
    t /= ntx;
    const int ty = t % nty;
    const int tz = t / nty;
    const int x = tx * ST_OX - 1 + lane, y = ty * ST_OY - 1 + w;
    if (lane < 1 || lane > ST_OX || w < 1 || w > ST_OY || x >= s.W || y >= s.H) return;
    const int zb = (c.zc + (int)gridDim.y - 1) / (int)gridDim.y;  // planes per grid row
    const int z0 = tz * c.zc + (int)blockIdx.y * zb, z1 = min(min(z0 + zb, tz * c.zc + c.zc), s.L);
    const int bs = c.box, r = c.r;
    const double wt = 1.0 / (double)((2 * bs + 1) * (2 * bs + 1));
    const float2 wh = dup2((float)wt), wl = dup2((float)(wt - (double)(float)wt));
    const size_t WH = (size_t)s.W * s.H, nvalid = (size_t)s.Wp * s.Hv * s.Lv;
    float *dfull = s.db + 2 * nvalid;
    const bool valid_xy = s.Wv > 0 && x >= r && x < r + s.Wv && y >= r && y < r + s.Hv;
    for (int z = z0; z < z1; ++z) {
        const size_t vi = (size_t)z * WH + (size_t)y * s.W + x;
        float fo = 1.0f, fi = 1.0f;
        if (valid_xy && z >= r && z < r + s.Lv) {
            const size_t di = ((size_t)(z - r) * s.Hv + (y - r)) * s.Wp + (x - r);
            fo = s.db[di];
            fi = s.db[nvalid + di];
        } else if (!DEBUG && c.lam_equal && !c.img_f32) {
            dfull[vi] = data_factor(0.0f, 0.0f, c.l1, c.l2, true);
            continue;
        }
        // fits of at least 2^-20 keep every nonzero difference above 2^-45 and
        // its square's residuals in the normal range
        const bool exact = fabsf(fo) >= 0x1p-20f && fabsf(fi) >= 0x1p-20f;
        const int q0 = max(z - bs, 0), nq = min(z + bs, s.L - 1) - q0 + 1;
        float2 e = make_float2(0.0f, 0.0f);
        for (int yy = max(y - bs, 0); yy <= min(y + bs, s.H - 1); ++yy) {
            for (int xx = max(x - bs, 0); xx <= min(x + bs, s.W - 1); ++xx) {
                const size_t i0 = (size_t)q0 * WH + (size_t)yy * s.W + xx;
                float2 sum = e;
                bool sure = exact;
                for (int qc = 0; qc < nq; qc += 3) {
                    float In[3];  // loads of three terms in flight together
#pragma unroll
                    for (int m = 0; m < 3; ++m)
                        In[m] = qc + m < nq ? load_img(s.img, i0 + (size_t)(qc + m) * WH, c.img_f32) : 0.0f;
#pragma unroll
                    for (int m = 0; m < 3; ++m) {
                        if (qc + m >= nq) break;
                        const float2 d = make_float2(__fsub_rn(In[m], fo), __fsub_rn(In[m], fi));
                        const float2 ph = mul2(d, d), pl = fma2(d, d, neg2(ph));
                        const float2 qh = mul2(wh, ph);
                        const float2 ql = fma2(wh, pl, fma2(wl, ph, fma2(wh, ph, neg2(qh))));
                        const float2 t = add2(sum, qh);
                        const float2 bb = sub2(t, sum);
                        const float2 tail = add2(add2(sub2(sum, sub2(t, bb)), sub2(qh, bb)), ql);
                        const float2 margin = mul2(t, dup2(0x1p-43f));
                        const float2 hi = add2(t, add2(tail, margin)), lo = add2(t, sub2(tail, margin));
                        sure = sure && hi.x == lo.x && hi.y == lo.y;
                        sum = hi;
                    }
                }
                e = sure ? sum : box_column_double(s.img, i0, WH, nq, c.img_f32, wt, fo, fi, e);
            }
        }
        const float s1 = e.x, s2 = e.y;
        dfull[vi] = data_factor(s1, s2, c.l1, c.l2, c.lam_equal != 0);
        if (DEBUG) {
            dbg.f[2 * dbg.n + vi] = s1;
            dbg.f[3 * dbg.n + vi] = s2;
        }
    }
}

// The debug step's stencil: the same arithmetic, one voxel per thread, with
// the intermediate fields written out.
template <Arith A>
__global__ void __launch_bounds__(ST_WARPS * 32, 2) stencil_debug_kernel(const SubVolDev *__restrict__ svs,
                                                                   const int *__restrict__ pre,
                                                                   const StepConst c, int parity,
                                                                   unsigned *__restrict__ flag, DebugOut dbg) {
    __shared__ float Pb[3][ST_WARPS + 2][32];
    __shared__ float2 Gb[3][ST_WARPS][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int b = blockIdx.x;
    const int sv = find_sv(pre, c.nsv, b);
    const SubVolDev &s = svs[sv];
    int t = b - __ldg(pre + sv);
    StencilCtx k;
    k.s = &s;
    k.W = s.W;
    k.H = s.H;
    k.L = s.L;
    k.r = c.r;
    const int ntx = (k.W + ST_OX - 1) / ST_OX, nty = (k.H + ST_OY - 1) / ST_OY;
    const int tx = t % ntx;
    t /= ntx;
    const int ty = t % nty;
    const int tz = t / nty;
    const int x0 = tx * ST_OX, y0 = ty * ST_OY;
    k.ref = c.boundary == 0;
    k.x = x0 - 1 + lane;
    k.y = y0 - 1 + w;
    k.w = w;
    k.lane = lane;
    k.z0 = tz * c.zc;
    k.z1 = min(k.z0 + c.zc, k.L);
    k.first = k.z0 - 2;
    k.in = k.x >= 0 && k.x < k.W && k.y >= 0 && k.y < k.H;
    k.outp = k.in && lane >= 1 && lane <= ST_OX && w >= 1 && w <= ST_OY;
    k.WH = (size_t)k.W * k.H;
    k.col = k.in ? (size_t)k.y * k.W + k.x : 0;
    k.phi = (parity ? s.phi[1] : s.phi[0]) + k.col;
    k.phi_out = parity ? s.phi[0] : s.phi[1];
    const bool valid = s.Wv > 0;
    const int r = k.r;
    k.inside_xy = valid && k.x >= r && k.x < k.W - r && k.y >= r && k.y < k.H - r;
    k.blk_inside = valid && x0 >= r && x0 + ST_OX - 1 < k.W - r && y0 >= r && y0 + ST_OY - 1 < k.H - r &&
                   k.z0 >= r && k.z1 - 1 < k.L - r;
    k.dplane = (size_t)s.Wp * s.Hv;
    k.dcol = k.inside_xy ? s.db + (size_t)(k.y - r) * s.Wp + (k.x - r) : s.db;
    if (c.full_data) {  // every voxel's data factor comes from the box or expanded data-term kernels
        k.blk_inside = true;
        k.dplane = k.WH;
        k.dcol = s.db + 2 * (size_t)s.Wp * s.Hv * s.Lv + k.col + (size_t)r * k.WH;
    }
    // The shuffles and shared rows supply every neighbour except: x-1 for
    // lane 0 and the previous linear element for x == 0 in the reference
    // mode, both at linear offset -1; x+1 for lane 31; y-1 / y+1 for the halo
    // rows.  Corner threads of the halo are never read.
    const bool halo_row = w == 0 || w == ST_WARPS - 1;
    const bool halo_col = lane == 0 || lane == 31;
    k.need_x = k.in && !(halo_row && halo_col) &&
               ((lane == 0) || (k.x == 0 && k.ref) || (lane == 31 && k.x + 1 < k.W));
    k.xoff = lane == 31 ? 1 : -1;
    k.need_y = k.in && halo_row && !halo_col && (w == 0 ? k.y > 0 : k.y + 1 < k.H);
    k.yoff = w == 0 ? -(ptrdiff_t)k.W : (ptrdiff_t)k.W;

    StencilState S;
    const int sp = k.first;
    S.P[0] = st_ld(k, sp);
    S.P[1] = st_ld(k, sp + 1);
    S.P[2] = st_ld(k, sp + 2);
    S.EX[1] = st_ldx(k, sp + 1);
    S.EY[1] = st_ldy(k, sp + 1);
    S.EX[2] = st_ldx(k, sp + 2);
    S.EY[2] = st_ldy(k, sp + 2);
    S.EX[0] = S.EY[0] = 0.0f;
    S.DT[0] = S.DT[1] = S.DT[2] = 0.0f;
    for (int i = 0; i < 3; ++i) S.G[i] = GN4{0.f, 0.f, 0.f, 0.f};
    Pb[1][w + 1][lane] = S.P[1];
    __syncthreads();
    const int count = k.z1 - k.first;
    for (int i = 0; i < count; i += 3) {
        stencil_step<0, A>(k, c, S, i, Pb, Gb, flag, dbg);
        if (i + 1 < count) stencil_step<1, A>(k, c, S, i + 1, Pb, Gb, flag, dbg);
        if (i + 2 < count) stencil_step<2, A>(k, c, S, i + 2, Pb, Gb, flag, dbg);
    }
}

}  // namespace rsf
