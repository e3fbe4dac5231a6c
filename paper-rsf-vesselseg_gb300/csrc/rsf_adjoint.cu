// rsf_adjoint.cu -- reverse-mode derivative of one RSF step, for a batch of
// volumes that share the step parameters.
//
// The forward step (CUDA_RSF/main.cpp:233-300, kernel.cu) maps phi to
//   phi' = phi + dt * ( -delta(phi) * data + nu * delta(phi) * kappa + mu * (Lap - kappa) )
// with data = lambda1 * e_out - lambda2 * e_in, e = (I - f)^2, f the ratios of
// Gaussian-blurred fields (I H, H, I (1-H), 1-H), kappa = sum_a D_a n_a,
// n = g / (|g| + 1e-6), g_a = D_a phi, Lap = sum_a D_a D_a phi, and D_a the
// central difference with the reference's boundary rules (kernel.cu:57-125).
// Given u = dL/dphi', this file computes dL/dphi and accumulates dL/dlambda1,
// dL/dlambda2, dL/dmu, dL/dnu.  The derivative is that of the exact real
// function above (H' = delta; delta' = -2 phi delta / (eps^2 + phi^2)), evaluated
// in FP32; it is not the derivative of the floating-point rounding.
//
// Chain, with pointwise adjoints written as bars:
//   data_bar  = -u dt delta       e_out_bar = lambda1 data_bar, e_in_bar = -lambda2 data_bar
//   f_bar     = -2 (I - f) e_bar  (valid region only; the border band holds f = 1)
//   B1_bar = f_out_bar / B2, B2_bar = -f_out_bar f_out / B2 (and B3, B4 from f_in)
//   H_bar  = I * G^T (B1_bar - B3_bar) + G^T (B2_bar - B4_bar)    (blur is linear)
//   kappa_bar = u dt (nu delta - mu), Lap_bar = u dt mu
//   n_bar_a = D_a^T kappa_bar;  g_bar_a = D_a^T Lap_bar + (n_bar_a - (n_bar . n) g_a/|g|) / (|g| + 1e-6)
//   phi_bar = u + delta H_bar + delta' u dt (-data + nu kappa) + sum_a D_a^T g_bar_a
// G^T of the valid correlation is the full correlation with the same
// (symmetric) taps.  D_a^T is gathered: voxel j collects 0.5 v(m) for every m
// among its three axis neighbours whose right index is j, and -0.5 v(m) for
// every m whose left index is j, so boundary rules transpose exactly.
//
// Kernels: the forward step's x- and y-passes and the z-pass's adjoint variant
// (zpass_adjoint_kernel, zchunk_adjoint_kernel), which the caller launches and
// which leave the data-term adjoint; then here transposed blur z, y, x (the x
// kernel forms H_bar); gradients; the pointwise terms with the parameter sums and
// the stencil adjoint w; the final D^T gather.  The blurs along y and z compute several
// consecutive outputs per thread; the last three kernels run on blocks of
// 32 x 8 voxels, the others on one item per thread.  Every kernel covers the
// whole batch in one launch: a block finds its volume in a block prefix
// array (one per kernel) and its tile within the volume.
//
// Scratch per volume (N = W H L; slices of the workspace pools of 1, 4 and
// 4 floats per voxel):
//   phi2 : H_bar
//   xs   : x fields (4 Wp H L), then [0, 2N) the valid-layout adjoint pair
//          (float2 per voxel) and [2N, 4N) e_out, e_in (w_z over e_out); then
//          g_x, g_y in [0, 2N)
//   ys   : y fields (4 Wp Hv L), then the z-transposed pair [0, 2N), the y-
//          transposed pair at 2N; later g_z, 1/(|g|+1e-6), w_x, w_y
#include <cuda_runtime.h>

#include "rsf_kernels.cuh"

namespace rsf {
namespace {

constexpr int kThreads = 256;

struct AdjConst {
    float2 taps2[MAXK];  // (g, g) pairs
    __device__ __forceinline__ unsigned long long tap2(int t) const { return pack2(taps2[t]); }
    int k, r;
    float eps, dt, mu, nu, l1, l2;
    int boundary;    // 0 reference (x = 0 reads the previous linear element), 1 clamp
    int img_f32;
    int nvol;
};

__device__ __forceinline__ float img_at(const void *img, long long i, int f32) {
    return f32 ? static_cast<const float *>(img)[i] : (float)static_cast<const unsigned char *>(img)[i];
}

// The volume of this block (binary search of the kernel's block prefix
// array) and the block's index within it.  Kernels copy their volume's
// descriptor by value, so that their stores cannot alias it and its fields
// are loaded once.
struct BlockVol {
    int v;
    long long t;
};
__device__ __forceinline__ BlockVol block_vol(const int *__restrict__ pre, int n) {
    const int b = blockIdx.x;
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(pre + mid) <= b) lo = mid;
        else hi = mid;
    }
    return {lo, (long long)(b - __ldg(pre + lo))};
}

// The stencil kernels run on blocks of 32 x 8 voxels of kWZ planes (gather) or of
// kPointZ planes (pointwise terms).
constexpr int kBX = 32, kBY = 8;
constexpr int kPointZ = 8;
constexpr int kWZ = 8;  // planes per block of adj_gather

// The difference rules of a voxel along one axis without branches (a warp that
// touches a face would otherwise take the general and the inner form one after
// the other).  D f = (f(i + r) - f(i - l)) / 2 with the offsets r, l.  Its
// transpose gathers D^T v = m v(i - l) + p v(i + r) with the same offsets: where a
// neighbour is missing the voxel's own value takes its place.  A value has no
// other part in it, so that an infinite one stays out of results that do not
// depend on it.
struct Axis {
    long long r, l;
    float m, p;
};
__device__ __forceinline__ Axis axis_plain(int q, int n, long long s) {
    const bool lo = q > 0, hi = q + 1 < n;
    return {hi ? s : 0, lo ? s : 0, lo ? 0.5f : -0.5f, hi ? -0.5f : 0.5f};
}
// Along x the neighbours are the ones in memory: in the reference boundary mode
// (kernel.cu:64-67) x = 0 reads the previous linear element, so the last voxel
// of a row is read by the first one of the next and, being its own right
// neighbour, by itself.  D^T v = m v(i - 1) + c v(i) + p v(i + 1), i > 0 and
// i + 1 < N decide at the volume's ends.
struct AxisX {
    int r, l;
    float m, c, p;
};
__device__ __forceinline__ AxisX axis_x(const AdjVol &a, int boundary, int x, long long i, long long N) {
    const bool lo = x > 0, hi = x + 1 < a.W;
    const bool left = boundary == 0 ? i > 0 : lo, right = boundary == 0 ? i + 1 < N : hi;
    return {hi, left, lo ? 0.5f : 0.0f, (hi ? 0.0f : 0.5f) - (left ? 0.0f : 0.5f), right ? -0.5f : 0.0f};
}
// The sum from the neighbours' values (0 where they have no weight) and the own.
__device__ __forceinline__ float gather_x(const AxisX &k, float vm, float v0, float vp) {
    return fmaf(k.p, vp, fmaf(k.c, k.c != 0.0f ? v0 : 0.0f, k.m * vm));
}

// delta(phi) with a fast division: the adjoint needs the derivative's value,
// not the forward's bit pattern.
__device__ __forceinline__ float dirac_fast(float phi, float eps) {
    return __fdividef(0.318309886183790672f * eps, fmaf(phi, phi, eps * eps));
}

// Running sums with their rounding errors (Knuth's two-sum; products with their
// residual), two at a time.  A parameter's derivative sums terms u (...) whose
// u of either sign cancels over the volume, so a plain FP32 sum keeps what its
// largest partial sums rounded off: dL/dmu of a 128^3 chain of 5 steps was
// 2.4e-3 from float64 with plain sums, 8e-4 so; the time of a training step did
// not change (3.04 ms for 4 volumes of 96x112x96 and 4 steps).
struct Sum2 {
    float2 s, e;
};
__device__ __forceinline__ float2 two_sum_error(float2 a, float2 b, float2 s) {
    const float2 bb = sub2(s, a);
    return add2(sub2(a, sub2(s, bb)), sub2(b, bb));
}
__device__ __forceinline__ void add_product(Sum2 &k, float2 a, float2 b) {
    const float2 t = mul2(a, b), r = fma2(a, b, neg2(t)), s = add2(k.s, t);
    k.e = add2(k.e, add2(two_sum_error(k.s, t, s), r));
    k.s = s;
}
__device__ __forceinline__ Sum2 add_sum(Sum2 a, Sum2 b) {
    const float2 s = add2(a.s, b.s);
    return {s, add2(add2(a.e, b.e), two_sum_error(a.s, b.s, s))};
}
__device__ __forceinline__ void add_sum(float &s, float &e, float bs, float be) {
    const float t = __fadd_rn(s, bs), bb = __fsub_rn(t, s);
    e = __fadd_rn(__fadd_rn(e, be), __fadd_rn(__fsub_rn(s, __fsub_rn(t, bb)), __fsub_rn(bs, bb)));
    s = t;
}
__device__ __forceinline__ float2 shfl2(float2 v, int o) {
    return make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
}

__device__ __forceinline__ long long nvox(const AdjVol &a) { return (long long)a.W * a.H * a.L; }
__device__ __forceinline__ long long item(const BlockVol &bv) { return bv.t * kThreads + threadIdx.x; }

// The transposed (full) correlations out[o] = sum_t g[t] in[o - t] over
// 0 <= o - t < n, both fields of the pair (P, Q) in packed multiply-adds, taps in
// chunks over a register window (conv_chunks of the forward kernels; the taps
// are symmetric, so ascending inputs take them in either order).  Inputs
// outside the range count 0.  4 x 96x112x96 voxels, 21 taps: z 40 -> 14 us, y
// 55 -> 17, x 85 -> 29 against scalar sums with an index test per multiply-add.
constexpr int kNB = 8;   // outputs per thread along z
constexpr int kNBy = 8;  // and along y

// z: xs (Wv, Hv, Lv) -> ys (Wv, Hv, L).
__global__ void __launch_bounds__(kThreads) adj_blurT_z(const __grid_constant__ AdjConst c,
                                                        const AdjVol *__restrict__ vols,
                                                        const int *__restrict__ pre) {
    const BlockVol bv = block_vol(pre, c.nvol);
    const AdjVol a = vols[bv.v];
    const long long plane = (long long)a.Wv * a.Hv;
    const int nzb = (a.L + kNB - 1) / kNB;
    const long long q = item(bv);
    if (q >= plane * nzb) return;
    const long long pxy = q % plane;
    const int z0 = (int)(q / plane) * kNB, first = z0 - c.k + 1;
    const unsigned long long *in = reinterpret_cast<const unsigned long long *>(a.xs) + pxy;
    unsigned long long u[kNB], *out = reinterpret_cast<unsigned long long *>(a.ys) + z0 * plane + pxy;
    conv_chunks<kNB>(c, [&](int i) {
        const int p = first + i;
        return p >= 0 && p < a.Lv ? __ldg(in + p * plane) : 0ull;
    }, u);
#pragma unroll
    for (int m = 0; m < kNB; ++m)
        if (z0 + m < a.L) out[m * plane] = u[m];
}

// y: ys (Wv, Hv, L) -> ys + 2N (Wv, H, L).
__global__ void __launch_bounds__(kThreads) adj_blurT_y(const __grid_constant__ AdjConst c,
                                                        const AdjVol *__restrict__ vols,
                                                        const int *__restrict__ pre) {
    const BlockVol bv = block_vol(pre, c.nvol);
    const AdjVol a = vols[bv.v];
    const int nyb = (a.H + kNBy - 1) / kNBy;
    const long long q = item(bv);
    if (q >= (long long)a.Wv * nyb * a.L) return;
    const int xv = (int)(q % a.Wv);
    const long long t1 = q / a.Wv;
    const int y0 = (int)(t1 % nyb) * kNBy, first = y0 - c.k + 1;
    const int z = (int)(t1 / nyb);
    const unsigned long long *in = reinterpret_cast<const unsigned long long *>(a.ys) + (long long)z * a.Hv * a.Wv + xv;
    unsigned long long u[kNBy], *out = reinterpret_cast<unsigned long long *>(a.ys + 2 * nvox(a)) +
                                       ((long long)z * a.H + y0) * a.Wv + xv;
    conv_chunks<kNBy>(c, [&](int i) {
        const int p = first + i;
        return p >= 0 && p < a.Hv ? __ldg(in + (long long)p * a.Wv) : 0ull;
    }, u);
#pragma unroll
    for (int m = 0; m < kNBy; ++m)
        if (y0 + m < a.H) out[(long long)m * a.Wv] = u[m];
}

// x, and H_bar = I * P~ + Q~ over the volume, into phi2 (0 for a volume without a
// valid region).  A warp takes a segment of 32 kNBx voxels of one row, whose
// inputs it stages in shared memory; a lane forms kNBx adjacent outputs (odd, so
// that the lanes' 64-bit loads fall into distinct banks).
constexpr int kNBx = 3;
constexpr int kTxWarps = 8;
__global__ void __launch_bounds__(32 * kTxWarps) adj_blurT_x_hbar(const __grid_constant__ AdjConst c,
                                                                  const AdjVol *__restrict__ vols,
                                                                  const int *__restrict__ pre) {
    constexpr int XT = 32 * kNBx;
    __shared__ unsigned long long slab_s[kTxWarps][XT + MAXK + 2 * kNBx];
    const BlockVol bv = block_vol(pre, c.nvol);
    const AdjVol a = vols[bv.v];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int ntx = (a.W + XT - 1) / XT;
    const long long row = bv.t / ntx * kTxWarps + w;
    if (row >= (long long)a.H * a.L) return;  // uniform per warp
    const int x0 = (int)(bv.t % ntx) * XT;
    const long long base = row * a.W;
    if (a.Wv == 0) {
        for (int x = x0 + lane; x < min(x0 + XT, a.W); x += 32) a.phi2[base + x] = 0.0f;
        return;
    }
    // slab[j]: input x0 - (k - 1) + j
    unsigned long long *slab = slab_s[w];
    const unsigned long long *in = reinterpret_cast<const unsigned long long *>(a.ys + 2 * nvox(a)) + row * a.Wv;
    const int first = x0 - c.k + 1, span = XT + c.k - 1;
    for (int j = lane; j < span; j += 32) {
        const int p = first + j;
        slab[j] = p >= 0 && p < a.Wv ? __ldg(in + p) : 0ull;
    }
    __syncwarp();
    // outputs top, top - 1, ..: input o - t is slab[o - x0 + k - 1 - t]
    const int top = kNBx * lane + kNBx - 1;
    unsigned long long u[kNBx];
    conv_chunks<kNBx>(c, [&](int i) { return slab[max(top + c.k - 1 - i, 0)]; }, u);
    __syncwarp();
#pragma unroll
    for (int m = 0; m < kNBx; ++m) slab[top - m] = u[m];
    __syncwarp();
#pragma unroll
    for (int m = 0; m < kNBx; ++m) {
        const int x = x0 + 32 * m + lane;
        const float2 pq = unpack2(slab[32 * m + lane]);
        if (x < a.W) a.phi2[base + x] = fmaf(img_at(a.img, base + x, c.img_f32), pq.x, pq.y);
    }
}

// Gradient g = D phi and 1 / (|g| + 1e-6), stored so that the kernels after it
// read them at their neighbours instead of recomputing (the unit normal is the
// product): g_x, g_y to xs, xs + N; g_z, 1 / (|g| + 1e-6) to ys, ys + N.
__global__ void __launch_bounds__(kThreads) adj_normals(AdjConst c, const AdjVol *__restrict__ vols,
                                                        const int *__restrict__ pre) {
    const BlockVol bv = block_vol(pre, c.nvol);
    const AdjVol a = vols[bv.v];
    const long long N = nvox(a);
    const long long i = item(bv);
    if (i >= N) return;
    const int x = (int)(i % a.W);
    const long long t1 = i / a.W;
    const int y = (int)(t1 % a.H);
    const int z = (int)(t1 / a.H);
    const AxisX ax = axis_x(a, c.boundary, x, i, N);
    const Axis ay = axis_plain(y, a.H, a.W), az = axis_plain(z, a.L, (long long)a.W * a.H);
    auto diff = [&](long long r, long long l) { return 0.5f * (a.phi[i + r] - a.phi[i - l]); };
    const float gx = diff(ax.r, ax.l), gy = diff(ay.r, ay.l), gz = diff(az.r, az.l);
    a.xs[i] = gx;
    a.xs[N + i] = gy;
    a.ys[i] = gz;
    a.ys[N + i] = __frcp_rn(sqrtf(gx * gx + gy * gy + gz * gz) + 1e-6f);
}

// The block's 32 x 8 column: x, y of this thread and the first z plane.
struct Col {
    int x, y, z0;
};
__device__ __forceinline__ Col col_of(const AdjVol &a, long long t, int zdepth) {
    const int nbx = (a.W + kBX - 1) / kBX, nby = (a.H + kBY - 1) / kBY;
    const long long t1 = t / nbx;
    return {(int)(t % nbx) * kBX + (int)threadIdx.x, (int)(t1 % nby) * kBY + (int)threadIdx.y,
            (int)(t1 / nby) * zdepth};
}

// Pointwise terms, parameter sums and the stencil adjoint:
//   out = u + delta H_bar + delta' u dt (nu kappa - data),
// with kappa = sum_a D_a n_a and Lap = sum_a D_a g_a from the stored fields, and
//   w_a = D_a^T Lap_bar + (n_bar_a - (n_bar . n) g_a/|g|) / (|g| + 1e-6),
// n_bar = D^T kappa_bar, kappa_bar = u dt (nu delta - mu), Lap_bar = u dt mu, to be
// gathered by D_a^T: w_x, w_y to ys + 2N, ys + 3N, w_z over e_out (read first, by
// the same thread).  A block covers a 32 x 8 column of kPointZ planes; kappa_bar
// of the three planes around the voxel, g_z and the z normals ride in
// registers, so each is formed once per column, and kappa_bar of the x and y
// neighbours is formed from phi and u at them (one pass over the fields
// instead of two with kappa_bar and the normals stored between them).  The
// parameter sums are reduced in the block and added with one double atomic per
// parameter and block (the same four addresses for every block, so their
// number matters).  4 x 96x112x96 voxels: 227 us as two kernels with branches for
// the face rules, 115 with three weights per axis, 100 so (the own value in a missing
// neighbour's place along y and z; the gather after it 21 and 26).  Planes per block,
// with three weights: 8 115 us, 16 122, 4 127; on one 43x58x67 volume 11.2, 18.6 and 8.0
// (9.4 with 8 now).
__global__ void __launch_bounds__(kBX * kBY, 2) adj_point(AdjConst c, const AdjVol *__restrict__ vols,
                                                       const int *__restrict__ pre,
                                                       double *grads) {
    const BlockVol bv = block_vol(pre, c.nvol);
    const AdjVol a = vols[bv.v];
    const long long N = nvox(a);
    const long long plane = (long long)a.W * a.H;
    const float *__restrict__ phi = a.phi, *__restrict__ uu = a.u;
    const float *__restrict__ gxa = a.xs, *__restrict__ gya = a.xs + N, *__restrict__ gza = a.ys, *__restrict__ rsa = a.ys + N;
    float *ez = a.xs + 2 * N;  // e_out, then w_z
    const float *__restrict__ ei_v = a.xs + 3 * N;
    float *__restrict__ wx = a.ys + 2 * N, *__restrict__ wy = a.ys + 3 * N;
    auto kbar = [&](long long m) { return uu[m] * c.dt * (c.nu * dirac_fast(phi[m], c.eps) - c.mu); };
    auto lbar = [&](long long m) { return uu[m] * c.dt * c.mu; };
    Sum2 s_l = {{0.0f, 0.0f}, {0.0f, 0.0f}}, s_mn = s_l;  // lambda1, lambda2; mu, nu
    const Col cl = col_of(a, bv.t, kPointZ);
    const int x = cl.x, y = cl.y;
    const int z1 = min(cl.z0 + kPointZ, a.L);
    if (x < a.W && y < a.H) {
        long long i = ((long long)cl.z0 * a.H + y) * a.W + x;
        const Axis ay = axis_plain(y, a.H, a.W);
        // of planes z - 1, z, z + 1: kappa_bar, Lap_bar, g_z and 1/(|g|+1e-6); the
        // voxel's own where there is no such plane
        float k1 = kbar(i), l1 = lbar(i), gz1 = gza[i], r1 = rsa[i];
        float k0 = k1, l0 = l1, gz0 = gz1, r0 = r1;
        if (cl.z0 > 0) {
            k0 = kbar(i - plane);
            l0 = lbar(i - plane);
            gz0 = gza[i - plane];
            r0 = rsa[i - plane];
        }
        for (int z = cl.z0; z < z1; ++z, i += plane) {
            float k2 = k1, l2 = l1, gz2 = gz1, r2 = r1;
            if (z + 1 < a.L) {
                k2 = kbar(i + plane);
                l2 = lbar(i + plane);
                gz2 = gza[i + plane];
                r2 = rsa[i + plane];
            }
            const float ph = phi[i], ui = uu[i];
            const float I = img_at(a.img, i, c.img_f32);
            const float gx = gxa[i], gy = gya[i];
            const float delta = dirac_fast(ph, c.eps);
            const float ddelta = __fdividef(-2.0f * ph * delta, fmaf(ph, ph, c.eps * c.eps));
            const AxisX ax = axis_x(a, c.boundary, x, i, N);
            const Axis az = axis_plain(z, a.L, plane);
            // curvature and "Laplacian"; the z neighbours are at hand
            const long long rx = i + ax.r, lx = i - ax.l, ry = i + ay.r, ly = i - ay.l;
            const float gxr = gxa[rx], gxl = gxa[lx], gyr = gya[ry], gyl = gya[ly];
            // The normals are rounded before they are subtracted, so that equal
            // neighbours cancel (a contracted multiply-add would leave the rounding
            // of one product, times u).
            const float kap = 0.5f * (__fmul_rn(gxr, rsa[rx]) - __fmul_rn(gxl, rsa[lx])) +
                              0.5f * (__fmul_rn(gyr, rsa[ry]) - __fmul_rn(gyl, rsa[ly])) +
                              0.5f * (__fmul_rn(gz2, r2) - __fmul_rn(gz0, r0));
            const float lap = 0.5f * (gxr - gxl) + 0.5f * (gyr - gyl) + 0.5f * (gz2 - gz0);
            // D^T of kappa_bar and Lap_bar
            auto kb = [&](float u, float p) { return u * (c.nu * dirac_fast(p, c.eps) - c.mu); };
            float um = 0.0f, up = 0.0f, pm = 0.0f, pp = 0.0f;
            if (ax.m != 0.0f) um = uu[i - 1] * c.dt, pm = phi[i - 1];
            if (ax.p != 0.0f) up = uu[i + 1] * c.dt, pp = phi[i + 1];
            const float nbx = gather_x(ax, kb(um, pm), k1, kb(up, pp)), lbx = gather_x(ax, um * c.mu, l1, up * c.mu);
            const float vm = uu[ly] * c.dt, vp = uu[ry] * c.dt;
            const float nby = fmaf(ay.p, kb(vp, phi[ry]), ay.m * kb(vm, phi[ly])), lby = fmaf(ay.p, vp * c.mu, ay.m * (vm * c.mu));
            const float nbz = fmaf(az.p, k2, az.m * k0), lbz = fmaf(az.p, l2, az.m * l0);
            const bool valid = a.Wv > 0 && x >= c.r && x < c.r + a.Wv && y >= c.r && y < c.r + a.Hv && z >= c.r &&
                               z < c.r + a.Lv;
            float eo, ei;
            if (valid) {
                eo = ez[i];
                ei = ei_v[i];
            } else {  // border band: f_out = f_in = 30 / 30
                eo = ei = (I - 1.0f) * (I - 1.0f);
            }
            const float data = c.l1 * eo - c.l2 * ei;
            a.out[i] = ui + delta * a.phi2[i] + ddelta * ui * c.dt * (c.nu * kap - data);
            const float ud = ui * c.dt, udd = ud * delta;
            add_product(s_l, make_float2(-udd, udd), make_float2(eo, ei));
            add_product(s_mn, make_float2(ud, udd), make_float2(lap - kap, kap));
            const float mag = sqrtf(gx * gx + gy * gy + gz1 * gz1);
            const float inv_mag = mag > 0.0f ? __frcp_rn(mag) : 0.0f;
            const float ndot = nbx * __fmul_rn(gx, r1) + nby * __fmul_rn(gy, r1) + nbz * __fmul_rn(gz1, r1);
            wx[i] = lbx + (nbx - ndot * gx * inv_mag) * r1;
            wy[i] = lby + (nby - ndot * gy * inv_mag) * r1;
            ez[i] = lbz + (nbz - ndot * gz1 * inv_mag) * r1;
            k0 = k1;
            k1 = k2;
            l0 = l1;
            l1 = l2;
            gz0 = gz1;
            gz1 = gz2;
            r0 = r1;
            r1 = r2;
        }
    }
    if (grads) {  // uniform: every thread reaches the shuffles and the barrier
        // Each step halves the sums a lane keeps: first the upper half-warp takes
        // (mu, nu) and the lower (lambda1, lambda2), then one value per quarter.
        __shared__ double part[kBY][4];
        const int ln = threadIdx.x;
        const bool up = ln & 16, up2 = ln & 8;
        const Sum2 give = up ? s_l : s_mn, keep = up ? s_mn : s_l;
        const Sum2 h = add_sum({keep.s, keep.e}, {shfl2(give.s, 16), shfl2(give.e, 16)});
        float hs = up2 ? h.s.y : h.s.x, he = up2 ? h.e.y : h.e.x;
        add_sum(hs, he, __shfl_xor_sync(0xffffffffu, up2 ? h.s.x : h.s.y, 8),
                __shfl_xor_sync(0xffffffffu, up2 ? h.e.x : h.e.y, 8));
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
            add_sum(hs, he, __shfl_xor_sync(0xffffffffu, hs, o), __shfl_xor_sync(0xffffffffu, he, o));
        // (an overflowed sum has no error term)
        if ((ln & 7) == 0) part[threadIdx.y][ln >> 3] = isfinite(he) ? (double)hs + (double)he : (double)hs;
        __syncthreads();
        if (threadIdx.y == 0 && threadIdx.x < 4) {
            double acc = 0.0;
            for (int w = 0; w < kBY; ++w) acc += part[w][threadIdx.x];
            atomicAdd(grads + threadIdx.x, acc);
        }
    }
}

// out += sum_a D_a^T w_a; a non-finite result sets kFlagAdjointNonFinite.
__global__ void __launch_bounds__(kBX * kBY) adj_gather(AdjConst c, const AdjVol *__restrict__ vols,
                                                        const int *__restrict__ pre, unsigned *flag) {
    const BlockVol bv = block_vol(pre, c.nvol);
    const AdjVol a = vols[bv.v];
    const long long N = nvox(a);
    const long long plane = (long long)a.W * a.H;
    const float *__restrict__ wx = a.ys + 2 * N, *__restrict__ wy = a.ys + 3 * N, *__restrict__ wz = a.xs + 2 * N;
    const Col cl = col_of(a, bv.t, kWZ);
    const int x = cl.x, y = cl.y;
    if (x >= a.W || y >= a.H) return;
    const int z1 = min(cl.z0 + kWZ, a.L);
    const Axis ay = axis_plain(y, a.H, a.W);
    long long i = ((long long)cl.z0 * a.H + y) * a.W + x;
    float bad = 0.0f;  // NaN once a result is not finite
    float zcv = wz[i], z0v = cl.z0 > 0 ? wz[i - plane] : zcv;  // w_z of planes z, z - 1
    for (int z = cl.z0; z < z1; ++z, i += plane) {
        const float z2v = z + 1 < a.L ? wz[i + plane] : zcv;
        const AxisX ax = axis_x(a, c.boundary, x, i, N);
        const Axis az = axis_plain(z, a.L, plane);
        const float d = gather_x(ax, ax.m != 0.0f ? wx[i - 1] : 0.0f, wx[i], ax.p != 0.0f ? wx[i + 1] : 0.0f) +
                        fmaf(ay.p, wy[i + ay.r], ay.m * wy[i - ay.l]) + fmaf(az.p, z2v, az.m * z0v);
        const float v = a.out[i] + d;
        a.out[i] = v;
        bad = fmaf(v, 0.0f, bad);
        z0v = zcv;
        zcv = z2v;
    }
    if (!isfinite(bad) && flag) atomicOr(flag, kFlagAdjointNonFinite);
}

long long cdiv(long long a, long long b) { return (a + b - 1) / b; }

}  // namespace

void adjoint_tiles(const AdjVol &v, int tiles[NADJ]) {
    const long long N = (long long)v.W * v.H * v.L;
    const bool valid = v.Wv > 0;
    const long long bxy = cdiv(v.W, kBX) * cdiv(v.H, kBY);
    long long t[NADJ] = {};
    if (valid) {
        t[ADJ_TZ] = cdiv((long long)v.Wv * v.Hv * cdiv(v.L, kNB), kThreads);
        t[ADJ_TY] = cdiv((long long)v.Wv * cdiv(v.H, kNBy) * v.L, kThreads);
    }
    t[ADJ_TX] = cdiv(v.W, 32 * kNBx) * cdiv((long long)v.H * v.L, kTxWarps);
    t[ADJ_NRM] = cdiv(N, kThreads);
    t[ADJ_PT] = bxy * cdiv(v.L, kPointZ);
    t[ADJ_G] = bxy * cdiv(v.L, kWZ);
    for (int j = 0; j < NADJ; j++) tiles[j] = t[j] > 0x7fffffffLL ? -1 : (int)t[j];
}

cudaError_t launch_step_adjoint(const float *taps, int k, const AdjScalars &s, const AdjVol *vols, const int *pre,
                                int n, const int *tot, double *grads, unsigned *flag, cudaStream_t st) {
    AdjConst c;
    for (int t = 0; t < MAXK; t++) c.taps2[t] = t < k ? make_float2(taps[t], taps[t]) : make_float2(0.0f, 0.0f);
    c.k = k;
    c.r = (k - 1) / 2;
    c.eps = s.eps;
    c.dt = s.dt;
    c.mu = s.mu;
    c.nu = s.nu;
    c.l1 = s.l1;
    c.l2 = s.l2;
    c.boundary = s.boundary;
    c.img_f32 = s.img_f32;
    c.nvol = n;
    const int n1 = n + 1;
    auto P = [&](int j) { return pre + (size_t)j * n1; };
    const dim3 b2(kBX, kBY, 1);
    if (tot[ADJ_TZ] > 0) adj_blurT_z<<<tot[ADJ_TZ], kThreads, 0, st>>>(c, vols, P(ADJ_TZ));
    if (tot[ADJ_TY] > 0) adj_blurT_y<<<tot[ADJ_TY], kThreads, 0, st>>>(c, vols, P(ADJ_TY));
    if (tot[ADJ_TX] > 0) adj_blurT_x_hbar<<<tot[ADJ_TX], 32 * kTxWarps, 0, st>>>(c, vols, P(ADJ_TX));
    if (tot[ADJ_NRM] > 0) adj_normals<<<tot[ADJ_NRM], kThreads, 0, st>>>(c, vols, P(ADJ_NRM));
    if (tot[ADJ_PT] > 0) adj_point<<<tot[ADJ_PT], b2, 0, st>>>(c, vols, P(ADJ_PT), grads);
    if (tot[ADJ_G] > 0) adj_gather<<<tot[ADJ_G], b2, 0, st>>>(c, vols, P(ADJ_G), flag);
    return cudaGetLastError();
}

}  // namespace rsf
