// rsf_sdf.cu -- the initial level set: the exact signed Euclidean distance of
// a seed region, on the device.
//
// The reference builds phi0 on the host: it subtracts 13 from the seed volume
// and calls tiralib's volume::sdf() (CUDA_RSF/main.cpp:174-183).  tiralib is
// not part of the reference checkout, so the transform is defined here on its
// own terms: a voxel is inside when seed > threshold; phi0 is +d(p, outside)
// at inside voxels and -d(p, inside) at outside voxels, d the Euclidean
// distance in voxels between voxel centres.  When one class is empty the
// other gets +-(W + H + L), larger than any distance in the box.
//
// Each class is one exact distance transform, computed separably on squared
// integer distances (Felzenszwalb & Huttenlocher, "Distance Transforms of
// Sampled Functions", Theory of Computing 8, 2012):
//   rows    (x) one warp per row: nearest feature to the left and right by
//               warp max/min scans, squared;
//   columns (y, then z) one thread per column: the lower envelope of the
//               parabolas (q - v)^2 + f(v), evaluated at every q.
// Envelope intersections are compared exactly in 64-bit integers, so the
// squared distances are exact and phi0 = sqrt of an integer, correctly rounded.
// Column threads are adjacent in x, so every access of a column step is
// coalesced across the warp; the envelope stacks live in device scratch laid
// out [k][column] for the same reason.
//
// Columns of up to kTileMax voxels take the tiled kernels instead: both
// classes at once (a voxel needs its distance to the other class only, so one
// signed value per voxel carries both transforms), a block holding 32 whole
// columns in shared memory and a thread per four rows.  The envelope is a serial
// chain of dependent loads per column, with one thread per column; here a
// thread searches outwards a few rows, which ends most voxels near a surface, and
// the others go by halving: for one class the nearest row's index grows with
// the voxel's (Aggarwal et al., "Geometric applications of a matrix-searching
// algorithm", Algorithmica 2, 1987), so a group of rows between two finished
// groups searches only the rows between their results.  That bounds the work per
// voxel whatever the seeds are, as the envelope's is.  256 x 448 x 512 voxels:
// winding vessels 3.84 ms with the envelopes, 0.82 here; an empty seed 2.04 and
// 1.32; a slanted plane 2.70 and 1.40 (3.94 with the search alone, blocks of 16 rows
// skipped where their smallest value cannot improve; on 500^3 9.5 ms, 4.7 with the
// envelopes, 3.3 here); sparse noise (1e-3) 2.65 and 1.27.
#include <cuda_runtime.h>

#include <climits>

#include "rsf_internal.h"

namespace rsf {
namespace {

constexpr unsigned kInf = 0xffffffffu;
constexpr int kRowWarps = 8;
constexpr int kColThreads = 128;

__device__ __forceinline__ bool is_inside(const void *seed, int f32, size_t i, float thr) {
    const float v = f32 ? static_cast<const float *>(seed)[i] : (float)static_cast<const unsigned char *>(seed)[i];
    return v > thr;
}

// Squared distance along x to the nearest feature of the row (kInf when the
// row has none).  Features are the voxels whose class equals feat_inside.
__global__ void __launch_bounds__(32 * kRowWarps) sdf_rows(const void *seed, int f32, float thr, int feat_inside,
                                                           unsigned *d, int W, long long rows) {
    const long long row = (long long)blockIdx.x * kRowWarps + threadIdx.x / 32;
    if (row >= rows) return;  // uniform per warp
    const int lane = threadIdx.x & 31;
    const size_t base = (size_t)row * W;
    int carry = -1;  // last feature at or left of the chunk start
    for (int x0 = 0; x0 < W; x0 += 32) {
        const int x = x0 + lane;
        const bool f = x < W && is_inside(seed, f32, base + x, thr) == (feat_inside != 0);
        int v = f ? x : -1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v = max(v, u);
        }
        v = max(v, carry);
        if (x < W) d[base + x] = (unsigned)v;
        carry = __shfl_sync(0xffffffffu, v, 31);
    }
    int rcarry = INT_MAX;  // first feature at or right of the chunk end
    for (int x0 = ((W - 1) / 32) * 32; x0 >= 0; x0 -= 32) {
        const int x = x0 + lane;
        const bool f = x < W && is_inside(seed, f32, base + x, thr) == (feat_inside != 0);
        int v = f ? x : INT_MAX;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_down_sync(0xffffffffu, v, o);
            if (lane + o < 32) v = min(v, u);
        }
        v = min(v, rcarry);
        if (x < W) {
            const int left = (int)d[base + x];
            long long best = -1;
            if (left >= 0) best = x - left;
            if (v != INT_MAX && (best < 0 || v - x < best)) best = v - x;
            d[base + x] = best < 0 ? kInf : (unsigned)(best * best);
        }
        rcarry = __shfl_sync(0xffffffffu, v, 0);
    }
}

struct ColArgs {
    unsigned *d;        // squared distances, transformed in place (not FINAL)
    unsigned *sv;       // envelope stack: sample positions, [k][column]
    unsigned *sf;       // envelope stack: sample values
    long long ncols;
    int W;              // columns are numbered c = a * W + x
    long long plane;    // element offset of a column: (c / W) * plane + c % W
    long long stride;   // element step along the column
    int n;              // column length
    // FINAL: write phi at the voxels of the evaluated class
    const void *seed;
    int f32;
    float thr;
    int feat_inside;
    float *phi;
    float fill;
};

template <bool FINAL>
__global__ void __launch_bounds__(kColThreads) sdf_cols(ColArgs a) {
    const long long c = (long long)blockIdx.x * kColThreads + threadIdx.x;
    if (c >= a.ncols) return;
    const size_t base = (size_t)(c / a.W) * (size_t)a.plane + (size_t)(c % a.W);
    const size_t nc = (size_t)a.ncols;
    // Lower envelope over the finite samples; the top two entries stay in
    // registers as (position, F = f + position^2).
    int top = -1;
    long long vt = 0, Ft = 0, vp = 0, Fp = 0;
    for (int q = 0; q < a.n; q++) {
        const unsigned f = a.d[base + (size_t)q * (size_t)a.stride];
        if (f == kInf) continue;
        const long long Fq = (long long)f + (long long)q * q;
        // the top parabola is hidden when the new one overtakes it no later
        // than it overtakes the one below it
        while (top >= 1 && (Fq - Ft) * (vt - vp) <= (Ft - Fp) * ((long long)q - vt)) {
            top--;
            vt = vp;
            Ft = Fp;
            if (top >= 1) {
                vp = a.sv[(size_t)(top - 1) * nc + c];
                Fp = (long long)a.sf[(size_t)(top - 1) * nc + c] + vp * vp;
            }
        }
        top++;
        a.sv[(size_t)top * nc + c] = (unsigned)q;
        a.sf[(size_t)top * nc + c] = f;
        vp = vt;
        Fp = Ft;
        vt = q;
        Ft = Fq;
    }
    int k = 0;
    long long v0 = 0, f0 = 0, v1 = 0, F1 = 0;
    if (top >= 0) {
        v0 = a.sv[c];
        f0 = a.sf[c];
    }
    if (top >= 1) {
        v1 = a.sv[nc + c];
        F1 = (long long)a.sf[nc + c] + v1 * v1;
    }
    for (int q = 0; q < a.n; q++) {
        // move right while the next parabola is lower at q
        while (k < top && F1 - (f0 + v0 * v0) < 2LL * q * (v1 - v0)) {
            k++;
            v0 = v1;
            f0 = F1 - v1 * v1;
            if (k < top) {
                v1 = a.sv[(size_t)(k + 1) * nc + c];
                F1 = (long long)a.sf[(size_t)(k + 1) * nc + c] + v1 * v1;
            }
        }
        const size_t idx = base + (size_t)q * (size_t)a.stride;
        const long long dq = q - v0;
        const unsigned D = top < 0 ? kInf : (unsigned)(dq * dq + f0);
        if (!FINAL) {
            a.d[idx] = D;
        } else if (is_inside(a.seed, a.f32, idx, a.thr) != (a.feat_inside != 0)) {
            const float mag = D == kInf ? a.fill : __fsqrt_rn(__uint2float_rn(D));
            a.phi[idx] = a.feat_inside ? -mag : mag;
        }
    }
}

// ---------------------------------------------------------------------------
// Tiled path.  Values are signed: positive inside, negative outside, the
// magnitude the distance to the other class so far.
// ---------------------------------------------------------------------------
constexpr int kTileMax = 1408;          // column length: 32 columns of 32-bit values and their groups' results in shared memory
constexpr int kShortMax = 144;          // columns up to here search more rows one by one (see launch_tile)
constexpr short kNone16 = 32767;        // no voxel of the other class in the row
constexpr int kNone = 1 << 28;          // nor in the plane; plus any squared offset it stays above every distance

// Signed distance along x to the other class: one warp per row.  The row's
// class words (32 voxels each) and, per word, the first voxel of each class
// to its right are gathered from the end; a second sweep carries the last
// ones to the left.
__global__ void __launch_bounds__(32 * kRowWarps) sdf_rows_tile(const void *seed, int f32, float thr, short *d, int W,
                                                                long long rows) {
    constexpr int kWords = (kTileMax + 31) / 32;
    __shared__ unsigned word_s[kRowWarps][kWords];
    __shared__ int next_s[kRowWarps][kWords][2];
    const long long row = (long long)blockIdx.x * kRowWarps + threadIdx.x / 32;
    if (row >= rows) return;  // uniform per warp
    const int lane = threadIdx.x & 31;
    unsigned *word = word_s[threadIdx.x / 32];
    int(*next)[2] = next_s[threadIdx.x / 32];
    const size_t base = (size_t)row * W;
    const int nw = (W + 31) / 32, far = 1 << 20;
    int nx[2] = {far, far};  // nearest outside / inside voxel to the right
    for (int i = nw - 1; i >= 0; --i) {
        const int x = 32 * i + lane;
        const unsigned in = __ballot_sync(0xffffffffu, x < W && is_inside(seed, f32, base + x, thr));
        const unsigned have = i < nw - 1 || (W & 31) == 0 ? 0xffffffffu : (1u << (W & 31)) - 1u;
        if (lane == 0) {
            word[i] = in;
            next[i][0] = nx[0];
            next[i][1] = nx[1];
        }
        if (~in & have) nx[0] = 32 * i + __ffs(~in & have) - 1;
        if (in) nx[1] = 32 * i + __ffs(in) - 1;
    }
    __syncwarp();
    int px[2] = {-far, -far};  // to the left
    for (int i = 0; i < nw; ++i) {
        const int x = 32 * i + lane;
        const unsigned in = word[i], have = i < nw - 1 || (W & 31) == 0 ? 0xffffffffu : (1u << (W & 31)) - 1u;
        const unsigned out = ~in & have;
        const int c = (in >> lane) & 1;
        const unsigned other = c ? out : in;
        const unsigned lo = other & ((1u << lane) - 1u), hi = other & ~((2u << lane) - 1u);
        const int left = lo ? 32 * i + 31 - __clz(lo) : px[1 - c];
        const int right = hi ? 32 * i + __ffs(hi) - 1 : next[i][1 - c];
        const int dist = min(min(x - left, right - x), (int)kNone16);
        if (x < W) d[base + x] = (short)(c ? dist : -dist);
        if (out) px[0] = 32 * i + 31 - __clz(out);
        if (in) px[1] = 32 * i + 31 - __clz(in);
    }
}

struct TileArgs {
    const void *in;     // signed row distances (int16), or squared plane distances (int32) for FINAL
    int *out;           // squared plane distances, signed
    float *phi;         // FINAL
    int W, n, ncols;    // columns are numbered c = a * W + x
    long long plane;    // element offset of a column: (c / W) * plane + c % W
    long long stride;   // element step along the column
    float fill;
};

// A group's state: the row that is nearest to its first row, or one of these.
constexpr unsigned short kNear = 0xffff;  // found within FINE rows
constexpr unsigned short kFar = 0xfffe;   // not found yet

// Squared distance along a strided axis added to the values in `in`, for 32
// columns per block (one per lane).  A thread takes groups of four consecutive
// rows, which share every value they read: rows y0 - t and y0 + 3 + t lie
// t .. t + 3 rows from them.  Every voxel searches TRY rows to either side, and FINE
// if its distance so far is at most one row more.
template <bool FINAL, int T, int TRY, int FINE>
__global__ void __launch_bounds__(T) sdf_cols_tile(TileArgs a) {
    extern __shared__ int sdf_sm[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    constexpr int NW = T / 32;
    int *v = sdf_sm + lane;  // the lane's column: row r at v[32 r]
    unsigned short *state = reinterpret_cast<unsigned short *>(sdf_sm + 32 * a.n) + lane;  // group g at state[32 g]
    const int col = blockIdx.x * 32 + lane;
    const bool have = col < a.ncols;
    const size_t base = (size_t)(col / a.W) * (size_t)a.plane + (size_t)(col % a.W);
    for (int r = w; r < a.n; r += NW) {
        int q = 1;
        if (have) {
            const size_t i = base + (size_t)r * (size_t)a.stride;
            if (FINAL) {
                q = __ldg(static_cast<const int *>(a.in) + i);
            } else {
                const int d = __ldg(static_cast<const short *>(a.in) + i);
                const int m = abs(d) == kNone16 ? kNone : d * d;
                q = d > 0 ? m : -m;
            }
        }
        v[32 * r] = q;
    }
    __syncthreads();
    int s[4], best[4];
    // a voxel of the other class counts 0, one of the same class its own distance
    auto take = [&](int q, int j, int d2) { best[j] = min(best[j], max(s[j] * q + d2, d2)); };
    auto worst = [&] { return max(max(best[0], best[1]), max(best[2], best[3])); };
    auto own = [&](int y0) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int q = v[32 * min(y0 + j, a.n - 1)];
            s[j] = q > 0 ? 1 : -1;
            best[j] = abs(q);
        }
    };
    auto store = [&](int y0) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!have || y0 + j >= a.n) continue;
            const size_t i = base + (size_t)(y0 + j) * (size_t)a.stride;
            if (FINAL) {
                const float mag = best[j] >= kNone ? a.fill : __fsqrt_rn(__int2float_rn(best[j]));
                a.phi[i] = s[j] > 0 ? mag : -mag;
            } else {
                a.out[i] = s[j] * best[j];
            }
        }
    };
    bool far = false;
    for (int y0 = 4 * w; y0 < a.n; y0 += 4 * NW) {
        own(y0);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int q = v[32 * min(y0 + i, a.n - 1)];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (i != j) take(q, j, (i - j) * (i - j));
        }
        // rows past an end repeat the last one at a larger offset, which never wins
        auto go_on = [&](int t) {
            const int wst = worst();
            return t * t < wst && (t <= TRY || wst <= (FINE + 1) * (FINE + 1));
        };
        for (int t = 1; t <= FINE && __any_sync(0xffffffffu, go_on(t)); ++t) {
            const int ql = v[32 * max(y0 - t, 0)], qr = v[32 * min(y0 + 3 + t, a.n - 1)];
            const int t0 = t * t, t1 = t0 + 2 * t + 1, t2 = t0 + 4 * t + 4, t3 = t0 + 6 * t + 9;
            take(ql, 0, t0);
            take(ql, 1, t1);
            take(ql, 2, t2);
            take(ql, 3, t3);
            take(qr, 3, t0);
            take(qr, 2, t1);
            take(qr, 1, t2);
            take(qr, 0, t3);
        }
        // (a far lane has four voxels of one class: mixed ones found each other)
        const bool fin = worst() <= (FINE + 1) * (FINE + 1);
        state[8 * y0] = fin ? kNear : kFar;
        if (fin) store(y0);
        else far = true;
    }
    if (!__syncthreads_or(far)) return;
    // The far groups by halving: groups are numbered from 1, those that are odd
    // multiples of `step` lie between two multiples of 2 step, which are finished (0
    // and numbers past the last stand for the column's ends).
    const int groups = (a.n + 3) / 4;
    int step = 1;
    while (2 * step <= groups) step *= 2;
    for (; step > 0; step /= 2) {
        for (int i = w;; i += NW) {
            const int below = 2 * step * i, above = below + 2 * step, g = below + step;
            if (g > groups) break;
            const bool todo = state[32 * (g - 1)] == kFar;
            if (!__any_sync(0xffffffffu, todo)) continue;
            const int y0 = 4 * (g - 1);
            int lo = y0, hi = y0, at = y0;
            if (todo) {
                own(y0);
                lo = 0;
                hi = a.n - 1;
                // a group found near lies at most FINE + 1 rows from its result; one of
                // the other class is its own
                if (below > 0) {
                    const int yn = 4 * (below - 1);
                    const unsigned short sn = state[8 * yn];
                    lo = sn == kNear ? max(yn + 2 - FINE, 0) : s[0] * v[32 * yn] > 0 ? sn : yn + 3;
                }
                if (above <= groups) {
                    const int yn = 4 * (above - 1);
                    const unsigned short sn = state[8 * yn];
                    hi = sn == kNear ? min(yn + FINE + 1, hi) : s[0] * v[32 * yn] > 0 ? sn : yn;
                }
            }
            // row r: its distance to the group's first row, and to all four
            auto row = [&](int r) {
                const int q = max(s[0] * v[32 * r], 0), d = r - y0, c = q + d * d;
                if (c < best[0]) {
                    best[0] = c;
                    at = r;
                }
                best[1] = min(best[1], c - 2 * d + 1);
                best[2] = min(best[2], c - 4 * d + 4);
                best[3] = min(best[3], c - 6 * d + 9);
            };
            if (todo) {
                row(lo);
                row(hi);
                // rows further away than the worst distance so far cannot improve any
                const int reach = (int)sqrtf((float)worst()) + 1;
                lo = max(lo, y0 - reach);
                hi = min(hi, y0 + 3 + reach);
            }
            const int last = __reduce_max_sync(0xffffffffu, hi - lo);
            if (todo) {
                for (int i = 0; i <= last; i += 4) {
#pragma unroll
                    for (int m = 0; m < 4; ++m) row(min(lo + i + m, hi));
                }
                state[8 * y0] = (unsigned short)at;
                store(y0);
            }
        }
        __syncthreads();
    }
}

size_t tile_smem(int n) { return 128 * (size_t)n + 64 * ((size_t)(n + 3) / 4); }

// Threads per block.  Three blocks share an SM at about 500 rows, and with 256
// threads leave it half of its warps: 256 x 448 x 512 voxels of winding vessels take 874
// us with 256 threads for the 448 rows, 818 with 512; 500^3 1897 and 1737, a single
// corner voxel there 3605 and 3396.  At 300 rows and below eight or more blocks of
// 256 fill it, and 512 threads share too few groups: 256^3 cut by a slanted plane 427 us
// and 486.
constexpr int kWideFrom = 400;

// TRY and FINE, by winding vessels (the first figure) and planes (the second), with 256
// threads: 4 and 24 take 0.87 and 1.45 ms on 256 x 448 x 512 voxels, 8 and 48 0.86 and 1.72.  In short
// columns the halving's levels, one after the other, are latency: 128^3 takes 76 and
// 125 us with 4 and 24, 69 and 177 with 8 and 48, 96^3 54 and 75, 49 and 94.
template <bool FINAL>
void launch_tile(const TileArgs &a, cudaStream_t st) {
    const unsigned blocks = (unsigned)((a.ncols + 31) / 32);
    const size_t sm = tile_smem(a.n);
    if (a.n >= kWideFrom) sdf_cols_tile<FINAL, 512, 4, 24><<<blocks, 512, sm, st>>>(a);
    else if (a.n > kShortMax) sdf_cols_tile<FINAL, 256, 4, 24><<<blocks, 256, sm, st>>>(a);
    else sdf_cols_tile<FINAL, 256, 8, 48><<<blocks, 256, sm, st>>>(a);
}

template <bool FINAL, int T>
cudaError_t allow_tile() {
    return cudaFuncSetAttribute(sdf_cols_tile<FINAL, T, 4, 24>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)tile_smem(T == 512 ? kTileMax : kWideFrom));
}

}  // namespace

cudaError_t config_signed_distance() {
    cudaError_t e = allow_tile<false, 256>();
    if (e == cudaSuccess) e = allow_tile<true, 256>();
    if (e == cudaSuccess) e = allow_tile<false, 512>();
    if (e == cudaSuccess) e = allow_tile<true, 512>();
    return e;
}

cudaError_t launch_signed_distance(const void *seed, int f32, float thr, float *phi, int W, int H, int L,
                                   unsigned *scratch, cudaStream_t st) {
    const size_t N = (size_t)W * H * L;
    unsigned *d = scratch, *sv = scratch + N, *sf = scratch + 2 * N;
    const long long rows = (long long)H * L;
    const float fill = (float)W + (float)H + (float)L;
    if (W <= kTileMax && H <= kTileMax && L <= kTileMax) {
        short *dx = reinterpret_cast<short *>(scratch + N);
        int *dxy = reinterpret_cast<int *>(scratch);
        sdf_rows_tile<<<(unsigned)((rows + kRowWarps - 1) / kRowWarps), 32 * kRowWarps, 0, st>>>(seed, f32, thr, dx, W,
                                                                                                rows);
        launch_tile<false>(TileArgs{dx, dxy, nullptr, W, H, W * L, (long long)W * H, W, fill}, st);
        launch_tile<true>(TileArgs{dxy, nullptr, phi, W, L, W * H, W, (long long)W * H, fill}, st);
        return cudaGetLastError();
    }
    for (int feat_inside = 0; feat_inside < 2; feat_inside++) {
        sdf_rows<<<(unsigned)((rows + kRowWarps - 1) / kRowWarps), 32 * kRowWarps, 0, st>>>(seed, f32, thr,
                                                                                           feat_inside, d, W, rows);
        ColArgs a{d, sv, sf, (long long)W * L, W, (long long)W * H, W, H, seed, f32, thr, feat_inside, phi, fill};
        sdf_cols<false><<<(unsigned)((a.ncols + kColThreads - 1) / kColThreads), kColThreads, 0, st>>>(a);
        a.ncols = (long long)W * H;
        a.plane = W;
        a.stride = (long long)W * H;
        a.n = L;
        sdf_cols<true><<<(unsigned)((a.ncols + kColThreads - 1) / kColThreads), kColThreads, 0, st>>>(a);
    }
    return cudaGetLastError();
}

}  // namespace rsf
