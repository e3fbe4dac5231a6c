// Compares the packed arithmetic of csrc/rsf_pair.cuh with the correctly rounded intrinsics and with the
// scalar arithmetic, over ranges of arguments (test_gpu_pair_arith.py).  A NaN's payload does not count.
#include <cuda_runtime.h>

#include "rsf_pair.cuh"

using namespace rsf;

namespace {
struct Result {
    unsigned long long bad;
    float arg[3];
};

__device__ bool differ(float a, float b) { return __float_as_uint(a) != __float_as_uint(b) && !(isnan(a) && isnan(b)); }
__device__ bool differ(float2 a, float2 b) { return differ(a.x, b.x) || differ(a.y, b.y); }
__device__ void report(Result *r, float a, float b = 0.0f, float c = 0.0f) {
    if (atomicAdd(&r->bad, 1ull) == 0ull) r->arg[0] = a, r->arg[1] = b, r->arg[2] = c;
}

// splitmix64 (Steele, Lea, Flood, "Fast splittable pseudorandom number generators", OOPSLA 2014)
__device__ unsigned long long mix(unsigned long long x) {
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}
// a float with exponent field in [lo, hi] and any mantissa and sign; one in eight is made of a power of two
// and up to two units in the last place
__device__ float random_float(unsigned long long h, int lo, int hi) {
    const unsigned e = lo + (unsigned)(h >> 40) % (unsigned)(hi - lo + 1);
    unsigned m = (unsigned)h & 0x7fffffu;
    if (((h >> 32) & 7u) == 0u) m = (m & 2u) ? m & 3u : 0x7fffffu - (m & 3u);
    return __uint_as_float((unsigned)(h >> 23 & 1u) << 31 | e << 23 | m);
}

enum { RCP, SQRT, DIRAC, HEAVISIDE, DIV, NORMALS };

// RCP .. HEAVISIDE: bit patterns lo .. lo + n - 1, each beside the next one of another block of patterns.
// DIV, NORMALS: n random arguments with exponent fields lo .. hi.
__global__ void sweep(int what, unsigned lo, unsigned hi, unsigned long long n, float eps, const PairConst c, Result *r) {
    const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n; i += step) {
        if (what <= HEAVISIDE) {
            const float2 x = make_float2(__uint_as_float(lo + (unsigned)i), __uint_as_float(lo + (unsigned)((i * 2654435761ull) % n)));
            float2 got, want;
            if (what == RCP) got = rcp2(x), want = make_float2(__frcp_rn(x.x), __frcp_rn(x.y));
            if (what == SQRT) got = sqrt2(x), want = make_float2(__fsqrt_rn(x.x), __fsqrt_rn(x.y));
            if (what == DIRAC)
                got = dirac2<Arith::Portable>(x, eps, c),
                want = make_float2(dirac<Arith::Portable>(x.x, eps), dirac<Arith::Portable>(x.y, eps));
            if (what == HEAVISIDE)
                got = heaviside2<Arith::Portable>(x, eps, c),
                want = make_float2(heaviside<Arith::Portable>(x.x, eps), heaviside<Arith::Portable>(x.y, eps));
            if (differ(got, want)) report(r, x.x, x.y, eps);
        } else if (what == DIV) {
            const float2 a = make_float2(random_float(mix(4 * i), lo, hi), random_float(mix(4 * i + 1), lo, hi));
            const float2 b = make_float2(random_float(mix(4 * i + 2), lo, hi), random_float(mix(4 * i + 3), lo, hi));
            if (differ(div2(a, b), make_float2(__fdiv_rn(a.x, b.x), __fdiv_rn(a.y, b.y)))) report(r, a.x, b.x, a.y);
        } else {
            float2 g[3];
            for (int k = 0; k < 3; ++k)
                g[k] = make_float2(random_float(mix(8 * i + 2 * k), lo, hi), random_float(mix(8 * i + 2 * k + 1), lo, hi));
            if (mix(8 * i + 6) & 1) g[1] = g[2] = make_float2(0.0f, 0.0f);
            unsigned small = 0xffffffffu;
            Normals2 got = normals2(g[0], g[1], g[2], small);
            if (normals_small(small)) got = normals2_rare(g[0], g[1], g[2]);
            const Normals2 want = normals2_scalar<Arith::Portable>(g[0], g[1], g[2]);
            if (differ(got.x, want.x) || differ(got.y, want.y) || differ(got.z, want.z)) report(r, g[0].x, g[1].x, g[2].x);
        }
    }
}
}  // namespace

// Mismatches, and an argument of the first one; -1 after a CUDA error.
extern "C" long long pair_sweep(int what, unsigned lo, unsigned hi, unsigned long long n, float eps, float *arg) {
    PairConst c;
    set_pair_const(c, eps, 0.1f, 0.1f, 0.1f);
    Result *d = nullptr, h = {};
    if (cudaMalloc(&d, sizeof h) != cudaSuccess || cudaMemset(d, 0, sizeof h) != cudaSuccess) return -1;
    sweep<<<1216, 256>>>(what, lo, hi, n, eps, c, d);
    const cudaError_t e = cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return -1;
    for (int k = 0; k < 3; ++k) arg[k] = h.arg[k];
    return (long long)h.bad;
}
