// rsf_stencil_pair.cuh -- the stencil / update kernel of the evolution:
// gradient, |gradient|, normalised gradient, curvature, the wide "Laplacian",
// delta and the explicit update (CUDA_RSF/kernel.cu:57-125, 173-189, 265-280,
// 365-387, 630-933), phi read and written once.
//
// What bounds it is instruction issue (about 70 correctly rounded FP32
// operations per voxel, among them a square root, a reciprocal and a
// quotient), so a thread carries the voxels of two adjacent rows and does
// their arithmetic in packed f32x2 instructions.  A block is SP_WARPS warps of
// 2 rows x 32 columns (rows y0-1 .. y0+14, columns x0-1 .. x0+30; the outer
// ones are halo) and streams c.zc planes.  Each step forms the gradient and normalised
// gradient of plane s+1 once per voxel and writes phi of plane s.  phi arrives
// through a ring of SP_RING planes in shared memory filled by cp.async,
// SP_RING - 2 steps ahead of its first use, so that no load's latency stalls a
// warp (and through it the block's barrier).  x neighbours of phi come from
// those rows, of the gradients by shuffles; y neighbours are the thread's own
// other row or come from shared memory; z neighbours are in registers (rings
// indexed by plane mod 3, compile-time slots of a 3-way unrolled plane loop).
// One barrier per plane.
//
// Measured per launch on the 48 sub-volumes cut from 512 x 1024 x 1024 voxels:
// 8.22 ms with one voxel per thread (32 warps per SM, 237 thread instructions
// per voxel, 67 % issue), 5.48 ms here (24 warps, 80 registers, 160 and 66 %).
// With phi loaded into registers one plane ahead its first form (5.64 ms) took
// 6.89 ms (long scoreboard stalls behind every barrier), with four rows per thread
// and 16 warps 8.80 ms, with 64 registers and 32 warps 6.75 ms (spills).
#pragma once
#include "rsf_kernels.cuh"

namespace rsf {

constexpr int SP_WARPS = (ST_OY + 2) / 2;         // one row pair each
constexpr int SP_RING = 6;                        // phi planes in shared memory
constexpr int SP_SLOT = (SP_WARPS + 2) * 34 * 2;  // floats of one
static_assert(SP_WARPS == 8, "warp 1 loads the outer x neighbours of 16 rows");

struct PairSmem {
    // phi, plane z0 - 2 + j in slot j mod SP_RING: [w + 1][lane + 1] holds the
    // warp's two rows; columns 0 and 33 the outer x neighbours, rows 0 (.y) and
    // SP_WARPS + 1 (.x) the outer y neighbours
    float2 P[SP_RING][SP_WARPS + 2][34];
    // n_y, g_y of the two rows at [w + 1]; rows 0 and SP_WARPS + 1 are read
    // only for results that are not used
    float2 NY[3][SP_WARPS + 2][32];
    float2 GY[3][SP_WARPS + 2][32];
};

// Per-thread state that does not change along z.  Row 0 is y0 - 1 + 2 w, row 1
// the next.  In the reference boundary mode the left neighbour of x = 0 is the
// previous linear element, so lane 0 of a block at x = 0 carries the column one
// element before lane 1's in memory: (W-1, y-1), and for y = 0 (W-1, H-1) of
// the previous plane, whose plane numbers lag by one (`wrap`, warp 0).
struct PairCtx {
    int W, L, rz, z0, z1, zend, lane, w;  // rz: planes of border band at each end; zend: end of the planes read
    size_t WH, dplane, iplane;            // steps between planes: phi, data factor, image (bytes)
    int dstep, istep;                     // steps between the rows: data factor, image (bytes)
    bool in0, in1;          // the rows' voxels exist
    bool out0, out1;        // and are outputs of this block
    bool val0, val1;        // inside the blur's valid region in x and y
    bool xl_self, xr_self;  // one-sided x differences
    int ytop, ybot;         // the row (0, 1 or another) without a row above / below
    bool self00;            // row 1 is voxel (0, 0): its left neighbour in plane 0 is itself
    int wrap;               // 1: this lane lags by one plane
    bool hwarp, hal;        // this warp loads outer neighbours, this thread one of them
    int hlow;               // first plane of the latter
};

struct PairState {
    float2 P[3];                        // phi of the planes
    float2 NX[3], GX[3], NZ[3], GZ[3];  // gradients of the planes
    float2 NY, GY;                      // n_y, g_y of plane sc
    float2 D[3];                        // data factor, or the image in the border band
};

struct PairPtr {
    const float *a;            // row 0 of plane sc + SP_RING (row 1 W elements on)
    const float *h;            // the thread's outer neighbour of the same plane
    float *s, *hs;             // their places in slot 0
    float *o;                  // row 0 of the output of plane sc
    const float *d;            // row 0 of the data factor of plane sc + 1
    const unsigned char *i;    // row 0 of the image of plane sc + 1
};

__device__ __forceinline__ float2 shfl_up2(float2 v) {
    return make_float2(__shfl_up_sync(0xffffffffu, v.x, 1), __shfl_up_sync(0xffffffffu, v.y, 1));
}
__device__ __forceinline__ float2 shfl_down2(float2 v) {
    return make_float2(__shfl_down_sync(0xffffffffu, v.x, 1), __shfl_down_sync(0xffffffffu, v.y, 1));
}

// Copies plane p of phi (at q.a and q.h) into slot `slot`, as one commit group
// (empty outside the planes that the block reads).
template <bool EDGE, bool FACE>
__device__ __forceinline__ void pair_fill(const PairCtx &k, const PairPtr &q, int p, int slot) {
    const int lag = EDGE ? k.wrap : 0;
    if (!EDGE || (p >= lag && p < k.zend + lag)) {
        float *d = q.s + slot * SP_SLOT;
        if (!FACE || k.in0) cp_async4(d, q.a);
        if (!FACE || k.in1) cp_async4(d + 1, q.a + k.W);
    }
    if (k.hwarp && k.hal && (!EDGE || (p >= k.hlow && p < k.zend))) cp_async4(q.hs + slot * SP_SLOT, q.h);
    cp_commit();
}

// The image word of a border voxel, and its data factor: f_out = f_in =
// 30/30 = 1 there (kernel.cu:300-325).
__device__ __forceinline__ float border_word(const unsigned char *ip, int img_f32) {
    return img_f32 ? __ldg(reinterpret_cast<const float *>(ip)) : __uint_as_float(__ldg(ip));
}
__device__ __forceinline__ float border_factor(float word, const StepConst &c) {
    const float I = c.img_f32 ? word : (float)__float_as_uint(word);
    const float d = __fsub_rn(I, 1.0f);
    const float e = __fmul_rn(d, d);
    return data_factor(e, e, c.l1, c.l2, c.lam_equal != 0);
}

// One plane.  INSIDE: every output of the step and the next lies in the blur's
// valid region.  EDGE: the step may meet the first or last plane of the
// volume or of the block.  FACE: the block touches an x or y face.  C: step
// mod 3 (slot of the register rings), half: 3 * (step / 3 mod 2).
template <int C, Arith A, bool INSIDE, bool EDGE, bool FACE>
__device__ __forceinline__ void pair_step(const PairCtx &k, const StepConst &c, PairState &S, PairPtr &q, int sc,
                                          int half, PairSmem &sm, float2 &acc) {
    constexpr int C1 = (C + 1) % 3, C2 = (C + 2) % 3;
    const int t1 = C == 2 ? 3 - half : C + 1 + half;       // slot of plane sc + 1
    const int t2 = C >= 1 ? C - 1 + (3 - half) : 2 + half; // slot of plane sc + 2
    const PairConst &pk = c.pk;
    // plane sc has been read by every warp: its slot takes plane sc + SP_RING
    pair_fill<EDGE, FACE>(k, q, sc + SP_RING, C + half);
    q.a += k.WH;
    if (k.hwarp) q.h += k.WH;
    // data factor of plane sc + 1 (read once, so from L2: 5.48 ms per launch on the 48
    // sub-volumes, 5.53 through L1), or the image in the border band
    float2 dn = make_float2(0.0f, 0.0f);
    if (INSIDE) {
        if (k.out0) dn.x = __ldcg(q.d);
        if (k.out1) dn.y = __ldcg(q.d + k.dstep);
    } else if (!EDGE || (sc + 1 >= k.z0 && sc + 1 < k.z1)) {
        const bool zin = sc + 1 >= k.rz && sc + 1 < k.L - k.rz;
        if (zin && k.val0) dn.x = __ldcg(q.d);
        else if (k.out0) dn.x = border_word(q.i, c.img_f32);
        if (zin && k.val1) dn.y = __ldcg(q.d + k.dstep);
        else if (k.out1) dn.y = border_word(q.i + k.istep, c.img_f32);
    }
    q.d += k.dplane;
    if (!INSIDE) q.i += k.iplane;
    // plane sc + 2 (filled SP_RING - 2 steps ago) has arrived
    asm volatile("cp.async.wait_group %0;" ::"n"(SP_RING - 2) : "memory");
    S.P[C2] = sm.P[t2][k.w + 1][k.lane + 1];
    // gradient of plane pn
    const int pn = sc + 1;
    const float2 p0 = S.P[C], p1 = S.P[C1];
    float2 l = sm.P[t1][k.w + 1][k.lane], r = sm.P[t1][k.w + 1][k.lane + 2];
    float u0 = sm.P[t1][k.w][k.lane + 1].y, d0 = p1.y;   // above and below row 0
    float u1 = p1.x, d1 = sm.P[t1][k.w + 2][k.lane + 1].x;  // row 1
    if (FACE) {
        if (k.xl_self) l = p1;
        if (k.xr_self) r = p1;
        if (k.ytop == 0) u0 = p1.x;
        if (k.ytop == 1) u1 = p1.y;
        if (k.ybot == 0) d0 = p1.x;
        if (k.ybot == 1) d1 = p1.y;
        if (EDGE && k.self00 && pn == 0) l.y = p1.y;
    }
    const int lag = EDGE ? k.wrap : 0;
    const float2 zl = (!EDGE || pn > lag) ? p0 : p1;
    const float2 zr = (!EDGE || pn < k.L - 1 + lag) ? S.P[C2] : p1;
    const float2 gx = half_diff2(r, l), gy = half_diff2(d0, u0, d1, u1), gz = half_diff2(zr, zl);
    unsigned small = 0xffffffffu;
    Normals2 n = A == Arith::Portable ? normals2(gx, gy, gz, small) : normals2_scalar<A>(gx, gy, gz);
    if (A == Arith::Portable && normals_small(small)) n = normals2_rare(gx, gy, gz);
    S.GX[C1] = gx;
    S.GZ[C1] = gz;
    S.NX[C1] = n.x;
    S.NZ[C1] = n.z;
    sm.NY[C1][k.w + 1][k.lane] = n.y;
    sm.GY[C1][k.w + 1][k.lane] = gy;
    __syncthreads();
    // output plane sc
    const float2 nc = S.NX[C], gc = S.GX[C], nyc = S.NY, gyc = S.GY;
    float2 nxl = shfl_up2(nc), nxr = shfl_down2(nc), gxl = shfl_up2(gc), gxr = shfl_down2(gc);
    float nu0 = sm.NY[C][k.w][k.lane].y, nd0 = nyc.y, nu1 = nyc.x, nd1 = sm.NY[C][k.w + 2][k.lane].x;
    float gu0 = sm.GY[C][k.w][k.lane].y, gd0 = gyc.y, gu1 = gyc.x, gd1 = sm.GY[C][k.w + 2][k.lane].x;
    if (FACE) {
        if (k.xl_self) nxl = nc, gxl = gc;
        if (k.xr_self) nxr = nc, gxr = gc;
        if (k.ytop == 0) nu0 = nyc.x, gu0 = gyc.x;
        if (k.ytop == 1) nu1 = nyc.y, gu1 = gyc.y;
        if (k.ybot == 0) nd0 = nyc.x, gd0 = gyc.x;
        if (k.ybot == 1) nd1 = nyc.y, gd1 = gyc.y;
        if (EDGE && k.self00 && sc == 0) nxl.y = nc.y, gxl.y = gc.y;
    }
    const bool zlo = !EDGE || sc > 0, zhi = !EDGE || sc < k.L - 1;
    const float2 nzl = zlo ? S.NZ[C2] : S.NZ[C], nzr = zhi ? n.z : S.NZ[C];
    const float2 gzl = zlo ? S.GZ[C2] : S.GZ[C], gzr = zhi ? gz : S.GZ[C];
    const float2 kap = add2(add2(half_diff2(nxr, nxl), half_diff2(nd0, nu0, nd1, nu1)), half_diff2(nzr, nzl));
    const float2 lap = add2(add2(half_diff2(gxr, gxl), half_diff2(gd0, gu0, gd1, gu1)), half_diff2(gzr, gzl));
    float2 data = S.D[C];
    if (!INSIDE) {
        const bool zin = sc >= k.rz && sc < k.L - k.rz;
        if (!(zin && k.val0)) data.x = border_factor(data.x, c);
        if (!(zin && k.val1)) data.y = border_factor(data.y, c);
    }
    const float2 out = update_phi2(p0, dirac2<A>(p0, c.eps, pk), data, kap, lap, pk);
    if ((!EDGE || sc >= k.z0) && k.out0) {
        q.o[0] = out.x;
        acc.x = __fmaf_rn(out.x, 0.0f, acc.x);
    }
    if ((!EDGE || sc >= k.z0) && k.out1) {
        q.o[k.W] = out.y;
        acc.y = __fmaf_rn(out.y, 0.0f, acc.y);
    }
    q.o += k.WH;
    S.NY = n.y;
    S.GY = gy;
    S.D[C1] = dn;
}

// The block's planes in groups of three (one per ring slot).  Groups that can
// meet no z rule and no end of the plane range run without the plane tests;
// `xyin`: the block's columns lie in the blur's valid region, so its groups
// clear of the border band in z do too.
template <Arith A, bool FACE>
__device__ __forceinline__ void pair_planes(const PairCtx &k, const StepConst &c, PairState &S, PairPtr &q,
                                            PairSmem &sm, float2 &acc, bool xyin) {
    const int first = k.z0 - 2, count = k.z1 - first;
    int half = 0;
    for (int i = 0; i < count; i += 3, half = 3 - half) {
        const int sc = first + i;
        if (i == 0 || sc <= 0 || sc + 2 + SP_RING >= k.zend) {
            pair_step<0, A, false, true, FACE>(k, c, S, q, sc, half, sm, acc);
            if (i + 1 < count) pair_step<1, A, false, true, FACE>(k, c, S, q, sc + 1, half, sm, acc);
            if (i + 2 < count) pair_step<2, A, false, true, FACE>(k, c, S, q, sc + 2, half, sm, acc);
        } else if (!FACE && xyin && sc >= k.rz && sc + 3 < k.L - k.rz) {
            pair_step<0, A, true, false, FACE>(k, c, S, q, sc, half, sm, acc);
            pair_step<1, A, true, false, FACE>(k, c, S, q, sc + 1, half, sm, acc);
            pair_step<2, A, true, false, FACE>(k, c, S, q, sc + 2, half, sm, acc);
            q.i += 3 * k.iplane;
        } else {
            pair_step<0, A, false, false, FACE>(k, c, S, q, sc, half, sm, acc);
            pair_step<1, A, false, false, FACE>(k, c, S, q, sc + 1, half, sm, acc);
            pair_step<2, A, false, false, FACE>(k, c, S, q, sc + 2, half, sm, acc);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

template <Arith A>
__global__ void __launch_bounds__(SP_WARPS * 32, 3) stencil_pair_kernel(const SubVolDev *__restrict__ svs,
                                                                                const int *__restrict__ pre,
                                                                                const __grid_constant__ StepConst c,
                                                                                int parity,
                                                                                unsigned *__restrict__ flag) {
    __shared__ PairSmem sm;
    const int b = blockIdx.x;
    const int sv = find_sv(pre, c.nsv, b);
    const SubVolDev s = svs[sv];
    int t = b - __ldg(pre + sv);
    PairCtx k;
    const int W = s.W, H = s.H, L = s.L, r = c.r;
    k.W = W;
    k.L = L;
    k.lane = threadIdx.x & 31;
    k.w = threadIdx.x >> 5;
    const int ntx = (W + ST_OX - 1) / ST_OX, nty = (H + ST_OY - 1) / ST_OY;
    const int x0 = (t % ntx) * ST_OX;
    t /= ntx;
    const int y0 = (t % nty) * ST_OY;
    k.z0 = (t / nty) * c.zc;
    k.z1 = min(k.z0 + c.zc, L);
    k.zend = min(k.z1 + 2, L);
    k.WH = (size_t)W * H;
    const ptrdiff_t WH = (ptrdiff_t)k.WH;
    const bool ref = c.boundary == 0, carried = ref && x0 == 0;
    const bool carry = carried && k.lane == 0;
    const int x = x0 - 1 + k.lane, ya = y0 - 1 + 2 * k.w;
    // the voxel carried in row 0: (x, ya), or one element back for the carry lane
    const int ex = carry ? W - 1 : x, ea = carry ? ya - 1 : ya;
    k.wrap = carry && ya == -1 ? 1 : 0;
    const bool xin = ex >= 0 && ex < W;
    k.in0 = xin && ((ea >= 0 && ea < H) || k.wrap);
    k.in1 = xin && ((ea >= -1 && ea + 1 < H) || k.wrap);
    const bool col_out = k.lane >= 1 && k.lane <= ST_OX && x < W;
    k.out0 = col_out && k.w > 0 && ya < H;
    k.out1 = col_out && k.w < SP_WARPS - 1 && ya + 1 < H;
    const bool xval = s.Wv > 0 && x >= r && x < W - r;
    k.val0 = k.out0 && xval && ya >= r && ya < H - r;
    k.val1 = k.out1 && xval && ya + 1 >= r && ya + 1 < H - r;
    k.rz = r;
    bool xyin = s.Wv > 0 && x0 >= r && x0 + ST_OX - 1 < W - r && y0 >= r && y0 + ST_OY - 1 < H - r;
    k.xl_self = !ref && ex == 0;
    k.xr_self = ex == W - 1;
    k.ytop = -ea;
    k.ybot = k.wrap ? 1 : H - 1 - ea;
    k.self00 = ref && x == 0 && ya == -1;
    // Offset of row 0 in its plane.  The carry lane's is the linear one of
    // x = -1, which is the previous element.
    const ptrdiff_t cola = (ptrdiff_t)ya * W + x;

    const float *phi = parity ? s.phi[1] : s.phi[0];
    float *phi_out = parity ? s.phi[0] : s.phi[1];
    const int esz = c.img_f32 ? 4 : 1;
    PairPtr q;
    q.a = phi + cola;
    // Outer neighbours: warp 0 loads the row above the block, the last warp
    // the row below, and warp 1 the two columns beside it (lane: 2 * row +
    // side).  They exist where the thread they serve has a voxel and the
    // neighbour is another one; the lagging row's needs planes 1 ..
    k.hlow = 0;
    ptrdiff_t hoff = 0;
    int hpair = 0, hcol = 0, hlane = 0;
    if (k.w == 0) {
        k.hal = xin && ea >= 1 && ea < H;
        hoff = cola - W;
        hpair = 0, hcol = k.lane + 1, hlane = 1;
    } else if (k.w == SP_WARPS - 1) {
        k.hal = xin && ea + 2 < H;
        hoff = cola + 2 * (ptrdiff_t)W;
        hpair = SP_WARPS + 1, hcol = k.lane + 1, hlane = 0;
    } else {
        const int row = k.lane >> 1, side = k.lane & 1, y = y0 - 1 + row;
        if (side) {
            k.hal = x0 + 31 < W && y >= 0 && y < H;
        } else if (carried) {  // (W - 2, y - 1)
            k.hlow = y == 0 ? 1 : 0;
            k.hal = y >= 0 && y <= H;
        } else {
            k.hal = x0 >= 2 && y >= 0 && y < H;
        }
        k.hal = k.hal && k.w == 1 && row < 2 * SP_WARPS;
        hoff = (ptrdiff_t)y * W + (side ? x0 + 31 : x0 - 2);
        hpair = min(row / 2, SP_WARPS - 1) + 1, hcol = side ? 33 : 0, hlane = row & 1;
    }
    k.hwarp = k.w <= 1 || k.w == SP_WARPS - 1;
    q.h = phi + hoff;
    q.hs = reinterpret_cast<float *>(&sm.P[0][hpair][hcol]) + hlane;
    q.s = reinterpret_cast<float *>(&sm.P[0][k.w + 1][k.lane + 1]);
    q.o = phi_out + cola + (ptrdiff_t)(k.z0 - 2) * WH;
    q.i = static_cast<const unsigned char *>(s.img) + (cola + (ptrdiff_t)(k.z0 - 1) * WH) * esz;
    k.istep = W * esz;
    k.iplane = k.WH * esz;
    k.dstep = s.Wp;
    k.dplane = (size_t)s.Wp * s.Hv;
    q.d = s.db + ((ptrdiff_t)(ya - r) * s.Wp + (x - r)) + (ptrdiff_t)(k.z0 - 1 - r) * (ptrdiff_t)k.dplane;
    if (c.full_data) {  // every voxel's data factor comes from the box or expanded data-term kernels
        xyin = true;
        k.rz = 0;
        k.val0 = k.out0;
        k.val1 = k.out1;
        k.dstep = W;
        k.dplane = k.WH;
        q.d = s.db + 2 * (size_t)s.Wp * s.Hv * s.Lv + cola + (ptrdiff_t)(k.z0 - 1) * WH;
    }

    // The first SP_RING planes from z0 - 2 on.
    pdl_wait();
    PairState S;
    const int first = k.z0 - 2;
    q.a += (ptrdiff_t)first * WH;
    q.h += (ptrdiff_t)first * WH;
#pragma unroll
    for (int j = 0; j < SP_RING; ++j) {
        pair_fill<true, true>(k, q, first + j, j);
        q.a += k.WH;
        q.h += k.WH;
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) S.NX[j] = S.GX[j] = S.NZ[j] = S.GZ[j] = S.D[j] = make_float2(0.0f, 0.0f);
    S.NY = S.GY = make_float2(0.0f, 0.0f);
    asm volatile("cp.async.wait_group %0;" ::"n"(SP_RING - 2) : "memory");
    S.P[0] = sm.P[0][k.w + 1][k.lane + 1];
    S.P[1] = sm.P[1][k.w + 1][k.lane + 1];
    __syncthreads();

    // x/y-interior blocks: every thread and outer neighbour exists, no face rule
    const bool face = !(x0 >= 2 && x0 + 32 <= W && y0 >= 2 && y0 + ST_OY + 2 <= H);
    float2 acc = make_float2(0.0f, 0.0f);  // NaN once an output is not finite
    if (face) pair_planes<A, true>(k, c, S, q, sm, acc, xyin);
    else pair_planes<A, false>(k, c, S, q, sm, acc, xyin);
    pdl_launch();
    if (!isfinite(acc.x + acc.y)) atomicOr(flag, kFlagNonFinite);
}

}  // namespace rsf
