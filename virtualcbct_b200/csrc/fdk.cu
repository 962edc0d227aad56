// fdk.cu -- FDK ramp filter (direct FP32 path) and voxel-driven cone-beam
// backprojection on sm_100a.
//
// Reference: Release_recon_from_forward_pro_float_CM/filterSinogram.cpp:67-131
// and reconstructImage.cpp:10-184 (OpenMP CPU code).
#include "internal.h"

#include <algorithm>
#include <climits>
#include <cstdlib>
#include <type_traits>

namespace vcbct {
namespace {

// Packed pairs of floats for Blackwell's f32x2 arithmetic: one instruction
// for two elements, each rounded exactly as the scalar instruction would
// round it.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 f2pack(float a, float b)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2unpack(f32x2 r, float& a, float& b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ f32x2 ffma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 fmul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fsub2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fadd2_rd(f32x2 a, f32x2 b)  // rounded toward -inf, as __fadd_rd
{
    f32x2 r;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// ------------------------------------------------------------------ filter --
// out[r][m] = Cm(v, n, m) * sum_k hT[k][m] * g[r][k],  g = -logf(p),  r = v*H + n,
// where hT already holds the diagonal coefficient (filterSinogram.cpp:103) and
// the ramp kernel (:106-110).  -logf is applied while staging g (the
// reference's log of a float is the float overload, :103/:108); every sum runs
// over k upward in one chain of fused multiply-adds.
//
// Bound by the FP32 pipe (2 W flops per output).  A block keeps a chunk of g
// of its 64 rows in shared memory, transposed (k-major), and goes over the
// columns in passes of 32 to 192: a thread makes 8 rows x TN columns as row
// pairs in packed f32x2, so that a pass takes the logarithm once per 32 TN
// columns and TN + 2 shared loads feed 4 TN packed instructions.  The passes
// split the detector's 32-column groups evenly (400 columns: 160 + 128 + 128),
// so at most 31 columns are padding.  Coefficients are fetched a stage ahead
// into registers; two blocks per SM overlap one's staging with the other's
// arithmetic.  360 x 400 x 400, half-fan weights, one B200: 3.00 ms with 4 x 4
// outputs a thread and 64-column tiles, 1.51 ms now; the same sums bit for
// bit.
constexpr int FT_M = 64;       // rows a block
constexpr int FT_K = 8;        // k per stage of the coefficients
constexpr int FT_TN = 6;       // most 32-column groups a pass
constexpr int FT_LD = FT_M + 4;   // floats of a transposed row of g
constexpr int FT_CHUNK = 256;  // most k of g staged at a time

struct FilterArgs {
    const float* proj;
    float* out;
    const float* hT;
    const FilterView* views;
    const float* wts;
    float pitch, sad;
    int M, H, W;
    int kc;             // k of g staged at a time
    int groups, npass;  // 32-column groups, column passes
    int per;            // passes a block makes
};

// g of k in [kb, kb + kn) into As
__device__ __forceinline__ void filter_stage(const FilterArgs& a, int r0, int kb, int kn, float* As)
{
    // 8 k x 4 rows a warp: whole sectors, and the 32 banks of the transposed
    // store (FT_LD = 4 mod 32); eight loads in flight per thread
    const int kl = threadIdx.x % 8, rl = threadIdx.x / 8;
    for (int rr = rl; rr < FT_M; rr += 32) {
        const int r = r0 + rr;
        const float* pr = a.proj + (size_t)r * a.W + kb;
        const float* wr = a.wts ? a.wts + (size_t)(r / a.H) * a.W + kb : nullptr;
        for (int kq = kl; kq < kn; kq += 64) {
            float p[8], w[8];
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int k = kq + 8 * q;
                const bool in = k < kn && r < a.M;
                p[q] = in ? __ldg(pr + k) : 1.0f;
                w[q] = in && wr ? __ldg(wr + k) : 1.0f;
            }
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int k = kq + 8 * q;
                float g = -logf(p[q]);
                if (wr) g *= w[q];
                if (k < kn) As[k * FT_LD + rr] = g;
            }
        }
    }
}

// The TN x 32 columns from n0 on; staged: the whole of g is in As already.
template <int TN>
__device__ __forceinline__ void filter_pass(const FilterArgs& a, int r0, int n0, bool staged, float* As, float* Bs)
{
    constexpr int BN = 32 * TN;
    const int tx = threadIdx.x % 32, ty = threadIdx.x / 32, W = a.W;
    f32x2 acc[4][TN];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = 0ull;
    for (int kb = 0; kb < W; kb += a.kc) {
        const int kn = min(a.kc, W - kb);
        if (!staged) {
            __syncthreads();
            filter_stage(a, r0, kb, kn, As);
        }
        // warp ty fetches row ty of the next stage before a stage's
        // arithmetic and stores it after
        float bn[TN];
        const float* hp = a.hT + (size_t)(kb + ty) * W + n0 + tx;
        auto fetch = [&](int k0) {
            const bool in = k0 + ty < kn;
#pragma unroll
            for (int j = 0; j < TN; j++) bn[j] = in && n0 + tx + 32 * j < W ? __ldg(hp + 32 * j) : 0.0f;
            hp += (size_t)FT_K * W;
        };
        float* bs = Bs + ty * BN + tx;
        auto store = [&](int buf) {
#pragma unroll
            for (int j = 0; j < TN; j++) bs[buf * FT_K * BN + 32 * j] = bn[j];
        };
        fetch(0);
        store(0);
        __syncthreads();
        for (int k0 = 0, buf = 0; k0 < kn; k0 += FT_K, buf ^= 1) {
            const bool more = k0 + FT_K < kn;
            if (more) fetch(k0 + FT_K);
            const float* Ak = As + (size_t)k0 * FT_LD + ty * 8;
            const float* Bk = Bs + buf * FT_K * BN + tx;
            auto step = [&](int kk) {
                const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(Ak + kk * FT_LD);
                const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(Ak + kk * FT_LD + 4);
                const f32x2 av[4] = {a0.x, a0.y, a1.x, a1.y};
                f32x2 b[TN];
#pragma unroll
                for (int j = 0; j < TN; j++) {
                    const float bj = Bk[kk * BN + 32 * j];
                    b[j] = f2pack(bj, bj);
                }
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < TN; j++) acc[i][j] = ffma2(av[i], b[j], acc[i][j]);
            };
            if (k0 + FT_K <= kn) {
#pragma unroll
                for (int kk = 0; kk < FT_K; kk++) step(kk);
            } else {
#pragma unroll 1
                for (int kk = 0; kk < kn - k0; kk++) step(kk);
            }
            if (more) store(buf ^ 1);
            __syncthreads();
        }
    }
    // epilogue: cosine factor Cm = D / sqrt(D^2 + pos1^2 + pos2^2) (:92-99)
    const float pitch = a.pitch, sad = a.sad;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int r = r0 + ty * 8 + i;
        if (r >= a.M) continue;
        const int v = r / a.H, n = r - v * a.H;
        const FilterView sh = a.views[v];
        const float pos2 = fabsf(sh.ycs + (float)n) * pitch;
#pragma unroll
        for (int j = 0; j < TN; j++) {
            const int m = n0 + tx + 32 * j;
            if (m >= W) continue;
            float lo, hi;
            f2unpack(acc[i / 2][j], lo, hi);
            const float pos1 = fabsf(sh.xcs + (float)m) * pitch;
            // rounded the same way whatever the pass width
            const float cm = sad / sqrtf(__fadd_rn(fmaf(pos1, pos1, __fmul_rn(sad, sad)), __fmul_rn(pos2, pos2)));
            a.out[(size_t)r * W + m] = ((i & 1) ? hi : lo) * cm;
        }
    }
}

// MAXTN: the widest pass; narrow passes leave registers for twice the blocks (of
// which three fit where a block stages 256 columns, four up to 192).
template <int MAXTN>
__global__ void __launch_bounds__(256, MAXTN <= 2 ? 4 : 2) filter_direct_kernel(const __grid_constant__ FilterArgs a)
{
    extern __shared__ __align__(16) float f_smem[];
    float* As = f_smem;                            // [kc][FT_LD]
    float* Bs = f_smem + (size_t)a.kc * FT_LD;     // [2][FT_K][32 x widest pass]
    const int r0 = blockIdx.x * FT_M;
    const int p0 = blockIdx.y * a.per, p1 = min(a.npass, p0 + a.per);
    const int w0 = a.groups / a.npass, more = a.groups % a.npass;  // the first `more` passes are a group wider
    for (int p = p0; p < p1; p++) {
        const int n0 = 32 * (p * w0 + min(p, more));
        const bool staged = p > p0 && a.kc >= a.W;
        const int tn = w0 + (p < more);
        if (tn == 1) filter_pass<1>(a, r0, n0, staged, As, Bs);
        else if (tn == 2) filter_pass<2>(a, r0, n0, staged, As, Bs);
        if constexpr (MAXTN > 2) {
            if (tn == 3) filter_pass<3>(a, r0, n0, staged, As, Bs);
            else if (tn == 4) filter_pass<4>(a, r0, n0, staged, As, Bs);
            else if (tn == 5) filter_pass<5>(a, r0, n0, staged, As, Bs);
            else if (tn == 6) filter_pass<6>(a, r0, n0, staged, As, Bs);
        }
    }
}

// ----------------------------------------------------------- backprojection --
// One thread per (x, y) voxel column and a chunk of ZB slices (register
// accumulators).  Per (x, y, view) the detector column coordinate U, its
// interpolation weight and the magnification are formed in FP64 (the floor
// of U decides which two detector columns are read and must agree with the
// reference); per slice the row coordinate ZETA is an exact integer base plus
// an FP32 fractional offset.  Bilinear interpolation is manual FP32 with the
// reference's edge rules and its weight quirk (the column weight is frac(U),
// not frac(UUU), reconstructImage.cpp:80-83).
// Register cap (minimum resident 256-thread blocks per SM) and slices per
// thread.  The packed f32x2 slice loop needs register pairs: with the launch
// constants in the parameter bank, 5 blocks (48 registers) and 6 (40) both
// run without spills on 270x270x200 from 360 half-fan views, and 5 is faster
// on B200 (3.05 vs 3.21 ms, the volume bitwise the same).  16 slices per
// thread at 4 or 3 blocks measured slower (3.55 / 3.49 vs 3.30 ms): more
// columns leave the interior loop at the cone's edges.
#ifndef VCBCT_BP_MIN_BLOCKS
#define VCBCT_BP_MIN_BLOCKS 5
#endif
#ifndef VCBCT_BP_TILE
#define VCBCT_BP_TILE 4  // warp tile width in voxel columns (4, 8, 16 or 32)
#endif
#ifndef VCBCT_BP_ZB
#define VCBCT_BP_ZB 8
#endif
// Per (backprojection block, view): may any column of the block's 32 x 8
// tile take the view in backproject_kernel?  U, g = 1 / (L2 pitch) and the
// row coordinate H/2 + z g are linear-fractional in (x, y) with a positive
// denominator, so over the tile's rectangle they take their extremes at its
// four corners.  A view whose corner values put every column left of column
// 0 or right of column W - 1 (the column test UU < 0 || UU > W - 1), or every
// slice of the block above or below the detector (the row test), is
// dropped; the margin is far above FP64 rounding, so a dropped view is one
// every column of the tile would have skipped.  One warp per (block, 32
// views): bit th & 31 of word th >> 5 of the block's mask.
template <int ZB>
__global__ void __launch_bounds__(256) bp_cull_kernel(FdkParams f, const BpView* __restrict__ views,
                                                      int gx, int gy, int nblocks, unsigned* __restrict__ keep)
{
    constexpr double kMargin = 1e-3;  // detector pixels
    const int nwords = (f.V + 31) >> 5;
    const long wid = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (wid >= (long)nblocks * nwords) return;
    const int lane = threadIdx.x & 31;
    const int blk = (int)(wid / nwords), word = (int)(wid % nwords);
    const int bx = blk % gx, by = (blk / gx) % gy, bz = blk / (gx * gy);
    const int th = word * 32 + lane;
    bool keep_it = false;
    if (th < f.V) {
        const double pitch = f.piso * f.mpn / f.W;
        const double cp = (double)f.N / 2.0 - 0.5;
        const double inv_sad = 1.0 / f.sad;
        const int xa = bx * 32, xb = min(xa + 31, f.N - 1);
        const int ya = by * 8, yb = min(ya + 7, f.N - 1);
        const double zza = f.zstart + (double)(bz * ZB) * f.step;
        const double zzl = zza + (double)(ZB - 1) * f.step;
        const BpView bv = views[th];
        double umin = 1e300, umax = -1e300, gmin = 1e300, gmax = -1e300;
        bool ok = true;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const double xx = (((c & 1) ? xb : xa) - cp) * f.scale;
            const double yy = -(((c & 2) ? yb : ya) - cp) * f.scale;
            const double X = xx * bv.cs + yy * bv.sn;
            const double L2 = 1.0 - (-xx * bv.sn + yy * bv.cs) * inv_sad;
            ok = ok && L2 > 1e-3;
            const double g = 1.0 / (L2 * pitch);
            const double u = bv.ushift + X * g;
            umin = fmin(umin, u);
            umax = fmax(umax, u);
            gmin = fmin(gmin, g);
            gmax = fmax(gmax, g);
        }
        keep_it = true;
        if (ok) {
            const bool left = umax < -kMargin, right = umin >= (double)f.W + kMargin;
            const double last_max = (double)(f.H / 2) + fmax(zzl * gmin, zzl * gmax);
            const double first_min = (double)(f.H / 2) + fmin(zza * gmin, zza * gmax);
            const bool below = last_max < -1.0 - kMargin, above = first_min > (double)f.H + 1.0 + kMargin;
            keep_it = !(left || right || below || above);
        }
    }
    const unsigned m = __ballot_sync(0xffffffffu, keep_it);
    if (lane == 0) keep[wid] = m;
}

// Launch constants of the backprojection, formed on the host in the same
// IEEE double operations as the device would (kernel parameters, so they
// are read from the constant bank instead of occupying registers).
struct BpConst {
    double pitch;    // piso * mpn / W: detector pitch at the isocentre
    double inv_sad;  // 1 / sad
    double cp;       // N / 2 - 0.5: the volume centre in voxels
};

static_assert(sizeof(BpView) == 32, "BpView is staged as four 8-byte words");

// Slice block of launch index i of n, from the middle of the volume out
// (c, c + 1, c - 1, c + 2, ... with c = (n - 1) / 2): the blocks near the
// slab's centre, seen by every view, are the longest and start first, the
// short ones at the cone's edges fill the last wave.
__device__ __forceinline__ int bp_zblock(int i, int n)
{
    const int c = (n - 1) / 2, off = (i + 1) >> 1;
    return (i & 1) ? c + off : c - off;
}

// ZS: slices of the ZB of a slice block that one thread makes (ZB, or a part
// of them where whole slice blocks would not fill the GPU).  Row coordinates
// are formed from the slice block's first slice either way, so the volume is
// the same bit for bit.
// SV: the view table is copied to shared memory at block start (the
// per-view loads at the head of each set-up chain then come from shared
// memory instead of through L1).
template <int ZB, int ZS, int MINB, bool SV>
__global__ void __launch_bounds__(256, MINB) backproject_kernel(
    FdkParams f, BpConst k, const BpView* __restrict__ views, const float* __restrict__ filt,
    float* __restrict__ vol_f32, short* __restrict__ vol_i16, const unsigned* __restrict__ keep)
{
    // each warp takes a TW x (32 / TW) tile of the block's 32 x 8 columns:
    // the detector's column-edge and cone-edge lines split fewer warps than
    // with 32 x 1 rows, and a warp's taps fall in fewer cache lines (B200,
    // 270x270x200 from 360 half-fan views: 3.35 ms with 4 x 8 tiles, 3.44
    // with 8 x 4, 3.59 with 16 x 2, 3.96 with 32 x 1; the volume is the same)
    constexpr int TW = VCBCT_BP_TILE, TH = 32 / TW, WX = 32 / TW;
    const int x = blockIdx.x * 32 + (threadIdx.y % WX) * TW + (threadIdx.x % TW);
    const int y = blockIdx.y * 8 + (threadIdx.y / WX) * TH + (threadIdx.x / TW);
    constexpr int PARTS = ZB / ZS;
    const int bz = bp_zblock(blockIdx.z / PARTS, gridDim.z / PARTS);
    const int is = (blockIdx.z % PARTS) * ZS;  // first slice of the block that this thread makes
    const float fis = (float)is;
    const int z0 = bz * ZB;
    const bool valid = x < f.N && y < f.N;
    const double R = (double)(f.N - 1) / 2.0;
    const bool inmask = valid && ((double)y - R) * ((double)y - R) + ((double)x - R) * ((double)x - R) <= R * R;
    float acc[ZS];
#pragma unroll
    for (int i = 0; i < ZS; i++) acc[i] = 0.0f;
    const double pitch = k.pitch;
    const double zz0 = f.zstart + z0 * f.step;
    const int W = f.W, H = f.H;
    // Slices of this block that no column of the mask sees in any view (the
    // cone's height is exceeded: |Y| <= rm over the mask, so the detector
    // row coordinate H/2 + z g lies between the bounds of g below) are left
    // at zero without looping over the views; block-uniform.
    bool seen = true;
    {
        const double rm = (f.N * 0.5 + 1.0) * f.scale;
        const double gmin = 1.0 / ((1.0 + rm / f.sad) * pitch), gmax = 1.0 / ((1.0 - rm / f.sad) * pitch);
        const double zzb = zz0 + (double)(min(ZB, f.Z - z0) - 1) * f.step;
        const double a = zz0 * gmin, b = zz0 * gmax, c = zzb * gmin, d = zzb * gmax;
        const double lo = (double)(H / 2) + fmin(fmin(a, b), fmin(c, d));
        const double hi = (double)(H / 2) + fmax(fmax(a, b), fmax(c, d));
        if (rm < f.sad && (hi < -1.0 || lo > (double)H + 1.0)) seen = false;
    }
    // Views this block's tile of columns can see (bp_cull_kernel): a view
    // that contributes nothing to any column of the tile is dropped for the
    // whole block.  The kept views are visited in order, so the accumulation
    // order and the volume are those of visiting every view.
    extern __shared__ __align__(16) unsigned char s_raw[];
    const BpView* s_bv = reinterpret_cast<const BpView*>(s_raw);  // SV: [V]
    unsigned* s_views = reinterpret_cast<unsigned*>(s_raw + (SV ? (size_t)f.V * sizeof(BpView) : 0));
    {
        const int tid = threadIdx.y * 32 + threadIdx.x;
        const int nwords = (f.V + 31) >> 5;
        const int blk = (bz * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
        for (int i = tid; i < nwords; i += 256) s_views[i] = __ldg(keep + (size_t)blk * nwords + i);
        if (SV) {
            const unsigned long long* src = reinterpret_cast<const unsigned long long*>(views);
            unsigned long long* dst = reinterpret_cast<unsigned long long*>(s_raw);
            for (int i = tid; i < f.V * 4; i += 256) dst[i] = __ldg(src + i);
        }
    }
    const double cp = k.cp;
    const double inv_sad = k.inv_sad;
    __syncthreads();
    if (!valid) return;
    const bool full = z0 + ZB <= f.Z;  // every slice of the block exists
    if (inmask && seen) {
        const double xx = (x - cp) * f.scale;
        const double yy = -(y - cp) * f.scale;
        // the kept views in order, one mask word at a time (the culled ones
        // cost nothing)
        const int nwords = (f.V + 31) >> 5;
        for (int wi = 0; wi < nwords; wi++)
        for (unsigned wd = s_views[wi]; wd != 0u;) {
            const int th = wi * 32 + __ffs(wd) - 1;
            wd &= wd - 1u;
            const BpView bv = SV ? s_bv[th] : views[th];
            const double cs = bv.cs, sn = bv.sn;
            // FP64 detector coordinates of this column (:76-83)
            const double X = xx * cs + yy * sn;
            const double Y = -xx * sn + yy * cs;
            const double L2 = 1.0 - Y * inv_sad;
            // the correctly rounded reciprocal: 1.0 / (L2 pitch) to the bit
            const double g = __drcp_rn(L2 * pitch);
            const double U = X * g;
            const double Uf = floor(U);
            const float wu = (float)(U - Uf);
            const double UUU = bv.ushift + U;
            // floor and conversion in one (round-down conversion; out of
            // range or NaN gives INT_MIN or INT_MAX, both rejected below)
            const int UU = __double2int_rd(UUU);
            if (UU < 0 || UU > W - 1) continue;
            const double zeta0 = (double)(H / 2) + zz0 * g;
            // every slice of the block projects above or below the detector
            if (zeta0 + (double)(ZB - 1) * f.step * g < -1.0 || zeta0 > (double)H + 1.0) continue;
            const double zf = floor(zeta0);
            const int Zi = (int)zf;
            const float Zf = (float)(zeta0 - zf);
            const float dz = (float)(f.step * g);
            const float iL = (float)(g * pitch);  // 1 / L2
            const float w2 = iL * iL * bv.dbeta * (float)f.xfactor;
            const bool lastc = (UU == W - 1);
            const float cw0 = lastc ? 1.0f : 1.0f - wu;
            const float cw1 = lastc ? 0.0f : wu;
            const int UU1 = lastc ? UU : UU + 1;
            const float* pv = filt + (size_t)th * H * W;
            if (!lastc && full && zeta0 >= 0.0 && zeta0 + (double)(ZB - 1) * f.step * g < (double)H - 2.5) {
                // every slice of the block projects between detector rows 0
                // and H - 2: no bounds or last-row tests.  Two slices per
                // step in packed f32x2 arithmetic (each element rounded as
                // the scalar operation would round it: the same volume, half
                // the floating-point instructions)
                const float* pc = pv + UU;
                const f32x2 dz2 = f2pack(dz, dz), zf2b = f2pack(Zf, Zf);
                const f32x2 cw0_2 = f2pack(cw0, cw0), cw1_2 = f2pack(cw1, cw1), w2_2 = f2pack(w2, w2);
                const f32x2 big2 = f2pack(12582912.0f, 12582912.0f), one2 = f2pack(1.0f, 1.0f);
#pragma unroll
                for (int i = 0; i < ZS; i += 2) {
                    const f32x2 zfrac = ffma2(f2pack(fis + (float)i, fis + (float)(i + 1)), dz2, zf2b);
                    const f32x2 tq = fadd2_rd(zfrac, big2);
                    const f32x2 wz = fsub2(zfrac, fsub2(tq, big2));
                    float tqa, tqb;
                    f2unpack(tq, tqa, tqb);
                    const float* ra = pc + (Zi + (__float_as_int(tqa) - 0x4B400000)) * W;
                    const float* rb = pc + (Zi + (__float_as_int(tqb) - 0x4B400000)) * W;
                    const f32x2 s0 = ffma2(cw1_2, f2pack(__ldg(ra + 1), __ldg(rb + 1)),
                                           fmul2(cw0_2, f2pack(__ldg(ra), __ldg(rb))));
                    const f32x2 s1 = ffma2(cw1_2, f2pack(__ldg(ra + W + 1), __ldg(rb + W + 1)),
                                           fmul2(cw0_2, f2pack(__ldg(ra + W), __ldg(rb + W))));
                    const f32x2 v = ffma2(wz, s1, fmul2(fsub2(one2, wz), s0));
                    f32x2 a2 = f2pack(acc[i], acc[i + 1]);
                    a2 = ffma2(v, w2_2, a2);
                    f2unpack(a2, acc[i], acc[i + 1]);
                }
                continue;
            }
            if (!lastc && full) {
                // some slices of the block project outside rows 0 .. H - 2:
                // the same packed pairs, a slice off the detector (NZ outside
                // 0 .. H - 1) adding an exact zero (its rows clamped, its
                // weight 0; the sums are never -0, so acc + 0 = acc), the last
                // row taking row weights (1, 0) as the scalar rule does
                const float* pc = pv + UU;
                const f32x2 dz2 = f2pack(dz, dz), zf2b = f2pack(Zf, Zf);
                const f32x2 cw0_2 = f2pack(cw0, cw0), cw1_2 = f2pack(cw1, cw1);
                const f32x2 big2 = f2pack(12582912.0f, 12582912.0f), one2 = f2pack(1.0f, 1.0f);
#pragma unroll
                for (int i = 0; i < ZS; i += 2) {
                    const f32x2 zfrac = ffma2(f2pack(fis + (float)i, fis + (float)(i + 1)), dz2, zf2b);
                    const f32x2 tq = fadd2_rd(zfrac, big2);
                    float wza, wzb, tqa, tqb;
                    f2unpack(fsub2(zfrac, fsub2(tq, big2)), wza, wzb);
                    f2unpack(tq, tqa, tqb);
                    const int NZa = Zi + (__float_as_int(tqa) - 0x4B400000);
                    const int NZb = Zi + (__float_as_int(tqb) - 0x4B400000);
                    const bool ina = (unsigned)NZa <= (unsigned)(H - 1), inb = (unsigned)NZb <= (unsigned)(H - 1);
                    const bool la = NZa == H - 1, lb = NZb == H - 1;
                    const int ra = min(max(NZa, 0), H - 1), rb = min(max(NZb, 0), H - 1);
                    const float* r0a = pc + ra * W;
                    const float* r0b = pc + rb * W;
                    const float* r1a = la || !ina ? r0a : r0a + W;
                    const float* r1b = lb || !inb ? r0b : r0b + W;
                    const f32x2 wz = f2pack(la ? 0.0f : wza, lb ? 0.0f : wzb);
                    const f32x2 s0 = ffma2(cw1_2, f2pack(__ldg(r0a + 1), __ldg(r0b + 1)),
                                           fmul2(cw0_2, f2pack(__ldg(r0a), __ldg(r0b))));
                    const f32x2 s1 = ffma2(cw1_2, f2pack(__ldg(r1a + 1), __ldg(r1b + 1)),
                                           fmul2(cw0_2, f2pack(__ldg(r1a), __ldg(r1b))));
                    const f32x2 v = ffma2(wz, s1, fmul2(fsub2(one2, wz), s0));
                    f32x2 a2 = f2pack(acc[i], acc[i + 1]);
                    a2 = ffma2(v, f2pack(ina ? w2 : 0.0f, inb ? w2 : 0.0f), a2);
                    f2unpack(a2, acc[i], acc[i + 1]);
                }
                continue;
            }
#pragma unroll
            for (int i = 0; i < ZS; i++) {
                const float zfrac = fmaf(fis + (float)i, dz, Zf);
                // floor through the adder instead of the conversion unit: the
                // round-down add of 1.5 * 2^23 leaves floor(zfrac) in the low
                // mantissa bits (|zfrac| < 2^22 here); bitwise the same as
                // floorf and (int), 3.5 % faster on B200
                const float tq = __fadd_rd(zfrac, 12582912.0f);
                const float fl = tq - 12582912.0f;
                const int NZ = Zi + (__float_as_int(tq) - 0x4B400000);
                const float wz = zfrac - fl;
                if (NZ < 0 || NZ > H - 1 || z0 + is + i >= f.Z) continue;
                const bool lastr = (NZ == H - 1);
                const float rw0 = lastr ? 1.0f : 1.0f - wz;
                const float rw1 = lastr ? 0.0f : wz;
                const int NZ1 = lastr ? NZ : NZ + 1;
                const float* r0p = pv + (size_t)NZ * W;
                const float* r1p = pv + (size_t)NZ1 * W;
                const float s0 = fmaf(cw1, __ldg(r0p + UU1), cw0 * __ldg(r0p + UU));
                const float s1 = fmaf(cw1, __ldg(r1p + UU1), cw0 * __ldg(r1p + UU));
                acc[i] = fmaf(fmaf(rw1, s1, rw0 * s0), w2, acc[i]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < ZS; i++) {
        const int z = z0 + is + i;
        if (z >= f.Z) break;
        const size_t o = ((size_t)z * f.N + y) * f.N + x;
        if (vol_f32) vol_f32[o] = acc[i];
        if (vol_i16) {
            // (short) of the reconstructed value: truncation toward zero
            // (R/main.cpp:184), saturated to the short range.
            float a = fminf(fmaxf(acc[i], -32768.0f), 32767.0f);
            vol_i16[o] = (short)__float2int_rz(a);
        }
    }
}

}  // namespace

}  // namespace vcbct

namespace vcbct {

cudaError_t launch_filter_direct(const float* proj, float* out, const float* hT,
                                 const FilterView* views, const float* wts, float pitch,
                                 float sad, int V, int H, int W, cudaStream_t st)
{
    const int M = V * H;
    FilterArgs a{proj, out, hT, views, wts, pitch, sad, M, H, W, 0, 0, 0, 0};
    a.kc = std::min((W + FT_K - 1) / FT_K * FT_K, FT_CHUNK);
    a.groups = (W + 31) / 32;
    a.npass = (a.groups + FT_TN - 1) / FT_TN;
    // One block makes every column pass of its rows, or a part of them where
    // the rows alone would not fill the GPU (two blocks an SM); narrower
    // passes where that is still so.
    const int rows = (M + FT_M - 1) / FT_M, want = std::max(1, 2 * kSMs / rows);
    if (a.npass < want) a.npass = std::min(a.groups, want);
    // (g does not stay staged from pass to pass beyond FT_CHUNK columns: then
    // every pass is a block of its own, and the last wave is shorter)
    a.per = W > FT_CHUNK ? 1 : (a.npass + want - 1) / want;
    const int widest = (a.groups + a.npass - 1) / a.npass;
    const size_t smem = ((size_t)a.kc * FT_LD + (size_t)2 * FT_K * 32 * widest) * sizeof(float);
    auto k = widest <= 2 ? filter_direct_kernel<2> : filter_direct_kernel<FT_TN>;
    const cudaError_t e = allow_smem(k, smem);
    if (e != cudaSuccess) return e;
    k<<<dim3((unsigned)rows, (unsigned)((a.npass + a.per - 1) / a.per)), 256, smem, st>>>(a);
    return cudaGetLastError();
}

size_t backproject_workspace_bytes(const FdkParams& f)
{
    constexpr int ZB = VCBCT_BP_ZB;
    const size_t nblocks = (size_t)((f.N + 31) / 32) * ((f.N + 7) / 8) * ((f.Z + ZB - 1) / ZB);
    return nblocks * (size_t)((f.V + 31) / 32) * sizeof(unsigned);
}

cudaError_t launch_backproject(const FdkParams& f, const BpView* d_views, const float* filt,
                               float* vol_f32, short* vol_i16, unsigned* keep, int* keep_ready,
                               cudaStream_t st)
{
    constexpr int ZB = VCBCT_BP_ZB;
    dim3 block(32, 8);
    dim3 grid((f.N + 31) / 32, (f.N + 7) / 8, (f.Z + ZB - 1) / ZB);
    BpConst k;
    k.pitch = f.piso * f.mpn / f.W;
    k.inv_sad = 1.0 / f.sad;
    k.cp = (double)f.N / 2.0 - 0.5;
    const int nblocks = (int)(grid.x * grid.y * grid.z);
    const long nwarps = (long)nblocks * ((f.V + 31) / 32);
    if (!keep_ready || !*keep_ready) {
        // the view masks follow the geometry and the views only: made once
        bp_cull_kernel<ZB><<<(unsigned)((nwarps * 32 + 255) / 256), 256, 0, st>>>(f, d_views, (int)grid.x,
                                                                                   (int)grid.y, nblocks, keep);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        if (keep_ready) *keep_ready = 1;
    }
    // the view table goes to shared memory where it fits the default 48 KB
    // with the view mask
    const size_t mask_bytes = (size_t)((f.V + 31) / 32) * sizeof(unsigned);
    const size_t table_bytes = (size_t)f.V * sizeof(BpView);
    const bool sv = table_bytes + mask_bytes <= 48 * 1024;
    const size_t smem = mask_bytes + (sv ? table_bytes : 0);
    // resident blocks per SM (the register cap): VCBCT_BP_MIN_BLOCKS by
    // default, 5 or 6 through the environment variable of the same name where
    // a thread makes a whole slice block
    int minb = VCBCT_BP_MIN_BLOCKS;
    if (const char* e = std::getenv("VCBCT_BP_MIN_BLOCKS")) minb = std::atoi(e) == 6 ? 6 : 5;
    auto launch = [&](auto zs) {
        constexpr int ZS = decltype(zs)::value;
        const dim3 gp(grid.x, grid.y, grid.z * (ZB / ZS));
        auto kernel = sv ? backproject_kernel<ZB, ZS, 5, true> : backproject_kernel<ZB, ZS, 5, false>;
        if constexpr (ZS == ZB)
            if (minb == 6) kernel = sv ? backproject_kernel<ZB, ZS, 6, true> : backproject_kernel<ZB, ZS, 6, false>;
        kernel<<<gp, block, smem, st>>>(f, k, d_views, filt, vol_f32, vol_i16, keep);
    };
    // Threads of fewer slices repeat the column's set-up, which is free while
    // SM slots (five an SM) stand idle.  Slices a thread 8 / 4 / 2, us on a B200:
    // 396 blocks (95x95x84) 151 / 154 / 154, 340 blocks 372 / 407 / 451, 231
    // blocks (86x86x51) 32 / 21 / 21, 190 blocks 33 / 25 / 21, 120 blocks
    // (80x80x27, 224 views of 793 x 720) 489 / 327 / 220, 128 blocks (58x58x64)
    // 341 / 249 / 295: two slices are not the best of every volume below 200
    // blocks, but better than eight.
    if (nblocks >= 300) launch(std::integral_constant<int, ZB>{});
    else if (nblocks >= 200) launch(std::integral_constant<int, ZB / 2>{});
    else launch(std::integral_constant<int, ZB / 4>{});
    return cudaGetLastError();
}

}  // namespace vcbct
