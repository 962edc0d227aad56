// internal.h -- shared declarations of libvcbct's CUDA translation units.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <string>

#include "vcbct.h"

namespace vcbct {

// Thread-local error message behind vcbct_last_error().
void set_error(const std::string& msg);
int fail(int code, const std::string& msg);
int cuda_fail(cudaError_t e, const char* what);

#define VCBCT_CUDA_TRY(call)                                  \
    do {                                                      \
        cudaError_t e__ = (call);                             \
        if (e__ != cudaSuccess) return ::vcbct::cuda_fail(e__, #call); \
    } while (0)

constexpr int kSMs = 148;  // of a B200, the only GPU this library is built for

// A launch whose blocks take more than 48 KB of dynamic shared memory needs its
// kernel's limit raised.  The limit is the kernel's (on a device), shared by
// every host thread and by launches prepared long before, so it is only ever
// set to `most`, what the kernel's largest launch takes, never to one call's
// size: that would lower it under another call's launch.
constexpr size_t kSmemDefault = 48 * 1024, kSmemMost = 227 * 1024;
template <class K>
cudaError_t allow_smem(K kernel, size_t bytes, size_t most = kSmemMost)
{
    if (bytes > most) return cudaErrorInvalidValue;
    if (bytes <= kSmemDefault) return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}

// Per-view geometry the projector kernels read (double, from the host
// tables of prepareTrigonometricTable, misc.cpp:10-37).
struct ViewGeom {
    double cs, sn, xc, yc;
};

// Scalar projection geometry passed by value to the kernels.
struct ProjParams {
    int N, Z, W, H, V, nmat;
    double s, step, pdet, piso, sad, dpn, xr, yr, zr;
};

// ---------------------------------------------------------------- MBFPA --
// Packed volume: voxel (x, y, z) at index (y*N + x)*Z + z, one 16-byte record
// of 8 uint16 element values (u16 form) or one 32-byte record of 8 floats
// (f32 form).  Elements beyond nmat are zero.  A volume keeps the form of
// the values it was loaded from: the march is bound by the L1's data path, and
// uint16 records are half the bytes (they convert exactly, once per slice and
// interval of a warp).  A projector's volume buffer holds either form; which
// one it holds is a word of device memory that the re-layout kernels write
// (VolRef::form), so a captured projection that is replayed after a volume of
// the other type was loaded reads what is there.
size_t packed_u16_bytes(int N, int Z);
size_t packed_f32_bytes(int N, int Z);

struct VolRef {
    const void* rec;   // packed records
    const int* form;   // device: kFormF32 / kFormU16; nullptr: as expected
    int expect;        // the form of the last load, which picks the kernel
};
enum { kFormF32 = 0, kFormU16 = 1 };

// uint16 slab [nz][nmat][N][N] -> slices [zoff, zoff + nz) of a u16-form
// volume of Z slices; form (may be nullptr) is set to kFormU16
cudaError_t launch_pack_u16(const uint16_t* src, int N, int nz, int zoff, int Z, int nmat, uint4* dst, int* form,
                            cudaStream_t st);
cudaError_t launch_pack_f32(const float* src, int N, int Z, int nmat, float4* dst, int* form, cudaStream_t st);
cudaError_t launch_unpack_grad(const float* planes, int N, int Z, int nmat, float* dst, cudaStream_t st);

// Spectral table: per bin 8 floats mu_k(E)/xfactor (zero padded) + pdf, and
// before the first bin's pdf the spectrum's floor: 2^-100 of its weight.
struct SpectrumDev {
    const float4* mu8;  // [NE][2] float4
    const float* pdf;   // [1 + NE]
    int NE;
};
inline float spectral_floor(const float* pdf, int NE)
{
    double w = 0.0;
    for (int e = 0; e < NE; e++) w += pdf[e] < 0.0f ? -(double)pdf[e] : (double)pdf[e];
    return (float)(w * 7.8886090522101181e-31);
}

struct ForwardArgs {
    ProjParams p;
    const ViewGeom* views;   // device [V]
    SpectrumDev spec;
    VolRef vol;
    float* out;              // [V][H][W] intensities (or nullptr)
    float* L_out;            // [V][H][W][nmat] path integrals (or nullptr)
    unsigned long long* seg_count;  // (or nullptr)
    int* err_flag;           // device fault flag
    int cols_per_block;
    int columns;             // sum by shared columns (march_shares_columns)
    // detector noise on `out` (kind 0: none, 1: Gaussian counts)
    int noise_kind;
    int view_offset;         // global index of view 0 of this launch (noise counters)
    int band0, nbands;       // detector row bands [band0, band0 + nbands) of 32 rows (nbands 0: all)
    double noise_i0, noise_max;
    unsigned long long noise_seed;
};
cudaError_t launch_forward(const ForwardArgs& a, cudaStream_t st);
// Whether a geometry's rays are summed by shared columns (several rays of a
// detector column per slice) or each on its own.
bool march_shares_columns(const ProjParams& p);
bool scatter_shares_columns(const ProjParams& p);
// Slice range [span[2b], span[2b+1]] the forward projection of detector row
// band b (rows 32b..32b+31, all views) can read; span must hold (Z, -1) per
// band on entry (bands that read nothing keep it).
cudaError_t launch_band_footprint(const ProjParams& P, const ViewGeom* d_views, int* d_span, cudaStream_t st);
cudaError_t launch_gaussian_noise(float* proj, size_t n, double max_pixvalue, unsigned long long seed,
                                  cudaStream_t st);

// Items of one single-launch batch, passed in the kernel's parameter block.
constexpr int kFlatItems = 40;
struct FlatBatch {
    int nitems;
    int ncolb[kFlatItems];
    long long begin[kFlatItems + 1];  // first tile of each item; begin[nitems] = total
    ForwardArgs fa[kFlatItems];
};
// Of the items of one launch, which are of one kind.
struct BatchShape {
    int NEmax, nmat_max;
    bool columns, u16;   // summed by shared columns; uint16 records
    int cols_per_block;
};
cudaError_t launch_flat_batch(const FlatBatch& b, const BatchShape& s, cudaStream_t st);

// The same items, which are walked, in one persistent launch of `blocks` blocks
// that take work tiles from `counter` (zeroed by the launch).
cudaError_t launch_persistent_batch(const FlatBatch& b, const BatchShape& s, int blocks, unsigned long long* counter,
                                    cudaStream_t st);
int batch_blocks_per_sm(const BatchShape& s);

struct AdjointArgs {
    ProjParams p;
    const ViewGeom* views;
    SpectrumDev spec;
    VolRef vol;              // read only to recompute path integrals
    const float* grad_out;   // [V][H][W] d loss / d intensity
    const float* L_in;       // [V][H][W][nmat] path integrals of the forward, or
                             // nullptr: recompute them (first march)
    float* grad_planes;      // float accumulator, z fastest, ceil(nmat/2) x 2 floats per voxel: groups of
                             // four elements [N*N*Z][4], the last a pair [N*N*Z][2] if it holds one or two
    int* err_flag;
    int cols_per_block;
    int columns;             // as the forward that L would come from
    int share;               // scatter by shared columns (scatter_shares_columns)
    int y0, y1;              // scatter only into volume rows iy in [y0, y1) (y1 <= y0: all)
};
cudaError_t launch_adjoint(const AdjointArgs& a, cudaStream_t st);

// ------------------------------------------------------ iterative recon --
// Geometry of lengthproj (the projector's, with the registration shifts the
// call uses).
struct LpParams {
    int N, Z, W, H;
    double s, step, pdet, piso, sad, dpn, xr, yr, zr;
};
size_t lengthproj_scratch_bytes(int n_views);
cudaError_t launch_lengthproj(const LpParams& q, const ViewGeom* d_views, int v0, int v1, const uint16_t* d_proj,
                              float* d_npf, void* d_scratch, cudaStream_t st);
cudaError_t launch_ir_update(int N, int Z, double scale, const short* d_before, float* d_out, const float* d_npf,
                             const float* d_npf_re, double wbefore, double weight_tv, double weight_prior,
                             cudaStream_t st);

// ------------------------------------------------------------------ FDK --
struct FdkParams {
    int W, H, V, N, Z, zstart, xfactor, redundancy;
    double step, scale, piso, pdet, mpn, sad;
};

// Per-view filter constants: detector centre shifts of filterSinogram.cpp:86-87.
struct FilterView {
    float xcs, ycs;
};
// Direct FP32 ramp filter.  hT: [W][W] float, hT[k][m] = h[m][k] + coeff*(m==k).
// wts: optional [V][W] redundancy weights applied to -log(p) before filtering.
cudaError_t launch_filter_direct(const float* proj, float* out, const float* hT,
                                 const FilterView* views, const float* wts, float pitch,
                                 float sad, int V, int H, int W, cudaStream_t st);

struct BpView {
    double cs, sn;   // cos / sin of the view angle
    double ushift;   // W/2 - 0.5 + xshift in pixels (reconstructImage.cpp:83)
    float dbeta;     // half the neighbouring angular gap (:45-71)
    float pad;
};
// keep: backproject_workspace_bytes(f) of device scratch holding the
// per-block view masks, a function of the geometry and the views only: with
// *keep_ready set they are taken as made and not redone; the launch sets it
// once it has queued them (keep_ready may be null: made every call).
size_t backproject_workspace_bytes(const FdkParams& f);
cudaError_t launch_backproject(const FdkParams& f, const BpView* d_views, const float* filt,
                               float* vol_f32, short* vol_i16, unsigned* keep, int* keep_ready,
                               cudaStream_t st);

// BF16 3-term split tensor-core ramp filter (tcgen05).  The workspace holds
// the split Toeplitz planes: with *b_ready set they are taken as already
// split from hT into this workspace and are not redone; the launch sets it
// once it has queued the split (b_ready may be null: split every call).
// The fused form (rows of `proj` and `out` 16-byte aligned: W % 4 == 0 and
// aligned bases, ramp_gemm_fused) splits -ln p inside the GEMM and stores
// through TMA; the other needs room for the split A planes as well: size the
// workspace with the same flag.
bool ramp_gemm_fused(const float* proj, const float* out, int W);
size_t ramp_gemm_workspace_bytes(int V, int H, int W, bool fused);
cudaError_t launch_ramp_gemm_bf16x3(const float* proj, float* out, const float* hT,
                                    const FilterView* views, const float* wts, float pitch,
                                    float sad, int V, int H, int W, void* workspace,
                                    int* b_ready, cudaStream_t st);
// The kernel's fault flag (1 after a bounded wait ran out; its output is then
// invalid), read synchronously on `st`; -1 if it cannot be read.
int ramp_gemm_error_flag(void* workspace, int V, int H, int W, cudaStream_t st);

}  // namespace vcbct
