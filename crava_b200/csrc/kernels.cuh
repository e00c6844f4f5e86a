// Kernel parameter blocks and launch helpers shared by the host API and the kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "fft_core.cuh"

namespace crava {

// Launches whose kernels follow one another in a stream overlap the next one's launch with the last one's
// end (programmatic dependent launch) where the grids they work on hold less than kDepBytes: there the
// launch gaps are a good part of the pass (64x64x128, 37 MB in all: 73.7 -> 65.1 us; 90x90x128, 73 MB: 120 -> 111).
// Larger ones run slower that way, the waiting CTAs taking room from the last wave (all launches so: 105x135x125 with 4
// to 16 realisations, 190 to 440 MB, 9 % slower; 160x160x160 10 %).  A job mixes both, each launch by its own
// grids; of 20 blocks of 37 to 500 MB none is slower than without at this limit, while 96 MB costs 90x90x125 3 %.
// dep_wait, before a kernel touches memory that another may have written or still reads, waits until the grids before
// it are over; dep_launch lets the next grid's CTAs take their places.
constexpr size_t kDepBytes = 64u << 20;
template <class... P, class... A>
inline cudaError_t launch_dep(size_t bytes, void (*fn)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st,
                              const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = bytes < kDepBytes ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, fn, args...);
}
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Schedule table: tile shapes and kernel choices by name and size (n), from the schedule
// file the library loads at first use (schedules.txt beside the library, written by
// crava_b200/autotune.py; CRAVA_SCHEDULES names another file) or set through
// crava_tuning_set.  An entry for n, else one for n = -1 (any size), else `fallback`.
int tuned(const char* key, int n, int fallback);

constexpr int kMaxGrids = 64;   // grids per batched transform launch
constexpr int kMaxTheta = 8;    // angle stacks per block
constexpr int kMaxSim = 16;     // realisations per job launch

// Grids of one batched transform launch.  p[] are the grids transformed in place;
// for the forward x pass src[] are the real inputs it reads (src[q] == p[q] is in place).
constexpr int kNumCounters = 5;
struct GridSet {
  float* p[kMaxGrids];
  const float* src[kMaxGrids];
  float scale[kMaxGrids];
  int n;
  unsigned long long* zero = nullptr;   // forward x pass: kNumCounters words it clears
  int plain = 0;   // 1: forward transforms in the scalar kernels' order of roundings (zpass.cuh says why)
};

// Per-kz operator tables of one block (device pointers), see the host-side builder.
struct KzTables {
  const float2* kw;     // nzp x nth : conj(W_l(k)) kD(k)
  const float2* e1;     // nzp x nth : conj(W_l(k)) / |w_l|
  const float2* e2;     // nzp x nth : conj(E3_l(k)) / |e3_l|
  const uint8_t* inv;   // nzp       : invert_frequency
  const double2* kwd;   // the same three tables in double, read by the FP64
  const double2* e1d;   //   re-factorisation of flagged bins
  const double2* e2d;
  const float* ed;      // nzp x nth : wnc errThetaCov_ll |e3_l(k)|^2 (e3 = 1 for constant
  const double* edd;    //   thickness); edd in double, null: the per-angle constants edd
};

// z transform plan of the pencil pass: nzp as a product of radices up to 20, stage by stage.
struct ZPlan {
  int n, ns;
  int8_t radix[10];
};
bool pencil_plan(int n, ZPlan& z);
// z lengths whose two-stage split is inlined in the pencil pass, its strides constants: the powers of two
// and the 5 x 2^6 that blocks are usually padded to.  The calls of the general stages cost a tenth of the instructions
// (pencil.cuh) and more of a small block's latency (64x60x320, prior grids: 178 against 140 us).
#define CRAVA_Z_INLINED(X) X(128, 16, 8) X(256, 16, 16) X(320, 20, 16)
constexpr bool z_inlined(int nzp) {
#define CRAVA_CASE(N, R0, R1) if (nzp == N) return true;
  CRAVA_Z_INLINED(CRAVA_CASE)
#undef CRAVA_CASE
  return false;
}
// kz at position p of a line after the forward stages (in place, digits reversed)
int pencil_kz(const ZPlan& z, int p);

struct ZParams {
  int nxp, nyp, nzp, cnxp;
  int W, NP, logNP, nIT;       // tile width in x-bins (power of two >= 2), pairs W / 2, tiles per x-row
  int SB;                      // realisations per batch
  int D, PS, swz;              // tile layout (pencil.cuh): slot of the diagonal, bytes per position,
                               // positions swapped within fours in the per-bin steps
  int vec;                     // 1: pairs of bins move as 16-byte words
  int logW, GT;                // k_zpass: log2 W, slots per z-transform call (3 SB <= GT)
  LinePlan zp;                 // k_zpass: the z transform's stages
  ZPlan z;
  int nth, nsim;
  int separable;               // 1: prior from cxy/ct factors, 0: from spectral grids
  int base_prior;              // grids: the six prior spectra are pv x one base spectrum, only
                               // cov[0] (= pv[0] x base) transformed
  int host_noise;              // 1: noise from `noise` grids
  int keep_resid;              // 1: write residual spectra into data grids
  int cov_spectral;            // 1: posterior covariance left as per-bin spectra
  int nxp_even;
  float2* data[kMaxTheta];
  float2* mean[3];
  float2* cov[6];              // out; in GRIDS mode also the prior spectra (in)
  const float2* errspec;       // GRIDS mode: error correlation spectrum
  float2* sim[3 * kMaxSim];
  const float2* noise[3 * kMaxSim];
  const float2* cxy;           // SEPARABLE: nyp x cnxp spectrum of corrXY
  const float2* ct;            // SEPARABLE: nzp spectrum of circCorrT
  const float2* septab;        // SEPARABLE: per-kz lower triangle of M2 (or null)
  float pv[6];                 // priorVar0: 00 11 22 01 02 12
  float A[kMaxTheta][3];
  float ec[kMaxTheta][kMaxTheta];  // 0.5 (1 - wnc) errThetaCov
  float ed[kMaxTheta];             // wnc errThetaCov_ll |e3_l|^2
  float G0[kMaxTheta][kMaxTheta];  // SEPARABLE: A P0 A^T
  float AP[kMaxTheta][3];          // SEPARABLE: A P0
  KzTables kz;
  const float2* twz;
  uint64_t seed;
  float fp64_threshold;            // > 0: re-factorise flagged bins in FP64
  double Ad[kMaxTheta][3];         // A, ec, ed in double for that path
  double ecd[kMaxTheta][kMaxTheta];
  double edd[kMaxTheta];
  // eigen form of the separable posterior (pencil.cuh): per-position rows of the per-kz
  // tables, float4 group g of position p at eig[g * nzp + p]; null: the Cholesky form
  const float4* eig;
  int n_inv_rows;                  // inverted kz (counted per tile, not per bin)
  unsigned long long* counters;    // [0] inverted bins [1] chol fallbacks [2] zero sim bins
                                   // [3] bins re-factorised in FP64 [4] pencil tiles whose
                                   // input spectra are not finite
};

// Local-noise shrinkage (localnoise.cu): per-trace maps of the posterior and realisations
// from the local noise scales; the matrices are job constants computed on the host.
struct LocalNoiseParams {
  int nx, ny, nz, nyp, rnxp, nth, nsim;
  const float* scale;                 // nth x ny x nx local noise scales, index i + nx (j + ny l)
  float* maps;                        // ny x nx x 18 floats: every trace's S and Msim (scratch)
  double inv_min[kMaxTheta];          // 1 / (smallest scale of angle l)
  double gsg[kMaxTheta][kMaxTheta];   // G Sm G^T
  double sth[kMaxTheta][kMaxTheta];   // SigmaTheta (errThetaCov)
  double b[kMaxTheta][3];             // G Sm
  double sm[3][3];                    // priorVar0
  double sdel[3][3];                  // (Sm - Smd)^-1/2, eigenvalues <= 1e-7 dropped
  double smdi[3][3];                  // Smd^-1/2, eigenvalues <= 0 dropped
  const float* prior_mean[3];         // real grids (FFTGrid layout)
  float* post[3];                     // posterior mean, corrected in place
  float* sim[3 * kMaxSim];            // realisations, corrected in place
};
cudaError_t launch_local_noise(const LocalNoiseParams& P, cudaStream_t st, int* nlaunch);

constexpr int kMaxFacies = 16;
constexpr int kMaxFaciesAngles = 4;   // local-noise angles of the facies densities (16 corners)
struct FaciesPrior { float p[kMaxFacies]; };
struct FaciesOut { float* p[kMaxFacies + 1]; };
struct FaciesBoxHost {
  int nb[3];
  double vmin[3];
  double dv[3];
  int rs;
  size_t fstride;
};

// Non-constant-thickness data pre-processing (thick.cu).  Per-angle tables of
// computeAdjustmentFactor over kz < cnzp: wamp the wavelet spectrum (cAmp), es3 the
// band-normalised spectrum of the third difference of the wavelet, tau2 |Re| of the
// reflection-coefficient covariance spectrum.
struct ThickParams {
  int nx, ny, nz, nxp, nyp, nzp, rnxp, cnzp;
  int W, logW, nIT;            // W complex lines (2W traces) per CTA, log2 W, tiles per row
  float* grid[kMaxTheta];      // the data grids, processed in place
  const double* rel_thick;     // nxp x nyp, Simbox::getRelThick(i, j)
  const float2* wamp;          // nth x cnzp
  const float2* es3;           // nth x cnzp
  const float* tau2;           // nth x cnzp
  const float2* glob;          // nth x cnzp: {0.05 wGlob2Adj, wGlob2Adj / (tau2 wGlob2 + sigma2Glob)}
  const float* ztaper;         // nzp: 1, or max(1 - dist^2, 0) for kz > nz
  const int* fillx;            // nxp, nyp: getFillNumber of every padded index
  const int* filly;
  const float* distx;          // nxp, nyp, nzp: getDistToBoundary of every padded index
  const float* disty;
  const float* distz;
  float wn2[kMaxTheta];        // (wavelet norm)^2
  float modW[kMaxTheta];       // norm^2 * maxfrequency / highCut
  float err_var[kMaxTheta];    // errThetaCov_ll
  float wnc, low_cut, high_cut;
  float rsq;                   // float(sqrt(float(nzp)))
  float inv_rsq;               // 1/rsq when rsq is a power of two (x/rsq == x*inv_rsq exactly),
                               // else 0: the kernel divides
  double lz;
  LinePlan zp;
  const float2* twz;
  // local wavelets (Wavelet1D with shift and gain grids): per angle and trace i + nx j the
  // shift in samples (shift / dz) and the gain; null: every local wavelet is the global one
  const float* wshift;
  const float* wgain;
  float2 es3_last[kMaxTheta];  // es3 at cnzp - 1 before the RMISSING that the table carries
  // 0: divideDataByScaleWavelet on every padded trace; 1: the wavelet convolution of
  // multiplyDataByScaleWaveletAndWriteToFile on the traces i < nx, j < ny
  int mode;
  float rsq_out;               // mode 1: float(sqrt(double(nzp))), its final divisor
  // 3D wavelets (Wavelet3D, src/wavelet3D.cpp:328-459): per angle and unpadded trace
  // i + nx j the dip adjustment of the trace's local wavelet (Wavelet3DFill), or null for
  // 1D wavelets
  const double* w3_mult;       // multiplyer = alpha1(phi, psi) cos(psi) cos(theta)
  const float4* w3_par;        // {Halpha, local stretch, norm^2 of the adjusted wavelet, gamma}
  const float2* wglob;         // nth x cnzp: the global (average) wavelets' half spectra
  double w3_den;               // double(nzp * dz * 1e-3): the bin spacing's reciprocal, 1/Hz
};
// Per-trace dip adjustment of 3D wavelets (Wavelet3D::getLocalStretch and
// createLocalWavelet1D -> extractLocalWaveletByDip1D -> dipAdjustWavelet, src/wavelet3D.cpp:
// 328-459; the filter surfaces are NRLib::RegularSurface<float> read by WaveletFilter,
// src/waveletfilter.cpp:60-75): for every angle and unpadded trace, from the structure depth
// gradients, phi, psi, the filter values alpha1 and Halpha, multiplyer and the stretch, then
// the norm^2 of the adjusted wavelet (Parseval over its half spectrum) and gamma, the factor
// that band-normalises the adjusted errorSmooth3 given the job's normalised table.
struct Wavelet3DFill {
  const float* gx;             // nx*ny depth gradients (i + nx j), or null: flat
  const float* gy;
  const float* alpha1;         // nth x ni*nj (i + ni j): phi (degrees) along i, psi along j
  const float* halpha;         // nth x ni*nj, or null: no damping
  int ni, nj;
  double x0, y0, dx, dy;       // surface origin and spacing (degrees)
  float theta[kMaxTheta];      // Wavelet::getTheta (radians)
  const float2* wamp;          // nth x cnzp: the 3D wavelets' own half spectra
  const float2* es3;           // nth x cnzp: band-normalised errorSmooth3 (RMISSING last), or null
  float2 es3_last[kMaxTheta];  // es3 at cnzp - 1 before the RMISSING
  int nx, ny, nzp, cnzp, loI, hiI;
  double den;                  // double(nzp * dz * 1e-3)
  double* mult;                // out: nth x nx*ny
  float4* par;                 // out: nth x nx*ny
};
// Prior grids of a GRIDS-mode job generated on the device (prior.cu): the six covariance
// grids fillInParamCorr x priorVar0 and the error-correlation grid fillInErrCorr.
struct PriorFill {
  float* cov[6];               // order Vp, Vs, Rho, VpVs, VpRho, VsRho
  float* err;
  const float* cxy;            // nxp x nyp corrXY
  const float* ct;             // nzp circCorrT
  float pv[6];                 // float(priorVar0(a, b)) in the grid order
  const float* act;            // estimated covariance: 6 x nzp circular auto-covariances in the
                               // grid order (FFTGrid::FillInLateralCorr; pv unused), or null
  float gi, gj;                // correlation gradients (samples per lateral index)
  int nxp, nyp, nzp, rnxp;
};
cudaError_t launch_fill_prior(const PriorFill& P, cudaStream_t st, int* nlaunch);

// One interpolateTrace: trace t (i + nx j) <- mean of nb[] (left, right, up, down; -1 absent)
struct TraceOp {
  int t;
  int nb[4];
  int nt;
};
size_t thick_smem_bytes(int W, int nzp);
int thick_tile_width(int nzp);
cudaError_t launch_thick_divide(const ThickParams& P, int nth, cudaStream_t st, int* nlaunch);
cudaError_t launch_wavelet3d_fill(const Wavelet3DFill& F, int nth, cudaStream_t st, int* nlaunch);
cudaError_t launch_trace_energy(const ThickParams& P, int nth, float* energy, int* nzero, cudaStream_t st,
                                int* nlaunch);
cudaError_t launch_trace_interp(float* g, int rnxp, int nyp, int nzp, int nx, const TraceOp* ops, int nops,
                                cudaStream_t st, int* nlaunch);
cudaError_t launch_extrapolate(const ThickParams& P, int l, const int box[4], cudaStream_t st, int* nlaunch);
float dist_to_boundary(int i, int n, int np);
int fill_number(int i, int n, int np);
void plan_trace_interpolation(const float* energy, int nx, int ny, float threshold, std::vector<TraceOp>& ops,
                              std::vector<int>& level_start, int box[4]);

// four-step launchers (fft4.cu): lengths of its size table only
bool four_step_supported(int n);
cudaError_t launch_line4(const GridSet& gs, int ni, int n, size_t pstride, int no, size_t ostride, const float2* tw,
                         float sign, cudaStream_t st, int* nlaunch);
cudaError_t launch_x4(bool fwd, const GridSet& gs, int nxp, int rows, const float2* tw, const float2* twn,
                      cudaStream_t st, int* nlaunch);
// launchers (kernels.cu)
// x transforms: pl/tw are the plan and table of length nxp/2 (even nxp) or nxp (odd);
// twn is the length-nxp table (its first nxp/2 entries are read; unused for odd nxp).
cudaError_t launch_x_r2c(const GridSet& gs, int nxp, int rows, const LinePlan& pl, const float2* tw,
                         const float2* twn, cudaStream_t st, int* nlaunch);
cudaError_t launch_x_c2r(const GridSet& gs, int nxp, int rows, const LinePlan& pl, const float2* tw,
                         const float2* twn, cudaStream_t st, int* nlaunch);
// Complex transform along a strided axis, in place, for all grids of gs:
//   element (i, p, o) at ((size_t)o * ostride + (size_t)p * pstride + i) complex,
//   0 <= i < ni (contiguous), 0 <= p < n (the transform axis), 0 <= o < no.
cudaError_t launch_line_fft(const GridSet& gs, int ni, int n, size_t pstride, int no, size_t ostride,
                            const LinePlan& pl, const float2* tw, float sign, cudaStream_t st, int* nlaunch);
// pencil.cu: the pencil pass.  pencil_shape sets zp's tile (W .. swz, nIT) and the threads per CTA
// from nzp, nth, nsim and the lateral size (schedule keys pencil_w, pencil_sb, pencil_threads, n =
// nzp * 16 + nth); false when no tile fits in shared memory.
bool pencil_shape(ZParams& zp, int* threads);
cudaError_t launch_pencil(const ZParams& zp, int threads, cudaStream_t st, int* nlaunch);
size_t pencil_smem_bytes(int W, int nzp, int nth, int SB);
// zpass.cu: the same with the scalar z transforms, for residual spectra; zpass_shape as pencil_shape
bool zpass_shape(ZParams& zp, int* threads);
cudaError_t launch_zpass(const ZParams& zp, int threads, cudaStream_t st, int* nlaunch);
size_t zpass_smem_bytes(int W, int nzp, int nth, int GT, int SB);
// Float layout of one position's row of the eigen tables: kw (2n floats), Lam (n), then per
// angle l a row of V (2n floats) and Q_l (6) + H_l (9); sections padded to 4 floats so the
// kernel reads them as float4 groups and streams one angle's row at a time.
struct EigLayout {
  int kw, lam, rows, vpad, rs, floats;
  explicit EigLayout(int n) {
    auto pad = [](int x) { return (x + 3) / 4 * 4; };
    kw = 0;
    lam = pad(2 * n);
    rows = lam + pad(n);
    vpad = pad(2 * n);
    rs = vpad + 16;
    floats = rows + n * rs;
  }
};
// facies.cu: prior[] and out[] are host arrays (copied into the launch parameters)
cudaError_t launch_facies_smoother(float* g, float* sum, int na, int nb, int nr, const double* dv, const double* S,
                                   cudaStream_t st, int* nlaunch);
cudaError_t launch_spec_mul(float2* a, const float2* b, size_t n, cudaStream_t st);
// gridio.cu: dst[e] = src[e] with the byte order of every 4-byte word reversed (dst == src
// allowed)
cudaError_t launch_bswap32(uint32_t* dst, const uint32_t* src, size_t n, cudaStream_t st);
// STORM grid files (gridio.cu): elements e0 .. e0+n-1 of the dense ordering (i fastest) of
// the nx x ny x nz region of a padded real grid (row pitch rnxp, nyp rows per slice) to
// big-endian words and back, and the linear padding fill of FFTGrid's StormContGrid
// constructor.
cudaError_t launch_storm_pack(uint32_t* dst, const float* grid, int nx, int ny, size_t e0, size_t n, int rnxp,
                              int nyp, cudaStream_t st);
cudaError_t launch_storm_unpack(float* grid, const uint32_t* src, int nx, int ny, size_t e0, size_t n, int rnxp,
                                int nyp, cudaStream_t st);
cudaError_t launch_pad_fill(float* grid, int nx, int ny, int nz, int nxp, int nyp, int nzp, int rnxp, cudaStream_t st,
                            int* nlaunch);
// SegY records (segy.cu): per record (inline/crossline order) the trace's grid column, its
// first and end regular samples with data, its top and grid sample spacing; hdr holds the 240-byte
// trace headers (60 words per record, already big-endian).
struct SegyTrace {
  int i, j, first, end;
  double ztop, gdz;
};
struct SegyPack {
  const float* grid;
  int rnxp, nyp, nz;
  int ns;
  float z0, dz;
  const SegyTrace* tr;
  const uint32_t* hdr;
};
cudaError_t launch_segy_pack(const SegyPack& P, size_t r0, int nr, uint32_t* out, cudaStream_t st);
struct FaciesCornersHost {
  int nang;
  bool pairs;                                     // cells packed in pairs (facies_pairs)
  const float* t;                                 // device, nang x ny x nx
  FaciesBoxHost box[1 << kMaxFaciesAngles];
  const float* dens[1 << kMaxFaciesAngles];       // device density volume of each corner
  float4* packed[1 << kMaxFaciesAngles];          // device scratch of facies_packed_bytes each
};
size_t facies_packed_bytes(const FaciesBoxHost& b, int nf, bool pairs);
// whether the volumes of hc.box are packed in pairs: neither small ones nor those that then pass the L2
bool facies_pairs(const FaciesCornersHost& hc, int nf);
// the probabilities from volumes already packed (launch_facies_prob_corners = pack + eval)
cudaError_t launch_facies_eval(const float* vp, const float* vs, const float* rho, int nx, int ny, int nz, int rnxp_in,
                               int nyp_in, int rnxp_out, const FaciesCornersHost& hc, int nf, const float* prior,
                               float undef_sum, float* const* out, float* seis_lh, cudaStream_t st);
// the facies-interleaved copies of every corner volume (hc.dens -> hc.packed)
cudaError_t launch_facies_pack(const FaciesCornersHost& hc, int nf, cudaStream_t st);
// What the inverse x transform of the posterior mean needs to evaluate the facies
// probabilities in the same pass (fft4_facies.cuh).
struct FaciesFuse {
  float* mean[3];        // the posterior-mean grids: half spectra in, real rows out, in place
  float scale;           // their FFTGrid inverse scale
  int nx, ny, nz, nyp;   // voxels evaluated; the grids' padded y size (rows j + nyp k)
  int rnxp_out;          // floats per row of the probability grids, 2 (nx / 2 + 1)
  int nf;
  float undef_sum;
  FaciesPrior pr;
  FaciesOut out;         // nf + 1 probability grids (the last the undefined class)
  float* seis_lh;        // the seismic likelihood, or null
};
// The fused pass for even nxp whose half length has a four-step split (four_step_supported);
// rows = nyp nzp.  The corner volumes must be packed already.
cudaError_t launch_x4_facies(const FaciesFuse& F, const FaciesCornersHost& hc, int nxp, int rows, const float2* tw,
                             const float2* twn, cudaStream_t st, int* nlaunch);
cudaError_t launch_facies_prob_corners(const float* vp, const float* vs, const float* rho, int nx, int ny, int nz,
                                       int rnxp_in, int nyp_in, int rnxp_out, const FaciesCornersHost& hc, int nf,
                                       const float* prior, float undef_sum, float* const* out, float* seis_lh,
                                       cudaStream_t st);

}  // namespace crava
