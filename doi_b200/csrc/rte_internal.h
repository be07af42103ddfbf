// rte_internal.h -- shared declarations between the host context (rte_host.cpp) and the
// sm_100a kernels (rte_*.cu).  Not part of the public ABI (include/rte_b200.h).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define RTE_MAX_L 7
#define RTE_PAIR_THREADS 128  // destination voxels per CTA (one per thread)
#define RTE_PAIR_TS 64        // source voxels staged in shared memory per step
#define RTE_MAX_MOM 48        // self-term power-series terms

// Stored pair kernel layout.  Sources in column order (slot = (y * nx + x) * nz + z), destinations in the same
// order with every column padded to nzp positions, a whole number of groups (one thread's destinations, see
// rte_column.cu).  A block holds the 32 * group positions of one warp of the column kernels, [source slot]
// [32 * group] with ld source rows, each row destination-major (the 32 lanes' first destinations, their
// second, ...): a warp's values of a run of sources are one contiguous block.
__host__ __device__ inline size_t kmat_index(size_t s, size_t p, size_t ld, int group) {
  const size_t kb = 32 * (size_t)group, o = p % kb;
  return (p / kb * ld + s) * kb + o % group * 32 + o / group;
}
// destination position of a slot
__host__ __device__ inline int kmat_pos(int slot, int nz, int nzp) { return slot / nz * nzp + slot % nz; }
// Destinations per thread of the column kernels.  Three at L <= 5, where four CTAs per SM still fit (33^3 L=5 launch:
// 2 per thread 2.93 ms, 3 2.41, 4 at two CTAs 3.11; FP64: 1 7.0 ms, 2 9.3, 3 5.6), two above.
#define RTE_COL_G(L) ((L) <= 5 ? 3 : 2)
// ... of a complex pair's kernel: the same, or one where two sets of sums exceed the registers
#define RTE_COL_GC(L, fp64) ((L) <= ((fp64) ? 3 : 5) ? RTE_COL_G(L) : 1)
// real right-hand sides per thread of an FP32 launch with an even number of them.  Two share the
// trigonometric rows, the kernel values and the copies, but take the registers of half the CTAs at L >= 4.  Solves of
// four sources and 20 terms, one -> two a thread: 33^3 L=1 92 -> 62 ms, L=2 111 -> 95, L=3 128 -> 111, L=5 203 -> 182;
// 29^3 L=4 79 -> 81, 25^3 L=6 76 -> 78, so these keep one.  (L = 7 would gain: 25^3 99.9 -> 96.9, 17^3 18.3 -> 17.2.)
#define RTE_COL_NB(L) (((L) >= 1 && (L) <= 3) || (L) == 5 ? 2 : 1)

// Plain FP64 pair operator (k_pair_fp64): sums over `chunk` sources per blockIdx.y.
struct PairArgs {
  int N, nx, ny, nz, Cfull;
  double dx, dy, dz;
  double prop_thresh;
  double kscale;        // dV / cm folded into the pair kernel
  const int* perm;      // thread -> voxel index
  const double* mut;    // mu_t per voxel
  const double* Win;    // [N][Cfull]
  double* part;         // partial sums [S][N][Cfull], indexed by voxel
  int chunk, nsplit;
};

// Pair-kernel precompute (rte_store.cu): rows of the source columns [col0, col1), destinations all.
struct StoreArgs {
  int N, nx, ny, nz;
  double dx, dy, dz, prop_thresh, kscale;
  const void* mu;     // mu_t in column order (T)
  void* K;            // T, row 0 is the first source of col0 (kmat_index with ld = Kld)
  size_t Kld;
  int nzp, group;
  int col0, col1;
  int ry;             // rows of columns up to which pairs are computed; what lies beyond is not read (rte_col_reach)
  const void* Kin;    // derivative mode: K of the same sources, whose slot 0 of this launch is row kin_slot (may be K)
  size_t Kin_ld;
  int kin_slot;
  int* counter;       // scratch: next unit of work
  // set by the launcher: column pairs per chunk, z block, chunks that share their lists, list entries of a batch,
  // blocks of z as units of their own
  int npair, zb, group_ch, cap, zsplit;
};

// Column form of the pair operator (rte_column.cu): sources and destinations in column order, one CTA per
// 128 threads' destinations, right-hand side and chunk of source columns.
struct ColArgs {
  int N, nx, ny, nz, Cfull;
  int nzp, group;     // destination positions per column, destinations per thread (ColDims)
  int nrhs;           // right-hand sides of this launch (1 for a complex pair)
  const void* W;      // source rows [nrhs][N][pitch] (T, slot order), coefficient c times N_c
  int pitch;
  const void* K;      // pair kernel (T), rows from source slot kslot0 (kmat_index with ld = Kld)
  size_t Kld;
  int kslot0;
  const void* tab;    // angle rows (rte_launch_col_table)
  int row, azn, csn, cls, pho, tg;
  void* part;         // chunk sums [S][N][vstride]: FP32 raw, or FP64 with N_c applied
  int vstride;
  int split0;         // first chunk-sum slice
  int col0, col1;     // source columns [col0, col1), `chunk` columns per blockIdx.y
  int ry;             // rows of columns within which voxels couple
  int chunk, nsplit;
  int* err;
  double* red;        // the epilogue's four norms, zeroed here for it
  // pair-by-pair form of flat grids (rte_flat.cu; tab: directions): entry of displacement 0, steps per column axis
  int d0, dsx, dsy, dsz;
  int tz, ncd;        // set by the launcher: sources per run, destination columns per CTA at most
};
struct ColDims {
  int pitch;                        // source rows
  int group, nzp;                   // destinations per thread, destination positions per column
  int row, azn, csn, nk, pho;       // angle rows: entries of csn values in tg residue classes of cls
  int tg, cls;
  int wide;                         // FP32 rows whose entries hold (cos theta, sin theta) in FP64
};
// chunk sums of a flat grid's exchanged frame (rte_flat.cu)
struct FlatArgs {
  int N, nx, ny, nz, Cfull, S, nb;
  int sx, sy, sz;       // voxel steps of the exchanged frame along the grid's axes
  const void* part;     // chunk sums [S][N][nb][Cfull] (ColArgs)
  const double* M;      // coefficients of the exchanged frame [Cfull][Cfull] (null: the same)
  double* out;          // [N][nb][Cfull]
};

struct ColTabArgs {
  int nx, ny, nz, nzp, L;
  double dx, dy, dz, kappa;
  int table, transpose;
  int row, azn, csn, nk, pho, tg, cls, wide;
};

// Self-voxel term of the epilogue: scale * D(mu_t(r)) W[r], D symmetric, from a table of the medium's distinct mu_t
// or the power series; W null: none.
struct SelfArgs {
  int K;
  const double* W;      // [N][nb][Cfull]
  const double* mut;
  const int* idx;       // voxel -> row of lut (null: power series)
  const double* lut;    // [ndistinct][Cfull][Cfull]
  const double* mom;    // [K][Cfull][Cfull]
  double scale;         // dV / cm
  int air_no_self;
  // derivative mode: scale * dmut(r) * dD/dmu(mu_t(r)) W (lut holds dD/dmu, or the series' derivative)
  const double* dmut;   // null: the self term itself
  // complex mu_t = mu_t + i kappa (intensity modulation): W holds (real, imaginary) pairs of rows,
  // lut_im the imaginary parts of the table (the power series takes the complex mu_t directly)
  double kappa;
  const double* lut_im;
};

struct EpiArgs {
  int N, nx, ny, nz, Cfull, S, nb;  // nb right-hand sides, layout [N][nb][Cfull]
  const double* part;   // [S][N][nb][Cfull]
  const float* partf;   // or FP32 chunk sums, times N_c here (then part is unused)
  SelfArgs self;
  const double* mus;
  int flag_scat;
  double scat[RTE_MAX_L + 1];  // per-l scatter factor (times mu_s of the voxel)
  double* Wout;         // FP64 result (may alias nothing else)
  void* rows;           // copy [nb][N][pitch] in slot order (times N_c) for the next pair launch (may be null)
  int rows64;           // rows are FP64 (else FP32)
  const int* islot;     // voxel -> slot
  int pitch;
  double* sum;          // running sum (null = do not accumulate)
  double* red;          // [0] ||Wout||^2 [1] ||sum||^2 [2] stop-layer sum of Wout [3] of sum
  int cplx;             // right-hand sides are (real, imaginary) pairs: odd ones are imaginary parts
};


struct ImgArgs {
  int nx, ny, nz, Cfull, L, vstride;
  const double* out;
  double wt[RTE_MAX_L + 1];  // transmission weights per l (m = 0 coefficient)
  double wr[RTE_MAX_L + 1];  // reflection weights per l
  const double* fball;       // ballistic flux per face pixel (z- first, z+ next); may be null
  const double* fball_im;    // its imaginary part under intensity modulation (may be null)
  const double* out_im;      // imaginary-part distribution, same layout as out (may be null)
  double* trans;  // nx*ny complex (re, im)
  double* ref;
};

// SH recurrence tables (host-computed, see rte_host.cpp) uploaded to __constant__.
struct ShTables {
  double A[64], B[64];   // q_l^m = A z q_{l-1}^m - B q_{l-2}^m, index l*(l+1)/2 + m
  double Q0[RTE_MAX_L + 1];  // q_m^m
};

#define RTE_MAX_SRC_COLS 512

struct SrcArgs {
  int nx, ny, nz, Cfull, L, kind, ncols;
  int face;                   // entry face (detector order: z-, z+, y-, y+, x-, x+)
  int cols[RTE_MAX_SRC_COLS]; // pixels of the entry face (row-major in the face) hit by the beam
  double coef[64];            // per real coefficient: scale * g^l * R_lm(beam direction)
  double scale, mag, dlen, dV, z_min, dz;
  int vstride;   // elements between consecutive voxels of W (Cfull for one right-hand side)
  const double* mut;
  const double* mus;
  double* W;     // N x vstride, zeroed by the caller
  double* fball; // ballistic exitant flux per face pixel (all six faces), zeroed by the caller
  // intensity modulation: attenuation with mu_t + i kappa; the imaginary part of the source goes to
  // W + Cfull (the second row of each voxel's pair) and that of the ballistic flux to fball_im
  double kappa;
  double* fball_im;
};

// detector faces and the adjoint gradient
struct FaceArgs {
  int nx, ny, nz, Cfull, vstride;
  const double* out;   // real basis [N][vstride]
  const double* h;     // [6][Cfull] exitant-flux weights of each face (area and cm included)
  const double* fball; // ballistic flux per face pixel, same layout as J (may be null)
  double* J;           // fluxes of all face pixels (z-, z+, y-, y+, x-, x+ concatenated)
  const double* rho;   // adjoint seed: dL/dJ per face pixel
  double* e;           // adjoint seed field [N][Cfull]
};

// Back-projection of the gradient (rte_backproject.cu); T is float for mixed contexts, double otherwise.
struct BpArgs {
  int N, nx, ny, nz, Cfull;
  double dx, dy, dz, prop_thresh, kscale;
  const int* islot;
  const double* mut;   // column order
  const void* y;       // T, destination-side field, column-order rows times N_c (rte_launch_rows), `pitch` apart
  const void* S;       // T, source-side field, likewise
  int pitch;
  const float* Kmat;   // stored pair kernel (both null: recompute the path integral)
  const double* Kmat64;
  size_t Kld;
  int nzp, group;      // layout of the stored kernel (ColDims)
  void* Q;             // T, weight of each unordered pair [source slot][destination slot > source slot]
  size_t ld;
  int accumulate;      // k_bp_weights: add to Q (later sources) instead of overwriting
  double* gcol;        // [N] column-order sums of the walk (scratch)
  double* g;           // gradient w.r.t. mu_t, accumulated [N]
  // set by the launchers: column pairs per chunk (weights) or three times as many (walk), chunks that share what
  // depends on the displacement, z block, list entries and |dz| rows of a batch, one batch for every displacement,
  // parts of a unit's z blocks or |dz| that are units of their own
  int jq, group_ch, zb, cap, rows, single, nparts;
};

struct GradLocalArgs {
  int N, Cfull, Cact;
  const double* y;      // e + D lambda
  const double* lam;    // adjoint field
  const double* S;      // forward running sum
  const double* out;    // A S
  const double* mus;
  const double* mut;
  const int* idx;       // voxel -> distinct mu_t (null: power series)
  const double* dlut;   // d Dself / d mu_t per distinct value [nd][C][C]
  const double* mom;
  int K;
  double scale;         // dV / cm
  int air_no_self;
  double scat[RTE_MAX_L + 1];
  double* gt;           // += self-term part of dL/dmu_t
  double* gs;           // += scatter part of dL/dmu_s
};

extern "C++" {
cudaError_t rte_launch_face_flux(const FaceArgs& a, cudaStream_t st);
cudaError_t rte_launch_adjoint_seed(const FaceArgs& a, cudaStream_t st);
cudaError_t rte_launch_parity(double* x, int N, int L, int vstride, cudaStream_t st);
cudaError_t rte_launch_axpy(double* y, const double* x, double alpha, size_t n, cudaStream_t st);
// ga[r] = sum_c fa[l] lam[r][c] out[r][c], gs[r] likewise with fs (N voxels, rows of (L+1)^2)
cudaError_t rte_launch_tangent_pair_dots(const double* lam, const double* out, const double* fa, const double* fs, int N,
                                         int L, double* ga, double* gs, cudaStream_t st);
cudaError_t rte_launch_y_field(double* y, const double* e, const double* lam, const double* mus, const double* scat,
                               int N, int L, int Cfull, cudaStream_t st);
// Symmetric back-projection in two passes: pair weights of one source added into Q, then one walk
// over every unordered pair scattering Q * length into the gradient.
cudaError_t rte_launch_bp_weights(const BpArgs& a, int LA, int fp64, cudaStream_t st);
cudaError_t rte_launch_bp_walk(const BpArgs& a, int fp64, cudaStream_t st);
// q = mus * scat_l * T + dmus * scat_l * out (per voxel and coefficient; q rows qstride apart)
cudaError_t rte_launch_tangent_rhs(double* q, int qstride, const double* T, const double* out, const double* mus,
                                   const double* dmus, const double* scat, int N, int L, cudaStream_t st);
cudaError_t rte_launch_scatter_add(double* dst, int dstride, const int* idx, const double* vals, int n, int C,
                                   cudaStream_t st);
cudaError_t rte_launch_strided_add(double* dst, const double* a, int astride, const double* b, int N, int C,
                                   cudaStream_t st);
cudaError_t rte_launch_masked_scale(const double* in, double* out, const uint8_t* mask, const double* fac, int N,
                                    int L, cudaStream_t st);
cudaError_t rte_launch_grad_local(const GradLocalArgs& a, cudaStream_t st);
// message returned by rte_last_error(NULL) on this thread
__attribute__((visibility("hidden"))) void rte_set_global_error(const char* msg);
cudaError_t rte_launch_source(const SrcArgs& a, cudaStream_t st);
// mutc / mutfc: mu_t in column order (islot), FP64 and FP32
cudaError_t rte_launch_medium(const double* mua, const double* mus, double* mut, double* mus_out,
                              double* mutc, float* mutfc, const int* islot, int N, double* red_max, cudaStream_t st);
cudaError_t rte_launch_fma_peak(int fp64, int iters, float* sink, cudaStream_t st, int blocks);
cudaError_t rte_upload_sh_tables(const ShTables& t);
// Uniform-medium convolution path (rte_fft.cpp): grid, padded grid, spacing, coupling distance,
// kernel scale, mu_t, and the pair range [p0, p1) of one sampling launch.
struct FftTabArgs {
  int nx, ny, nz, Mx, My, Mz;
  double dx, dy, dz, prop_thresh, kscale, mut;
  int p0, p1;
};
cudaError_t rte_launch_fft_table(const FftTabArgs& a, int L, int table, double* T, size_t M, cudaStream_t st);
cudaError_t rte_launch_fft_pad(const double* W, int vstride, int Cfull, int Cact, int nb, const FftTabArgs& a, double* F,
                               size_t M, cudaStream_t st);
cudaError_t rte_launch_fft_extract(const void* spec, double* tau, int p0, int np, int C, size_t Mk, cudaStream_t st);
cudaError_t rte_launch_fft_product(const void* That, const void* Wh, void* Oh, int C, int Cact, int nb, size_t Mk,
                                   int complex_table, cudaStream_t st);
cudaError_t rte_launch_fft_crop(const double* F, int Cfull, int Cact, int nb, const FftTabArgs& a, double* part,
                                size_t M, cudaStream_t st);
struct FftState;
cudaError_t rte_fft_prepare(FftState** s, const FftTabArgs& a, int L, int table, int nbmax, cudaStream_t st);
cudaError_t rte_fft_apply(FftState* s, const double* W, int vstride, int Cfull, int LA, int nb, double* part,
                          cudaStream_t st);
size_t rte_fft_bytes(int nx, int ny, int nz, int L, int nbmax);
cudaError_t rte_fft_warm(FftState* s, int nf);
uintptr_t rte_fft_signature(const FftState* s);
void rte_fft_destroy(FftState* s);

// host copies: the recurrence tables and the real SH R_c at a unit direction (index l*l + l + m)
ShTables make_sh_tables();
void sh_real_host(const ShTables& t, int L, double x, double y, double z, double* R);
cudaError_t rte_launch_pair_fp64(const PairArgs& a, int LA, cudaStream_t st);
cudaError_t rte_launch_store_kernel(const StoreArgs& a, cudaStream_t st, int fp64);
cudaError_t rte_launch_epilogue(const EpiArgs& a, int LA, cudaStream_t st);
cudaError_t rte_launch_images(const ImgArgs& a, cudaStream_t st);
// complex basis -> real parts; u1/u2 rows ostride apart (0: C)
cudaError_t rte_launch_to_real(const double* cplx, double* u1, double* u2, int N, int L, double* red,
                               cudaStream_t st, int ostride = 0);
cudaError_t rte_launch_to_cplx(const double* u1, const double* u2, double* cplx, int N, int L,
                               cudaStream_t st, int ustride = 0);
cudaError_t rte_launch_layer_sums(const double* W, const double* S, int N, int nx, int ny, int nz, int Cfull,
                                  double* red, cudaStream_t st, int cplx = 0);
// FP64 [N][vstride] (voxel order) -> source rows of the pair kernels in slot order (FP32, or FP64),
// coefficient c times the monic SH normalisation N_c
cudaError_t rte_launch_rows(const double* w, void* rows, const int* islot, int N, int nb, int pitch, int Cfull,
                            int fp64, cudaStream_t st);
ColDims rte_col_dims(int C, int L, int nz, int fp64, int cplx);
cudaError_t rte_launch_rows_rot(const double* w, void* rows, const double* M, const int* islot, int N, int nb, int pitch,
                                int Cfull, int fp64, cudaStream_t st);
cudaError_t rte_launch_sums_rot(const FlatArgs& a, int LA, int fp64, cudaStream_t st);
size_t rte_dirs_bytes(int nx, int ny, int nz, int L, int fp64);
cudaError_t rte_launch_dirs_table(int nx, int ny, int nz, double dx, double dy, double dz, int transpose, int L, int fp64,
                                  void* tab, cudaStream_t st);
cudaError_t rte_launch_pair_dirs(const ColArgs& a, int LA, int fp64, cudaStream_t st, int* occ = nullptr);
// rows of columns beyond its own that a launch reads the pair kernel of, where voxels couple over ry rows
int rte_col_reach(int nx, int nzp, int group, int ry);
cudaError_t rte_launch_col_table(const ColTabArgs& a, void* tab, int fp64, cudaStream_t st);
// launches, or with occ != null only reports the CTAs per SM
cudaError_t rte_launch_column(const ColArgs& a, int LA, int fp64, int cplx, cudaStream_t st, int* occ = nullptr);
}
