// ek_internal.h -- shared definitions of libekpnp's kernels and C ABI.
//
// Device memory of one channel (all planes ny rows x nxp columns, nxp = nx
// rounded up to 32, rows of FP64 256-byte aligned; 16 for nx <= 16, where a row of
// FP16 starts 32-byte aligned):
//   pops[2]   27 planes each, ping-pong: species-major (fluid f, c+ h, c- t),
//             then direction 0..8 in the reference numbering (LBM.cu:831-834).
//             Between steps a buffer holds POST-collision populations; the next
//             step pulls them (streaming fused into the load).  Right after
//             ek_init_equilibrium it holds pre-collision populations at their
//             own node ("state_pre"), and the first step reads them in place.
//   fields    9 planes: rho, ux, uy, c+, c-, psi, Ex, Ey, and the Poisson
//             right-hand side.
//   spec      (ny-2) x mp complex: x-spectrum of the interior rows (mp >= nx/2+1)
//   piv       (ny-2) x mp: pivots of the per-mode tridiagonal y-solve
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "../../include/ekpnp.h"

namespace ek {

// Programmatic dependent launch.  A kernel started by launch_pdl may be
// scheduled while the kernel before it in the stream is still draining; its
// first statement is pdl_wait(), which waits for that kernel's completion
// and the visibility of its writes, then lets the next kernel be scheduled
// in turn.  A kernel launched the ordinary way passes pdl_wait() at once.
// Used for a channel's one-wave row transform after the LBM step (measured
// at 4096 x 1024: -2.6 us a step) and for every kernel of a small channel's step
// (launch_chain); on the many-wave LBM kernel of a large channel the per-block
// wait cost ~40 us a step (the batched passes run many waves: not used there).
__device__ __forceinline__ void pdl_wait() {
#if defined(__CUDA_ARCH__)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#endif
}

// Loads of what the kernel just before in the stream wrote.  A chained kernel starts
// while that one still runs, so these values are not constant over its lifetime:
// the read-only path (__ldg, a const __restrict__ parameter) is not for them, and
// nothing may move their loads above pdl_wait().  Volatile statements stay in order,
// wait included.
__device__ __forceinline__ double ld_fresh(const double *p) {
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_fresh(const float *p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float2 ld_fresh(const float2 *p) {
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_fresh(const float4 *p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// Field-plane bytes (right-hand side + psi of every channel stepped together)
// that the evict_last stores may pin, out of the 126 MB L2: above it the
// planes are stored the ordinary way.
constexpr size_t KEEP_L2_BYTES = (size_t)80 << 20;
inline bool keep_l2_fits(size_t bytes) { return bytes <= KEEP_L2_BYTES; }

// Stores of field planes that the next kernel reads back (the Poisson
// right-hand side written by the LBM step, psi written by the inverse row
// pass): with keep set they carry an L2 evict_last policy, so the plane
// stays in L2 while the step's populations stream through it.
__device__ __forceinline__ void st_field_f(float *p, float v, bool keep) {
#if defined(__CUDA_ARCH__)
    if (keep) {
        unsigned long long pol;
        asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
        asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(p), "f"(v), "l"(pol) : "memory");
        return;
    }
#endif
    *p = v;
}

__device__ __forceinline__ void st_field_f4(float *p, float4 v, bool keep) {
#if defined(__CUDA_ARCH__)
    if (keep) {
        unsigned long long pol;
        asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
        asm volatile("st.global.L2::cache_hint.v4.f32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z),
                     "f"(v.w), "l"(pol)
                     : "memory");
        return;
    }
#endif
    *(float4 *)p = v;
}

__device__ __forceinline__ void st_field_f2(float *p, float2 v, bool keep) {
#if defined(__CUDA_ARCH__)
    if (keep) {
        unsigned long long pol;
        asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
        asm volatile("st.global.L2::cache_hint.v2.f32 [%0], {%1, %2}, %3;" ::"l"(p), "f"(v.x), "f"(v.y), "l"(pol) : "memory");
        return;
    }
#endif
    *(float2 *)p = v;
}

template <typename... Exp, typename... Act>
cudaError_t launch_attrs(const cudaLaunchAttribute *at, int nat, void (*kern)(Exp...), dim3 grid, dim3 block, size_t smem,
                         cudaStream_t s, Act &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = const_cast<cudaLaunchAttribute *>(at);
    cfg.numAttrs = nat;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<Act>(args)...);
}

template <typename... Exp, typename... Act>
cudaError_t launch_pdl(void (*kern)(Exp...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Act &&...args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    return launch_attrs(at, 1, kern, grid, block, smem, s, std::forward<Act>(args)...);
}

// A kernel of a small channel's step (PDL_NODES): launch_pdl where chain is
// set, an ordinary launch otherwise.  Chained kernels overlap on the SMs and so share one split
// of L1 and shared memory: all ask for the same small share of shared memory,
// since the LBM step lives on L1 (its pulls read every line twice or more).
// A kernel scheduled while another holds the largest share gets the L1 that is
// left: on B200 that cost a batch of 64 channels 27 % of its step.
// 1000 x 257 FP64 on B200: 46 us a step at 7 to 25 %, 53 at 100 %.
constexpr unsigned CHAIN_SMEM_PERCENT = 25;
template <typename... Exp, typename... Act>
cudaError_t launch_chain(bool chain, void (*kern)(Exp...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Act &&...args) {
    if (!chain) {
        kern<<<grid, block, smem, s>>>(std::forward<Act>(args)...);
        return cudaGetLastError();
    }
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at[1].val.sharedMemCarveout = CHAIN_SMEM_PERCENT;
    return launch_attrs(at, 2, kern, grid, block, smem, s, std::forward<Act>(args)...);
}
// Channels of at most this many nodes: every kernel of a step is about one
// wave of blocks, and the step a chain of launch latencies.  Time of a step chained
// over that with ordinary launches (pass A always early), FP64 and FP32 on B200: 256 x
// 128 0.69, 0.69; 1000 x 257 0.83, 0.83; 512 x 512 0.82, 0.79.  Above the line powers of
// two still gain (512 x 1024 0.89, 0.85; 1024 x 1024 0.96, 0.93; 2048 x 2000 1.02,
// 1.02), but mixed lengths, whose blocks then wait in the others' place, lose: 1000 x
// 500 1.05, 1.05; 1500 x 800 1.13, 1.16.
constexpr size_t PDL_NODES = (size_t)1 << 18;
// The LBM kernel of a step: by itself (many waves of blocks); of a small
// channel, letting pass A be scheduled early; the same, itself scheduled while
// the kernel before drains.  CHAIN_NEXT gathers its populations before the wait
// for that kernel, so it is only for a step right after another one's Poisson
// solve (the populations were written three kernels earlier).
enum StepChain { CHAIN_NONE = 0, CHAIN_FIRST = 1, CHAIN_NEXT = 2 };

// D2Q9 velocity set in the reference numbering:  6 2 5 / 3 0 1 / 7 4 8
__host__ __device__ constexpr int cxd(int d) {
    return d == 1 || d == 5 || d == 8 ? 1 : (d == 3 || d == 6 || d == 7 ? -1 : 0);
}
__host__ __device__ constexpr int cyd(int d) {
    return d == 2 || d == 5 || d == 6 ? 1 : (d == 4 || d == 7 || d == 8 ? -1 : 0);
}
__host__ __device__ constexpr int oppd(int d) { return d == 0 ? 0 : (d <= 4 ? (d + 1) % 4 + 1 : (d - 3) % 4 + 5); }
static_assert(oppd(1) == 3 && oppd(2) == 4 && oppd(3) == 1 && oppd(4) == 2, "opp straight");
static_assert(oppd(5) == 7 && oppd(6) == 8 && oppd(7) == 5 && oppd(8) == 6, "opp diagonal");

constexpr double W0 = 4.0 / 9.0, WS = 1.0 / 9.0, WD = 1.0 / 36.0;  // LBM.h:105-107

// Relaxation and wall constants, evaluated on the device with the reference's
// expressions (LBM.cu:336-341, 745-746, 812-813) so they round as it does.
struct Rates {
    double wp, wm;    // fluid omega+*dt, omega-*dt
    double wcp, wcm;  // c+  (minus set by diffu, plus by VC)
    double wtp, wtm;  // c-  (minus set by D, plus by VT)
    double sp, sm;    // Guo source factors 1 - dt*omega/2
    double ms, md;    // moving top wall terms
};

// Reciprocals of a channel's constants and the weights over cs2 (LBM.cu:556-572),
// rounded once: the FP64 step divides by the constants through them.
struct Recips {
    double cs2, cfl, dx, dy, eps;
    double w0_cs2, ws_cs2, wd_cs2, ci2_cs2;  // W / cs2, (1/cfl)^2 / cs2
};

// Per-channel constants, passed by value to every kernel.
struct Chan {
    int nx, ny, nxp, flags;
    size_t plane;  // ny * nxp
    double dx, dy, dt, cfl, cs2, rho0, c0;
    double mob_p, mob_n, f_charge, eps, ext_x, exf;
    Rates r;
    Recips inv;
    const double *zlo, *zhi, *cplo, *cphi, *cnlo, *cnhi;  // per-x wall values (nx each)
    // Shifted storage only: per-row reference densities divided by 36, three
    // rows of ny floats (fluid, c+, c-).  A population of species s stored at
    // row y holds f - w_i * 36 * kref[s*ny + y]; every kref value is a
    // multiple of 2^-q, so 36 w_i (kref[y'] - kref[y]) is exact in FP32.
    const float *kref;
    // Shifted storage only: per-x ion frames of the wall nodes (/36), per
    // population buffer, and half their defect (see ChanF::kwall).
    const float *kwall;
    const float *wdelta;
    // Shifted storage only: the step's field planes (PoissonPlan::rhsf, psif, psim),
    // and the x-fluctuation of the wall lifting, (zeta(x) - zeta_mean)/dy^2,
    // lower wall then upper (2 nx floats), which rows 1 and ny-2 subtract
    // from rhsf.
    float *rhsf;
    const float *psif;
    const double *psim;
    const float *lift;
    int keep_l2;   // right-hand side and psi planes held in L2 between kernels
};

enum Field { F_RHO = 0, F_UX, F_UY, F_CP, F_CN, F_PSI, F_EX, F_EY, F_RHS, F_COUNT };

// ---- launchers (ek_lbm_f64.cu) ----
cudaError_t launch_rates(const ek_params &p, Rates *dev_out, cudaStream_t s);
cudaError_t launch_init_f64(const Chan &c, double *pops, const double *fields, bool explicit_e,
                            cudaStream_t s);
// chain: how the step's kernel is launched (StepChain)
cudaError_t launch_step_f64(const Chan &c, const double *src, double *dst, double *fields,
                            bool first, bool explicit_e, bool moments, int chain, cudaStream_t s);
cudaError_t launch_efield_f64(const Chan &c, double *fields, cudaStream_t s);
cudaError_t launch_rhs_from_moments_f64(const Chan &c, double *fields, cudaStream_t s);

// ---- Poisson-Boltzmann start (ek_init.cu) ----
cudaError_t launch_pb_fill(const Chan &c, double *fields, double *psi_old, cudaStream_t s);
cudaError_t launch_pb_conc(const Chan &c, double e_kt, double *fields, cudaStream_t s);
cudaError_t launch_pb_relax(const Chan &c, double omega, double *fields, double *psi_old, cudaStream_t s);
// Newton Poisson-Boltzmann start: ncol columns (walls[q] = {zeta_lo, zeta_hi})
// solved on the device (psi, cp, dp: ny x ncol scratch, ok: ncol flags), then
// the fields of every node from its column colmap[x].
cudaError_t launch_pb_newton(const Chan &c, double dy, double g, double a, const double2 *walls, int ncol,
                             double *psi, double *cp, double *dp, int *ok, const int *colmap, double *fields,
                             cudaStream_t s);

// ---- shifted-storage forms (ek_lbm_f32.cu); storage = EK_STORE_F32 or _F16 ----
// sbuf: index (0/1) of the population buffer that src is (it names the wall
// ions' frames); buf: the buffer that pops is.
cudaError_t launch_step_shifted(const Chan &c, int storage, const void *src, void *dst, double *fields,
                                bool first, bool explicit_e, bool moments, int sbuf, int chain, cudaStream_t s);
cudaError_t launch_init_shifted(const Chan &c, int storage, void *pops, const double *fields, bool explicit_e,
                                int buf, cudaStream_t s);
// Wall frames of the ions from the fields' wall rows (initialisation; buf is
// the buffer the initial populations go to), and their defect after the wall
// concentrations change.
cudaError_t launch_wall_frames(const Chan &c, const double *fields, int qp, int qn, int buf, float *kwall,
                               float *wdelta, cudaStream_t s);
cudaError_t launch_wall_delta(const Chan &c, const float *kwall, float *wdelta, cudaStream_t s);
// Row means of rho, c+, c- rounded to the grid K 2^-q, stored /36 in
// kout[3*ny] (ek_lbm_f32.cu); q per species.
cudaError_t launch_row_refs(const Chan &c, const double *fields, int qf, int qp, int qn, float *kout,
                            cudaStream_t s);
// Re-express stored shifted populations against a new reference profile.
cudaError_t launch_rebase(const Chan &c, int storage, void *pops, const float *kold, const float *knew,
                          cudaStream_t s);
// ---- TMA-fed persistent form of the shifted step (ek_lbm_tma.cu) ----
// map_out: a 128-byte CUtensorMap (64-byte aligned) over one population buffer.
cudaError_t make_pop_tensor_map(int storage, const void *pops, int nxp, int ny, void *map_out);
cudaError_t launch_step_tma(const Chan &c, int storage, const void *map, const void *src, void *dst, double *fields,
                            bool first, bool explicit_e, bool moments, int sbuf, int *err, long long wait_cycles,
                            cudaStream_t s);
// map_out: a CUtensorMap over a row-major BF16 matrix (ld elements a row, 16-byte
// aligned rows), boxes of box_rows x box_cols with 128-byte swizzle.
cudaError_t make_matrix_tensor_map(const void *p, int rows, int cols, int ld, int box_rows, int box_cols, void *map_out);
inline size_t pop_elem_bytes(int storage) { return storage == EK_STORE_F64 ? 8 : (storage == EK_STORE_F32 ? 4 : 2); }

// ---- Poisson (ek_poisson.cu) ----
struct PoissonPlan {
    int nx, ny, n, mp, log2nx;  // n = ny-2 interior rows
    bool pow2;
    double dy2;                 // dy*dy
    double2 *tw;                // nx twiddles exp(-2 pi i k/nx)
    double *piv;                // n x mp pivots
    double2 *spec;              // n x mp spectrum
    // FP32 form (shifted storage): modes >= 1 in FP32, the zero mode in FP64
    // (column 0 of spec); null where the form is not set up
    float2 *twf;                // FP32 row transforms: per-pass twiddle tables (< nx entries)
    float *pivf;                // n x mp pivots, FP32 (mode 1 starts a sector)
    float2 *specf;              // n x mp spectrum, FP32 (the same from nx = 32 on)
    double *rowmean;            // n row means of the last solve: the offset removed before the FP32 FFT
    int *rowmean_ok;            // set by the first solve's pass C; before it pass A takes exact means
    // Field planes of the shifted-storage step (every shifted context; the
    // FP32 form reads and writes them directly, the FP64 form through
    // compose/split kernels):
    //   rhsf  (ny x nxp) FP32: the right-hand side minus its row constant,
    //         rhs_q (c+ - c- - (R+ - R-)); the constant rhs_q (R+ - R-) of the
    //         row references and the wall lifting are added in FP64 by pass A
    //   psif  (ny x nxp) FP32: psi minus its row mean
    //   psim  (ny) FP64: the row means of psi (the zero mode, walls included)
    float *rhsf;
    float *psif;
    double *psim;
    double zlo_mean, zhi_mean;  // x-means of the wall potentials (psim of the wall rows)
    int keep_l2;                // psi stores ask L2 to keep the plane (see st_field_f)
};
// pass 0: row FFTs, 1: tridiagonal column solve, 2: inverse row FFTs + walls
cudaError_t poisson_pass_f64(int pass, const PoissonPlan &pp, const Chan &c, double *fields, cudaStream_t s);
// Same passes with the right-hand side and psi planes given directly.
cudaError_t poisson_pass_f64_at(int pass, const PoissonPlan &pp, const Chan &c, const double *rhs, double *psi,
                                cudaStream_t s);
size_t poisson_smem_bytes_f64(int nx);
// FP32 form of the passes (power-of-two nx >= 16, n <= 8192, twf/pivf/specf
// set): the row FFTs and the column solves of the modes >= 1 in FP32 on the
// fluctuation about each row's mean; the row sums (the zero mode), its
// column solve and the mean of psi in FP64.
bool poisson_f32_supported(const PoissonPlan &pp);
// Passes 0 and 2 (pass 1 is poisson_tridiag_f32): pass 0 reads
// pp.rhsf with the row constants of c.kref and the wall lifting; pass 2 writes
// pp.psif and pp.psim, and the FP64 psi plane too when write_f64.
cudaError_t poisson_pass_f32(int pass, const PoissonPlan &pp, const Chan &c, double *psi, bool write_f64,
                             cudaStream_t s);
// Shifted storage with the FP64 passes: the FP64 right-hand side from rhsf
// (before pass 0), and psif/psim from the FP64 psi (after pass 2, and
// whenever psi was set from outside).
cudaError_t launch_compose_rhs(const PoissonPlan &pp, const Chan &c, double *rhs, cudaStream_t s);
// The FP64 row constant of the right-hand side of row y (1 <= y <= ny-2):
// rhs_q (R+ - R-) of the row references, minus zeta_mean/dy^2 on rows 1 and
// ny-2 (the x-mean of the wall lifting; its fluctuation is Chan::lift).
__host__ __device__ inline double rhs_row_constant(const PoissonPlan &pp, const Chan &c, int y) {
    const double rq = -c.f_charge / c.eps, inv_dy2 = 1.0 / (c.dy * c.dy);
    double v = rq * (36.0 * (double)c.kref[c.ny + y] - 36.0 * (double)c.kref[2 * c.ny + y]);
    if (y == 1) v -= pp.zlo_mean * inv_dy2;
    if (y == c.ny - 2) v -= pp.zhi_mean * inv_dy2;
    return v;
}
cudaError_t launch_split_psi(const PoissonPlan &pp, const Chan &c, const double *psi, cudaStream_t s);
// rhsf from the c+, c- moments (a solve outside the step, FP32 form).
cudaError_t launch_rhsf_from_moments(const PoissonPlan &pp, const Chan &c, const double *fields, cudaStream_t s);
// Pass B of the FP32 form, one kernel: the FP64 zero mode in its first
// block, the FP32 modes in the others.  Batched: items int3 {channel, first
// mode, modes per block}, modes per block 0 naming a channel's zero mode.
cudaError_t poisson_tridiag_f32(const PoissonPlan &pp, cudaStream_t s);
cudaError_t batch_tridiag_f32(const PoissonPlan *plans, const void *items, int nitems, cudaStream_t s);
// Batched Poisson passes of the FP32 form over many channels (ek_batch.cu
// builds the items): pass 0/2 items int2 {channel, first row pair}
// (each block/(nx/16) row pairs; power-of-two nx from 16 to 4096); pass 1 is batch_tridiag_f32.  write_f64 as poisson_pass_f32.
// block: the threads a block, batch_row_block of the widest channel.
cudaError_t batch_poisson(int pass, const PoissonPlan *plans, const Chan *chans, double *const *fields,
                          const void *items, int nitems, int block, bool write_f64, cudaStream_t s);
int batch_row_block(int nx_max);
// The whole solve of a small channel in one launch, by one cluster of `blocks`
// blocks: poisson_cluster_blocks of the plan (0: the separate passes), looked up
// outside a capture.
int poisson_cluster_blocks(const PoissonPlan &pp, bool f32);
cudaError_t poisson_cluster(const PoissonPlan &pp, const Chan &c, bool f32, const double *rhs, double *psi, bool write_f64,
                            int blocks, cudaStream_t s);
int poisson_tridiag_modes(int n, int nx);
// Steady-state residual sums (ek_residual.cu): per channel 8 FP64 sums,
// (q - q_snap)^2 then q^2 for q in (ux, c+, c-, psi); the snapshot is updated.
cudaError_t launch_residual_f64(const Chan &c, const double *fields, double *snap, double *part,
                                int nblocks, double *out8, cudaStream_t s);
int residual_blocks(const Chan &c);
// Many channels: items int4 {channel, block, blocks of the channel, first
// partial}, ranges int2 {first partial, blocks} per channel, out8 8 per channel.
cudaError_t launch_batch_residual(const Chan *chans, double *const *fields, double *const *snaps, const int4 *items,
                                  int nitems, const int2 *ranges, int nch, double *part, double *out8,
                                  cudaStream_t s);
// Record an error message for ek_last_error() (ek_api.cu).
void set_last_error(const char *msg);
// Shared-memory attributes of the row kernels: of one plan's length (its sizes and
// specf set), of all FP64 passes (ek_poisson_noalloc), of a batch's.
cudaError_t poisson_set_smem_limits(const PoissonPlan &pp);
cudaError_t poisson_load_f64();
cudaError_t batch_set_smem_limits(int block);

}  // namespace ek
