// Kernels of the batched 3DI fitting path (sm_100a). Built with -fmad=false: every formula
// below is evaluated in the operand order of the 3DI sources it restates, without FMA
// contraction, so each per-fragment quantity is bit-identical to the CPU oracle's.
#include "tdi_internal.cuh"
#include "tdi_async.cuh"
#include "tdi_cholesky.cuh"

#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cfloat>
#include <cmath>

namespace tdi {

// ------------------------------------------------------------------------------------------
// Rotation R(u) and dR/du_i (rotation_header.cu:46-151).

__device__ __forceinline__ void mul33(const float *A, const float *B, float *C)
{
    C[0] = (A[0] * B[0] + A[3] * B[1]) + A[6] * B[2];
    C[1] = (A[1] * B[0] + A[4] * B[1]) + A[7] * B[2];
    C[2] = (A[2] * B[0] + A[5] * B[1]) + A[8] * B[2];
    C[3] = (A[0] * B[3] + A[3] * B[4]) + A[6] * B[5];
    C[4] = (A[1] * B[3] + A[4] * B[4]) + A[7] * B[5];
    C[5] = (A[2] * B[3] + A[5] * B[4]) + A[8] * B[5];
    C[6] = (A[0] * B[6] + A[3] * B[7]) + A[6] * B[8];
    C[7] = (A[1] * B[6] + A[4] * B[7]) + A[7] * B[8];
    C[8] = (A[2] * B[6] + A[5] * B[7]) + A[8] * B[8];
}

__device__ __forceinline__ void skew(float *S, const float *u)
{
    S[0] = 0; S[1] = u[2]; S[2] = -u[1];
    S[3] = -u[2]; S[4] = 0; S[5] = u[0];
    S[6] = u[1]; S[7] = -u[0]; S[8] = 0;
}

// R(u) alone, by the operations of rotation() (a line search's trials need no derivative).
__device__ __forceinline__ void rotation_r(const float *u, float *R)
{
    const float theta = sqrtf((u[0] * u[0] + u[1] * u[1]) + u[2] * u[2]);
    const float un[3] = {u[0] / theta, u[1] / theta, u[2] / theta};
    float Sn[9], Sn2[9];
    skew(Sn, un);
    const float st = (float)sin((double)theta);
    const float cis = 1.0f - (float)cos((double)theta);
    mul33(Sn, Sn, Sn2);
#pragma unroll
    for (int i = 0; i < 9; ++i)
        R[i] = i % 4 == 0 ? (cis * Sn2[i] + 1.0f) + st * Sn[i] : cis * Sn2[i] + st * Sn[i];
}

__device__ void rotation(const float *u, float *R, float *dR)
{
    float theta = sqrtf((u[0] * u[0] + u[1] * u[1]) + u[2] * u[2]);
    float un[3] = {u[0] / theta, u[1] / theta, u[2] / theta};
    float R1[3][9], Sn[9], Sn2[9];
    skew(R1[0], u); skew(R1[1], u); skew(R1[2], u);
    skew(Sn, un);
    float st = (float)sin((double)theta);
    float cis = 1.0f - (float)cos((double)theta);
    float tinv2 = 1.0f / (theta * theta);
    for (int a = 0; a < 3; ++a)
        for (int i = 0; i < 9; ++i) R1[a][i] *= u[a];
    mul33(Sn, Sn, Sn2);
    for (int i = 0; i < 9; ++i) {
        if (i == 0 || i == 4 || i == 8)
            R[i] = (cis * Sn2[i] + 1.0f) + st * Sn[i];
        else
            R[i] = cis * Sn2[i] + st * Sn[i];
    }
    float IR[9];
    for (int i = 0; i < 9; ++i) IR[i] = R[i] * -1.0f;
    IR[0] += 1; IR[4] += 1; IR[8] += 1;
    for (int a = 0; a < 3; ++a) {
        float R2[9], R3[9];
        const float *c = IR + 3 * a;
        R2[0] = u[0] * c[0]; R2[1] = u[0] * c[1]; R2[2] = u[0] * c[2];
        R2[3] = u[1] * c[0]; R2[4] = u[1] * c[1]; R2[5] = u[1] * c[2];
        R2[6] = u[2] * c[0]; R2[7] = u[2] * c[1]; R2[8] = u[2] * c[2];
        for (int i = 0; i < 9; ++i) R1[a][i] += R2[i];
        R3[0] = R1[a][0] - R2[0]; R3[1] = R1[a][1] - R2[3]; R3[2] = R1[a][2] - R2[6];
        R3[3] = R1[a][3] - R2[1]; R3[4] = R1[a][4] - R2[4]; R3[5] = R1[a][5] - R2[7];
        R3[6] = R1[a][6] - R2[2]; R3[7] = R1[a][7] - R2[5]; R3[8] = R1[a][8] - R2[8];
        mul33(R3, R, dR + 9 * a);
        for (int i = 0; i < 9; ++i) dR[9 * a + i] *= tinv2;
    }
}

// Kernel ids for live profiling (tdi_batch_profile).
enum KernelId : int32_t { KID_VERTEX = 1, KID_RASTER = 2, KID_RENDER = 3, KID_NEIGHBOURS = 4,
                          KID_JACOBIAN = 5, KID_NORMAL_EQ = 6, KID_BARRIER = 7, KID_SOLVE = 8,
                          KID_RESOLVE = 9 };

__device__ __forceinline__ void prof_count(const DBatch &b, int id, unsigned long long n = 1)
{
    if (b.prof_id == id) atomicAdd(b.prof_frames, n);
}

// ------------------------------------------------------------------------------------------
// Stage control.

// Frames running the stage this round: the host's count, or the device count the previous
// round's compaction wrote (rounds replayed from a CUDA graph, whose grids are sized for a
// capacity; blocks past the count return at once).
__device__ __forceinline__ int active_n(const DBatch &b) { return b.dnact ? *b.dnact : b.nact; }

__device__ void end_shape_stage(const Cfg &c, FrameCtl &ctl, int stage, int outer)
{
    ctl.active = 0;
    ctl.render = 0;
    ctl.need_jac = 0;
    if (stage == ST_RIGID) ctl.iters_rigid += outer; else ctl.iters_finetune += outer;
    if (stage == ST_RIGID) ctl.stage_ok = outer > c.niters_success;
}

// Line-search rejection (model_fitter.cu:325-355) by a whole block: shrink t, stop below the
// threshold, otherwise place the next trial x_ls = x + t d over the entries the stage updates. A
// trial with tau_z < 0 ends the stage: the reference's line search then breaks without terminating,
// and every later outer iteration repeats the same trial (the frame is stuck at x,
// model_fitter.cu:255-259). s_t: a shared float.
__device__ void shape_reject(const DModel &m, const DBatch &b, const Cfg &c, int f, int stage, float *s_t)
{
    FrameCtl &ctl = b.ctl[f];
    const int maxit = stage == ST_RIGID ? c.max_iters_rigid : c.max_iters_finetune;
    if (threadIdx.x == 0) {
        const float t = ctl.t * 0.8f;
        ctl.t = t;
        *s_t = t;
        if (t < 0.075f) end_shape_stage(c, ctl, stage, ctl.outer < maxit ? ctl.outer + 1 : ctl.outer);
    }
    __syncthreads();
    const float t = *s_t;
    if (t < 0.075f) return;
    const int n_upd = stage == ST_FINETUNE ? m.K : m.KT;
    const float *x = b.x + (size_t)f * m.KTP, *d = b.d + (size_t)f * m.KTP;
    float *xl = b.x_ls + (size_t)f * m.KTP;
    for (int a = threadIdx.x; a < n_upd; a += blockDim.x) xl[a] = x[a] + t * d[a];
    __syncthreads();
    if (threadIdx.x == 0 && xl[m.K + 2] < 0.0f) {
        ctl.flags |= FLAG_STUCK_NEG_TZ;
        end_shape_stage(c, ctl, stage, maxit);
    }
}

// Lists of a round, built by atomic appends (a kernel's result does not depend on their order): the
// frames that render, and those whose accepted point gets its normal equations.
__device__ __forceinline__ int render_n(const DBatch &b) { return b.rcount[0]; }
__device__ __forceinline__ int jac_n(const DBatch &b) { return b.rcount[1]; }

constexpr int SS_THREADS = 96;                   // start of a stage: a block per frame copies its states

__global__ void __launch_bounds__(SS_THREADS) k_stage_start(DModel m, DBatch b, Cfg c, int stage)
{
    const int f = blockIdx.x, tid = threadIdx.x;
    if (f == 0 && tid == 0) b.rcount[0] = b.rcount[1] = 0;
    if (f >= b.F) return;
    if (tid == 0) {
        FrameCtl &ctl = b.ctl[f];
        const bool dead = (ctl.flags & (FLAG_RENDER_SKIPPED | FLAG_OVERFLOW)) != 0;
        ctl.active = dead ? 0 : 1;
        ctl.mode = M_FULL;
        ctl.render = 0;
        ctl.need_jac = 0;
        ctl.t = 1.0f;
        ctl.inner = 0;
        ctl.outer = 1;
    }
    if (stage == ST_LAMBDA && tid < 3) b.lam_ls[f * 4 + tid] = b.lam[f * 4 + tid];
    // fit_3DMM_lambdas copies ov.betas into ov_linesearch (model_fitter.cu:991) and so
    // does fit_to_video_frame before each shape fit (video_fitter.cu:570-574); the
    // finetune keeps the line-search state the last shape fit left.
    if (stage == ST_RIGID || stage == ST_LAMBDA)
        for (int a = tid; a < m.KT; a += SS_THREADS) b.x_ls[(size_t)f * m.KTP + a] = b.x[(size_t)f * m.KTP + a];
}

// ------------------------------------------------------------------------------------------
// Vertex stage: X0 = mean + E*eps (sequential fmaf over k), camera transform and
// projection (renderer.cu:806-861, funcs.cu:395-453). A block owns up to 96 frames (fewer
// for bases too wide for that, vt_frames; coefficients, rotations, translations, cameras and render flags staged in shared memory) and walks a
// strided set of 32-vertex tiles; each tile's basis rows (32 x 3 x KP floats, contiguous in
// HBM) are brought into shared memory by the TMA engine, one bulk copy per vertex row,
// double-buffered so that the next tile streams in while this one is computed. A thread
// owns one vertex x 2 to 12 frames (3 FMA chains each). geo[f][slot] = (X0, Y0, Z0, albedo);
// proj[f][slot] = (xp, yp, camera Z, 0).
// The grid is one-dimensional (about two blocks per SM) and is split on the device by the
// number of frames that render this round (known only there): ftiles frame tiles x groups
// vertex-tile stripes, so that every block has work whatever share of the active frames
// the pre-render checks rejected. The frames are dealt evenly to the tiles and warps, and a warp
// runs the loop compiled for its number of frame pairs: 77 frames are one tile of 10 per thread
// (64-frame tiles carried 51 idle ones), and a warp without a frame only keeps the buffers moving.
// Full rounds are bound by the packed multiply-adds and the projection's divisions (814 us for 1,024
// frames, 16 per thread spill and take 869); 77 frames 112 -> 75 us, one frame 10.5 -> 6.9 us, where
// the frames' coefficients, stored with all lanes in one bank, also took a part.

// Two IEEE fused multiply-adds in one instruction (sm_100 packed FP32): d.x = fma(a.x, b.x, c.x),
// d.y = fma(a.y, b.y, c.y), round to nearest, denormals kept -- the same results as two fmaf.
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c)
{
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<unsigned long long &>(d))
        : "l"(reinterpret_cast<const unsigned long long &>(a)), "l"(reinterpret_cast<const unsigned long long &>(b)),
          "l"(reinterpret_cast<const unsigned long long &>(c)));
    return d;
}

__device__ __forceinline__ float2 fmul2(float2 a, float2 b)
{
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<unsigned long long &>(d))
        : "l"(reinterpret_cast<const unsigned long long &>(a)), "l"(reinterpret_cast<const unsigned long long &>(b)));
    return d;
}

// 1 in both halves, from a zero the compiler does not know to be one. Packed products and
// packed sums are contracted into packed fused multiply-adds by the assembler, .rn or not (measured:
// every result equals fma's); a sum written as fma(p, 1, s) with an unknown 1 keeps the product's
// own rounding and rounds as p + s.
__device__ __forceinline__ float2 packed_one(int zero)
{
    const float u = __int_as_float(0x3f800000 | zero);
    return make_float2(u, u);
}

constexpr int VT_V = 32;                                   // vertices per tile (one per lane)
constexpr int VT_F = 96;                                    // frames of a block, at most (12 per thread)
constexpr int VT_SMEM = 200 * 1024;                         // shared memory of a block, at most
constexpr int VT_FR = 16;                                   // per-frame floats: R(9), tau(3), cam(4)
constexpr int VT_BLOCKS_PER_SM = 2;
constexpr int VT_WARPS = 8;                                 // computing warps; one more issues the copies
constexpr int VT_THREADS = (VT_WARPS + 1) * 32;

__host__ __device__ __forceinline__ int vt_row(int KP) { return 3 * KP + 4; }   // basis row pitch (floats)
__host__ __device__ __forceinline__ size_t vt_smem(int KP, int NF)
{
    return ((size_t)2 * VT_V * vt_row(KP) + (size_t)NF * KP + (size_t)NF * VT_FR) * sizeof(float);
}

// Frames of a tile: what shared memory holds beside two tiles of basis rows, 96 up to 168 expressions,
// 64 up to 192, 32 up to 224, 16 up to 240; 0 when the rows leave no room. (Counts at which the warps'
// coefficients take no more than their frames': 2, 4, 8 or 12 per warp.)
inline int vt_frames(int KP)
{
    for (int nf : {VT_F, 64, 32, 16})
        if (vt_smem(KP, nf) <= VT_SMEM) return nf;
    return 0;
}

// A thread's coefficients at one k as NP frame pairs (16-byte loads, a last 8-byte one).
template <int NP>
__device__ __forceinline__ void vt_load_x(float2 (&xv)[NP], const float *p)
{
#pragma unroll
    for (int q = 0; q + 1 < NP; q += 2) {
        const float4 x = *reinterpret_cast<const float4 *>(p + 2 * q);
        xv[q] = make_float2(x.x, x.y);
        xv[q + 1] = make_float2(x.z, x.w);
    }
    if (NP & 1) xv[NP - 1] = *reinterpret_cast<const float2 *>(p + 2 * (NP - 1));
}

// Floats of a warp's coefficients at one k: its NP pairs, rounded up to 16 bytes (a single pair is read
// in 8-byte loads).
__device__ __forceinline__ constexpr int vt_pitch(int NP) { return NP == 1 ? 2 : 4 * ((NP + 1) / 2); }

struct VtShared {
    int any, issued;
    volatile int abort;
    int render[VT_F], frame[VT_F];
    __align__(8) uint64_t full[2], empty[2];
};

// A computing warp's tiles: vertex v of the lane, 2 NP frames.
template <int NP>
__device__ __forceinline__ void vt_tiles(const DModel &m, const DBatch &b, VtShared &sh, const float *Eb, const float *Xs,
                                         const float *Fs, int gy, int groups, int ntiles)
{
    constexpr int XP = VT_WARPS * vt_pitch(NP);
    const int KP = m.KP, K = m.K, ER = vt_row(KP);
    const int vl = threadIdx.x;
    const float *xr = Xs + threadIdx.y * vt_pitch(NP);    // this warp's frames at k: xr[k * XP + q]
    const int fl0 = threadIdx.y * 2 * NP;
    bool busy = false;
    for (int q = 0; q < 2 * NP; ++q) busy = busy || sh.render[fl0 + q];
    for (int j = 0;; ++j) {
        const int t = gy + j * groups;
        if (t >= ntiles) break;
        const int buf = j & 1;
        const int v = t * VT_V + vl;
        // the epilogue's per-vertex inputs, loaded before the wait
        float mx = 0.0f, my = 0.0f, mz = 0.0f, tx = 0.0f;
        if (busy && v < m.V) { mx = m.mean[v]; my = m.mean[m.V + v]; mz = m.mean[2 * m.V + v]; tx = m.tex[v]; }
        const bool w = mbar_wait(smem_addr(&sh.full[buf]), (uint32_t)((j >> 1) & 1));
        if (!__all_sync(0xffffffffu, w)) {
            if (threadIdx.x == 0) { sh.abort = 1; atomicOr(b.err, 2); }
            break;
        }
        // Sequential fused multiply-add over k for every output (the order the oracle uses),
        // two frames per instruction: each half of fma.rn.f32x2 is an IEEE fused
        // multiply-add, so every chain rounds exactly as fmaf would.
        float2 acc[NP][3];
#pragma unroll
        for (int q = 0; q < NP; ++q) acc[q][0] = acc[q][1] = acc[q][2] = make_float2(0.0f, 0.0f);
        if (busy) {
            const float *er = Eb + (size_t)(buf * VT_V + vl) * ER;
            int k = 0;
#pragma unroll 1
            for (; k + 4 <= K; k += 4) {
                const float4 ex = *reinterpret_cast<const float4 *>(er + k);
                const float4 ey = *reinterpret_cast<const float4 *>(er + KP + k);
                const float4 ez = *reinterpret_cast<const float4 *>(er + 2 * KP + k);
                const float exv[4] = {ex.x, ex.y, ex.z, ex.w}, eyv[4] = {ey.x, ey.y, ey.z, ey.w};
                const float ezv[4] = {ez.x, ez.y, ez.z, ez.w};
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    float2 xv[NP];
                    vt_load_x<NP>(xv, xr + (k + jj) * XP);
                    const float2 e0 = make_float2(exv[jj], exv[jj]), e1 = make_float2(eyv[jj], eyv[jj]);
                    const float2 e2 = make_float2(ezv[jj], ezv[jj]);
#pragma unroll
                    for (int q = 0; q < NP; ++q) {
                        acc[q][0] = ffma2(e0, xv[q], acc[q][0]);
                        acc[q][1] = ffma2(e1, xv[q], acc[q][1]);
                        acc[q][2] = ffma2(e2, xv[q], acc[q][2]);
                    }
                }
            }
#pragma unroll 1
            for (; k < K; ++k) {
                const float ex = er[k], ey = er[KP + k], ez = er[2 * KP + k];
                float2 xv[NP];
                vt_load_x<NP>(xv, xr + k * XP);
#pragma unroll
                for (int q = 0; q < NP; ++q) {
                    acc[q][0] = ffma2(make_float2(ex, ex), xv[q], acc[q][0]);
                    acc[q][1] = ffma2(make_float2(ey, ey), xv[q], acc[q][1]);
                    acc[q][2] = ffma2(make_float2(ez, ez), xv[q], acc[q][2]);
                }
            }
        }
        __syncwarp();                          // this warp is done with the buffer
        if (threadIdx.x == 0) mbar_arrive(smem_addr(&sh.empty[buf]));
        if (busy && v < m.V) {
#pragma unroll
            for (int q = 0; q < 2 * NP; ++q) {
                if (!sh.render[fl0 + q]) continue;
                const int f = sh.frame[fl0 + q];
                const float *R = Fs + (fl0 + q) * VT_FR, *tau = R + 9, *cam = R + 12;
                const float2 *a = acc[q >> 1];
                const float X0 = mx + ((q & 1) ? a[0].y : a[0].x);
                const float Y0 = my + ((q & 1) ? a[1].y : a[1].x);
                const float Z0 = mz + ((q & 1) ? a[2].y : a[2].x);
                const float X3 = ((R[0] * X0 + R[3] * Y0) + R[6] * Z0) + tau[0];
                const float Y3 = ((R[1] * X0 + R[4] * Y0) + R[7] * Z0) + tau[1];
                const float Z3 = ((R[2] * X0 + R[5] * Y0) + R[8] * Z0) + tau[2];
                b.geo[(size_t)f * m.V + v] = make_float4(X0, Y0, Z0, tx);
                b.proj[(size_t)f * m.V + v] = make_float4((cam[0] * X3) / Z3 + cam[2], (cam[1] * Y3) / Z3 + cam[3], Z3, 0.0f);
            }
        }
    }
}

// The round's frames are dealt evenly to tiles of at most nf (vt_frames), a tile's frames to the warps,
// 2 NP each.
__global__ void __launch_bounds__(VT_THREADS, VT_BLOCKS_PER_SM) k_vertex(DModel m, DBatch b, int nf)
{
    extern __shared__ __align__(16) float vsm[];
    const int KP = m.KP, K = m.K, ER = vt_row(KP);
    float *Eb = vsm;                           // [2][VT_V][ER]: basis rows of two tiles
    float *Fs = Eb + 2 * VT_V * ER;            // [nf][VT_FR]
    float *Xs = Fs + nf * VT_FR;               // [K][VT_WARPS][pitch]: coefficients, the frames innermost
    __shared__ VtShared sh;
    const int ntiles = (m.V + VT_V - 1) / VT_V;
    const int rc = b.rcount[0];
    const int ftiles = (rc + nf - 1) / nf;
    if (ftiles == 0) return;
    const int groups = max(1, min(ntiles, (int)gridDim.x / ftiles));
    if ((int)blockIdx.x >= ftiles * groups) return;
    const int gy = blockIdx.x / ftiles;        // vertex-tile stripe
    const int tf = (rc + ftiles - 1) / ftiles;                        // frames of a tile
    const int np = (tf + 2 * VT_WARPS - 1) / (2 * VT_WARPS);          // frame pairs of a warp
    const int f0 = (blockIdx.x - gy * ftiles) * tf;
    const int tid = threadIdx.y * 32 + threadIdx.x;
    const bool producer = threadIdx.y == VT_WARPS;
    if (tid == 0) { sh.any = 0; sh.abort = 0; sh.issued = 0; }
    __syncthreads();
    if (tid < VT_F) {
        const int ai = f0 + tid;
        const int f = tid < tf && ai < rc ? b.rlist[ai] : -1;
        const int r = f >= 0 && b.ctl[f].render;
        sh.frame[tid] = f;
        sh.render[tid] = r;
        if (r) {
            sh.any = 1;
            if (gy == 0) prof_count(b, KID_VERTEX);
        }
    }
    if (tid == 0) {
        mbar_init(smem_addr(&sh.full[0]), 1);
        mbar_init(smem_addr(&sh.full[1]), 1);
        mbar_init(smem_addr(&sh.empty[0]), VT_WARPS);
        mbar_init(smem_addr(&sh.empty[1]), VT_WARPS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (!sh.any) return;
    const int rowbytes = 3 * KP * (int)sizeof(float);
    const uint32_t eb_addr = smem_addr(Eb);
    if (!producer) {
        // lane = frame, four coefficients at a time: conflict-free stores
        const int wp = vt_pitch(np), xp = VT_WARPS * wp;
        const int fg = (tf + 31) / 32, kq = (K + 3) / 4;
        for (int i = threadIdx.y; i < fg * kq; i += VT_WARPS) {
            const int g = i / kq, k = 4 * (i - g * kq), fl = g * 32 + threadIdx.x;
            if (fl >= 2 * VT_WARPS * np) continue;
            const int f = fl < tf ? sh.frame[fl] : -1;
            float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (f >= 0) x = *reinterpret_cast<const float4 *>(b.xe + (size_t)f * m.KTP + k);
            const int w = fl / (2 * np);
            float *o = Xs + k * xp + w * wp + (fl - w * 2 * np);
            o[0] = x.x;
            o[xp] = x.y;
            o[2 * xp] = x.z;
            o[3 * xp] = x.w;
        }
        for (int i = tid; i < tf * VT_FR; i += VT_WARPS * 32) {
            const int fl = i / VT_FR, e = i % VT_FR, f = sh.frame[fl];
            float v = 0.0f;
            if (f >= 0) v = e < 9 ? b.R[f * 9 + e] : e < 12 ? b.xe[(size_t)f * m.KTP + K + (e - 9)] : b.cam[f * 4 + (e - 12)];
            Fs[i] = v;
        }
    } else if (threadIdx.x == 0) {
        // the first two tiles stream in while the coefficients are staged
        for (int j = 0; j < 2; ++j) {
            const int t = gy + j * groups;
            if (t >= ntiles) break;
            const int nv = min(VT_V, m.V - t * VT_V);
            const uint32_t bar = smem_addr(&sh.full[j]);
            mbar_expect_tx(bar, (uint32_t)(nv * rowbytes));
            for (int r = 0; r < nv; ++r)
                bulk_g2s(eb_addr + (uint32_t)((j * VT_V + r) * ER) * 4u, m.E + (size_t)(t * VT_V + r) * 3 * KP,
                         (uint32_t)rowbytes, bar);
        }
    }
    __syncthreads();                           // coefficients staged
    if (producer) {
        if (threadIdx.x == 0) {
            // tile j into buffer j & 1 once the computing warps have released tile j - 2
            int j = 2;
            for (;; ++j) {
                const int t = gy + j * groups;
                if (t >= ntiles || sh.abort) break;
                const int buf = j & 1;
                if (!mbar_wait(smem_addr(&sh.empty[buf]), (uint32_t)(((j - 2) >> 1) & 1))) {
                    sh.abort = 1;
                    atomicOr(b.err, 2);
                    break;
                }
                const int nv = min(VT_V, m.V - t * VT_V);
                const uint32_t bar = smem_addr(&sh.full[buf]);
                mbar_expect_tx(bar, (uint32_t)(nv * rowbytes));
                for (int r = 0; r < nv; ++r)
                    bulk_g2s(eb_addr + (uint32_t)((buf * VT_V + r) * ER) * 4u, m.E + (size_t)(t * VT_V + r) * 3 * KP,
                             (uint32_t)rowbytes, bar);
            }
            sh.issued = min(j, (ntiles - gy + groups - 1) / groups);
        }
    } else {
        switch (np) {
        case 1: vt_tiles<1>(m, b, sh, Eb, Xs, Fs, gy, groups, ntiles); break;
        case 2: vt_tiles<2>(m, b, sh, Eb, Xs, Fs, gy, groups, ntiles); break;
        case 3: vt_tiles<3>(m, b, sh, Eb, Xs, Fs, gy, groups, ntiles); break;
        case 4: vt_tiles<4>(m, b, sh, Eb, Xs, Fs, gy, groups, ntiles); break;
        case 5: vt_tiles<5>(m, b, sh, Eb, Xs, Fs, gy, groups, ntiles); break;
        default: vt_tiles<6>(m, b, sh, Eb, Xs, Fs, gy, groups, ntiles); break;
        }
    }
    __syncthreads();
    if (sh.abort && tid == VT_WARPS * 32) {
        // copies of the last two issued tiles may still be in flight: wait for them (bounded)
        // before the block's shared memory is released
        for (int j = max(0, sh.issued - 2); j < sh.issued; ++j)
            mbar_wait(smem_addr(&sh.full[j & 1]), (uint32_t)((j >> 1) & 1));
    }
}

// ------------------------------------------------------------------------------------------
// Barrier objective of a state (logbarrier_initializer.cu:1921-2093 with compute_Gs :456-520):
// expression bounds, then the four landmark box constraints. Landmark 3D points are the
// vertex-stage object coordinates at the landmark vertices (same formula as the reference's
// p0L + EL*eps). The -log terms are FP64 logarithms rounded to FP32, summed in FP64: strides of the
// block, then a tree over the lanes, then the warps. The oracle adds them one after the other; the two
// sums agree to FP64 rounding, and the objective is their FP32 rounding.

__device__ __forceinline__ void landmark_G(const DModel &m, const DBatch &b, int f, const float *x,
                                           const float *R, int i, const float *p, float G[4])
{
    const float *tau = x + m.K;
    const float *cam = b.cam + f * 4;
    const float fs = b.face_size[f];
    const float *bnd = b.bounds + (size_t)f * 4 * NL;
    const float xl = b.xl[f * NL + i], yl = b.yl[f * NL + i];
    const float p0 = p[0], p1 = p[1], p2 = p[2];
    const float r1p = (R[0] * p0 + R[3] * p1) + R[6] * p2;
    const float r2p = (R[1] * p0 + R[4] * p1) + R[7] * p2;
    const float r3p = (R[2] * p0 + R[5] * p1) + R[8] * p2;
    const float xproj = cam[0] * ((r1p + tau[0]) / (r3p + tau[2])) + cam[2];
    const float yproj = cam[1] * ((r2p + tau[1]) / (r3p + tau[2])) + cam[3];
    G[0] = 0.0f - ((xl + bnd[0 * NL + i] * fs) - xproj);
    G[1] = 0.0f - ((yl + bnd[1 * NL + i] * fs) - yproj);
    G[2] = 0.0f - ((xproj - bnd[2 * NL + i] * fs) - xl);
    G[3] = 0.0f - ((yproj - bnd[3 * NL + i] * fs) - yl);
}

// The evaluation point of every active frame, one block per frame: the state x or x_ls, R(u) and
// dR/du; with check, the face-size check (renderer.cu:838-857), the barrier objective and the
// pre-render decisions of a trial (model_fitter.cu:237-300): tau_z, face size, NaN barrier, then
// -g.d < 3e-4. These need only the 51 landmark vertices, so they run before the vertex stage: the
// landmark object points and projections are formed here with the vertex stage's arithmetic (the
// same values bit for bit), and a trial rejected here costs no vertex stage and no raster. Frames
// that go on are appended to the round's list.
// Latency-bound (every frame has its block): a thread per landmark coordinate runs one fused
// multiply-add chain with its basis row loaded ahead, another warp forms the rotation meanwhile,
// the logarithms spread over the block. As a warp per frame with the landmark rows staged per
// block, the rotation and the list in launches of their own, a round spent 31 us here;
// 8 us in this form (77 frames).
constexpr int PT_THREADS = 192;
constexpr int PT_E4 = 10;                        // 16-byte loads of a basis row in flight

__host__ __device__ __forceinline__ size_t point_smem(int K, int KTP)
{
    return ((size_t)KTP + 4 + 2 * K + 4 * NL) * sizeof(float);   // the state (padded), the barrier terms
}

__global__ void __launch_bounds__(PT_THREADS) k_point(DModel m, DBatch b, Cfg c, int stage, int check)
{
    extern __shared__ __align__(16) float psm[];
    __shared__ float s_R[9], s_dR[27], s_lm[NL][3], s_xp[NL], s_yp[NL], s_t;
    __shared__ double s_ob[PT_THREADS / 32];
    __shared__ int s_go;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (blockIdx.x == 0 && tid == 0) b.rcount[1] = 0;     // the last round's normal equations are done
    if ((int)blockIdx.x >= active_n(b)) return;
    const int f = b.act[blockIdx.x];
    FrameCtl &ctl = b.ctl[f];
    const bool active = ctl.active != 0, full = ctl.mode == M_FULL;
    __syncthreads();                             // (every thread has read the flags)
    if (tid == 0) {
        ctl.need_jac = 0;
        if (!active) ctl.render = 0;
    }
    if (!active) return;
    const int K = m.K, KP = m.KP, KT = m.KT;
    float *xs = psm, *term = psm + m.KTP + 4;
    const float *src = (full || stage == ST_LAMBDA ? b.x : b.x_ls) + (size_t)f * m.KTP;
    float *xe = b.xe + (size_t)f * m.KTP;
    for (int a = tid; a < KT; a += PT_THREADS) {
        const float v = src[a];
        xs[a] = v;
        xe[a] = v;
    }
    __syncthreads();
    if (warp == PT_THREADS / 32 - 1) {
        if (lane == 0) rotation(xs + K + 3, s_R, s_dR);
        __syncwarp();
        if (lane < 9) b.R[f * 9 + lane] = s_R[lane];
        if (lane < 27) b.dR[f * 27 + lane] = s_dR[lane];
        if (!check) {
            if (lane == 0) {
                ctl.render = 1;
                b.rlist[atomicAdd(b.rcount, 1)] = f;
            }
            return;
        }
    } else {
        if (!check) return;
        if (tid < 3 * NL) {
            const int li = tid / 3, cc = tid - 3 * li, v = m.lis[li];
            const float4 *e4 = reinterpret_cast<const float4 *>(m.E + ((size_t)v * 3 + cc) * KP);
            float acc = 0.0f;
            for (int k0 = 0; k0 < K; k0 += 4 * PT_E4) {
                float4 e[PT_E4];
#pragma unroll
                for (int u = 0; u < PT_E4; ++u) e[u] = k0 + 4 * u < K ? __ldg(e4 + (k0 >> 2) + u) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                for (int u = 0; u < PT_E4; ++u) {
                    const int k = k0 + 4 * u;
                    if (k < K) acc = fmaf(e[u].x, xs[k], acc);
                    if (k + 1 < K) acc = fmaf(e[u].y, xs[k + 1], acc);
                    if (k + 2 < K) acc = fmaf(e[u].z, xs[k + 2], acc);
                    if (k + 3 < K) acc = fmaf(e[u].w, xs[k + 3], acc);
                }
            }
            s_lm[li][cc] = m.mean[(size_t)cc * m.V + v] + acc;
        }
    }
    // the expression bounds' terms need only the state
    const bool ft = stage == ST_FINETUNE;
    const float *lb = m.eps_b + (ft ? 2 : 0) * K, *ub = m.eps_b + (ft ? 3 : 1) * K;
    __syncthreads();
    const float *tau = xs + K;
    const float *cam = b.cam + f * 4;
    if (tid < NL) {
        const float X0 = s_lm[tid][0], Y0 = s_lm[tid][1], Z0 = s_lm[tid][2];
        const float X3 = ((s_R[0] * X0 + s_R[3] * Y0) + s_R[6] * Z0) + tau[0];
        const float Y3 = ((s_R[1] * X0 + s_R[4] * Y0) + s_R[7] * Z0) + tau[1];
        const float Z3 = ((s_R[2] * X0 + s_R[5] * Y0) + s_R[8] * Z0) + tau[2];
        s_xp[tid] = (cam[0] * X3) / Z3 + cam[2];
        s_yp[tid] = (cam[1] * Y3) / Z3 + cam[3];
        float G[4];
        landmark_G(m, b, f, xs, s_R, tid, s_lm[tid], G);
        for (int s = 0; s < 4; ++s) term[2 * K + s * NL + tid] = G[s];
    } else {
        for (int k = tid - NL; k < K; k += PT_THREADS - NL) {
            const float fub = xs[k] - ub[k];
            const float flb = lb[k] - xs[k];
            term[2 * k] = -flb;
            term[2 * k + 1] = -fub;
        }
    }
    __syncthreads();
    double ob = 0.0;
    for (int q = tid; q < 2 * K + 4 * NL; q += PT_THREADS) ob += (double)(-(float)log((double)term[q]));
    for (int o = 16; o > 0; o >>= 1) ob += __shfl_down_sync(0xffffffffu, ob, o);
    if (lane == 0) s_ob[warp] = ob;
    __syncthreads();
    if (tid == 0) {
        const float d_iod = fabsf(s_xp[9] - s_xp[0]);
        const float d_lem = fabsf(s_yp[0] - s_yp[40]);
        const float d_rem = fabsf(s_yp[9] - s_yp[40]);
        const double lim = (double)c.ref_face_size * 2;
        const int face_ok = !((double)d_iod > lim || (double)d_lem > lim || (double)d_rem > lim);
        ob = 0.0;
        for (int w = 0; w < PT_THREADS / 32; ++w) ob += s_ob[w];
        ctl.face_ok = face_ok;
        ctl.obj_b = (float)ob;
        int go = 1;                              // 0: the trial is rejected; -1: the stage ends
        if (!full) {
            if (!face_ok || isnan(ob)) go = 0;
            else if ((double)(-ctl.l2base) < 0.0003) go = -1;
        }
        ctl.render = go > 0;
        if (go > 0) b.rlist[atomicAdd(b.rcount, 1)] = f;
        if (go < 0) {
            const int maxit = stage == ST_RIGID ? c.max_iters_rigid : c.max_iters_finetune;
            end_shape_stage(c, ctl, stage, ctl.outer < maxit ? ctl.outer + 1 : ctl.outer);
        }
        s_go = go;
    }
    __syncthreads();
    if (s_go == 0) shape_reject(m, b, c, f, stage, &s_t);
}

// ------------------------------------------------------------------------------------------
// Visibility (get_pixels_to_render + keep_only_minZ + remove_if, funcs.cu:900-1029,
// renderer.cu:650-680) in two kernels.
//
// k_raster_depth: every triangle enumerates its <= 4 fragments in bounding-box order, folds a
// 64-bit key [epoch tag | depth bits | triangle id] into the frame's z-buffer with atomicMin
// and appends the fragment to the frame's candidates. Neither depends on the visiting
// order, so triangles are visited in Morton order of their centroids and their corners (vertex
// slots) lie close in memory.
//
// k_raster_resolve, one block per frame: the candidates whose depth equals their pixel's minimum
// survive. Slot order is (row r, then triangle): every survivor sets its bit in one bit set per
// row over the triangles, and its slot is the number of bits before its own. The pixel owner is
// the minimum key (smallest triangle among depth ties). Slot 0 is dropped, as remove_if(is_zero)
// does. The epoch tag makes earlier renders' keys lose to this one's without clearing the
// z-buffer; it is cleared once the tag range is used up.

// True when alpha + beta, formed as fl(fl(na / denom) + fl(nb / denom)), is certainly above
// 1 for na, nb of denom's (nonzero) sign, so the two divisions can be skipped. With u = 2^-24:
// a finite s = fl(na + nb) beyond lim = fl(denom (1 + 16u)) gives (na + nb) / denom > 1 + 13u
// exactly, and the rounded quotients and their rounded sum then still exceed 1. Cases the bound
// cannot settle (and |denom| below 1e-30) return false and take the exact test.
__device__ __forceinline__ bool sum_exceeds_one(float na, float nb, float denom, bool dpos)
{
    constexpr float GROW = 1.0f + 16.0f * 5.9604644775390625e-8f;
    const float s = na + nb, lim = denom * GROW;
    const bool beyond = dpos ? s > lim : s < lim;
    return beyond && fabsf(denom) >= 1e-30f && fabsf(s) <= 3.4028234663852886e38f;
}

// Samples of one triangle with corners b, c, a (rows 0, 1, 2 of the triangle list) in the
// reference's order: x-major over the integer points of the bounding box, at most NTMP.
// emit(r, pix, alpha, beta) receives each, pix wrapped to 16 bits as the reference's
// ushort index is; the count is returned.
template <class Emit>
__device__ __forceinline__ int tri_samples(float bx, float by, float cx, float cy, float ax, float ay,
                                           int x0, int y0, uint32_t &flags, Emit &&emit)
{
    const float xhi = ceilf(fmaxf(fmaxf(bx, cx), ax));
    const float yhi = ceilf(fmaxf(fmaxf(by, cy), ay));
    float xlo_f = floorf(fminf(fminf(bx, cx), ax));
    float ylo_f = floorf(fminf(fminf(by, cy), ay));
    if (!(xlo_f >= 0.0f) || !(ylo_f >= 0.0f) || xhi > 65535.0f || yhi > 65535.0f) {
        flags |= FLAG_OUT_OF_DOMAIN;
        if (!(xhi <= 65535.0f && yhi <= 65535.0f)) return 0;
        xlo_f = xlo_f >= 0.0f ? xlo_f : 0.0f;
        ylo_f = ylo_f >= 0.0f ? ylo_f : 0.0f;
    }
    // A triangle whose box exceeds the whole crop only arises from a vertex near the camera
    // plane; the reference would walk the whole box. It is skipped and flagged instead.
    if ((xhi - xlo_f) * (yhi - ylo_f) > 65536.0f) {
        flags |= FLAG_OUT_OF_DOMAIN;
        return 0;
    }
    // The reference recomputes these per sample point; they do not depend on it.
    const float v0x = bx - ax, v1x = cx - ax;
    const float v0y = by - ay, v1y = cy - ay;
    const float d00 = v0x * v0x + v0y * v0y;
    const float d01 = v0x * v1x + v0y * v1y;
    const float d11 = v1x * v1x + v1y * v1y;
    const float denom = d00 * d11 - d01 * d01;
    // With a zero or NaN denominator no sample can pass (alpha, beta become inf/NaN and
    // alpha + beta <= 1 fails).
    if (!(denom > 0.0f) && !(denom < 0.0f)) return 0;
    const bool dpos = denom > 0.0f;
    int ridx = 0;
    // Boxes of at most 2 x 2 sample points (almost every triangle of a dense face mesh): the
    // same points with the same FP32 operations, evaluated without branches (the candidates'
    // products are formed once and shared, which rounds exactly as per point). Points whose
    // alpha + beta certainly exceeds 1 are dropped before the divisions; the rest take the
    // exact test in x-major order. At most 4 fragments, so the NTMP cap cannot bind.
    if (xhi - xlo_f <= 2.0f && yhi - ylo_f <= 2.0f) {
        const int xi0 = (int)xlo_f, yi0 = (int)ylo_f;
        const float xf1 = xlo_f + 1.0f, yf1 = ylo_f + 1.0f;
        // (the reference stops at the first coordinate outside the box; xf1 < xhi implies
        // xlo_f < xhi, so these select the same points)
        const bool okx[2] = {xlo_f < xhi, xf1 < xhi}, oky[2] = {ylo_f < yhi, yf1 < yhi};
        const float v2x[2] = {xlo_f - ax, xf1 - ax}, v2y[2] = {ylo_f - ay, yf1 - ay};
        float p0x[2], p1x[2], p0y[2], p1y[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            p0x[i] = v0x * v2x[i]; p1x[i] = v1x * v2x[i];
            p0y[i] = v0y * v2y[i]; p1y[i] = v1y * v2y[i];
        }
        float na[4], nb[4];
        uint32_t cand = 0;
#pragma unroll
        for (int ix = 0; ix < 2; ++ix)
#pragma unroll
            for (int iy = 0; iy < 2; ++iy) {
                const int k = 2 * ix + iy;
                const float d20 = p0x[ix] + p0y[iy];
                const float d21 = p1x[ix] + p1y[iy];
                na[k] = d11 * d20 - d01 * d21;
                nb[k] = d00 * d21 - d01 * d20;
                const bool sa = dpos ? na[k] > 0.0f : na[k] < 0.0f;
                const bool sb = dpos ? nb[k] > 0.0f : nb[k] < 0.0f;
                const bool c = okx[ix] && oky[iy] && sa && sb && !sum_exceeds_one(na[k], nb[k], denom, dpos);
                cand |= c ? (1u << k) : 0u;
            }
        while (cand) {
            const int k = __ffs(cand) - 1;
            cand &= cand - 1;
            const float nak = k == 0 ? na[0] : k == 1 ? na[1] : k == 2 ? na[2] : na[3];
            const float nbk = k == 0 ? nb[0] : k == 1 ? nb[1] : k == 2 ? nb[2] : nb[3];
            const float alpha = nak / denom;
            const float beta = nbk / denom;
            if (alpha > 0 && beta > 0 && (alpha + beta <= 1)) {
                const int px = ((yi0 + (k & 1)) - y0) + ((xi0 + (k >> 1)) - x0) * DIM;
                if (px < 0 || px >= NPIX) flags |= FLAG_OUT_OF_DOMAIN;
                emit(ridx, (uint32_t)(uint16_t)px, alpha, beta);
                ridx++;
            }
        }
        return ridx;
    }
    // Loop counters are kept as floats (integers below 2^24 are exact), which is what the
    // reference's ushort counters are converted to in every comparison and subtraction.
    int xi = (int)xlo_f;
    for (float xf = xlo_f; xf < xhi && ridx < NTMP; xf += 1.0f, ++xi) {
        const float v2x = xf - ax;
        int yi = (int)ylo_f;
        for (float yf = ylo_f; yf < yhi && ridx < NTMP; yf += 1.0f, ++yi) {
            const float v2y = yf - ay;
            const float d20 = v0x * v2x + v0y * v2y;
            const float d21 = v1x * v2x + v1y * v2y;
            // alpha = na/denom > 0 and beta = nb/denom > 0 need na, nb to have denom's sign
            // (a quotient of opposite signs, of a zero or of a NaN is not > 0): samples that
            // fail this skip the divisions; the rest take the exact test.
            const float na = d11 * d20 - d01 * d21;
            if (!(dpos ? na > 0.0f : na < 0.0f)) continue;
            const float nb = d00 * d21 - d01 * d20;
            if (!(dpos ? nb > 0.0f : nb < 0.0f)) continue;
            if (sum_exceeds_one(na, nb, denom, dpos)) continue;
            const float alpha = na / denom;
            const float beta = nb / denom;
            if (alpha > 0 && beta > 0 && (alpha + beta <= 1)) {
                const int px = (yi - y0) + (xi - x0) * DIM;
                if (px < 0 || px >= NPIX) flags |= FLAG_OUT_OF_DOMAIN;
                emit(ridx, (uint32_t)(uint16_t)px, alpha, beta);
                ridx++;
            }
        }
    }
    return ridx;
}

// The geometry terms of a fragment's shading: unit normal of its triangle and barycentric
// point p in model coordinates, interpolated albedo t (corners b, c, a as geometry records).
__device__ __forceinline__ void shade_geometry(const float4 &gb, const float4 &gc, const float4 &ga4, float al,
                                               float be, float (&nn)[3], float (&p)[3], float &t)
{
    const float ga = (1 - al) - be;
    const float b0x = gb.x, b0y = gb.y, b0z = gb.z;
    const float c0x = gc.x, c0y = gc.y, c0z = gc.z;
    const float a0x = ga4.x, a0y = ga4.y, a0z = ga4.z;
    const float n_vx = b0x - a0x, n_vy = b0y - a0y, n_vz = b0z - a0z;
    const float n_wx = c0x - a0x, n_wy = c0y - a0y, n_wz = c0z - a0z;
    const float nrx = n_vy * n_wz - n_vz * n_wy;
    const float nry = n_vz * n_wx - n_vx * n_wz;
    const float nrz = n_vx * n_wy - n_vy * n_wx;
    const float normn = sqrtf((nrx * nrx + nry * nry) + nrz * nrz);
    nn[0] = nrx / normn; nn[1] = nry / normn; nn[2] = nrz / normn;
    p[0] = (b0x * al + c0x * be) + a0x * ga;
    p[1] = (b0y * al + c0y * be) + a0y * ga;
    p[2] = (b0z * al + c0z * be) + a0z * ga;
    t = (gb.w * al + gc.w * be) + ga4.w * ga;
}

// The shading inputs of a fragment as records: (unit normal, n . p), and the albedo t.
__device__ __forceinline__ float4 shade_record(const float4 &gb, const float4 &gc, const float4 &ga, float al, float be,
                                               float &t)
{
    float nn[3], p[3];
    shade_geometry(gb, gc, ga, al, be, nn, p, t);
    return make_float4(nn[0], nn[1], nn[2], (nn[0] * p[0] + nn[1] * p[1]) + nn[2] * p[2]);
}

__device__ __forceinline__ unsigned long long zkey(uint32_t tag, float Z, int tri)
{
    return ((unsigned long long)tag << (31 + TRI_BITS)) |
           ((unsigned long long)(__float_as_uint(Z) & 0x7FFFFFFFu) << TRI_BITS) |
           (unsigned long long)(uint32_t)tri;
}

__device__ __forceinline__ bool survives(unsigned long long k, uint32_t tag, uint32_t zbits)
{
    return (uint32_t)(k >> (31 + TRI_BITS)) == tag && (uint32_t)((k >> TRI_BITS) & 0x7FFFFFFFu) == zbits;
}

constexpr int RD_THREADS = 256;             // depth pass: threads per block
constexpr int RD_BLOCKS = 8;                // depth pass: blocks per frame (at least)
constexpr int RD_MAX_BLOCKS = 128;          // depth pass: blocks per frame when few frames render
constexpr int RD_SPREAD = 2400;             // blocks of a launch of few frames: four waves of four per SM
constexpr int RR_THREADS = 1024;            // resolve: one block per frame
constexpr int RR_WARPS = RR_THREADS / 32;
constexpr int RR_U = 4;                     // resolve: candidates per thread in flight together
constexpr int RD_CAND = 640;                // depth pass: candidates a block collects before it appends them

// A fragment of the raster in flight. A raster's working set lies in the frame's chunk partials of the
// normal equations (idle but between the normal equations and their reduction): the candidate of every
// slot, then the candidates, in the room of KC floats per fragment of capacity (104,857 candidates from 23
// expressions on); a frame with more takes the resolve's general path. What an evaluation leaves for
// tdi_batch_read (neighbours, gradients, Jacobian) is not touched.
struct __align__(16) Candidate {
    uint32_t pix_row;                       // pixel | row << 16
    int32_t tri;
    float al, be;
};

struct CandidateSpan {
    Candidate *c;
    float4 *sn;                             // shading inputs: unit normal and n . p
    float *t;                               // and interpolated albedo
    float *z;                               // camera Z of the triangle's first corner
    int cap;
};

constexpr size_t RASTER_WORK = (size_t)NMAX * (CAND_COLS + 1) * sizeof(float);    // bytes per frame (4.1 MB)

__device__ __forceinline__ uint32_t *raster_slots(const DBatch &b, int f)
{
    return reinterpret_cast<uint32_t *>(reinterpret_cast<char *>(b.ne_part) + (size_t)f * RASTER_WORK);   // [NMAX]
}

__device__ __forceinline__ CandidateSpan candidates(const DModel &m, const DBatch &b, int f)
{
    CandidateSpan s;
    const size_t bytes = (size_t)NMAX * m.KC * sizeof(float);
    s.cap = (int)(bytes / (sizeof(Candidate) + sizeof(float4) + 2 * sizeof(float)));
    s.c = reinterpret_cast<Candidate *>(raster_slots(b, f) + NMAX);
    s.sn = reinterpret_cast<float4 *>(s.c + s.cap);
    s.t = reinterpret_cast<float *>(s.sn + s.cap);
    s.z = s.t + s.cap;
    return s;
}

// True when no sample point of the triangle can be a fragment, decided without evaluating one: the
// box has a single sample column (or row), and it lies left of (above) every corner by a gap that
// rounding cannot bridge for a triangle of this shape. (With two columns the second lies inside the
// corners' range.)
// Why no evaluation could accept such a point (u = 2^-24; l0 = |b - a|, l1 = |c - a|, s the sine
// between them, D = (l0 l1 s)^2 the exact denominator; the corner differences carry one rounding
// each): a point outside the range by g in a coordinate in which the triangle is at most 1 wide has
// a barycentric coordinate of at most -e, e = g / 2 (1 - 1e-3). FP32 forms na and nb within
// 13 u l1^2 l0 l2 and 13 u l0^2 l1 l2 and the denominator within 13 u l0^2 l1^2, l2 <= 3.2 the
// distance of the point from a (the triangle is at most 2 wide in the other coordinate). alpha
// (beta) <= -e then gives na (nb) the wrong sign, and alpha + beta >= 1 + e leaves the rounded sum
// above 1, whenever g min(l0, l1) s^3 > 2 x 173 u (1 + 1e-3) = 2.1e-5; the test below asks for
// 4.5e-5 (squared: RC_SHAPE), and for a gap that is large against the rounding of the differences
// (RC_GAP). Any NaN makes the shape test fail and takes the full path, as do boxes outside
// the domain.
constexpr float RC_GAP = 1.0f / 4096.0f;
constexpr float RC_SHAPE = 2.025e-9f;

__device__ __forceinline__ bool no_sample_inside(float bx, float by, float cx, float cy, float ax, float ay)
{
    const float xmax = fmaxf(fmaxf(bx, cx), ax), xmin = fminf(fminf(bx, cx), ax);
    const float ymax = fmaxf(fmaxf(by, cy), ay), ymin = fminf(fminf(by, cy), ay);
    const bool dom = fminf(xmin, ymin) >= 0.0f && fmaxf(xmax, ymax) <= 65535.0f &&
                     fmaxf(xmax - xmin, ymax - ymin) <= 2.0f;
    const float xlo = floorf(xmin), ylo = floorf(ymin);
    const float gx = xmax <= xlo + 1.0f ? xmin - xlo : 0.0f;
    const float gy = ymax <= ylo + 1.0f ? ymin - ylo : 0.0f;
    const float g = fmaxf(gx, gy);
    const float v0x = bx - ax, v1x = cx - ax, v0y = by - ay, v1y = cy - ay;
    const float d00 = v0x * v0x + v0y * v0y, d01 = v0x * v1x + v0y * v1y, d11 = v1x * v1x + v1y * v1y;
    const float q = d00 * d11, denom = q - d01 * d01;
    const bool shape = (denom * denom) * (denom * fminf(d00, d11)) * (g * g) > RC_SHAPE * ((q * q) * q);
    return dom && g > RC_GAP && shape;
}

// Blocks per frame for rc rendering frames of T triangles (a block has at least one per thread), and
// the largest grid that up to `frames` of them can ask for.
__host__ __device__ __forceinline__ int raster_parts(int rc, int T)
{
    const int p = RD_SPREAD / rc, most = T < RD_THREADS * RD_MAX_BLOCKS ? (T + RD_THREADS - 1) / RD_THREADS : RD_MAX_BLOCKS;
    const int q = p < RD_BLOCKS ? RD_BLOCKS : p;
    return q > most ? most : q;
}
inline int raster_grid(int frames)
{
    const int spread = frames * RD_MAX_BLOCKS < RD_SPREAD ? frames * RD_MAX_BLOCKS : RD_SPREAD;
    return frames * RD_BLOCKS > spread ? frames * RD_BLOCKS : spread;
}

// A dense face mesh has about 25 triangles per visible fragment, most of them smaller than a
// pixel, so the pass is bound by the instructions spent on triangles without a sample
// point. Each warp therefore first tests its triangles with no_sample_inside (about 50
// instructions instead of about 230) and queues the others' corners in shared memory (12-15% of the
// 53,490-vertex mesh's); a full warp's worth of queued triangles is then evaluated densely. RD_ILP
// triangles per lane have their gathers in flight together (1,024 frames in one launch: 1 875 us,
// 2 707, 3 671). 64 registers and 47 KB of shared memory are four blocks per SM (at 70 registers, three
// blocks, 795 us); shared memory admits no fifth.
// 1,024 frames of the 53,490-vertex model in one launch: 1,192 us with every sample evaluated in
// place, 671 with the queue, the candidates and their shading inputs included (which the resolve
// formed before). What is left is issue (0.68 per cycle) and the latency of the gathers.
constexpr int RD_WARPS = RD_THREADS / 32;
constexpr int RD_ILP = 3;                   // triangles per lane and step
constexpr int RD_QUEUE = 32 * (RD_ILP + 1); // a warp's queue: what a step adds to a remainder below 32

__global__ void __launch_bounds__(RD_THREADS) k_raster_depth(DModel m, DBatch b)
{
    // the blocks are split between the frames that render: RD_BLOCKS each, or more when few do
    const int rc = render_n(b);
    if (rc == 0) return;
    const int parts = raster_parts(rc, m.T);
    const int fi = blockIdx.x / parts, part = blockIdx.x - fi * parts;
    if (fi >= rc) return;
    const int f = b.rlist[fi];
    const FrameCtl &ctl = b.ctl[f];
    if (part == 0 && threadIdx.x == 0) prof_count(b, KID_RASTER);
    __shared__ float4 s_qa[RD_WARPS][RD_QUEUE];     // bx, by, cx, cy
    __shared__ float4 s_qb[RD_WARPS][RD_QUEUE];     // ax, ay, camera Z of b, place in the Morton order (bits)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float4 *qa = s_qa[warp], *qb = s_qb[warp];
    const uint32_t tag = TAG_MAX - (ctl.epoch + 1);
    const float4 *pj = b.proj + (size_t)f * m.V;
    unsigned long long *zb = b.zbuf + (size_t)f * NPIX;
    const int x0 = b.x0y0[2 * f], y0 = b.x0y0[2 * f + 1];
    const int T = m.T;
    // candidates are collected per block and appended together: one global counter update per
    // block. Their shading inputs are formed then, for every render of this raster: here the corners'
    // geometry lies close together in Morton order and the gathers are spread over all SMs.
    __shared__ Candidate s_cand[RD_CAND];
    __shared__ float s_cz[RD_CAND];
    __shared__ int s_cs[RD_CAND];
    const CandidateSpan cs = candidates(m, b, f);
    const float4 *geo = b.geo + (size_t)f * m.V;
    auto append = [&](int g, const Candidate &cd, float z, int place) {
        if (g >= cs.cap) return;
        const int4 tq = __ldg(m.tlo4 + place);
        float t;
        cs.sn[g] = shade_record(__ldg(geo + tq.x), __ldg(geo + tq.y), __ldg(geo + tq.z), cd.al, cd.be, t);
        cs.t[g] = t;
        cs.c[g] = cd;
        cs.z[g] = z;
    };
    __shared__ int s_nc, s_base;
    if (threadIdx.x == 0) s_nc = 0;
    __syncthreads();
    // each block a contiguous range of the Morton order
    const int per_block = (T + parts - 1) / parts;
    const int s_begin = part * per_block, s_end = min(T, s_begin + per_block);
    uint32_t flags = 0;
    int queued = 0;                                 // entries of the warp's queue
    auto evaluate = [&](int e) {
        const float4 A = qa[e], B = qb[e];
        const int place = __float_as_int(B.w), idx = __ldg(&m.tlo4[place].w);
        const unsigned long long key = zkey(tag, B.z, idx);
        const int nf = tri_samples(A.x, A.y, A.z, A.w, B.x, B.y, x0, y0, flags,
                                   [&](int r, uint32_t px, float al, float be) {
                                       atomicMin(zb + px, key);
                                       const Candidate cd{px | ((uint32_t)r << 16), idx, al, be};
                                       const int k = atomicAdd(&s_nc, 1);
                                       if (k < RD_CAND) {
                                           s_cand[k] = cd;
                                           s_cz[k] = B.z;
                                           s_cs[k] = place;
                                       } else {
                                           append(atomicAdd(b.ccount + f, 1), cd, B.z, place);
                                       }
                                   });
        if (nf && !(B.z > 0.0f)) flags |= FLAG_OUT_OF_DOMAIN;
    };
    for (int base = s_begin + (int)threadIdx.x; base - lane < s_end; base += RD_THREADS * RD_ILP) {
        int4 tq[RD_ILP];
        float4 pb[RD_ILP], pc[RD_ILP], pa[RD_ILP];
#pragma unroll
        for (int h = 0; h < RD_ILP; ++h) tq[h] = __ldg(m.tlo4 + min(base + RD_THREADS * h, T - 1));
#pragma unroll
        for (int h = 0; h < RD_ILP; ++h) {
            pb[h] = __ldg(pj + tq[h].x);
            pc[h] = __ldg(pj + tq[h].y);
            pa[h] = __ldg(pj + tq[h].z);
        }
#pragma unroll
        for (int h = 0; h < RD_ILP; ++h) {
            const bool take = base + RD_THREADS * h < s_end &&
                              !no_sample_inside(pb[h].x, pb[h].y, pc[h].x, pc[h].y, pa[h].x, pa[h].y);
            const unsigned msk = __ballot_sync(0xffffffffu, take);
            if (take) {
                const int e = queued + __popc(msk & ((1u << lane) - 1u));
                qa[e] = make_float4(pb[h].x, pb[h].y, pc[h].x, pc[h].y);
                qb[e] = make_float4(pa[h].x, pa[h].y, pb[h].z, __int_as_float(base + RD_THREADS * h));
            }
            queued += __popc(msk);
        }
        __syncwarp();
        while (queued >= 32) {
            queued -= 32;
            evaluate(queued + lane);
            __syncwarp();
        }
    }
    if (lane < queued) evaluate(lane);
    if (flags) atomicOr(&b.ctl[f].flags, flags);
    __syncthreads();
    const int nc = min(s_nc, RD_CAND);
    if (threadIdx.x == 0 && nc) s_base = atomicAdd(b.ccount + f, nc);
    __syncthreads();
    for (int e = threadIdx.x; e < nc; e += RD_THREADS) append(s_base + e, s_cand[e], s_cz[e], s_cs[e]);
}

// Block-wide exclusive scan of one value per thread (RR_THREADS threads); returns the
// thread's offset and writes the total to *total. Uses s_w[RR_WARPS].
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t *s_w, uint32_t *total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) s_w[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = lane < RR_WARPS ? s_w[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < RR_WARPS) s_w[lane] = wi - w;
        if (lane == 31) s_w[RR_WARPS] = wi;
    }
    __syncthreads();
    const uint32_t off = s_w[warp] + inc - v;
    *total = s_w[RR_WARPS];
    __syncthreads();
    return off;
}

// Words of the resolve's working set: NTMP bit sets over the triangles and as many offsets. In shared
// memory when they fit (two blocks per SM for 106,466 triangles), else in the frame's buffer.
constexpr int RR_SMEM = 224 * 1024;
__host__ __device__ __forceinline__ int resolve_words(int T) { return 2 * NTMP * mask_words(T); }
__host__ __device__ __forceinline__ size_t resolve_smem(int T)
{
    const size_t bytes = (size_t)resolve_words(T) * sizeof(uint32_t);
    return bytes <= RR_SMEM ? bytes : 0;
}

// What bounds it is latency (a candidate's record, then its pixel's key, twice), so RR_U candidates
// per thread are in flight together. Listing the triangles with fragments from a bit mask,
// re-evaluating their samples, staging the survivors and forming their shading inputs here took 40 us
// for 77 frames (319 us for 1,024); most of it was gathering the corners' geometry through one
// SM, which the depth pass's blocks now do with their candidates. 16 us (176) with
// k_raster_slots.
__global__ void __launch_bounds__(RR_THREADS) k_raster_resolve(DModel m, DBatch b)
{
    if ((int)blockIdx.x >= render_n(b)) return;
    const int f = b.rlist[blockIdx.x];
    FrameCtl &ctl = b.ctl[f];
    if (threadIdx.x == 0) prof_count(b, KID_RESOLVE);
    extern __shared__ __align__(16) uint32_t rrs[];
    __shared__ uint32_t s_w[RR_WARPS + 1];
    __shared__ int s_bbox[4];
    const int tid = threadIdx.x, lane = tid & 31;
    const int T = m.T, W = mask_words(T);
    uint32_t *bits = resolve_smem(T) ? rrs : b.tri_work + (size_t)f * resolve_words(T);   // [NTMP][W]
    uint32_t *pre = bits + NTMP * W;                                                       // bits before each word
    const uint32_t epoch = ctl.epoch + 1;
    const uint32_t tag = TAG_MAX - epoch;
    unsigned long long *zb = b.zbuf + (size_t)f * NPIX;
    const float4 *pj = b.proj + (size_t)f * m.V;
    const float4 *geo = b.geo + (size_t)f * m.V;
    const int x0 = b.x0y0[2 * f], y0 = b.x0y0[2 * f + 1];
    const CandidateSpan cs = candidates(m, b, f);
    const int nc = b.ccount[f];
    const bool listed = nc <= cs.cap;
    if (tid == 0) {
        s_bbox[0] = s_bbox[2] = 1 << 30;
        s_bbox[1] = s_bbox[3] = -1;
    }
    for (int w = tid; w < NTMP * W; w += RR_THREADS) bits[w] = 0u;
    __syncthreads();
    // visit(c, z, key, i): every candidate with its pixel's key and its place in the list
    auto for_candidates = [&](auto &&visit) {
        if (listed) {
            for (int i0 = tid; i0 < nc; i0 += RR_THREADS * RR_U) {
                Candidate cd[RR_U];
                float z[RR_U];
                unsigned long long key[RR_U];
#pragma unroll
                for (int u = 0; u < RR_U; ++u) {
                    const int i = i0 + u * RR_THREADS;
                    if (i < nc) { cd[u] = cs.c[i]; z[u] = cs.z[i]; }
                }
#pragma unroll
                for (int u = 0; u < RR_U; ++u)
                    if (i0 + u * RR_THREADS < nc) key[u] = __ldcg(zb + (cd[u].pix_row & 0xFFFFu));
#pragma unroll
                for (int u = 0; u < RR_U; ++u)
                    if (i0 + u * RR_THREADS < nc) visit(cd[u], z[u], key[u], i0 + u * RR_THREADS);
            }
        } else {
            // more candidates than the buffer holds: every triangle's samples again
            for (int idx = tid; idx < T; idx += RR_THREADS) {
                const int4 tc = __ldg(m.tl4 + idx);
                const float4 pb = __ldg(pj + tc.x), pc = __ldg(pj + tc.y), pa = __ldg(pj + tc.z);
                uint32_t fl2 = 0;
                tri_samples(pb.x, pb.y, pc.x, pc.y, pa.x, pa.y, x0, y0, fl2, [&](int r, uint32_t px, float al, float be) {
                    visit(Candidate{px | ((uint32_t)r << 16), idx, al, be}, pb.z, __ldcg(zb + px), -1);
                });
            }
        }
    };
    auto survivor = [&](const Candidate &c, float z, unsigned long long key) -> bool {
        return survives(key, tag, __float_as_uint(z) & 0x7FFFFFFFu) && !(c.tri == 0 && (c.pix_row >> 16) == 0);
    };
    int bx0 = 1 << 30, bx1 = -1, by0 = 1 << 30, by1 = -1;
    for_candidates([&](const Candidate &c, float z, unsigned long long key, int) {
        if (!survivor(c, z, key)) return;
        atomicOr(bits + (c.pix_row >> 16) * W + (c.tri >> 5), 1u << (c.tri & 31));
        const int px = (int)((c.pix_row >> 8) & 255u), py = (int)(c.pix_row & 255u);
        bx0 = min(bx0, px); bx1 = max(bx1, px);
        by0 = min(by0, py); by1 = max(by1, py);
    });
    bx0 = __reduce_min_sync(0xffffffffu, bx0); bx1 = __reduce_max_sync(0xffffffffu, bx1);
    by0 = __reduce_min_sync(0xffffffffu, by0); by1 = __reduce_max_sync(0xffffffffu, by1);
    if (lane == 0 && bx1 >= 0) {
        atomicMin(&s_bbox[0], bx0); atomicMax(&s_bbox[1], bx1);
        atomicMin(&s_bbox[2], by0); atomicMax(&s_bbox[3], by1);
    }
    __syncthreads();
    // bits before every word, in slot order (row by row): each thread a contiguous run of words
    const int wpt = (NTMP * W + RR_THREADS - 1) / RR_THREADS;
    const int w_begin = min(NTMP * W, tid * wpt), w_end = min(NTMP * W, w_begin + wpt);
    uint32_t nz = 0;
    for (int w = w_begin; w < w_end; ++w) nz += __popc(bits[w]);
    uint32_t total;
    uint32_t run = block_scan(nz, s_w, &total);
    for (int w = w_begin; w < w_end; ++w) {
        pre[w] = run;
        run += __popc(bits[w]);
    }
    __syncthreads();
    uint32_t fl = 0;
    if (total > (uint32_t)NMAX) fl |= FLAG_OVERFLOW;
    if (total < 1000u || total > 52000u) fl |= FLAG_RENDER_SKIPPED;
    if (total > 25600u) fl |= FLAG_OUT_OF_DOMAIN;
    const bool refused = (fl & (FLAG_RENDER_SKIPPED | FLAG_OVERFLOW)) != 0;
    // Every survivor's slot: the candidate of each slot for k_raster_slots, or (when the candidates
    // did not fit) the fragment itself with its shading inputs.
    Fragment *out = b.frag + (size_t)f * NMAX;
    float4 *shc = b.shc + (size_t)f * NMAX;
    float *sht = b.sht + (size_t)f * NMAX;
    uint32_t *slot = raster_slots(b, f);
    for_candidates([&](const Candidate &c, float z, unsigned long long key, int i) {
        if (!survivor(c, z, key)) return;
        const int w = (int)(c.pix_row >> 16) * W + (c.tri >> 5);
        const uint32_t p = pre[w] + __popc(bits[w] & ((1u << (c.tri & 31)) - 1u));
        if (p >= (uint32_t)NMAX) return;
        const uint32_t owner = key == zkey(tag, z, c.tri) ? 0x80000000u : 0u;
        if (i >= 0) {
            slot[p] = (uint32_t)i | owner;
            return;
        }
        const Fragment fr{(c.pix_row & 0xFFFFu) | owner, c.tri, c.al, c.be};
        const int4 tq = __ldg(m.tl4 + c.tri);
        float t;
        out[p] = fr;
        shc[p] = shade_record(geo[tq.x], geo[tq.y], geo[tq.z], c.al, c.be, t);
        sht[p] = t;
    });
    if (epoch == TAG_MAX) {
        // tag range used up: the next raster starts from a cleared z-buffer
        __syncthreads();
        for (int p = tid; p < NPIX; p += RR_THREADS) zb[p] = ~0ull;
    }
    if (tid == 0) {
        ctl.N = (int)min(total, (uint32_t)NMAX);
        ctl.epoch = epoch == TAG_MAX ? 0u : epoch;
        ctl.flags |= fl;
        ctl.renders += 1;
        for (int q = 0; q < 4; ++q) ctl.bbox[q] = s_bbox[q];
        if (s_bbox[1] >= 0 && (s_bbox[0] < 1 || s_bbox[1] > DIM - 2 || s_bbox[2] < 1 || s_bbox[3] > DIM - 2))
            ctl.flags |= FLAG_OUT_OF_DOMAIN;
        if (refused) ctl.render = 0;
        ctl.slots = listed;
        b.ccount[f] = 0;                     // (every thread has read it: barriers above)
    }
}

// The fragments of a raster in slot order with their shading inputs for its renders (unit normal and
// n . p in shc, interpolated albedo in sht, so that the renders shade from coalesced records;
// R, tau and the light enter per render). Slot order follows the triangle numbering, which has
// nothing to do with the order in which candidates were found: three scattered records per
// fragment, which took one SM 17 us per frame inside the resolve and here are spread over RS_PARTS
// blocks per frame.
constexpr int RS_THREADS = 256, RS_PARTS = 16;

__global__ void __launch_bounds__(RS_THREADS) k_raster_slots(DModel m, DBatch b)
{
    const int rc = render_n(b);
    for (int it = blockIdx.x; it < rc * RS_PARTS; it += gridDim.x) {
        const int f = b.rlist[it / RS_PARTS];
        const FrameCtl &ctl = b.ctl[f];
        if (!ctl.slots) continue;
        const int N = ctl.N;
        const CandidateSpan cs = candidates(m, b, f);
        const uint32_t *slot = raster_slots(b, f);
        for (int p = (it % RS_PARTS) * RS_THREADS + threadIdx.x; p < N; p += RS_PARTS * RS_THREADS) {
            const uint32_t s = slot[p];
            const int i = (int)(s & 0x7FFFFFFFu);
            const Candidate c = cs.c[i];
            const float4 sn = cs.sn[i];
            const float t = cs.t[i];
            b.frag[(size_t)f * NMAX + p] = Fragment{(c.pix_row & 0xFFFFu) | (s & 0x80000000u), c.tri, c.al, c.be};
            b.shc[(size_t)f * NMAX + p] = sn;
            b.sht[(size_t)f * NMAX + p] = t;
        }
    }
}

// ------------------------------------------------------------------------------------------
// Render of one frame from its fragments, one block per frame: shading
// (fill_diffuse_component_and_populate_texture_and_shape, newfuncs.cu:18-167), owners
// painted into a zeroed image (fill_tex_im1, funcs.cu:800-817), the 15-tap separable blur
// (newfuncs.cu:539-715) over the fragment box plus its 8-pixel margin (the image is zero
// outside that box, so the result equals the full-image blur there), then the
// normalised gradients of render and target at every fragment (fill_grads, funcs.cu:842-897)
// and the correlation sum.

__device__ __forceinline__ void camera_coords(const float *R, const float *tau, float X0, float Y0,
                                              float Z0, float &X, float &Y, float &Z)
{
    X = ((R[0] * X0 + R[3] * Y0) + R[6] * Z0) + tau[0];
    Y = ((R[1] * X0 + R[4] * Y0) + R[7] * Z0) + tau[1];
    Z = ((R[2] * X0 + R[5] * Y0) + R[8] * Z0) + tau[2];
}

// Normalised central-difference gradient of one pixel from its four neighbours as
// fill_grads forms them (index 0 past the crop border): r, l = x + 1, x - 1; d, u = y + 1, y - 1.
__device__ __forceinline__ void grad_of(float r, float l, float d, float u, float &gx, float &gy,
                                        float &h, float &gxn, float &gyn)
{
    const float a = 0.5f * (r - l);
    const float bb = 0.5f * (d - u);
    const float hh = 1e-16f + sqrtf((4 * a) * a + (4 * bb) * bb);
    gx = a; gy = bb; h = hh;
    gxn = (2.0f * a) / hh;
    gyn = (2.0f * bb) / hh;
}

__device__ __forceinline__ void neighbour_pixels(int p, int &kr, int &kl, int &kd, int &ku)
{
    const int y = p & 255, x = p >> 8;
    kr = (x < DIM - 1) ? (x + 1) * DIM + y : 0;
    kl = (x > 0) ? (x - 1) * DIM + y : 0;
    ku = (y > 0) ? x * DIM + y - 1 : 0;
    kd = (y < DIM - 1) ? x * DIM + y + 1 : 0;
}

// Region of the render: the fragment box + 8 px, or the whole crop when the fragments touch
// its border (a border pixel's neighbour is pixel 0). Blur taps are summed in ascending
// offset order with zeros outside the region (rows along y, then columns along x).
// The region buffers carry zero lines on the blurred side, so the taps need no bounds test:
// A[xl][RPAD + yl] (pitch pb + 2 RPAD) holds the shaded image and later the blurred one,
// B[KRAD + xl][yl] (pitch pb, rh rounded up to even) the row pass. They live in shared memory
// when they fit, else in the frame's global buffer.
// Each blur thread forms a run of outputs along the taps' direction from a sliding window (a
// value is read (RUN + 14) / RUN times instead of 15) on two lines at once, with packed FP32
// products and sums (each half rounds as the scalar operation does). Runs of 9 along y put a
// warp's lanes on distinct banks; the last run of a line is moved back to end at the line's end
// (its first outputs are formed twice, with the same values).

constexpr int LIGHT_THREADS = 1024;               // the light fit's renders
constexpr int RENDER_SMEM_FLOATS = 27 * 1024;     // padded region buffers (108 KB)
constexpr int RENDER_GU = 4;                      // fragments in flight in the gradient pass
constexpr int RENDER_SU = 4;                      // and in the shading
constexpr int RPAD = 8;                           // zero columns left and right of A's lines (KRAD used)
constexpr int RUN_Y = 9, RUN_X = 8;               // outputs per thread and line of the row and column pass
constexpr int RIMG = 2 * DIM * (DIM + 2 * RPAD);  // per-frame floats of the global fallback

struct Region {
    int rx0, ry0, rw, rh, pb, ph;
    float *A, *B;
    __device__ __forceinline__ int at(int p) const { return ((p >> 8) - rx0) * ph + RPAD + ((p & 255) - ry0); }
};

// The frame's region; its buffers at smem when they fit, else in the frame's global buffer.
__device__ __forceinline__ Region make_region(const FrameCtl &ctl, float *smem, float *global)
{
    const bool border = ctl.bbox[0] < 1 || ctl.bbox[1] > DIM - 2 || ctl.bbox[2] < 1 || ctl.bbox[3] > DIM - 2;
    Region r;
    r.rx0 = border ? 0 : max(0, ctl.bbox[0] - 8);
    r.ry0 = border ? 0 : max(0, ctl.bbox[2] - 8);
    r.rw = (border ? DIM - 1 : min(DIM - 1, ctl.bbox[1] + 8)) - r.rx0 + 1;
    r.rh = (border ? DIM - 1 : min(DIM - 1, ctl.bbox[3] + 8)) - r.ry0 + 1;
    r.pb = (r.rh + 1) & ~1;
    r.ph = r.pb + 2 * RPAD;
    // (an odd region's last row pair reads one line past A: B's first)
    r.A = r.rw * r.ph + (r.rw + 2 * KRAD) * r.pb <= RENDER_SMEM_FLOATS ? smem : global;
    r.B = r.A + r.rw * r.ph;
    return r;
}

// A zeroed; with pads, B's zero lines too (they stay zero).
template <int NT>
__device__ __forceinline__ void region_clear(const Region &r, bool pads)
{
    float2 *A = reinterpret_cast<float2 *>(r.A);
    for (int i = threadIdx.x; i < r.rw * (r.ph >> 1); i += NT) A[i] = make_float2(0.0f, 0.0f);
    if (pads)
        for (int i = threadIdx.x; i < KRAD * r.pb; i += NT) {
            r.B[i] = 0.0f;
            r.B[(KRAD + r.rw) * r.pb + i] = 0.0f;
        }
}

// Row pass A -> B, column pass B -> A (the shaded image in A, then the blurred one).
template <int NT>
__device__ __forceinline__ void region_blur(const Region &r, const Cfg &c)
{
    const int tid = threadIdx.x;
    const float2 one = packed_one(c.normal_eq & 2);      // (normal_eq is 0 or 1)
    float2 tap[NTAPS];                                   // tap[j]: the weight of offset j - KRAD, in both halves
#pragma unroll
    for (int j = 0; j < NTAPS; ++j) tap[j] = make_float2(c.taps[2 * KRAD - j], c.taps[2 * KRAD - j]);
    {
        const int nrun = (r.rh + RUN_Y - 1) / RUN_Y, npair = (r.rw + 1) >> 1;
        for (int i = tid; i < npair * nrun; i += NT) {
            const int xl = i / nrun, y0 = min((i - xl * nrun) * RUN_Y, r.rh - RUN_Y);
            const float *a0 = r.A + 2 * xl * r.ph + RPAD - KRAD + y0, *a1 = a0 + r.ph;   // a0[t] = A(2 xl, y0 - KRAD + t)
            float2 s[RUN_Y];
#pragma unroll
            for (int o = 0; o < RUN_Y; ++o) s[o] = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int t = 0; t < RUN_Y + 2 * KRAD; ++t) {
                const float2 v = make_float2(a0[t], a1[t]);
#pragma unroll
                for (int o = 0; o < RUN_Y; ++o)
                    if (t >= o && t - o <= 2 * KRAD) s[o] = ffma2(fmul2(tap[t - o], v), one, s[o]);
            }
            float *q = r.B + (KRAD + 2 * xl) * r.pb + y0;
#pragma unroll
            for (int o = 0; o < RUN_Y; ++o) q[o] = s[o].x;
            if (2 * xl + 1 < r.rw) {
#pragma unroll
                for (int o = 0; o < RUN_Y; ++o) q[r.pb + o] = s[o].y;
            }
        }
    }
    __syncthreads();
    {
        const int nrun = (r.rw + RUN_X - 1) / RUN_X, npair = r.pb >> 1;
        for (int i = tid; i < npair * nrun; i += NT) {
            const int g = i / npair, yl = 2 * (i - g * npair), x0 = min(g * RUN_X, r.rw - RUN_X);
            const float *bp = r.B + x0 * r.pb + yl;                    // bp[t pb] = B(x0 - KRAD + t, yl)
            float2 s[RUN_X];
#pragma unroll
            for (int o = 0; o < RUN_X; ++o) s[o] = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int t = 0; t < RUN_X + 2 * KRAD; ++t) {
                const float2 v = *reinterpret_cast<const float2 *>(bp + t * r.pb);
#pragma unroll
                for (int o = 0; o < RUN_X; ++o)
                    if (t >= o && t - o <= 2 * KRAD) s[o] = ffma2(fmul2(tap[t - o], v), one, s[o]);
            }
            float *q = r.A + x0 * r.ph + RPAD + yl;
#pragma unroll
            for (int o = 0; o < RUN_X; ++o) *reinterpret_cast<float2 *>(q + o * r.ph) = s[o];
        }
    }
    __syncthreads();
}

// The rotated light R^T (lambda - tau) of a render.
__device__ __forceinline__ void light_terms(const float *R, const float *tau, const float *lam, float (&q)[3])
{
    const float d0 = lam[0] - tau[0], d1 = lam[1] - tau[1], d2 = lam[2] - tau[2];
    q[0] = (R[0] * d0 + R[1] * d1) + R[2] * d2;
    q[1] = (R[3] * d0 + R[4] * d1) + R[5] * d2;
    q[2] = (R[6] * d0 + R[7] * d1) + R[8] * d2;
}

// Owners shaded into the cleared region. Each fragment's unit normal, n . p and interpolated
// albedo depend only on the geometry of the raster: the depth pass forms them for every
// raster (k_raster_slots places them, shc and sht). A render forms the rotated light once and the same FP32 operations as
// the reference's shading: Id = (n0 q0 + n1 q1) + n2 q2 - n.p, I = t + (L t) Id. RENDER_SU fragments per thread:
// each one's pixel word and shading terms are loaded together.
template <int NT>
__device__ __forceinline__ void region_shade(const Region &r, const Fragment *frags, const float4 *shc,
                                             const float *sht, int N, const float (&q)[3], float Lint)
{
    for (int n0 = threadIdx.x; n0 < N; n0 += NT * RENDER_SU) {
        uint32_t po[RENDER_SU];
        float4 sn[RENDER_SU];
        float t[RENDER_SU];
#pragma unroll
        for (int u = 0; u < RENDER_SU; ++u) {
            const int n = n0 + u * NT;
            po[u] = 0u;
            if (n < N) {
                po[u] = frags[n].pix_owner;
                sn[u] = shc[n];
                t[u] = sht[n];
            }
        }
#pragma unroll
        for (int u = 0; u < RENDER_SU; ++u)
            if (po[u] & 0x80000000u) {
                const float Id = ((sn[u].x * q[0] + sn[u].y * q[1]) + sn[u].z * q[2]) - sn[u].w;
                r.A[r.at(po[u] & 0xFFFF)] = t[u] + (Lint * t[u]) * Id;
            }
    }
}

// FP64 sum of a block's values: shuffles, then the warps in order; the total in thread 0. The order is
// that of RENDER_SUMS threads with one value each, whatever the block: thread t of a smaller one holds
// the values of threads t, t + NT, ..., so that a frame's sum does not depend on the block size.
constexpr int RENDER_SUMS = 1024;
template <int NT>
__device__ __forceinline__ double render_sum(double (&v)[RENDER_SUMS / NT], double *s_red)
{
#pragma unroll
    for (int h = 0; h < RENDER_SUMS / NT; ++h) {
        for (int o = 16; o > 0; o >>= 1) v[h] += __shfl_down_sync(0xffffffffu, v[h], o);
        if ((threadIdx.x & 31) == 0) s_red[(threadIdx.x >> 5) + h * (NT / 32)] = v[h];
    }
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < RENDER_SUMS / 32; ++w) s += s_red[w];
    return s;
}

// Normalised gradients of the blurred targets at every pixel, once per fit: a render reads one
// 8-byte value per fragment instead of forming them from four gathered pixels.
__global__ void k_target_grad(const float *target, float2 *tgn, int F)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)F * NPIX) return;
    const int p = (int)(i & (NPIX - 1));
    const float *t = target + (i - p);
    int kr, kl, kd, ku;
    neighbour_pixels(p, kr, kl, kd, ku);
    float gx, gy, h;
    float2 g;
    grad_of(t[kr], t[kl], t[kd], t[ku], gx, gy, h, g.x, g.y);
    tgn[i] = g;
}

// NT threads per frame: 512 (two blocks per SM) for full rounds, 1,024 when the frames do not
// fill the SMs and a block's own latency is the round's. Both give the same bits (render_sum).
template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT) k_render_t(DModel m, DBatch b, Cfg c, int stage)
{
    if ((int)blockIdx.x >= render_n(b)) return;
    const int f = b.rlist[blockIdx.x];
    FrameCtl &ctl = b.ctl[f];
    const int tid = threadIdx.x;
    if (!ctl.render) {                           // the resolve refused the raster
        if (tid == 0) end_shape_stage(c, ctl, stage, ctl.outer);
        return;
    }
    if (tid == 0) prof_count(b, KID_RENDER);
    extern __shared__ __align__(16) float rsm[];
    __shared__ double s_red[RENDER_SUMS / 32];
    __shared__ int s_take;
    __shared__ float s_t;
    const Region r = make_region(ctl, rsm, b.img + (size_t)f * RIMG);
    const int N = ctl.N;
    const Fragment *frags = b.frag + (size_t)f * NMAX;
    region_clear<NT>(r, true);
    float q[3];
    light_terms(b.R + f * 9, b.xe + (size_t)f * m.KTP + m.K, b.lam + f * 4, q);
    __syncthreads();
    region_shade<NT>(r, frags, b.shc + (size_t)f * NMAX, b.sht + (size_t)f * NMAX, N, q, b.Lint[f]);
    __syncthreads();
    region_blur<NT>(r, c);
    const float2 *tgn = b.tgn + (size_t)f * NPIX;
    float *fg = b.fgrad + (size_t)f * 5 * NMAX;
    constexpr int NS = RENDER_SUMS / NT;         // sums per thread: of the fragments tid + NT h modulo RENDER_SUMS
    static_assert(RENDER_GU % NS == 0, "a thread's u-th fragment belongs to its sum u % NS");
    double corr[NS] = {};
    for (int n0 = tid; n0 < N; n0 += NT * RENDER_GU) {
        int pv[RENDER_GU];
        float2 tg[RENDER_GU];
#pragma unroll
        for (int u = 0; u < RENDER_GU; ++u) {
            const int n = n0 + u * NT;
            pv[u] = n < N ? (int)(frags[n].pix_owner & 0xFFFF) : -1;
        }
#pragma unroll
        for (int u = 0; u < RENDER_GU; ++u) tg[u] = pv[u] >= 0 ? tgn[pv[u]] : make_float2(0.0f, 0.0f);
#pragma unroll
        for (int u = 0; u < RENDER_GU; ++u) {
            if (pv[u] < 0) break;
            const int n = n0 + u * NT;
            int kr, kl, kd, ku;                // (pixel 0 lies outside a region that is not the crop)
            neighbour_pixels(pv[u], kr, kl, kd, ku);
            float gx, gy, h, gxn, gyn;
            grad_of(r.A[r.at(kr)], r.A[r.at(kl)], r.A[r.at(kd)], r.A[r.at(ku)], gx, gy, h, gxn, gyn);
            fg[n] = gx; fg[NMAX + n] = gy; fg[2 * NMAX + n] = h;
            fg[3 * NMAX + n] = tg[u].x; fg[4 * NMAX + n] = tg[u].y;
            corr[u % NS] += (double)gxn * (double)tg[u].x + (double)gyn * (double)tg[u].y;
        }
    }
    const double total = render_sum<NT>(corr, s_red);
    // The decision (model_fitter.cu:215-356): objective -(tau*corr - barrier); Armijo test.
    if (tid == 0) {
        const int maxit = stage == ST_RIGID ? c.max_iters_rigid : c.max_iters_finetune;
        const float tau_img = 5.0f * 5.0f;
        ctl.corr = total;
        float gc = tau_img * (float)total;
        gc = gc + (-ctl.obj_b);
        const float obj = -gc;
        int take = 1, jac = 1;                   // the point is kept; it gets its normal equations
        if (ctl.mode == M_FULL) {
            take = 2;                            // (already x)
        } else {
            ctl.inner++;
            float l2 = ctl.l2base;
            l2 = l2 * (0.4f * ctl.t);
            if (obj < ctl.obj0 + l2) {
                if (ctl.outer >= maxit) { end_shape_stage(c, ctl, stage, ctl.outer); jac = 0; }
                else ctl.outer++;
            } else {
                take = jac = 0;
            }
        }
        if (take) { ctl.obj0 = obj; ctl.objective = obj; }
        if (jac) {
            ctl.need_jac = 1;
            b.jlist[atomicAdd(b.rcount + 1, 1)] = f;
        }
        s_take = take;
    }
    __syncthreads();
    if (s_take == 1) {
        for (int a = tid; a < m.KT; a += NT) b.x[(size_t)f * m.KTP + a] = b.x_ls[(size_t)f * m.KTP + a];
    } else if (s_take == 0) {
        shape_reject(m, b, c, f, stage, &s_t);
    }
}

// ------------------------------------------------------------------------------------------
// Neighbour maps (derivative_computer.cu:43-72; funcs.cu:81-131, 288-343), one block per
// frame. The reference stable-sorts fragments by pixel and derives, for sorted position i,
// left = i - (cum[p] - cum[p-256]) (0 when not positive, clamped to N-1),
// right = i + cum[p+256] - cum[p], above/below = i -+ 1 (16-bit wrap), position 0 and N-1
// all 0, where cum counts distinct covered pixels up to a pixel. Here the sort is replaced by
// a counting placement: sorted position = distinct pixels below p + extra (tied) fragments
// below p + rank among the fragments of p in slot order.
// The counting atomics also build the per-word masks (covered pixels, pixels with 2+
// fragments) and extra-fragment counts, so only 2,048 words are scanned. Sorted positions
// and the inverse permutation are held in shared memory as 16-bit indices (NMAX = 32768).
// A pixel hit by several fragments (rare) first gets its fragments placed in arbitrary order
// inside its group, then each of them counts the group members with a lower slot index,
// which gives the stable order; frames without such pixels skip those passes.

constexpr int NB_U = 4;                 // fragment pixels loaded per thread before use
__host__ __device__ constexpr size_t neigh_smem()
{
    return (size_t)(NPIX / 2 + 4 * (NPIX / 32)) * sizeof(uint32_t) + (size_t)NMAX * sizeof(uint16_t);
}

__device__ __forceinline__ uint32_t cnt_at(const uint32_t *cnt, int p)
{
    return (cnt[p >> 1] >> ((p & 1) * 16)) & 0xFFFFu;
}

__global__ void __launch_bounds__(1024) k_neighbours(DBatch b, int all_frames)
{
    if ((int)blockIdx.x >= (all_frames ? render_n(b) : jac_n(b))) return;
    const int f = (all_frames ? b.rlist : b.jlist)[blockIdx.x];
    FrameCtl &ctl = b.ctl[f];
    if (!(all_frames ? ctl.render : ctl.need_jac)) return;
    if (threadIdx.x == 0) prof_count(b, KID_NEIGHBOURS);
    extern __shared__ __align__(16) uint32_t nsm[];
    uint32_t *cnt = nsm;                    // 32768 words: two 16-bit counts each
    uint16_t *perm = reinterpret_cast<uint16_t *>(nsm);   // replaces cnt: sorted position -> fragment
    uint32_t *bits = cnt + NPIX / 2;        // 2048 words: covered pixels
    uint32_t *tieb = bits + NPIX / 32;      // 2048 words: pixels with 2+ fragments
    uint32_t *wU = tieb + NPIX / 32;        // 2048: distinct pixels before the word
    uint32_t *wE = wU + NPIX / 32;          // 2048: extra fragments in (then before) the word
    uint16_t *spos = reinterpret_cast<uint16_t *>(wE + NPIX / 32);   // [NMAX]: fragment -> sorted position
    __shared__ uint32_t s_wsum[2][32];
    __shared__ uint32_t s_flags;
    __shared__ int s_ties;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int N = ctl.N;
    const Fragment *frags = b.frag + (size_t)f * NMAX;
    auto pix_of = [&](int n) -> int { return (int)(frags[n].pix_owner & 0xFFFF); };
    auto load_pix = [&](int n0, int pv[NB_U]) {
#pragma unroll
        for (int u = 0; u < NB_U; ++u) {
            const int n = n0 + u * 1024;
            pv[u] = n < N ? pix_of(n) : 0;
        }
    };
    if (tid == 0) { s_flags = 0; s_ties = 0; }
    {
        uint4 *z = reinterpret_cast<uint4 *>(nsm);          // cnt, bits, tieb
        for (int i = tid; i < (NPIX / 2 + 2 * (NPIX / 32)) / 4; i += 1024) z[i] = make_uint4(0u, 0u, 0u, 0u);
        for (int i = tid; i < NPIX / 32; i += 1024) wE[i] = 0;
    }
    __syncthreads();
    for (int n0 = tid; n0 < N; n0 += 1024 * NB_U) {
        int pv[NB_U];
        load_pix(n0, pv);
#pragma unroll
        for (int u = 0; u < NB_U; ++u) {
            if (n0 + u * 1024 >= N) break;
            const int p = pv[u], w = p >> 5;
            const uint32_t bm = 1u << (p & 31), sh = (p & 1) * 16;
            const uint32_t old = (atomicAdd(&cnt[p >> 1], 1u << sh) >> sh) & 0xFFFFu;
            if (old == 0) {
                atomicOr(&bits[w], bm);
            } else {
                atomicAdd(&wE[w], 1u);
                if (old == 1) { atomicOr(&tieb[w], bm); s_ties = 1; }
            }
        }
    }
    __syncthreads();
    // exclusive scans of the distinct and extra counts over the 2048 words
    uint32_t u2[2], e2[2];
    for (int q = 0; q < 2; ++q) { u2[q] = __popc(bits[tid * 2 + q]); e2[q] = wE[tid * 2 + q]; }
    uint32_t us = u2[0] + u2[1], es = e2[0] + e2[1];
    uint32_t ui = us, ei = es;   // inclusive warp scans
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, ui, o), c2 = __shfl_up_sync(0xffffffffu, ei, o);
        if (lane >= o) { ui += a; ei += c2; }
    }
    if (lane == 31) { s_wsum[0][warp] = ui; s_wsum[1][warp] = ei; }
    __syncthreads();                       // also orders every read of wE above before its rewrite
    if (tid < 32) {
        uint32_t a = s_wsum[0][tid], c2 = s_wsum[1][tid];
        uint32_t ai = a, ci = c2;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t1 = __shfl_up_sync(0xffffffffu, ai, o), t2 = __shfl_up_sync(0xffffffffu, ci, o);
            if (tid >= o) { ai += t1; ci += t2; }
        }
        s_wsum[0][tid] = ai - a;
        s_wsum[1][tid] = ci - c2;
    }
    __syncthreads();
    {
        const uint32_t ubase = s_wsum[0][warp] + ui - us, ebase = s_wsum[1][warp] + ei - es;
        wU[tid * 2] = ubase; wE[tid * 2] = ebase;
        wU[tid * 2 + 1] = ubase + u2[0]; wE[tid * 2 + 1] = ebase + e2[0];
    }
    __syncthreads();
    const bool ties = s_ties != 0;
    auto cum = [&](int p) -> int {                     // covered pixels q <= p
        const int w = p >> 5, bit = p & 31;
        return (int)(wU[w] + __popc(bits[w] & ((2u << bit) - 1u)));
    };
    auto tied = [&](int p) -> bool { return (tieb[p >> 5] >> (p & 31)) & 1u; };
    // first sorted position of pixel p's fragments
    auto group_start = [&](int p) -> int {
        const int w = p >> 5;
        const uint32_t below = (1u << (p & 31)) - 1u;
        uint32_t pos = wU[w] + __popc(bits[w] & below) + wE[w];
        uint32_t tb = tieb[w] & below;
        while (tb) {
            const int j = __ffs(tb) - 1;
            tb &= tb - 1;
            pos += cnt_at(cnt, w * 32 + j) - 1;
        }
        return (int)pos;
    };
    for (int n0 = tid; n0 < N; n0 += 1024 * NB_U) {
        int pv[NB_U];
        load_pix(n0, pv);
#pragma unroll
        for (int u = 0; u < NB_U; ++u) {
            const int n = n0 + u * 1024;
            if (n < N) spos[n] = (uint16_t)group_start(pv[u]);
        }
    }
    if (ties) {
        // distinct slots inside each group, in arbitrary order: the counts are taken back one
        // by one (nothing reads them after the barrier)
        __syncthreads();
        for (int n = tid; n < N; n += 1024) {
            const int p = pix_of(n);
            if (!tied(p)) continue;
            const uint32_t sh = (p & 1) * 16;
            const uint32_t old = (atomicSub(&cnt[p >> 1], 1u << sh) >> sh) & 0xFFFFu;
            spos[n] = (uint16_t)(spos[n] + old - 1);
        }
    }
    __syncthreads();                       // the counts are no longer read: perm replaces them
    for (int n = tid; n < N; n += 1024) perm[spos[n]] = (uint16_t)n;
    __syncthreads();
    if (ties) {
        // stable order inside each group: rank = group members with a lower slot index
        for (int n = tid; n < N; n += 1024) {
            const int p = pix_of(n);
            if (!tied(p)) continue;
            const int i = spos[n];
            int r = 0, j = i - 1;
            for (; j >= 0; --j) {
                const int q = perm[j];
                if (pix_of(q) != p) break;
                r += q < n;
            }
            const int start = j + 1;
            for (j = i + 1; j < N; ++j) {
                const int q = perm[j];
                if (pix_of(q) != p) break;
                r += q < n;
            }
            spos[n] = (uint16_t)(start + r);
        }
        __syncthreads();
        for (int n = tid; n < N; n += 1024)
            if (tied(pix_of(n))) perm[spos[n]] = (uint16_t)n;
        __syncthreads();
    }
    int32_t *nb = b.nb + (size_t)f * 4 * NMAX;
    for (int n0 = tid; n0 < N; n0 += 1024 * NB_U) {
        int pv[NB_U];
        load_pix(n0, pv);
#pragma unroll
        for (int u = 0; u < NB_U; ++u) {
            const int n = n0 + u * 1024;
            if (n >= N) continue;
            const int i = spos[n], p = pv[u];
            int S[4] = {0, 0, 0, 0};
            if (i != 0 && i != N - 1) {
                const int y = p & 255, x = p >> 8;
                const int right = (x < DIM - 1) ? (x + 1) * DIM + y : 0;
                const int left = (x > 0) ? (x - 1) * DIM + y : 0;
                const int dl = cum(p) - cum(left);
                int kl = (i > dl) ? (i - dl) : 0;
                kl = (uint16_t)kl;
                if (kl >= N - 1) kl = N - 1;
                S[0] = kl;
                S[1] = (uint16_t)(i + cum(right) - cum(p));
                S[2] = (uint16_t)(i - 1);
                S[3] = (uint16_t)(i + 1);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                int sq = S[q];
                if (sq >= N) { atomicOr(&s_flags, FLAG_OUT_OF_DOMAIN); sq = 0; }
                nb[q * NMAX + n] = perm[sq];
            }
        }
    }
    __syncthreads();
    if (tid == 0 && s_flags) ctl.flags |= s_flags;
}

// ------------------------------------------------------------------------------------------
// Jacobian rows dI/dtheta (newfuncs.cu:173-299, funcs.cu:224-282). A block takes chunks of
// JAC_CH fragments of one frame: one thread per fragment forms the interpolated point, its
// camera coordinates and the pose columns, and leaves the per-fragment factors in shared
// memory (each twice, as the operand of a packed operation); then the chunk's (fragment, four
// expression columns) items are spread over all threads, consecutive items being consecutive
// columns of a fragment, so that the nine basis rows of an item are read in 16-byte loads,
// coalesced and in flight together. Two columns per packed FP32 instruction, each half rounding as
// the scalar operation (products and sums kept apart, see packed_one).
// It was bound by issue (one column per item: 922,000 warp instructions per frame, 62% issue active,
// 1,389 us for 1,024 frames); now by the reads of the basis rows (10.6 MB per frame, mostly L2):
// 1,087 us (3 blocks per SM 1,153, 2 blocks 1,417). (Taking the chunks in pixel order, so that a chunk's triangles share corners, measured
// 3% slower before.)

constexpr int JAC_THREADS = 256;
constexpr int JAC_CH = 128;                  // fragments per chunk
constexpr int JAC_BPF = 32;                  // blocks per frame

__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }

// two columns of a Jacobian row from the basis pairs of the three corners (b, c, a; x, y, z each)
struct JacFactors {
    float2 al, be, ga, gx, vx, vy, vz, gy, cx, cy;
};

__device__ __forceinline__ float2 jac_pair(const float2 (&e)[3][3], const JacFactors &q, const float2 (&R)[9], float2 one,
                                           float2 mone)
{
    float2 t[3];
#pragma unroll
    for (int j = 0; j < 3; ++j)
        t[j] = ffma2(ffma2(fmul2(e[0][j], q.al), one, fmul2(e[1][j], q.be)), one, fmul2(e[2][j], q.ga));
    float2 r[3];                             // (tx R[i] + ty R[3 + i]) + tz R[6 + i]
#pragma unroll
    for (int i = 0; i < 3; ++i)
        r[i] = ffma2(ffma2(fmul2(t[0], R[i]), one, fmul2(t[1], R[3 + i])), one, fmul2(t[2], R[6 + i]));
    const float2 nwx = fmul2(q.cx, ffma2(fmul2(r[2], q.vx), mone, fmul2(r[0], q.vz)));
    const float2 nwy = fmul2(q.cy, ffma2(fmul2(r[2], q.vy), mone, fmul2(r[1], q.vz)));
    const float2 s = ffma2(fmul2(q.gx, nwx), one, fmul2(q.gy, nwy));
    return make_float2(-s.x, -s.y);
}

__global__ void __launch_bounds__(JAC_THREADS, 4) k_jacobian(DModel m, DBatch b)
{
    if ((int)blockIdx.y >= jac_n(b)) return;
    const int f = b.jlist[blockIdx.y];
    const FrameCtl &ctl = b.ctl[f];
    if (blockIdx.x == 0 && threadIdx.x == 0) prof_count(b, KID_JACOBIAN);
    __shared__ float4 s_f[5][JAC_CH];        // factor pairs: (al, be), (ga, gx), (vx, vy), (vz, gy), (cx, cy), each twice
    __shared__ int4 s_e[JAC_CH];             // basis row offsets of b, c, a (16-byte units); Jacobian row offset
    const int N = ctl.N, K = m.K, KP = m.KP, V = m.V, KTP = m.KTP;
    const int tid = threadIdx.x;
    const float4 *geo = b.geo + (size_t)f * V;
    const float *Rg = b.R + f * 9, *dR = b.dR + f * 27;
    const float *tau = b.xe + (size_t)f * KTP + K;
    const float phix = b.cam[f * 4], phiy = b.cam[f * 4 + 1];
    const Fragment *frags = b.frag + (size_t)f * NMAX;
    const float *fg = b.fgrad + (size_t)f * 5 * NMAX;
    float *Jf = b.J + (size_t)f * NMAX * KTP;
    const float2 one = packed_one(ctl.need_jac & 2), mone = make_float2(-one.x, -one.y);   // (need_jac is 1)
    float2 R2[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) R2[i] = dup2(Rg[i]);
    const int Q = KP >> 2;                               // column quads of a row
    const uint32_t mg = Q > 1 ? 0xFFFFFFFFu / (uint32_t)Q + 1u : 0u;   // i / Q = umulhi(i, mg) for i < 2^16
    const float4 *E4 = reinterpret_cast<const float4 *>(m.E);
    for (int c0 = blockIdx.x * JAC_CH; c0 < N; c0 += gridDim.x * JAC_CH) {
        const int cnt = min(JAC_CH, N - c0);
        if (tid < cnt) {
            const int n = c0 + tid;
            const Fragment fr = frags[n];
            const int4 tc = __ldg(m.tl4 + fr.tri);
            const int ib = tc.x, ic = tc.y, ia = tc.z;
            const float al = fr.al, be = fr.be, ga = (1 - fr.al) - fr.be;
            const float4 gb = geo[ib], gc = geo[ic], ga4 = geo[ia];
            const float px = (gb.x * al + gc.x * be) + ga4.x * ga;
            const float py = (gb.y * al + gc.y * be) + ga4.y * ga;
            const float pz = (gb.z * al + gc.z * be) + ga4.z * ga;
            float R[9];
#pragma unroll
            for (int i = 0; i < 9; ++i) R[i] = R2[i].x;
            float bX, bY, bZ, cX, cY, cZ, aX, aY, aZ;
            camera_coords(R, tau, gb.x, gb.y, gb.z, bX, bY, bZ);
            camera_coords(R, tau, gc.x, gc.y, gc.z, cX, cY, cZ);
            camera_coords(R, tau, ga4.x, ga4.y, ga4.z, aX, aY, aZ);
            const float vx = (bX * al + cX * be) + aX * ga;
            const float vy = (bY * al + cY * be) + aY * ga;
            const float vz = (bZ * al + cZ * be) + aZ * ga;
            const float ivz = 1.0f / vz, ivz2 = ivz * ivz;
            const float gx = fg[n], gy = fg[NMAX + n];
            const float cx = phix * ivz2, cy = phiy * ivz2;
            s_f[0][tid] = make_float4(al, al, be, be);
            s_f[1][tid] = make_float4(ga, ga, gx, gx);
            s_f[2][tid] = make_float4(vx, vx, vy, vy);
            s_f[3][tid] = make_float4(vz, vz, gy, gy);
            s_f[4][tid] = make_float4(cx, cx, cy, cy);
            s_e[tid] = make_int4(ib * 3 * Q, ic * 3 * Q, ia * 3 * Q, n * KTP);
            float *row = Jf + (size_t)n * KTP;
            row[K + 0] = -(gx * (phix * ivz) + gy * 0.0f);
            row[K + 1] = -(gx * 0.0f + gy * (phiy * ivz));
            row[K + 2] = -(gx * (((-phix) * vx) * ivz2) + gy * (((-phiy) * vy) * ivz2));
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const float *d = dR + 9 * j;
                const float dvx = (d[0] * px + d[3] * py) + d[6] * pz;
                const float dvy = (d[1] * px + d[4] * py) + d[7] * pz;
                const float dvz = (d[2] * px + d[5] * py) + d[8] * pz;
                const float dWx = (phix * ivz2) * (vz * dvx - vx * dvz);
                const float dWy = (phiy * ivz2) * (vz * dvy - vy * dvz);
                row[K + 3 + j] = -(gx * dWx + gy * dWy);
            }
            for (int j = m.KT; j < KTP; ++j) row[j] = 0.0f;
        }
        __syncthreads();
        for (int i = tid; i < cnt * Q; i += JAC_THREADS) {
            const int nl = Q > 1 ? (int)__umulhi((uint32_t)i, mg) : i, kq = i - nl * Q;
            const int4 o = s_e[nl];
            float4 e[3][3];
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                e[0][j] = __ldg(E4 + o.x + j * Q + kq);
                e[1][j] = __ldg(E4 + o.y + j * Q + kq);
                e[2][j] = __ldg(E4 + o.z + j * Q + kq);
            }
            const float4 f0 = s_f[0][nl], f1 = s_f[1][nl], f2 = s_f[2][nl], f3 = s_f[3][nl], f4 = s_f[4][nl];
            const JacFactors q{make_float2(f0.x, f0.y), make_float2(f0.z, f0.w), make_float2(f1.x, f1.y),
                               make_float2(f1.z, f1.w), make_float2(f2.x, f2.y), make_float2(f2.z, f2.w),
                               make_float2(f3.x, f3.y), make_float2(f3.z, f3.w), make_float2(f4.x, f4.y),
                               make_float2(f4.z, f4.w)};
            float2 lo[3][3], hi[3][3];
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    lo[c][j] = make_float2(e[c][j].x, e[c][j].y);
                    hi[c][j] = make_float2(e[c][j].z, e[c][j].w);
                }
            const float2 r0 = jac_pair(lo, q, R2, one, mone), r1 = jac_pair(hi, q, R2, one, mone);
            float *dst = Jf + o.w + 4 * kq;
            if (4 * kq + 3 < K) {
                *reinterpret_cast<float4 *>(dst) = make_float4(r0.x, r0.y, r1.x, r1.y);
            } else {                                     // the last quad: columns from K on are the pose's
                if (4 * kq < K) dst[0] = r0.x;
                if (4 * kq + 1 < K) dst[1] = r0.y;
                if (4 * kq + 2 < K) dst[2] = r1.x;
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------
// Normal equations of the image term (derivative_computer.cu:135-164): rows of
// d(gx/|g|)/dtheta and d(gy/|g|)/dtheta, H = tau * sum(row row^T), g = -tau * sum(w row).
// The reference sums with cublasSgemm in the library's order; the order here is fixed and
// shared with the oracle: fragments in chunks of NE_CH, each chunk summed from zero with one
// FP64 fused multiply-add per row and entry in fragment order (x row, then y row), the chunk
// sums then added in chunk order. The rows are floats, so every product is exact in FP64.
// k_normal_eq writes one partial per chunk (NE_BPF blocks per frame, each looping over
// chunks); rows are staged 32 fragments at a time in shared memory as doubles. k_normal_eq_reduce
// adds the chunk partials.

constexpr int NE_THREADS = 256;
constexpr int NE_CH = 256;                   // fragments per chunk (the unit of the sum order)
constexpr int NE_SUB = 32;                   // fragments staged in shared memory at a time
constexpr int NE_BPF = 32;                   // blocks per frame
constexpr int NE_MAXCH = NMAX / NE_CH;       // chunk partials per frame at most
constexpr int NE_SPREAD = 148;               // chunks of a round up to which their tiles are split over two blocks
static_assert(NE_THREADS == NE_CH && NE_SUB == 32 && NE_THREADS == 8 * 32, "thread mapping of the row build");

// Chunk partials are sized for the widest layout the normal-equation kernels have used:
// 132 tiles of 4 x 8 doubles plus a row (KTP <= 88); the 8 x 8 tensor-core tiles need less.
constexpr int NE_TILES = 132;

__host__ __device__ __forceinline__ int ne_part_stride(int KTP)
{
    return NE_TILES * 32 + KTP;   // the widest partial layout of the normal-equation kernels
}

// Rows of one chunk of NE_CH fragments: per-fragment scalars and neighbour indices are
// staged once per chunk (one thread per fragment); a thread then builds fragment
// 4*warp + lane/8 of each 32-fragment stage at columns 8*g + lane%8, its four neighbour
// rows of J loaded one stage ahead.
constexpr int NE_GRP = 11;                   // column groups of 8: KTP <= 88 (K <= 82)

struct ChunkHead {
    int nb[4][NE_CH];
    float pre[NE_CH], dx[NE_CH], dy[NE_CH];
    double w[2 * NE_CH];
};

__device__ __forceinline__ void chunk_head(ChunkHead &hd, const float *fg, const int32_t *nb, int c0, int cnt, int q)
{
    const int n = c0 + q;
    float pre = 0.0f, dx = 0.0f, dy = 0.0f, wx = 0.0f, wy = 0.0f;
    int k0 = 0, k1 = 0, k2 = 0, k3 = 0;
    if (q < cnt) {
        const float gx = fg[n], gy = fg[NMAX + n], h = fg[2 * NMAX + n];
        pre = (float)(1.0 / (0.001 + (double)(h * h * h)));
        dx = 2 * gx;
        dy = 2 * gy;
        wx = fg[3 * NMAX + n];
        wy = fg[4 * NMAX + n];
        k0 = nb[n]; k1 = nb[NMAX + n]; k2 = nb[2 * NMAX + n]; k3 = nb[3 * NMAX + n];
    }
    hd.pre[q] = pre; hd.dx[q] = dx; hd.dy[q] = dy;
    hd.nb[0][q] = k0; hd.nb[1][q] = k1; hd.nb[2][q] = k2; hd.nb[3][q] = k3;
    hd.w[2 * q] = (double)wx;
    hd.w[2 * q + 1] = (double)wy;
}

template <int GRP>
__device__ __forceinline__ void chunk_prefetch(float (&v)[GRP][4], const ChunkHead &hd, const float *Jf,
                                               int KT, int KTP, int q, int cnt, int a_low)
{
    const bool live = q < cnt;
    const int r0 = hd.nb[0][q], r1 = hd.nb[1][q], r2 = hd.nb[2][q], r3 = hd.nb[3][q];
#pragma unroll
    for (int g = 0; g < GRP; ++g) {
        const int a = 8 * g + a_low;
        const bool use = live && a < KT;
        v[g][0] = use ? __ldg(Jf + (size_t)r0 * KTP + a) : 0.0f;
        v[g][1] = use ? __ldg(Jf + (size_t)r1 * KTP + a) : 0.0f;
        v[g][2] = use ? __ldg(Jf + (size_t)r2 * KTP + a) : 0.0f;
        v[g][3] = use ? __ldg(Jf + (size_t)r3 * KTP + a) : 0.0f;
    }
}

// Chain rule through the normalised gradient (newfuncs.cu:417-463) at one column.
__device__ __forceinline__ void chain_value(const float (&vv)[4], float pre, float diffx, float diffy,
                                            float &ox, float &oy)
{
    const float dh = vv[1] - vv[0];
    const float dv = vv[3] - vv[2];
    const float X = (-diffy) * (-dh) - (-diffx) * (-dv);
    ox = ((-pre) * (-diffy)) * X;
    oy = (pre * (-diffx)) * X;
}

// FP64 tensor-core form of the exact sum: mma.sync m8n8k4 f64 updates an 8x8 tile with four
// rows k = 0..3 as the fused multiply-add chain d = fma(a3, b3, fma(a2, b2, fma(a1, b1,
// fma(a0, b0, c)))) (checked on B200 against CPU emulation: no mismatch in 4.2M entries; the
// parity tests check H and g bit for bit). Four rows are two fragments' x and y rows in
// order, so the chain is exactly the oracle's. Tiles of 8x8 cover the upper triangle of a
// P8 x P8 matrix whose column KT holds the weights w (so the column KT of the sum is g).
constexpr int NE_P8 = 88;                    // padded width: parameters + weight column, <= 88
constexpr int NE_T8 = NE_P8 / 8;             // 11 tile rows / columns
constexpr int NE_NT8 = NE_T8 * (NE_T8 + 1) / 2;   // 66 tiles

__device__ __forceinline__ void ne_tile8(int t, int &bi, int &bj)
{
    bi = 0;
    while (t >= NE_T8 - bi) { t -= NE_T8 - bi; ++bi; }
    bj = bi + t;
}

__host__ __device__ constexpr inline int ne_part_stride8() { return NE_NT8 * 64; }
static_assert(RASTER_WORK <= (size_t)NE_MAXCH * ne_part_stride8() * sizeof(double), "a raster's working set lies there");

__device__ __forceinline__ void dmma_884(double &d0, double &d1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1) : "d"(a), "d"(b));
}

// Rows are staged in shared memory as doubles (converted once when built), row pitch NE_PD:
// 92 doubles puts the four rows a warp reads at once on disjoint bank groups.
constexpr int NE_PD = NE_P8 + 4;

// Tile list in ne_tile8's order, as a compile-time table.
struct NeTiles {
    int bi[NE_NT8], bj[NE_NT8];
};
__host__ __device__ constexpr NeTiles make_ne_tiles()
{
    NeTiles t{};
    int k = 0;
    for (int i = 0; i < NE_T8; ++i)
        for (int j = i; j < NE_T8; ++j) { t.bi[k] = i; t.bj[k] = j; ++k; }
    return t;
}

// Half of a block's warps build rows, the other half run the tensor cores, two stages of rows
// between them (named barriers: full and empty per stage), so that the neighbour rows' gathers, the
// chain rule and the conversions of one stage hide behind the updates of the one before. With
// one updating warp per SM sub-partition a row value loaded once feeds 16 tiles instead of 8 (the
// shared-memory reads were 0.67 of the tensor time). All warps building, then all updating, took 2,874 us
// for 1,024 frames; this form 2,498 us (26.6 TFLOP/s in the tiles; the pipe gives 37 measured alone).
// With few frames a chunk's tiles are split over NE_SPLIT blocks, each building all rows: one frame is
// 15 chunks, and 148 SMs (38 -> 24 us).
constexpr int NE_MMA_WARPS = 4;              // one per SM sub-partition
constexpr int NE_BUILDERS = NE_THREADS - 32 * NE_MMA_WARPS;
constexpr int NE_SPLIT = 2;
constexpr int NE_FULL = 1, NE_EMPTY = 3, NE_HEAD = 5;   // named barriers: full and empty by stage, the builders' own

__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }

// Share W of the upper triangle's tiles. For whole blocks (S = 1) the four shares are cut so that each
// touches few of the 11 column blocks (6, 6, 9 and 8 instead of 11 each, for 17, 17, 16 and 16 tiles),
// since every column block touched is a shared-memory read per fragment pair; split blocks take
// every 4 S-th tile.
__host__ __device__ constexpr int ne_share(int t, int bi, int bj, int S)
{
    if (S > 1) return t % (NE_MMA_WARPS * S);
    if (bj <= 4) return 0;
    if (bi >= 6) return 1;
    if (bj == 5) return bi <= 1 ? 0 : bi == 2 ? 2 : 3;
    if (bi == 5) return bj <= 7 ? 1 : 3;
    return bi <= 2 ? 2 : 3;
}
constexpr int NE_SHARE = 17;                 // tiles of a share at most
struct NeList {
    int n, t[NE_SHARE], bi[NE_SHARE], bj[NE_SHARE];
    unsigned used;                           // column blocks touched
};
__host__ __device__ constexpr NeList make_ne_list(int W, int S)
{
    NeList l{};
    constexpr NeTiles TT = make_ne_tiles();
    for (int t = 0; t < NE_NT8; ++t)
        if (ne_share(t, TT.bi[t], TT.bj[t], S) == W) {
            l.t[l.n] = t; l.bi[l.n] = TT.bi[t]; l.bj[l.n] = TT.bj[t];
            l.used |= 1u << TT.bi[t] | 1u << TT.bj[t];
            ++l.n;
        }
    return l;
}

// The updates of one stage's fragment pairs for the tiles of share W: a lane loads its row's value in
// each column block of the share once per pair and feeds every tile from those registers.
template <int W, int S>
__device__ __forceinline__ void ne_pairs(double (&acc)[NE_SHARE][2], const double *rows, int cn, int kr, int fr8)
{
    constexpr NeList LS = make_ne_list(W, S);
    for (int q = 0; q + 2 <= cn; q += 2) {
        const double *rk = rows + (size_t)(2 * q + kr) * NE_PD + fr8;
        double v[NE_T8];
#pragma unroll
        for (int c = 0; c < NE_T8; ++c)
            if (LS.used >> c & 1u) v[c] = rk[8 * c];
#pragma unroll
        for (int j = 0; j < LS.n; ++j) dmma_884(acc[j][0], acc[j][1], v[LS.bi[j]], v[LS.bj[j]]);
    }
    // an odd last fragment: this thread's two entries of each tile, the same chain
    if (cn & 1) {
        const double *rx = rows + (size_t)(2 * (cn - 1)) * NE_PD, *ry = rx + NE_PD;
#pragma unroll
        for (int j = 0; j < LS.n; ++j) {
            const int r = 8 * LS.bi[j] + fr8, c = 8 * LS.bj[j] + 2 * kr;
#pragma unroll
            for (int i = 0; i < 2; ++i) acc[j][i] = fma(ry[r], ry[c + i], fma(rx[r], rx[c + i], acc[j][i]));
        }
    }
}

template <int W, int S>
__device__ __forceinline__ void ne_update(const double *rows, double *parts, int N, int ch0, int step, int total, int lane)
{
    constexpr NeList LS = make_ne_list(W, S);
    const int kr = lane & 3, fr8 = lane >> 2;            // fragment row k and tile row/column
    int g = 0;                                           // stages so far
    for (int ch = ch0; ch * NE_CH < N; ch += step) {
        double acc[NE_SHARE][2];
#pragma unroll
        for (int j = 0; j < LS.n; ++j) acc[j][0] = acc[j][1] = 0.0;
        const int cnt = min(N - ch * NE_CH, NE_CH), nsub = (cnt + NE_SUB - 1) / NE_SUB;
        for (int it = 0; it < nsub; ++it, ++g) {
            bar_sync(NE_FULL + (g & 1), NE_THREADS);
            ne_pairs<W, S>(acc, rows + (size_t)(g & 1) * 2 * NE_SUB * NE_PD, min(NE_SUB, cnt - it * NE_SUB), kr, fr8);
            if (g + 2 < total) bar_arrive(NE_EMPTY + (g & 1), NE_THREADS);
        }
        double *part = parts + (size_t)ch * (NE_NT8 * 64);
#pragma unroll
        for (int j = 0; j < LS.n; ++j)
            *reinterpret_cast<double2 *>(part + LS.t[j] * 64 + fr8 * 8 + 2 * kr) = make_double2(acc[j][0], acc[j][1]);
    }
}

// Rows of one fragment's x and y gradients at four consecutive columns a0 ... a0 + 3, from its
// neighbours' Jacobian rows; the weight in column KT, zeros right of it.
__device__ __forceinline__ void ne_build4(double *rx, double *ry, const float4 (&v)[4], int a0, int KT, bool live, float pre,
                                          float diffx, float diffy, float wx, float wy)
{
    const float e[4][4] = {{v[0].x, v[1].x, v[2].x, v[3].x}, {v[0].y, v[1].y, v[2].y, v[3].y},
                           {v[0].z, v[1].z, v[2].z, v[3].z}, {v[0].w, v[1].w, v[2].w, v[3].w}};
    double ox[4], oy[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float x, y;
        chain_value(e[i], pre, diffx, diffy, x, y);
        const bool col = live && a0 + i < KT;
        x = col ? x : 0.0f;
        y = col ? y : 0.0f;
        if (live && a0 + i == KT) { x = wx; y = wy; }
        ox[i] = (double)x;
        oy[i] = (double)y;
    }
    *reinterpret_cast<double2 *>(rx) = make_double2(ox[0], ox[1]);
    *reinterpret_cast<double2 *>(rx + 2) = make_double2(ox[2], ox[3]);
    *reinterpret_cast<double2 *>(ry) = make_double2(oy[0], oy[1]);
    *reinterpret_cast<double2 *>(ry + 2) = make_double2(oy[2], oy[3]);
}

__global__ void __launch_bounds__(NE_THREADS, 2) k_normal_eq(DModel m, DBatch b)
{
    const int jn = jac_n(b);
    if ((int)blockIdx.y >= jn) return;
    const int f = b.jlist[blockIdx.y];
    const FrameCtl &ctl = b.ctl[f];
    if (blockIdx.x == 0 && threadIdx.x == 0) prof_count(b, KID_NORMAL_EQ);
    extern __shared__ __align__(16) double nesd[];  // rows [2][2*NE_SUB][NE_PD]
    const int KTP = m.KTP, KT = m.KT;
    __shared__ ChunkHead hd;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int N = ctl.N;
    const int nch = (N + NE_CH - 1) / NE_CH;
    // the blocks of a frame: all of a chunk's tiles each, or half of them while the chunks of the round
    // are fewer than half the blocks that fit (NE_SPREAD)
    const bool split = jn * nch <= NE_SPREAD;
    const int ch0 = split ? blockIdx.x / NE_SPLIT : blockIdx.x, half = split ? blockIdx.x % NE_SPLIT : 0;
    const int step = split ? gridDim.x / NE_SPLIT : gridDim.x;
    if (ch0 >= nch) return;
    int total = 0;                                   // stages of this block
    for (int ch = ch0; ch < nch; ch += step) total += (min(N - ch * NE_CH, NE_CH) + NE_SUB - 1) / NE_SUB;
    if (tid < 32 * NE_MMA_WARPS) {
        double *parts = b.ne_part + (size_t)f * NE_MAXCH * ne_part_stride8();
        if (!split) {
            switch (warp) {
            case 0: ne_update<0, 1>(nesd, parts, N, ch0, step, total, lane); break;
            case 1: ne_update<1, 1>(nesd, parts, N, ch0, step, total, lane); break;
            case 2: ne_update<2, 1>(nesd, parts, N, ch0, step, total, lane); break;
            default: ne_update<3, 1>(nesd, parts, N, ch0, step, total, lane); break;
            }
        } else {
            switch (warp + NE_MMA_WARPS * half) {
            case 0: ne_update<0, 2>(nesd, parts, N, ch0, step, total, lane); break;
            case 1: ne_update<1, 2>(nesd, parts, N, ch0, step, total, lane); break;
            case 2: ne_update<2, 2>(nesd, parts, N, ch0, step, total, lane); break;
            case 3: ne_update<3, 2>(nesd, parts, N, ch0, step, total, lane); break;
            case 4: ne_update<4, 2>(nesd, parts, N, ch0, step, total, lane); break;
            case 5: ne_update<5, 2>(nesd, parts, N, ch0, step, total, lane); break;
            case 6: ne_update<6, 2>(nesd, parts, N, ch0, step, total, lane); break;
            default: ne_update<7, 2>(nesd, parts, N, ch0, step, total, lane); break;
            }
        }
        return;
    }
    // a builder lane forms four columns (of every 32) of one fragment: its neighbours' rows come in
    // 16-byte loads, all of a fragment's in flight together
    constexpr int NG = (NE_P8 + 31) / 32, NF = NE_BUILDERS / 8;   // column groups; fragments built side by side
    const int bt = tid - 32 * NE_MMA_WARPS, a_low = 4 * (lane & 7), q_me = 4 * (bt >> 5) + (lane >> 3);
    const float *Jf = b.J + (size_t)f * NMAX * KTP;
    const int32_t *nb = b.nb + (size_t)f * 4 * NMAX;
    const float *fg = b.fgrad + (size_t)f * 5 * NMAX;
    int g = 0;
    for (int ch = ch0; ch < nch; ch += step) {
        const int c0 = ch * NE_CH, cnt = min(N, c0 + NE_CH) - c0;
        const int nsub = (cnt + NE_SUB - 1) / NE_SUB;
        bar_sync(NE_HEAD, NE_BUILDERS);              // the previous chunk's rows are built
        for (int q = bt; q < NE_CH; q += NE_BUILDERS) chunk_head(hd, fg, nb, c0, cnt, q);
        bar_sync(NE_HEAD, NE_BUILDERS);
        for (int it = 0; it < nsub; ++it, ++g) {
            double *rows = nesd + (size_t)(g & 1) * 2 * NE_SUB * NE_PD;
            float4 v[NE_SUB / NF][NG][4];
#pragma unroll
            for (int h = 0; h < NE_SUB / NF; ++h) {
                const int q = it * NE_SUB + q_me + h * NF;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float *row = Jf + (size_t)hd.nb[u][q] * KTP;
#pragma unroll
                    for (int gg = 0; gg < NG; ++gg) {
                        const int a = 32 * gg + a_low;
                        v[h][gg][u] = a < KTP ? __ldg(reinterpret_cast<const float4 *>(row + a)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    }
                }
            }
            if (g >= 2) bar_sync(NE_EMPTY + (g & 1), NE_THREADS);
#pragma unroll
            for (int h = 0; h < NE_SUB / NF; ++h) {
                const int ql = q_me + h * NF, q = it * NE_SUB + ql;
                const float pre = hd.pre[q], diffx = hd.dx[q], diffy = hd.dy[q];
                const float wx = (float)hd.w[2 * q], wy = (float)hd.w[2 * q + 1];
#pragma unroll
                for (int gg = 0; gg < NG; ++gg) {
                    const int a = 32 * gg + a_low;
                    if (a < NE_P8)
                        ne_build4(rows + (2 * ql) * NE_PD + a, rows + (2 * ql + 1) * NE_PD + a, v[h][gg], a, KT, q < cnt, pre,
                                  diffx, diffy, wx, wy);
                }
            }
            bar_arrive(NE_FULL + (g & 1), NE_THREADS);
        }
    }
}

// Sum of the chunk partials in chunk order: H = tau*S, g = -tau*(column KT of S).
__global__ void __launch_bounds__(NE_THREADS) k_normal_eq_reduce(DModel m, DBatch b)
{
    if ((int)blockIdx.y >= jac_n(b)) return;
    const int f = b.jlist[blockIdx.y];
    const FrameCtl &ctl = b.ctl[f];
    const int KTP = m.KTP, KT = m.KT;
    const int stride = ne_part_stride8();
    const int nch = (ctl.N + NE_CH - 1) / NE_CH;
    const double *part = b.ne_part + (size_t)f * NE_MAXCH * stride;
    const double tau = 25.0;
    float *H = b.H + (size_t)f * KTP * KTP;
    const float *Hb = b.Hb + (size_t)f * KTP * KTP;
    // one entry per thread: tile t, position p; the chunk values are loaded eight at a time
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < NE_NT8 * 64; e += gridDim.x * blockDim.x) {
        const int t = e >> 6, pos = e & 63;
        int bi, bj;
        ne_tile8(t, bi, bj);
        const int a = 8 * bi + (pos >> 3), c = 8 * bj + (pos & 7);
        if (a > c || c > KT || a >= KT) continue;
        const double *p = part + e;
        double s = 0.0;
        int q = 0;
        for (; q + 8 <= nch; q += 8) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = p[(size_t)(q + u) * stride];
#pragma unroll
            for (int u = 0; u < 8; ++u) s += v[u];
        }
        for (; q < nch; ++q) s += p[(size_t)q * stride];
        if (c < KT) {
            const float v = (float)(tau * s) + Hb[(size_t)a * KTP + c];
            H[(size_t)a * KTP + c] = v;
            H[(size_t)c * KTP + a] = v;
        } else {
            b.g[(size_t)f * KTP + a] = (float)(-tau * s) + b.gb[(size_t)f * KTP + a];
        }
    }
}

// ------------------------------------------------------------------------------------------
// Log-barrier gradient and Gauss-Newton Hessian (logbarrier_initializer.cu:1272-1843), one block per
// frame. They need only the accepted point, so they are formed beside the Jacobian and the
// normal equations of the image (on a stream of their own in the replayed rounds) and left in gb
// and the upper triangle of Hb; the reduction of the image's chunk sums adds them. 31 us per
// round (77 frames) that the round waited for before.

// The constraint rows are P columns wide: 88 for up to 87 unknowns, 128 for the wider systems of the
// tensor-core normal equations.
constexpr int BAR_WIDE = 128;
template <int P>
struct BarTiles {
    static constexpr int T8 = P / 8, NT8 = T8 * (T8 + 1) / 2, TPW = (NT8 + 7) / 8;
    int bi[NT8], bj[NT8];
};
template <int P>
__host__ __device__ constexpr BarTiles<P> make_bar_tiles()
{
    BarTiles<P> t{};
    int k = 0;
    for (int i = 0; i < BarTiles<P>::T8; ++i)
        for (int j = i; j < BarTiles<P>::T8; ++j) { t.bi[k] = i; t.bj[k] = j; ++k; }
    return t;
}

// The barrier Hessian's tensor-core updates of warp W over the 4 x 51 constraint rows (FP32
// in shared memory, pitch P), four consecutive rows per step.
template <int P, int W>
__device__ __forceinline__ void bar_hessian(double (&acc)[BarTiles<P>::TPW][2], const float *Fm, int kr, int fr8)
{
    constexpr BarTiles<P> TT = make_bar_tiles<P>();
    constexpr int NT = (BarTiles<P>::NT8 - W + 7) / 8;
    for (int t = 0; t < 4 * NL; t += 4) {
        const float *rk = Fm + (size_t)(t + kr) * P + fr8;
        double v[BarTiles<P>::T8];
#pragma unroll
        for (int c = 0; c < BarTiles<P>::T8; ++c) v[c] = (double)rk[8 * c];
#pragma unroll
        for (int j = 0; j < NT; ++j) dmma_884(acc[j][0], acc[j][1], v[TT.bi[W + 8 * j]], v[TT.bj[W + 8 * j]]);
    }
}

template <int P>
__global__ void __launch_bounds__(256) k_barrier_full(DModel m, DBatch b, int ft_bounds)
{
    constexpr int NE_P8 = P, NE_NT8 = BarTiles<P>::NT8, NE_TPW = BarTiles<P>::TPW, NE_T8 = BarTiles<P>::T8;
    if ((int)blockIdx.x >= jac_n(b)) return;
    const int f = b.jlist[blockIdx.x];
    if (threadIdx.x == 0) prof_count(b, KID_BARRIER);
    extern __shared__ float bsm[];
    const int KT = m.KT, KTP = m.KTP, K = m.K;
    float *Fm = bsm;                              // [4*NL][NE_P8], zeros right of KT
    __shared__ float G[4][NL];
    __shared__ float s_p[NL][3];
    __shared__ float s_v[NL][3], s_ivz[NL], s_ivz2[NL];
    __shared__ int s_lis[NL];
    __shared__ float s_R[9], s_dR[27];
    const int tid = threadIdx.x;
    const float *x = b.x + (size_t)f * KTP;       // the accepted point (= evaluation point)
    const float *R = b.R + f * 9, *dR = b.dR + f * 27;
    const float *tau = x + K;
    const float4 *geo = b.geo + (size_t)f * m.V;
    const float *cam = b.cam + f * 4;
    const float phix = cam[0], phiy = cam[1], cx = cam[2], cy = cam[3];
    const float fs = b.face_size[f];
    const float *bnd = b.bounds + (size_t)f * 4 * NL;
    const float *xl = b.xl + f * NL, *yl = b.yl + f * NL;
    if (tid >= 64 && tid < 64 + 36) {
        const int q = tid - 64;
        if (q < 9) s_R[q] = R[q]; else s_dR[q - 9] = dR[q - 9];
    }
    if (tid < NL) {
        const int v = m.lis[tid];
        s_lis[tid] = v;
        const float4 pv = geo[v];
        const float p0 = pv.x, p1 = pv.y, p2 = pv.z;
        s_p[tid][0] = p0; s_p[tid][1] = p1; s_p[tid][2] = p2;
        const float r1p = (R[0] * p0 + R[3] * p1) + R[6] * p2;
        const float r2p = (R[1] * p0 + R[4] * p1) + R[7] * p2;
        const float r3p = (R[2] * p0 + R[5] * p1) + R[8] * p2;
        const float xproj = phix * ((r1p + tau[0]) / (r3p + tau[2])) + cx;
        const float yproj = phiy * ((r2p + tau[1]) / (r3p + tau[2])) + cy;
        G[0][tid] = 0.0f - ((xl[tid] + bnd[0 * NL + tid] * fs) - xproj);
        G[1][tid] = 0.0f - ((yl[tid] + bnd[1 * NL + tid] * fs) - yproj);
        G[2][tid] = 0.0f - ((xproj - bnd[2 * NL + tid] * fs) - xl[tid]);
        G[3][tid] = 0.0f - ((yproj - bnd[3 * NL + tid] * fs) - yl[tid]);
        // camera point of the landmark and its inverse depth, once per landmark
        const float vx = r1p + tau[0], vy = r2p + tau[1], vz = r3p + tau[2];
        s_v[tid][0] = vx; s_v[tid][1] = vy; s_v[tid][2] = vz;
        const float ivz = 1.0f / vz;
        s_ivz[tid] = ivz;
        s_ivz2[tid] = ivz * ivz;
    }
    __syncthreads();
    // rows of the constraint gradients: warps take landmarks (i = warp + 8 q), lanes take
    // columns (a = lane + 32 c). Per column the basis values of all the warp's landmarks are
    // loaded before any is used, so that their loads are in flight together; the rotation and
    // its derivatives come from shared memory.
    constexpr int BQ = (NL + 7) / 8;
    const int warp = tid >> 5;
    for (int a = tid & 31; a < NE_P8; a += 32) {
        float eb[BQ][3];
#pragma unroll
        for (int q = 0; q < BQ; ++q) {
            const int i = warp + 8 * q;
            eb[q][0] = eb[q][1] = eb[q][2] = 0.0f;
            if (i < NL && a < K) {
                const float *ex = m.E + (size_t)s_lis[i] * 3 * m.KP;
                eb[q][0] = __ldg(ex + a);
                eb[q][1] = __ldg(ex + m.KP + a);
                eb[q][2] = __ldg(ex + 2 * m.KP + a);
            }
        }
#pragma unroll
        for (int q = 0; q < BQ; ++q) {
            const int i = warp + 8 * q;
            if (i >= NL) continue;
            const float p0 = s_p[i][0], p1 = s_p[i][1], p2 = s_p[i][2];
            const float vx = s_v[i][0], vy = s_v[i][1], vz = s_v[i][2];
            const float ivz = s_ivz[i], ivz2 = s_ivz2[i];
            float wx = 0.0f, wy = 0.0f;
            if (a < K) {
                const float RIX = eb[q][0], RIY = eb[q][1], RIZ = eb[q][2];
                const float dvx = (RIX * s_R[0] + RIY * s_R[3]) + RIZ * s_R[6];
                const float dvy = (RIX * s_R[1] + RIY * s_R[4]) + RIZ * s_R[7];
                const float dvz = (RIX * s_R[2] + RIY * s_R[5]) + RIZ * s_R[8];
                wx = (phix * ivz2) * (dvx * vz - dvz * vx);
                wy = (phiy * ivz2) * (dvy * vz - dvz * vy);
            } else if (a < KT) {
                const int cidx = a - K;
                if (cidx == 0) { wx = phix * ivz; wy = 0.0f; }
                else if (cidx == 1) { wx = 0.0f; wy = phiy * ivz; }
                else if (cidx == 2) { wx = ((-phix) * vx) * ivz2; wy = ((-phiy) * vy) * ivz2; }
                else {
                    const float *d = s_dR + 9 * (cidx - 3);
                    const float dvx = (d[0] * p0 + d[3] * p1) + d[6] * p2;
                    const float dvy = (d[1] * p0 + d[4] * p1) + d[7] * p2;
                    const float dvz = (d[2] * p0 + d[5] * p1) + d[8] * p2;
                    wx = (phix * ivz2) * (vz * dvx - vx * dvz);
                    wy = (phiy * ivz2) * (vz * dvy - vy * dvz);
                }
            }
            const bool live = a < KT;
            Fm[(0 * NL + i) * NE_P8 + a] = live ? -wx / G[0][i] : 0.0f;
            Fm[(1 * NL + i) * NE_P8 + a] = live ? -wy / G[1][i] : 0.0f;
            Fm[(2 * NL + i) * NE_P8 + a] = live ? wx / G[2][i] : 0.0f;
            Fm[(3 * NL + i) * NE_P8 + a] = live ? wy / G[3][i] : 0.0f;
        }
    }
    __syncthreads();
    const float *lb = m.eps_b + (ft_bounds ? 2 : 0) * K;
    const float *ub = m.eps_b + (ft_bounds ? 3 : 1) * K;
    float *H = b.Hb + (size_t)f * KTP * KTP;
    float *gv = b.gb + (size_t)f * KTP;
    // gradient: column sums over landmarks, set by set (the oracle's order)
    if (tid < KT) {
        const int a = tid;
        double gs = 0.0;
        for (int i = 0; i < NL; ++i)
            for (int s = 0; s < 4; ++s) gs += (double)Fm[(s * NL + i) * NE_P8 + a];
        float ga = (float)gs;
        if (a < K) {
            const float fub = x[a] - ub[a];
            const float flb = lb[a] - x[a];
            ga = ga + (-1.0f / fub + 1.0f / flb);
        }
        gv[a] = ga;
    }
    // Hessian: H = sum over the 204 constraint rows (set, then landmark) of F_t^T F_t, each entry
    // one FP64 fused multiply-add chain in row order, the oracle's order (the terms are
    // products of floats, exact in FP64). On the FP64 tensor cores: mma.sync m8n8k4 adds four
    // consecutive rows to an 8x8 tile as fma(a3, b3, fma(a2, b2, fma(a1, b1, fma(a0, b0, c)))),
    // the same chain; 66 tiles of the upper triangle, warp W taking tiles W, W + 8, ...
    {
        const int lane = tid & 31, warp = tid >> 5;
        const int kr = lane & 3, fr8 = lane >> 2;
        double acc[NE_TPW][2];
#pragma unroll
        for (int j = 0; j < NE_TPW; ++j) acc[j][0] = acc[j][1] = 0.0;
        switch (warp) {
        case 0: bar_hessian<P, 0>(acc, Fm, kr, fr8); break;
        case 1: bar_hessian<P, 1>(acc, Fm, kr, fr8); break;
        case 2: bar_hessian<P, 2>(acc, Fm, kr, fr8); break;
        case 3: bar_hessian<P, 3>(acc, Fm, kr, fr8); break;
        case 4: bar_hessian<P, 4>(acc, Fm, kr, fr8); break;
        case 5: bar_hessian<P, 5>(acc, Fm, kr, fr8); break;
        case 6: bar_hessian<P, 6>(acc, Fm, kr, fr8); break;
        default: bar_hessian<P, 7>(acc, Fm, kr, fr8); break;
        }
#pragma unroll
        for (int j = 0; j < NE_TPW; ++j) {
            const int t = warp + 8 * j;
            if (t >= NE_NT8) continue;
            int bi = 0, bj = t;                  // tile t: row by row of the upper triangle
            while (bj >= NE_T8 - bi) { bj -= NE_T8 - bi; ++bi; }
            bj += bi;
            const int a = 8 * bi + fr8;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int c = 8 * bj + 2 * kr + i;
                if (a > c || c >= KT) continue;
                float hv = (float)acc[j][i];
                if (a == c && a < K) {
                    const float fub = x[a] - ub[a];
                    const float flb = lb[a] - x[a];
                    const float nu = (float)(-1.0 / ((double)fub + 1e-12));
                    const float nl = (float)(1.0 / ((double)flb + 1e-12));
                    hv = hv + (nu * nu + nl * nl);
                }
                H[(size_t)a * KTP + c] = hv;
            }
        }
    }
}

// ------------------------------------------------------------------------------------------
// FP64 Cholesky solve (solver.h:70-105) of the shape system, one block per frame
// (tdi_cholesky.cuh), then the first trial of the line search.

constexpr int SV_THREADS = CH_THREADS;

__host__ __device__ __forceinline__ int sv_blocks(int n) { return n < 96 ? 6 : 8; }   // register blocks: n < 16 of them
// the solve, then the direction and the gradient (floats) and their products (doubles)
__host__ __device__ __forceinline__ size_t solve_smem(int n) { return chol_smem(n, sv_blocks(n)); }

template <int RB>
__device__ __forceinline__ void solve_frame(const DModel &m, const DBatch &b, const Cfg &c, int stage, int f,
                                            FrameCtl &ctl, double *sm)
{
    const int n = m.KT, KTP = m.KTP, K = m.K;
    const int tid = threadIdx.x;
    const float *H = b.H + (size_t)f * KTP * KTP;
    const float *gv = b.g + (size_t)f * KTP;
    float *d = b.d + (size_t)f * KTP;
    const double lam_d = (double)c.damping;      // damped solve: H + lambda I (0: undamped)
    double *xs;
    const bool ok = chol_solve<RB, false>(
        n, sm,
        [&](int i, int l) {
            const double h = (double)H[(size_t)l * KTP + i];
            return i == l ? h + lam_d : h;
        },
        [&](int l) { return (double)gv[l]; }, xs);
    if (!ok) {                                   // block-uniform
        for (int i = tid; i < n; i += SV_THREADS) d[i] = __int_as_float(0x7fc00000);
        if (tid == 0) {
            ctl.flags |= FLAG_CHOL_FAILED | FLAG_NAN_DIRECTION;
            end_shape_stage(c, ctl, stage, ctl.outer);
        }
        return;
    }
    // direction, its slope and the first trial point (the factor's memory is free again)
    double *prod = sm;
    float *dsm = reinterpret_cast<float *>(sm + n);
    if (tid < n) {
        const float dv = (float)(-xs[tid]);
        d[tid] = dv;
        dsm[tid] = dv;
        prod[tid] = (double)dv * (double)gv[tid];
    }
    __syncthreads();
    if (isnan(dsm[0])) {
        if (tid == 0) {
            ctl.flags |= FLAG_NAN_DIRECTION;
            end_shape_stage(c, ctl, stage, ctl.outer);
        }
        return;
    }
    const int n_upd = stage == ST_FINETUNE ? K : n;
    const float t = 1.0f;
    const float *x = b.x + (size_t)f * KTP;
    float *xl = b.x_ls + (size_t)f * KTP;
    for (int a = tid; a < n_upd; a += SV_THREADS) xl[a] = x[a] + t * dsm[a];
    if (tid == 0) {
        double dg = 0.0;
#pragma unroll 8
        for (int a = 0; a < n; ++a) dg += prod[a];       // (the products are exact)
        ctl.l2base = (float)dg;
        ctl.mode = M_TRIAL;
        ctl.t = t;
        const int maxit = stage == ST_RIGID ? c.max_iters_rigid : c.max_iters_finetune;
        // the trial's tau_z (left as it was when the stage does not update the pose)
        const float tz = n_upd > K + 2 ? x[K + 2] + t * dsm[K + 2] : xl[K + 2];
        if (tz < 0.0f) {
            ctl.flags |= FLAG_STUCK_NEG_TZ;
            end_shape_stage(c, ctl, stage, maxit);
        }
    }
}

// RB = 6 register blocks for up to 95 unknowns, 8 up to 127: one kernel each, so that the
// smaller system is not held to the larger one's register count
template <int RB>
__global__ void __launch_bounds__(SV_THREADS, RB == 6 ? 2 : 1) k_solve_t(DModel m, DBatch b, Cfg c, int stage)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) b.rcount[0] = 0;    // the round's renders are done
    if ((int)blockIdx.x >= jac_n(b)) return;
    const int f = b.jlist[blockIdx.x];
    FrameCtl &ctl = b.ctl[f];
    if (threadIdx.x == 0) prof_count(b, KID_SOLVE);
    extern __shared__ double ssm[];
    solve_frame<RB>(m, b, c, stage, f, ctl, ssm);
}

// ------------------------------------------------------------------------------------------
// Light fit (model_fitter.cu:981-1073), one block per frame, every render and decision of the
// frame's line search in one launch: objective -corr, Armijo test with alpha = beta = 0.5, the light
// system (derivative_computer.cu:235-312) as dI/dlambda = L t (R n), chain rule, 3x3 normal
// equations in FP64, Cholesky.
//
// The fit moves only the light: the raster, its neighbour maps, every fragment's dI/dlambda and
// so the neighbour differences of the chain rule stay as they are. They are formed once (32
// bytes per fragment, LightTerm); the shading terms and pixel positions stay in shared memory when
// they fit beside the region. An iteration is a render (shade, blur, gradients) whose
// gradient pass also sums the light system: nearly every trial is accepted (151 of 159 in a
// long fit), so a second pass over the fragments only for accepted trials costs more.
// It is bound by the latency of one block (a fit of 160 iterations in a batch of 77 decides the
// launch). As rounds over all frames, four launches each, that light fit took 6.7 ms; with a
// 512-thread block per frame and a separate pass for the system 2.8 ms; this form 1.8 ms
// (3.8 ms of a 1,024-frame fit, most of it one frame of 270 iterations).

struct __align__(16) LightTerm {
    float dh[3], dv[3];      // differences of dI/dlambda between the right/left, below/above neighbours
    float sxn, syn;          // normalised target gradient
};

struct LightSearch {
    double corr;
    float obj0, l2base, t, lam[3], dlam[3], glam[3];
    int iters, inner, trials;
};

constexpr int LIGHT_SMEM = 216 * 1024;       // the region, then 24 bytes per fragment when they fit
constexpr int LF_SUMS = 10;                  // the correlation, 6 entries of H's upper triangle, 3 of the right-hand side

__device__ __forceinline__ int light_region_bytes(const Region &r) { return (r.rw * r.ph + (r.rw + 2 * KRAD) * r.pb) * 4; }

// d = -(H^-1 g) of the 3x3 light system in the oracle's order (upper triangle of H in row order);
// NaN when a pivot is not positive.
__device__ __forceinline__ void light_solve(const float (&h)[6], const float (&g)[3], float (&d)[3])
{
    const double a00 = h[0], a10 = h[1], a20 = h[2], a11 = h[3], a21 = h[4], a22 = h[5];
    bool ok = a00 > 0.0;
    const double l00 = sqrt(a00), l10 = a10 / l00, l20 = a20 / l00;
    const double s1 = a11 - l10 * l10;
    ok = ok && s1 > 0.0;
    const double l11 = sqrt(s1), l21 = (a21 - l20 * l10) / l11;
    const double s2 = (a22 - l20 * l20) - l21 * l21;
    ok = ok && s2 > 0.0;
    const double l22 = sqrt(s2);
    const double y0 = (double)g[0] / l00, y1 = ((double)g[1] - l10 * y0) / l11;
    const double y2 = (((double)g[2] - l20 * y0) - l21 * y1) / l22;
    const double x2 = y2 / l22, x1 = (y1 - l21 * x2) / l11, x0 = ((y0 - l10 * x1) - l20 * x2) / l00;
    const float nan = __int_as_float(0x7fc00000);
    d[0] = ok ? (float)(-x0) : nan;
    d[1] = ok ? (float)(-x1) : nan;
    d[2] = ok ? (float)(-x2) : nan;
}

__global__ void __launch_bounds__(LIGHT_THREADS, 1) k_light_fit(DModel m, DBatch b, Cfg c, long max_rounds)
{
    constexpr int NT = LIGHT_THREADS;
    if ((int)blockIdx.x >= render_n(b)) return;
    const int f = b.rlist[blockIdx.x];
    FrameCtl &ctl = b.ctl[f];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (!ctl.render) {                           // the resolve refused the raster
        if (tid == 0) ctl.active = 0;
        return;
    }
    extern __shared__ __align__(16) float rsm[];
    __shared__ double s_sum[NT / 32][LF_SUMS];
    __shared__ double s_tot[LF_SUMS];
    __shared__ float s_q[3];                 // the rotated light of the next render
    __shared__ float s_lam[3];               // and the light itself
    __shared__ float s_R[9], s_tau[3];
    __shared__ LightSearch st;               // thread 0's, written back when the fit ends
    __shared__ int s_next;                   // after a render: 0 = done, 1 = another trial
    const Region r = make_region(ctl, rsm, b.img + (size_t)f * RIMG);
    const int N = ctl.N;
    const Fragment *frags = b.frag + (size_t)f * NMAX;
    const float4 *shc = b.shc + (size_t)f * NMAX;
    const float *sht = b.sht + (size_t)f * NMAX;
    const float Lint = b.Lint[f];
    // shading terms and region positions (-1: not the pixel's owner) in shared memory when they fit
    const int rbytes = r.A == rsm ? (light_region_bytes(r) + 15) & ~15 : 0;
    const bool cached = rbytes + N * 24 <= LIGHT_SMEM;
    float4 *c_sn = reinterpret_cast<float4 *>(reinterpret_cast<char *>(rsm) + rbytes);
    float *c_t = reinterpret_cast<float *>(c_sn + N);
    int *c_at = reinterpret_cast<int *>(c_t + N);
    if (tid < 9) s_R[tid] = b.R[f * 9 + tid];
    if (tid < 3) {
        s_tau[tid] = b.x[(size_t)f * m.KTP + m.K + tid];
        const float v = b.lam[f * 4 + tid];
        s_lam[tid] = v;
        st.lam[tid] = v;
        st.dlam[tid] = st.glam[tid] = 0.0f;
    }
    if (tid == 0) {
        st.obj0 = st.l2base = 0.0f;
        st.t = 1.0f;
        st.iters = ctl.iters_lambda;
        st.inner = ctl.inner;
        st.trials = 0;
    }
    region_clear<NT>(r, true);
    __syncthreads();
    // the terms (in the Jacobian's buffer), and while they are formed the rows dI/dlambda
    LightTerm *terms = reinterpret_cast<LightTerm *>(b.J + (size_t)f * NMAX * m.KTP);
    float4 *rows = reinterpret_cast<float4 *>(b.fgrad + (size_t)f * 5 * NMAX);
    for (int n = tid; n < N; n += NT) {
        const float4 sn = shc[n];
        const float t = sht[n];
        const float Lt = Lint * t;
        const float r0 = Lt * sn.x, r1 = Lt * sn.y, r2 = Lt * sn.z;
        float v[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) v[j] = (r0 * s_R[j] + r1 * s_R[j + 3]) + r2 * s_R[j + 6];
        rows[n] = make_float4(v[0], v[1], v[2], 0.0f);
        if (cached) {
            const uint32_t po = frags[n].pix_owner;
            c_sn[n] = sn;
            c_t[n] = t;
            c_at[n] = r.at(po & 0xFFFF) | (int)(po & 0x80000000u);
        }
    }
    __syncthreads();
    const float2 *tgn = b.tgn + (size_t)f * NPIX;
    const int32_t *nb = b.nb + (size_t)f * 4 * NMAX;
    for (int n = tid; n < N; n += NT) {
        const float4 k0 = rows[nb[n]], k1 = rows[nb[NMAX + n]], k2 = rows[nb[2 * NMAX + n]], k3 = rows[nb[3 * NMAX + n]];
        const float2 tg = tgn[frags[n].pix_owner & 0xFFFF];
        LightTerm t;
        t.dh[0] = k1.x - k0.x; t.dh[1] = k1.y - k0.y; t.dh[2] = k1.z - k0.z;
        t.dv[0] = k3.x - k2.x; t.dv[1] = k3.y - k2.y; t.dv[2] = k3.z - k2.z;
        t.sxn = tg.x; t.syn = tg.y;
        terms[n] = t;
    }
    if (tid == 0) {
        float q[3];
        light_terms(s_R, s_tau, s_lam, q);
        for (int j = 0; j < 3; ++j) s_q[j] = q[j];
    }
    __syncthreads();
    // a border pixel's neighbours wrap to pixel 0; elsewhere they lie beside it in the region
    const bool border = r.rw == DIM && r.rh == DIM;
    for (long round = 0; round < max_rounds; ++round) {
        const float q[3] = {s_q[0], s_q[1], s_q[2]};
        if (cached) {
            for (int n = tid; n < N; n += NT) {
                const int at = c_at[n];
                if (at < 0) {
                    const float4 sn = c_sn[n];
                    const float t = c_t[n];
                    const float Id = ((sn.x * q[0] + sn.y * q[1]) + sn.z * q[2]) - sn.w;
                    r.A[at & 0x7FFFFFFF] = t + (Lint * t) * Id;
                }
            }
        } else {
            region_shade<NT>(r, frags, shc, sht, N, q, Lint);
        }
        __syncthreads();
        region_blur<NT>(r, c);
        double acc[LF_SUMS];
#pragma unroll
        for (int e = 0; e < LF_SUMS; ++e) acc[e] = 0.0;
        for (int n = tid; n < N; n += NT) {
            const LightTerm t = terms[n];
            float v[4];
            if (cached && !border) {
                const int at = c_at[n] & 0x7FFFFFFF;
                v[0] = r.A[at + r.ph]; v[1] = r.A[at - r.ph]; v[2] = r.A[at + 1]; v[3] = r.A[at - 1];
            } else {
                int kr, kl, kd, ku;
                neighbour_pixels((int)(frags[n].pix_owner & 0xFFFF), kr, kl, kd, ku);
                v[0] = r.A[r.at(kr)]; v[1] = r.A[r.at(kl)]; v[2] = r.A[r.at(kd)]; v[3] = r.A[r.at(ku)];
            }
            float gx, gy, h, gxn, gyn;
            grad_of(v[0], v[1], v[2], v[3], gx, gy, h, gxn, gyn);
            const float pre = (float)(1.0 / (0.001 + (double)(h * h * h)));
            const float diffx = 2 * gx, diffy = 2 * gy;
            double ox[3], oy[3];
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const float X = (-diffy) * (-t.dh[j]) - (-diffx) * (-t.dv[j]);
                ox[j] = (double)(((-pre) * (-diffy)) * X);
                oy[j] = (double)((pre * (-diffx)) * X);
            }
            // (the products of floats are exact in FP64: a fused multiply-add rounds as their sum)
            const double sx = t.sxn, sy = t.syn;
            acc[0] += fma((double)gxn, sx, (double)gyn * sy);
            acc[1] += fma(ox[0], ox[0], oy[0] * oy[0]);
            acc[2] += fma(ox[0], ox[1], oy[0] * oy[1]);
            acc[3] += fma(ox[0], ox[2], oy[0] * oy[2]);
            acc[4] += fma(ox[1], ox[1], oy[1] * oy[1]);
            acc[5] += fma(ox[1], ox[2], oy[1] * oy[2]);
            acc[6] += fma(ox[2], ox[2], oy[2] * oy[2]);
            acc[7] += fma(sx, ox[0], sy * oy[0]);
            acc[8] += fma(sx, ox[1], sy * oy[1]);
            acc[9] += fma(sx, ox[2], sy * oy[2]);
        }
#pragma unroll
        for (int e = 0; e < LF_SUMS; ++e) {
            double v = acc[e];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) s_sum[warp][e] = v;
        }
        __syncthreads();
        if (warp == 0) {
            if (lane < LF_SUMS) {
                double v = 0.0;
#pragma unroll
                for (int w = 0; w < NT / 32; ++w) v += s_sum[w][lane];
                s_tot[lane] = v;
            }
            __syncwarp();
            if (lane == 0) {
                st.corr = s_tot[0];
                const float obj = -(float)s_tot[0];
                int next = 2;                            // accepted: a new direction
                if (round == 0) {
                    st.obj0 = obj;
                    st.iters++;
                } else {
                    st.inner++;
                    float l2 = st.l2base;
                    l2 = l2 * (0.5f * st.t);
                    if (obj < st.obj0 + l2) {
                        for (int j = 0; j < 3; ++j) st.lam[j] = s_lam[j];
                        st.obj0 = obj;
                        if (st.iters >= c.max_iters_lambda) next = 0; else st.iters++;
                    } else {
                        next = 1;
                        st.t = st.t * 0.5f;
                        if (st.t < 0.01f) next = 0;
                        else
                            for (int j = 0; j < 3; ++j) s_lam[j] = st.lam[j] + st.t * st.dlam[j];
                    }
                }
                if (next == 2) {
                    float h[6], g[3], dl[3];
                    for (int e = 0; e < 6; ++e) h[e] = (float)s_tot[1 + e];
                    for (int j = 0; j < 3; ++j) g[j] = (float)(-s_tot[7 + j]);
                    light_solve(h, g, dl);
                    const float l2 = (float)((double)dl[0] * g[0] + (double)dl[1] * g[1] + (double)dl[2] * g[2]);
                    st.l2base = l2;
                    st.trials = 1;
                    st.t = 1.0f;
                    for (int j = 0; j < 3; ++j) {
                        st.dlam[j] = dl[j];
                        st.glam[j] = g[j];
                        s_lam[j] = st.lam[j] + 1.0f * dl[j];
                    }
                    // the first trial's -g.d test (model_fitter.cu:1044-1048) does not depend on the trial
                    next = !((double)(-l2) < 0.0003 || !(l2 == l2));
                }
                float qn[3];
                light_terms(s_R, s_tau, s_lam, qn);
                for (int j = 0; j < 3; ++j) s_q[j] = qn[j];
                s_next = next;
            }
        }
        region_clear<NT>(r, false);          // for the next render (the gradients are read)
        __syncthreads();
        if (!s_next) break;
    }
    if (tid == 0) {
        ctl.active = 0;
        ctl.need_jac = 0;
        ctl.corr = st.corr;
        ctl.obj0 = st.obj0;
        ctl.iters_lambda = st.iters;
        ctl.inner = st.inner;
        ctl.l2base = st.l2base;
        ctl.t = st.t;
        if (st.trials) ctl.mode = M_TRIAL;
        for (int j = 0; j < 3; ++j) {
            b.lam[f * 4 + j] = st.lam[j];
            b.lam_ls[f * 4 + j] = s_lam[j];
            if (st.trials) { b.dlam[f * 4 + j] = st.dlam[j]; b.glam[f * 4 + j] = st.glam[j]; }
        }
    }
}

// Unblurred image and owner-triangle map of every rendering frame (renderer.cu:635-696), into a zero
// image and a map of -1. The shading terms are the raster's (shc, sht).
__global__ void __launch_bounds__(256) k_paint(DModel m, DBatch b, float *images, int32_t *tri_map)
{
    const int f = blockIdx.y;
    const FrameCtl &ctl = b.ctl[f];
    if (!ctl.render) return;
    float q[3];
    light_terms(b.R + f * 9, b.xe + (size_t)f * m.KTP + m.K, b.lam + f * 4, q);
    const float Lint = b.Lint[f];
    const size_t n0 = (size_t)f * NMAX;
    for (int n = blockIdx.x * 256 + threadIdx.x; n < ctl.N; n += gridDim.x * 256) {
        const Fragment fr = b.frag[n0 + n];
        if (!(fr.pix_owner & 0x80000000u)) continue;
        const float4 sn = b.shc[n0 + n];
        const float t = b.sht[n0 + n];
        const float Id = ((sn.x * q[0] + sn.y * q[1]) + sn.z * q[2]) - sn.w;
        const int p = fr.pix_owner & 0xFFFF;
        images[(size_t)f * NPIX + p] = t + (Lint * t) * Id;
        tri_map[(size_t)f * NPIX + p] = fr.tri;
    }
}

// Frames still running the current stage, in ascending order (one block, block-wide scan).
__global__ void __launch_bounds__(1024) k_compact_active(DBatch b, int *out)
{
    __shared__ int s_warp[32];
    __shared__ int s_base;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_base = 0;
    __syncthreads();
    for (int f0 = 0; f0 < b.F; f0 += 1024) {
        const int f = f0 + tid;
        const int a = (f < b.F) ? b.ctl[f].active : 0;
        const unsigned mask = __ballot_sync(0xffffffffu, a);
        if (lane == 0) s_warp[warp] = __popc(mask);
        __syncthreads();
        if (tid < 32) {
            int v = s_warp[tid], incl = v;
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (tid >= o) incl += t;
            }
            s_warp[tid] = incl - v;
        }
        __syncthreads();
        if (a) b.act[s_base + s_warp[warp] + __popc(mask & ((1u << lane) - 1u))] = f;
        __syncthreads();
        if (tid == 1023) s_base += s_warp[31] + __popc(mask);
        __syncthreads();
    }
    if (tid == 0) {
        out[0] = s_base;
        out[1] = *b.err;
    }
}

// ------------------------------------------------------------------------------------------
// The subject's shape and albedo (renderer.cu:866-883,941-951): one thread per coordinate of a
// vertex (rows 0..3V-1: X, Y, Z planes) or albedo entry (rows 3V..4V-1); the basis row is a
// sequential fused multiply-add chain over k from 0, then added to the mean. In place on m, t.

__global__ void k_apply_identity(int V, int KA, int KB, float *m, const float *I, const float *alpha, float *t,
                                 const float *T, const float *beta)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= 4 * V) return;
    if (r < 3 * V) {
        const float *row = I + (size_t)r * KA;
        float acc = 0.0f;
        for (int k = 0; k < KA; ++k) acc = fmaf(row[k], alpha[k], acc);
        if (KA) m[r] = m[r] + acc;
    } else {
        const int v = r - 3 * V;
        const float *row = T + (size_t)v * KB;
        float acc = 0.0f;
        for (int k = 0; k < KB; ++k) acc = fmaf(row[k], beta[k], acc);
        if (KB) t[v] = t[v] + acc;
    }
}

}  // namespace tdi
