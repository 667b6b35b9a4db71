// Differentiable render loss and its hand-written adjoint (tdi_batch_loss, tdi_batch_loss_backward).
//
// Loss of a frame: L = -sum_n (gxn_n gxsn_n + gyn_n gysn_n), the negated normalised-gradient
// correlation of 3DI's image term (funcs.cu:842-897, renderer.cu:725-729; the shape fit
// minimises tau_img L plus its barriers), evaluated in FP64 over a frozen set of fragments: the
// visibility (which triangle is sampled at which pixel, and the owner of each pixel) comes from
// the library's raster at the evaluation point; barycentrics, vertex geometry, shading, the
// 15-tap blur and the gradients are recomputed in FP64 from the state. With the visibility held,
// L is a smooth function of (epsilon, tau, u, lambda, L_intensity), and its gradient is exact.
//
// Backward pass (every buffer is recomputed from the state, nothing is kept from the forward):
//   1. per fragment: dL/d(normalised gradients) -> dL/d(gx, gy) through the normalisation ->
//      scattered into dL/d(blurred image) at the four neighbour pixels;
//   2. the transposed blur (the taps are symmetric and the border zero, so the transpose is the
//      same separable filter, applied in the opposite order);
//   3. per owner fragment: dL/d(pixel value) through the shading to the light (lambda, L), the
//      translation and rotation (through R^T (lambda - tau)), the object coordinates of its three
//      corners (normal and interpolated point) and the barycentrics; through those to the projected
//      corners, the camera coordinates and again the object coordinates. Everything after the
//      pixel is linear in it, so each fragment carries its own 3 x 3 object-coordinate terms
//      and nothing is accumulated per vertex (only about a fifth of the vertices have a fragment);
//   4. object coordinates -> expression coefficients by the basis-transpose product
//      dL/deps_k = sum_n sum_c E[v(n, c)][:,k] . dL/dP0(n, c); 5. dL/dR -> dL/du through dR/du.
// Steps 1 and 2 and the forward's image run in one kernel with a block per frame and the image
// region in shared memory (k_adj_image). 96 frames of the 53,490-vertex model, loss and gradients:
// 4.55 ms of kernels with dense per-vertex passes and whole-crop FP64 blurs in global memory,
// 1.49 ms in this form.
// Rotation in FP64: the reference's formula (rotation_header.cu:46-151) evaluated in double.

namespace tdi {

constexpr int AD_THREADS = 256;
constexpr int AD_GLOB = 16;   // per-frame FP64 accumulators: dR[9], dtau[3], dlam[3], dL

__device__ __forceinline__ double wsum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ void rotation_d(const float *uf, double *R, double *dR)
{
    const double u[3] = {uf[0], uf[1], uf[2]};
    const double th = sqrt((u[0] * u[0] + u[1] * u[1]) + u[2] * u[2]);
    const double un[3] = {u[0] / th, u[1] / th, u[2] / th};
    auto skew = [](double *S, const double *w) {
        S[0] = 0; S[1] = w[2]; S[2] = -w[1];
        S[3] = -w[2]; S[4] = 0; S[5] = w[0];
        S[6] = w[1]; S[7] = -w[0]; S[8] = 0;
    };
    auto mul = [](const double *A, const double *B, double *C) {
        for (int j = 0; j < 3; ++j)
            for (int i = 0; i < 3; ++i) C[3 * j + i] = A[i] * B[3 * j] + A[3 + i] * B[3 * j + 1] + A[6 + i] * B[3 * j + 2];
    };
    double Sn[9], Sn2[9], R1[3][9];
    skew(Sn, un);
    mul(Sn, Sn, Sn2);
    const double st = sin(th), cis = 1.0 - cos(th), tinv2 = 1.0 / (th * th);
    for (int i = 0; i < 9; ++i) R[i] = cis * Sn2[i] + ((i % 4 == 0) ? 1.0 : 0.0) + st * Sn[i];
    double IR[9];
    for (int i = 0; i < 9; ++i) IR[i] = ((i % 4 == 0) ? 1.0 : 0.0) - R[i];
    for (int a = 0; a < 3; ++a) {
        skew(R1[a], u);
        for (int i = 0; i < 9; ++i) R1[a][i] *= u[a];
        double R2[9], R3[9];
        const double *c = IR + 3 * a;
        for (int r = 0; r < 3; ++r)
            for (int q = 0; q < 3; ++q) R2[3 * r + q] = u[r] * c[q];
        for (int i = 0; i < 9; ++i) R1[a][i] += R2[i];
        for (int r = 0; r < 3; ++r)
            for (int q = 0; q < 3; ++q) R3[3 * r + q] = R1[a][3 * r + q] - R2[3 * q + r];
        mul(R3, R, dR + 9 * a);
        for (int i = 0; i < 9; ++i) dR[9 * a + i] *= tinv2;
    }
}

// Per frame: R, dR/du in FP64 (one thread per frame).
__global__ void k_adj_rot(DModel m, DBatch b, const float *x, int F, double *R64)
{
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= F) return;
    rotation_d(x + (size_t)f * m.KT + m.K + 3, R64 + (size_t)f * 36, R64 + (size_t)f * 36 + 9);
}

// FP64 vertex stage: object coordinates P0 = mean + E eps, geo64 [F][V][3]. (Camera coordinates and
// projections are formed by the fragments that need them: 24 bytes per vertex instead of 64.)
// A block takes AV_V vertices x 8 FPT frames with their basis rows and coefficients in shared
// memory as doubles, converted once; a thread forms one vertex of FPT frames by fused
// multiply-add chains over k. Bound by shared-memory reads (6 + FPT / 2 wavefronts per 3 FPT
// multiply-adds), so FPT is 8 for batches that fill it.
constexpr int AV_V = 32;

__host__ __device__ __forceinline__ size_t adj_vertex_smem(int KP, int FPT)
{
    return ((size_t)AV_V * 3 * (KP + 1) + (size_t)8 * FPT * KP) * sizeof(double);
}

template <int FPT>
__global__ void __launch_bounds__(256) k_adj_vertex_tiled(DModel m, const float *x, int F, double *geo64)
{
    extern __shared__ __align__(16) double avs[];
    constexpr int NF = 8 * FPT;
    const int KP = m.KP, K = m.K, KT = m.KT, W = KP + 1;    // row pitch KP + 1: lanes (vertices) on distinct banks
    double *Xs = avs;                                         // [KP][NF]
    double *Es = Xs + (size_t)NF * KP;                        // [AV_V][3][W]
    const int v0 = blockIdx.x * AV_V, f0 = blockIdx.y * NF, tid = threadIdx.x;
    const int vl = tid & 31, fg = tid >> 5, v = v0 + vl;
    const int nrow = min(AV_V, m.V - v0) * 3;
    {
        const int Q = KP >> 2;
        const uint32_t mq = 0xFFFFFFFFu / (uint32_t)Q + 1u;      // i / Q = umulhi(i, mq) for i < 2^16
        const float4 *e4 = reinterpret_cast<const float4 *>(m.E + (size_t)v0 * 3 * KP);
#pragma unroll 4
        for (int i = tid; i < nrow * Q; i += 256) {
            const int r = Q > 1 ? (int)__umulhi((uint32_t)i, mq) : i, k = 4 * (i - r * Q);
            const float4 e = __ldg(e4 + i);
            double *o = Es + (size_t)r * W + k;
            o[0] = e.x; o[1] = e.y; o[2] = e.z; o[3] = e.w;
        }
        // lanes take frames, so that the transposed coefficients are stored side by side
        for (int fl = tid % NF; fl < NF; fl += 256) {
            const float *xr = x + (size_t)min(f0 + fl, F - 1) * KT;
#pragma unroll 4
            for (int k = tid / NF; k < K; k += 256 / NF) Xs[(size_t)k * NF + fl] = (double)xr[k];
        }
    }
    __syncthreads();
    if (f0 + fg * FPT >= F || v >= m.V) return;
    const double *e0 = Es + (size_t)vl * 3 * W, *e1 = e0 + W, *e2 = e1 + W, *xk = Xs + fg * FPT;
    double acc[FPT][3];
#pragma unroll
    for (int q = 0; q < FPT; ++q) acc[q][0] = acc[q][1] = acc[q][2] = 0.0;
#pragma unroll 2
    for (int k = 0; k < K; ++k, xk += NF) {
        const double a0 = e0[k], a1 = e1[k], a2 = e2[k];
        double xv[FPT];
        if constexpr (FPT == 1) {
            xv[0] = xk[0];
        } else {
#pragma unroll
            for (int q = 0; q < FPT; q += 2) {
                const double2 t = *reinterpret_cast<const double2 *>(xk + q);
                xv[q] = t.x; xv[q + 1] = t.y;
            }
        }
#pragma unroll
        for (int q = 0; q < FPT; ++q) {
            acc[q][0] = fma(a0, xv[q], acc[q][0]);
            acc[q][1] = fma(a1, xv[q], acc[q][1]);
            acc[q][2] = fma(a2, xv[q], acc[q][2]);
        }
    }
    const double mean[3] = {(double)m.mean[v], (double)m.mean[(size_t)m.V + v], (double)m.mean[2 * (size_t)m.V + v]};
#pragma unroll
    for (int q = 0; q < FPT; ++q) {
        const int f = f0 + fg * FPT + q;
        if (f >= F) break;
        double *g = geo64 + ((size_t)f * m.V + v) * 3;
        for (int c = 0; c < 3; ++c) g[c] = mean[c] + acc[q][c];
    }
}

// Barycentrics of sample s in triangle (b, c, a) by Cramer's rule: s - a = alpha (b - a) + beta (c - a)
// (the same values as the reference's dot-product form, funcs.cu:961-977, in exact arithmetic),
// and their derivatives with respect to the three projected corners when d != nullptr:
// d[0..5] = dalpha/d(b, c, a) (x, y each), d[6..11] = dbeta/d(b, c, a).
__device__ __forceinline__ void bary_d(const double *pb, const double *pc, const double *pa, double sx, double sy,
                                       double &al, double &be, double *d)
{
    const double v0x = pb[0] - pa[0], v0y = pb[1] - pa[1], v1x = pc[0] - pa[0], v1y = pc[1] - pa[1];
    const double v2x = sx - pa[0], v2y = sy - pa[1];
    const double D = v0x * v1y - v0y * v1x;
    al = (v2x * v1y - v2y * v1x) / D;
    be = (v0x * v2y - v0y * v2x) / D;
    if (!d) return;
    // dD/dv0 = (v1y, -v1x), dD/dv1 = (-v0y, v0x)
    const double a0x = -al * v1y / D, a0y = al * v1x / D;                            // dalpha/dv0
    const double a1x = (-v2y + al * v0y) / D, a1y = (v2x - al * v0x) / D;            // dalpha/dv1
    const double a2x = v1y / D, a2y = -v1x / D;                                       // dalpha/dv2
    const double b0x = (v2y - be * v1y) / D, b0y = (-v2x + be * v1x) / D;            // dbeta/dv0
    const double b1x = be * v0y / D, b1y = -be * v0x / D;                             // dbeta/dv1
    const double b2x = -v0y / D, b2y = v0x / D;                                       // dbeta/dv2
    d[0] = a0x; d[1] = a0y; d[2] = a1x; d[3] = a1y; d[4] = -(a0x + a1x + a2x); d[5] = -(a0y + a1y + a2y);
    d[6] = b0x; d[7] = b0y; d[8] = b1x; d[9] = b1y; d[10] = -(b0x + b1x + b2x); d[11] = -(b0y + b1y + b2y);
}

struct AdjFrame {                 // a frame's inputs to the FP64 render
    const double *geo, *R;        // [V][3], [9] (then dR [27])
    const float *x, *lam, *cam;   // state [KT], light [3], camera [4]
    float L;
    int x0, y0, N, K;
    const Fragment *fr;
};

__device__ __forceinline__ AdjFrame adj_frame(const DModel &m, const DBatch &b, const float *x, const float *lam,
                                              const float *Lint, const double *geo64, const double *R64, int f)
{
    AdjFrame a;
    a.geo = geo64 + (size_t)f * m.V * 3;
    a.R = R64 + (size_t)f * 36;
    a.x = x + (size_t)f * m.KT;
    a.lam = lam + (size_t)f * 3;
    a.cam = b.cam + (size_t)f * 4;
    a.L = Lint[f];
    a.x0 = b.x0y0[2 * f];
    a.y0 = b.x0y0[2 * f + 1];
    a.N = b.ctl[f].N;
    a.K = m.K;
    a.fr = b.frag + (size_t)f * NMAX;
    return a;
}

// A fragment's corner: object coordinates, camera coordinates X = R P + tau, projection.
struct AdjCorner {
    double P[3], X[3], s[2];
};

__device__ __forceinline__ AdjCorner adj_corner(const AdjFrame &a, int v)
{
    AdjCorner c;
    const double *g = a.geo + (size_t)v * 3;
    for (int k = 0; k < 3; ++k) c.P[k] = g[k];
    for (int i = 0; i < 3; ++i)
        c.X[i] = (a.R[i] * c.P[0] + a.R[3 + i] * c.P[1]) + a.R[6 + i] * c.P[2] + (double)a.x[a.K + i];
    c.s[0] = (double)a.cam[0] * c.X[0] / c.X[2] + (double)a.cam[2];
    c.s[1] = (double)a.cam[1] * c.X[1] / c.X[2] + (double)a.cam[3];
    return c;
}

// The image of one frame in FP64 and its loss, one block per frame, the region around the fragments
// (their box + 8 px; beyond it the render is zero and the target does not reach a fragment's
// gradient) in shared memory with zero lines and columns around it:
//   the owner fragments' values painted into a zero image (fill_tex_im1, funcs.cu:800-817), the
//   15-tap blur, the gradients of render
//   and target at every fragment (fill_grads, funcs.cu:842-897), the loss; with BACK the adjoint of
//   the gradients scattered into dL/d(blurred image), the transposed blur, and dL/d(pixel value)
//   of every fragment's pixel out in dI.
// Both blur passes work in place (a thread's inputs are in registers before any output of its lines is
// written), so that one FP64 buffer of the region suffices: a face's region of up to 150 x 150 fits.
constexpr int AI_THREADS = 512;
constexpr int AI_SMEM = 216 * 1024;
constexpr size_t AI_GLOBAL = (size_t)(DIM + 2 * KRAD) * (DIM + 2 * RPAD);   // doubles of a region that does not fit
constexpr int AI_RUN_Y = 5;                            // row pass: outputs per lane (odd: lanes on distinct banks)
constexpr int AI_CHUNK = 32 * AI_RUN_Y;                // outputs of a line per warp and chunk; two chunks cover the crop
constexpr int AI_RUN_X = 16;                           // column pass: outputs per thread
static_assert(2 * AI_CHUNK >= DIM, "row pass covers a line in two chunks");

struct RegionD {                                       // [KRAD + rw + KRAD][ph], the image at (KRAD + x, RPAD + y)
    int rx0, ry0, rw, rh, ph;
    double *A;
    __device__ __forceinline__ int at(int p) const { return (KRAD + (p >> 8) - rx0) * ph + RPAD + ((p & 255) - ry0); }
};

// along y: a warp per line
__device__ __forceinline__ void adj_blur_rows(const RegionD &r, const double (&tap)[NTAPS])
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool two = r.rh > AI_CHUNK;
    for (int xl = warp; xl < r.rw; xl += AI_THREADS / 32) {
        double *line = r.A + (KRAD + xl) * r.ph + RPAD;
        double s[2][AI_RUN_Y];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int y0 = h * AI_CHUNK + lane * AI_RUN_Y;
#pragma unroll
            for (int o = 0; o < AI_RUN_Y; ++o) s[h][o] = 0.0;
            if (h == 0 ? y0 < r.rh : two && y0 < r.rh) {
#pragma unroll
                for (int t = 0; t < AI_RUN_Y + 2 * KRAD; ++t) {
                    // (a run that reaches past the line's padding reads zeros instead)
                    const double v = y0 + t - KRAD < r.rh + RPAD ? line[y0 + t - KRAD] : 0.0;
#pragma unroll
                    for (int o = 0; o < AI_RUN_Y; ++o)
                        if (t >= o && t - o <= 2 * KRAD) s[h][o] = fma(tap[t - o], v, s[h][o]);
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int o = 0; o < AI_RUN_Y; ++o) {
                const int y = h * AI_CHUNK + lane * AI_RUN_Y + o;
                if (y < r.rh) line[y] = s[h][o];
            }
    }
    __syncthreads();
}

// along x: a thread per column and segment, all segments of a column in the same step
__device__ __forceinline__ void adj_blur_cols(const RegionD &r, const double (&tap)[NTAPS])
{
    const int nseg = (r.rw + AI_RUN_X - 1) / AI_RUN_X, ncol = AI_THREADS / nseg;
    const int seg = threadIdx.x / ncol, yl = threadIdx.x - seg * ncol, x0 = seg * AI_RUN_X;
    for (int y0 = 0; y0 < r.rh; y0 += ncol) {
        const bool live = seg < nseg && y0 + yl < r.rh;
        double *col = r.A + x0 * r.ph + RPAD + y0 + yl;    // col[t ph]: the image at x0 - KRAD + t
        double s[AI_RUN_X];
        if (live) {
#pragma unroll
            for (int o = 0; o < AI_RUN_X; ++o) s[o] = 0.0;
#pragma unroll
            for (int t = 0; t < AI_RUN_X + 2 * KRAD; ++t) {
                const double v = x0 + t < r.rw + 2 * KRAD ? col[t * r.ph] : 0.0;
#pragma unroll
                for (int o = 0; o < AI_RUN_X; ++o)
                    if (t >= o && t - o <= 2 * KRAD) s[o] = fma(tap[t - o], v, s[o]);
            }
        }
        __syncthreads();
        if (live) {
#pragma unroll
            for (int o = 0; o < AI_RUN_X; ++o)
                if (x0 + o < r.rw) col[(KRAD + o) * r.ph] = s[o];
        }
    }
    __syncthreads();
}

// FP64 shading of the owner fragments (fill_diffuse_component..., newfuncs.cu:18-167), one value per
// fragment: 13 scattered loads each, so spread over the SMs instead of the image kernel's one block
// per frame (where they took 26 us of its 46).
__global__ void __launch_bounds__(AD_THREADS) k_adj_shade(DModel m, DBatch b, const float *x, const float *lam,
                                                          const float *Lint, const double *geo64, const double *R64,
                                                          double *shade)
{
    const int f = blockIdx.y;
    const AdjFrame a = adj_frame(m, b, x, lam, Lint, geo64, R64, f);
    for (int n = blockIdx.x * AD_THREADS + threadIdx.x; n < a.N; n += gridDim.x * AD_THREADS) {
        const Fragment fr = a.fr[n];
        if (!(fr.pix_owner >> 31)) continue;
        const int pix = fr.pix_owner & 0xFFFF;
        const int4 tq = __ldg(m.tl4 + fr.tri);
        const AdjCorner cb = adj_corner(a, tq.x), cc = adj_corner(a, tq.y), ca = adj_corner(a, tq.z);
        double al, be;
        bary_d(cb.s, cc.s, ca.s, (double)(a.x0 + (pix >> 8)), (double)(a.y0 + (pix & 255)), al, be, nullptr);
        const double gm = 1.0 - al - be;
        double v[3], w[3], nr[3];
        for (int k = 0; k < 3; ++k) { v[k] = cb.P[k] - ca.P[k]; w[k] = cc.P[k] - ca.P[k]; }
        nr[0] = v[1] * w[2] - v[2] * w[1]; nr[1] = v[2] * w[0] - v[0] * w[2]; nr[2] = v[0] * w[1] - v[1] * w[0];
        const double nn = sqrt(nr[0] * nr[0] + nr[1] * nr[1] + nr[2] * nr[2]);
        double Id = 0.0;
        for (int k = 0; k < 3; ++k) {
            double q = 0.0;
            for (int j = 0; j < 3; ++j) q += a.R[3 * k + j] * ((double)a.lam[j] - (double)a.x[m.K + j]);
            Id += nr[k] / nn * (q - (cb.P[k] * al + cc.P[k] * be + ca.P[k] * gm));
        }
        const double t = (double)m.tex[tq.x] * al + (double)m.tex[tq.y] * be + (double)m.tex[tq.z] * gm;
        shade[(size_t)f * NMAX + n] = t + (double)a.L * t * Id;
    }
}

template <bool BACK>
__global__ void __launch_bounds__(AI_THREADS, 1) k_adj_image(DBatch b, Cfg c, const double *shade,
                                                             const float *target, double *region, double *grads,
                                                             const double *gloss, double *loss, double *dI)
{
    extern __shared__ __align__(16) double ais[];
    __shared__ double s_red[AI_THREADS / 32];
    const int f = blockIdx.x, tid = threadIdx.x;
    const int N = b.ctl[f].N;
    const Fragment *frs = b.frag + (size_t)f * NMAX;
    if (N == 0) {
        if (tid == 0 && loss) loss[f] = 0.0;
        return;
    }
    const Region rf = make_region(b.ctl[f], nullptr, nullptr);
    RegionD r{rf.rx0, rf.ry0, rf.rw, rf.rh, rf.ph, nullptr};
    const size_t need = (size_t)(r.rw + 2 * KRAD) * r.ph;
    r.A = need * sizeof(double) <= AI_SMEM ? ais : region + (size_t)f * AI_GLOBAL;
    double tap[NTAPS];
#pragma unroll
    for (int j = 0; j < NTAPS; ++j) tap[j] = (double)c.taps[2 * KRAD - j];
    auto clear = [&](double *p, int n) { for (int i = tid; i < n; i += AI_THREADS) p[i] = 0.0; };
    clear(r.A, (int)need);                               // the zero lines and columns stay zero
    __syncthreads();
    const double *sh = shade + (size_t)f * NMAX;
#pragma unroll 4
    for (int n = tid; n < N; n += AI_THREADS) {
        const uint32_t po = frs[n].pix_owner;
        const double v = sh[n];
        if (po >> 31) r.A[r.at(po & 0xFFFF)] = v;
    }
    __syncthreads();
    adj_blur_rows(r, tap);
    adj_blur_cols(r, tap);
    // the render's gradients, kept while the target takes the region
    double *gr = grads + (size_t)f * 2 * NMAX;
    for (int n = tid; n < N; n += AI_THREADS) {
        int kr, kl, kd, ku;
        neighbour_pixels((int)(frs[n].pix_owner & 0xFFFF), kr, kl, kd, ku);
        gr[n] = 0.5 * (r.A[r.at(kr)] - r.A[r.at(kl)]);
        gr[NMAX + n] = 0.5 * (r.A[r.at(kd)] - r.A[r.at(ku)]);
    }
    __syncthreads();
    const float *tg = target + (size_t)f * NPIX;
    for (int i = tid; i < r.rw * r.rh; i += AI_THREADS) {
        const int xl = i / r.rh, yl = i - xl * r.rh;
        r.A[(KRAD + xl) * r.ph + RPAD + yl] = (double)tg[(r.rx0 + xl) * DIM + r.ry0 + yl];
    }
    __syncthreads();
    adj_blur_rows(r, tap);
    adj_blur_cols(r, tap);
    double part = 0.0;
    const double gl = BACK ? gloss[f] : 0.0;
    for (int n = tid; n < N; n += AI_THREADS) {
        int kr, kl, kd, ku;
        neighbour_pixels((int)(frs[n].pix_owner & 0xFFFF), kr, kl, kd, ku);
        const double gx = gr[n], gy = gr[NMAX + n];
        const double rr = sqrt(4.0 * gx * gx + 4.0 * gy * gy), h = 1e-16 + rr;
        const double sx = 0.5 * (r.A[r.at(kr)] - r.A[r.at(kl)]), sy = 0.5 * (r.A[r.at(kd)] - r.A[r.at(ku)]);
        const double hs = 1e-16 + sqrt(4.0 * sx * sx + 4.0 * sy * sy);
        const double sxn = 2.0 * sx / hs, syn = 2.0 * sy / hs;
        part += -((2.0 * gx / h) * sxn + (2.0 * gy / h) * syn);
        if (BACK) {
            const double dgxn = -gl * sxn, dgyn = -gl * syn;         // dL/d(2 gx / h), dL/d(2 gy / h)
            const double dh = rr > 0.0 ? 1.0 / rr : 0.0;
            const double hx = 4.0 * gx * dh, hy = 4.0 * gy * dh;     // dh/dgx, dh/dgy
            const double dgx = dgxn * (2.0 / h - 2.0 * gx * hx / (h * h)) + dgyn * (-2.0 * gy * hx / (h * h));
            const double dgy = dgxn * (-2.0 * gx * hy / (h * h)) + dgyn * (2.0 / h - 2.0 * gy * hy / (h * h));
            gr[n] = 0.5 * dgx;                           // in place of the render's gradient
            gr[NMAX + n] = 0.5 * dgy;
        }
    }
    if (loss) {
        part = wsum(part);
        if ((tid & 31) == 0) s_red[tid >> 5] = part;
        __syncthreads();
        if (tid < 32) {
            const double t = wsum(tid < AI_THREADS / 32 ? s_red[tid] : 0.0);
            if (tid == 0) loss[f] = t;
        }
    }
    if (!BACK) return;
    __syncthreads();
    // dL/d(blurred image), then the transposed blur: the column pass first, then the row pass
    clear(r.A, (int)need);
    __syncthreads();
    for (int n = tid; n < N; n += AI_THREADS) {
        int kr, kl, kd, ku;
        neighbour_pixels((int)(frs[n].pix_owner & 0xFFFF), kr, kl, kd, ku);
        const double dgx = gr[n], dgy = gr[NMAX + n];
        atomicAdd(r.A + r.at(kr), dgx);
        atomicAdd(r.A + r.at(kl), -dgx);
        atomicAdd(r.A + r.at(kd), dgy);
        atomicAdd(r.A + r.at(ku), -dgy);
    }
    __syncthreads();
    adj_blur_cols(r, tap);
    adj_blur_rows(r, tap);
    double *out = dI + (size_t)f * NMAX;
    for (int n = tid; n < N; n += AI_THREADS) {
        const uint32_t po = frs[n].pix_owner;
        out[n] = (po >> 31) ? r.A[r.at(po & 0xFFFF)] : 0.0;
    }
}

// Adjoint of the shading of the owner fragments: dL/dpixel -> light, pose, and the object coordinates
// of the three corners (dP [N][9]: corners b, c, a), through the normal and the interpolated point,
// and through the barycentrics, the projections and the camera coordinates. Per-frame terms
// (glob: dR[9], dtau[3], dlam[3], dL) summed per block, one atomic per block and entry.
__global__ void __launch_bounds__(AD_THREADS) k_adj_frag_back(DModel m, DBatch b, const float *x, const float *lam,
                                                              const float *Lint, const double *geo64, const double *R64,
                                                              const double *dI, double *dP0, double *glob)
{
    __shared__ double s_acc[AD_THREADS / 32][AD_GLOB];
    const int f = blockIdx.y;
    const AdjFrame a = adj_frame(m, b, x, lam, Lint, geo64, R64, f);
    if ((int)(blockIdx.x * AD_THREADS) >= a.N) return;
    double acc[AD_GLOB];
#pragma unroll
    for (int i = 0; i < AD_GLOB; ++i) acc[i] = 0.0;
    double dl[3];
    for (int j = 0; j < 3; ++j) dl[j] = (double)a.lam[j] - (double)a.x[m.K + j];
    for (int n = blockIdx.x * AD_THREADS + threadIdx.x; n < a.N; n += gridDim.x * AD_THREADS) {
        double dP[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
        const double dIn = dI[(size_t)f * NMAX + n];
        if (dIn != 0.0) {
            const Fragment fr = a.fr[n];
            const int pix = fr.pix_owner & 0xFFFF;
            const int4 tq = __ldg(m.tl4 + fr.tri);
            const AdjCorner cr[3] = {adj_corner(a, tq.x), adj_corner(a, tq.y), adj_corner(a, tq.z)};    // b, c, a
            double al, be, db[12];
            bary_d(cr[0].s, cr[1].s, cr[2].s, (double)(a.x0 + (pix >> 8)), (double)(a.y0 + (pix & 255)), al, be, db);
            const double gm = 1.0 - al - be;
            double v[3], w[3], nr[3], nh[3], q[3], p[3];
            for (int k = 0; k < 3; ++k) { v[k] = cr[0].P[k] - cr[2].P[k]; w[k] = cr[1].P[k] - cr[2].P[k]; }
            nr[0] = v[1] * w[2] - v[2] * w[1]; nr[1] = v[2] * w[0] - v[0] * w[2]; nr[2] = v[0] * w[1] - v[1] * w[0];
            const double nn = sqrt(nr[0] * nr[0] + nr[1] * nr[1] + nr[2] * nr[2]);
            double Id = 0.0;
            for (int k = 0; k < 3; ++k) {
                nh[k] = nr[k] / nn;
                q[k] = 0.0;
                for (int j = 0; j < 3; ++j) q[k] += a.R[3 * k + j] * dl[j];
                p[k] = cr[0].P[k] * al + cr[1].P[k] * be + cr[2].P[k] * gm;
                Id += nh[k] * (q[k] - p[k]);
            }
            const double tb = m.tex[tq.x], tc = m.tex[tq.y], ta = m.tex[tq.z];
            const double t = tb * al + tc * be + ta * gm, L = a.L;
            const double dt = dIn * (1.0 + L * Id), dId = dIn * L * t;
            acc[15] += dIn * t * Id;                                         // dL/dL_intensity
            double dal = dt * (tb - ta), dbe = dt * (tc - ta);
            double dn[3];
            for (int k = 0; k < 3; ++k) {
                dn[k] = dId * (q[k] - p[k]);
                const double dq = dId * nh[k], dp = -dId * nh[k];
                for (int j = 0; j < 3; ++j) {
                    acc[3 * k + j] += dq * dl[j];                            // dR[3k + j]
                    const double dd = dq * a.R[3 * k + j];
                    acc[12 + j] += dd;                                       // dlambda_j
                    acc[9 + j] -= dd;                                        // dtau_j
                }
                dal += dp * (cr[0].P[k] - cr[2].P[k]);
                dbe += dp * (cr[1].P[k] - cr[2].P[k]);
                dP[0][k] += al * dp; dP[1][k] += be * dp; dP[2][k] += gm * dp;
            }
            const double nd = nh[0] * dn[0] + nh[1] * dn[1] + nh[2] * dn[2];
            double dnr[3];
            for (int k = 0; k < 3; ++k) dnr[k] = (dn[k] - nh[k] * nd) / nn;
            // nr = v x w: dL/dv = w x dnr, dL/dw = dnr x v
            const double dv[3] = {w[1] * dnr[2] - w[2] * dnr[1], w[2] * dnr[0] - w[0] * dnr[2], w[0] * dnr[1] - w[1] * dnr[0]};
            const double dw[3] = {dnr[1] * v[2] - dnr[2] * v[1], dnr[2] * v[0] - dnr[0] * v[2], dnr[0] * v[1] - dnr[1] * v[0]};
            for (int k = 0; k < 3; ++k) {
                dP[0][k] += dv[k];
                dP[1][k] += dw[k];
                dP[2][k] -= dv[k] + dw[k];
            }
            // projected corners -> camera coordinates -> translation, rotation, object coordinates
            for (int ci = 0; ci < 3; ++ci) {
                const double sx = dal * db[2 * ci] + dbe * db[6 + 2 * ci], sy = dal * db[2 * ci + 1] + dbe * db[6 + 2 * ci + 1];
                const double X = cr[ci].X[0], Y = cr[ci].X[1], Z = cr[ci].X[2];
                const double gx = sx * a.cam[0], gy = sy * a.cam[1];
                const double gc[3] = {gx / Z, gy / Z, -(gx * X + gy * Y) / (Z * Z)};
                for (int j = 0; j < 3; ++j) {
                    double s = 0.0;
                    for (int i = 0; i < 3; ++i) {
                        acc[i + 3 * j] += gc[i] * cr[ci].P[j];               // dR[i + 3j] (X = R P0 + tau)
                        s += gc[i] * a.R[i + 3 * j];
                    }
                    dP[ci][j] += s;
                    acc[9 + j] += gc[j];
                }
            }
        }
        double *o = dP0 + ((size_t)f * NMAX + n) * 9;
        for (int ci = 0; ci < 3; ++ci)
            for (int j = 0; j < 3; ++j) o[3 * ci + j] = dP[ci][j];
    }
#pragma unroll
    for (int i = 0; i < AD_GLOB; ++i) {
        const double w = wsum(acc[i]);
        if ((threadIdx.x & 31) == 0) s_acc[threadIdx.x >> 5][i] = w;
    }
    __syncthreads();
    if (threadIdx.x < AD_GLOB) {
        double t = 0.0;
        for (int w = 0; w < AD_THREADS / 32; ++w) t += s_acc[w][threadIdx.x];
        atomicAdd(glob + (size_t)f * AD_GLOB + threadIdx.x, t);
    }
}

// Basis-transpose product dL/deps_k = sum_n sum_c sum_j E[v(n, c)][j][k] dP0[n][c][j]: a block takes a
// share of one frame's fragments, a thread four columns of every FL-th fragment (nine 16-byte
// basis loads in flight); the block's sums are added with one atomic per column. Bound by the
// basis rows' reads (2.8 KB per fragment, mostly from L2) and the conversions to FP64.
constexpr int AE_THREADS = 256, AE_CH = 64;

__global__ void __launch_bounds__(AE_THREADS) k_adj_eps(DModel m, DBatch b, const double *dP0, double *geps)
{
    extern __shared__ __align__(16) double aes[];        // [FL][KP] the threads' sums
    __shared__ double s_d[AE_CH * 9];
    __shared__ int s_v[AE_CH * 3];
    const int f = blockIdx.y, tid = threadIdx.x, N = b.ctl[f].N;
    const int Q = m.KP >> 2, FL = AE_THREADS / Q;        // column groups; fragments taken side by side
    const int kq = tid % Q, fl = tid / Q;
    const Fragment *frs = b.frag + (size_t)f * NMAX;
    if ((int)blockIdx.x * AE_CH >= N) return;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int c0 = blockIdx.x * AE_CH; c0 < N; c0 += gridDim.x * AE_CH) {
        const int cnt = min(AE_CH, N - c0);
        for (int i = tid; i < cnt * 9; i += AE_THREADS) s_d[i] = dP0[((size_t)f * NMAX + c0) * 9 + i];
        if (tid < cnt) {
            const int4 tq = __ldg(m.tl4 + frs[c0 + tid].tri);
            s_v[3 * tid] = tq.x; s_v[3 * tid + 1] = tq.y; s_v[3 * tid + 2] = tq.z;
        }
        __syncthreads();
        if (fl < FL)
            for (int n = fl; n < cnt; n += FL) {
                float4 e[9];
#pragma unroll
                for (int q = 0; q < 9; ++q)
                    e[q] = __ldg(reinterpret_cast<const float4 *>(m.E + ((size_t)s_v[3 * n + q / 3] * 3 + q % 3) * m.KP) + kq);
#pragma unroll
                for (int q = 0; q < 9; ++q) {
                    const double d = s_d[9 * n + q];
                    acc[0] = fma((double)e[q].x, d, acc[0]);
                    acc[1] = fma((double)e[q].y, d, acc[1]);
                    acc[2] = fma((double)e[q].z, d, acc[2]);
                    acc[3] = fma((double)e[q].w, d, acc[3]);
                }
            }
        __syncthreads();
    }
    if (fl < FL) {
#pragma unroll
        for (int j = 0; j < 4; ++j) aes[(size_t)fl * m.KP + 4 * kq + j] = acc[j];
    }
    __syncthreads();
    for (int k = tid; k < m.K; k += AE_THREADS) {
        double t = 0.0;
        for (int q = 0; q < FL; ++q) t += aes[(size_t)q * m.KP + k];
        atomicAdd(geps + (size_t)f * m.K + k, t);
    }
}

// Gradients out: x [F][K+6] (epsilon, tau, u through dR/du), lambda [F][3], L [F]; one block per frame.
__global__ void k_adj_final(DModel m, const double *R64, const double *glob, const double *geps, double *gx,
                            double *glam, double *gL)
{
    const int f = blockIdx.x, tid = threadIdx.x;
    const double *G = glob + (size_t)f * AD_GLOB, *dR = R64 + (size_t)f * 36 + 9;
    double *o = gx + (size_t)f * m.KT;
    for (int k = tid; k < m.K; k += blockDim.x) o[k] = geps[(size_t)f * m.K + k];
    if (tid < 3) {
        o[m.K + tid] = G[9 + tid];
        double s = 0.0;
        for (int i = 0; i < 9; ++i) s += G[i] * dR[9 * tid + i];
        o[m.K + 3 + tid] = s;
        if (glam) glam[(size_t)f * 3 + tid] = G[12 + tid];
    }
    if (tid == 0 && gL) gL[f] = G[15];
}

// The caller's states [F][K+6] into the batch's evaluation states (pitch KTP).
__global__ void k_adj_set_x(DModel m, DBatch b, const float *x, int F)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= F * m.KT) return;
    const int f = i / m.KT, a = i - f * m.KT;
    b.x[(size_t)f * m.KTP + a] = x[i];
    b.x_ls[(size_t)f * m.KTP + a] = x[i];
}

}  // namespace tdi
