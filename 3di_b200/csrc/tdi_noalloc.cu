// Visibility of one frame without any device allocation (tdi_raster_noalloc in tdi.h).
//
// Some callers of this library cannot call cudaMalloc: a plugin hosted by an application
// that owns every byte of device memory through its own pool and only lends out buffers,
// code that runs with a device-memory budget fixed before it starts, or a per-frame loop
// that must not stall on the allocator. tdi_batch_raster needs a batch, and a batch
// allocates its working set. This entry point takes the frame's projected vertices and
// triangles and writes the fragment list into buffers the caller already owns; its own
// working memory -- the 64-bit depth-key buffer of the 256x256 crop and one fragment count
// per triangle -- is a fixed array compiled into the library's device image.
//
// Limits and sharing rules:
//  * at most NOALLOC_MAX_TRIANGLES (131,072) triangles; larger meshes are rejected;
//  * the array costs 640 KiB on every device that loads the library, until the process ends;
//  * every call on a device uses the same array. Each call first resets the depth keys, so
//    nothing carries over between calls, but two calls whose kernels overlap on the GPU
//    (different streams, or different host threads) race on the array and give undefined
//    fragments. Serialise calls on one stream.
//  * the triangle corners are caller-owned device memory that the host cannot check: a
//    triangle with a corner outside [0, n_vertices) is skipped on the device before any
//    vertex is read and the call's flags get TDI_FLAG_BAD_INDEX;
//  * every call looks up the array's device address (cudaGetSymbolAddress, which allocates
//    nothing) with the caller's device current, so a device reset between calls is safe. The
//    first call on a device also loads the library's device code there; make that first call
//    before any stream capture begins.

namespace tdi {

constexpr int NOALLOC_MAX_TRIANGLES = 131072;
constexpr int NA_RC = 8;          // blocks of the resolve's cluster
constexpr int NA_WARPS = 32;      // warps per block of the resolve
constexpr int NA_PER_WARP = ((NOALLOC_MAX_TRIANGLES + NA_RC * NA_WARPS * 32 - 1) / (NA_RC * NA_WARPS * 32)) * 32;

struct NoAllocScratch {
    unsigned long long zbuf[NPIX];                 // depth keys of the crop (512 KiB)
    uint8_t tri_cnt[NOALLOC_MAX_TRIANGLES];        // fragments per triangle (128 KiB)
};

static __device__ __align__(256) NoAllocScratch g_noalloc_scratch;

// One frame is three launches in the caller's stream, each as wide as its work: the depth keys
// reset, the depth pass over all SMs, and the resolve in one cluster. As one cluster of 8
// blocks that evaluated every triangle's samples up to three times the frame took 111 us; it is
// latency that bounds it, so the depth pass decides most triangles early (no_sample_inside) and the
// resolve gathers the triangles that have fragments into dense warps: 25 us with the launches' gaps.

// The array keeps the previous call's keys: reset them (every key compares smaller).
__global__ void __launch_bounds__(256) k_noalloc_reset(NoAllocScratch *scr, uint32_t *flags_out)
{
    ulonglong2 *z = reinterpret_cast<ulonglong2 *>(scr->zbuf);
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < NPIX / 2) z[i] = make_ulonglong2(~0ull, ~0ull);
    if (i == 0) *flags_out = 0u;
}

__global__ void __launch_bounds__(256) k_noalloc_depth(const float *xp, const float *yp, const float *zc,
                                                       const int32_t *tl, int V, int T, int x0, int y0,
                                                       NoAllocScratch *scr, uint32_t *flags_out)
{
    unsigned long long *zb = scr->zbuf;
    uint32_t flags = 0;
    for (int idx = blockIdx.x * 256 + threadIdx.x; idx < T; idx += gridDim.x * 256) {
        const int ib = __ldg(tl + idx), ic = __ldg(tl + T + idx), ia = __ldg(tl + 2 * T + idx);
        int nf = 0;
        // corners outside the vertex arrays: the triangle has no fragments and no vertex is read; the
        // resolve skips it through its zero count
        if ((uint32_t)ib < (uint32_t)V && (uint32_t)ic < (uint32_t)V && (uint32_t)ia < (uint32_t)V) {
            const float bx = __ldg(xp + ib), by = __ldg(yp + ib), cx = __ldg(xp + ic), cy = __ldg(yp + ic);
            const float ax = __ldg(xp + ia), ay = __ldg(yp + ia), Z = __ldg(zc + ib);
            if (!no_sample_inside(bx, by, cx, cy, ax, ay)) {
                const unsigned long long key = zkey(0, Z, idx);
                nf = tri_samples(bx, by, cx, cy, ax, ay, x0, y0, flags,
                                 [&](int, uint32_t px, float, float) { atomicMin(zb + px, key); });
                if (nf && !(Z > 0.0f)) flags |= FLAG_OUT_OF_DOMAIN;
            }
        } else {
            flags |= FLAG_BAD_INDEX;
        }
        scr->tri_cnt[idx] = (uint8_t)nf;
    }
    if (flags) atomicOr(flags_out, flags);
}

// Survivors in slot order with the batch raster's owner rule, as one cluster: each warp takes a
// contiguous range of triangles, lists those with fragments and evaluates them 32 at a time, once to
// count the survivors per slot row and once to write them (16-byte records: pixel | owner<<31,
// triangle, float bits of alpha and beta).
__global__ void __cluster_dims__(NA_RC, 1, 1) __launch_bounds__(1024)
k_raster_noalloc(const float *xp, const float *yp, const float *zc, const int32_t *tl, int T, int x0, int y0,
                 const NoAllocScratch *scr, int32_t *frags, int capacity, int32_t *count, uint32_t *flags_out)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    __shared__ uint16_t s_list[NA_WARPS][NA_PER_WARP];     // offsets in the warp's range
    __shared__ uint32_t s_cnt[NA_WARPS][NTMP];
    __shared__ uint32_t s_off[NA_WARPS][NTMP];
    __shared__ uint32_t s_blk[NTMP];
    __shared__ int s_bbox[4];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    const unsigned long long *zb = scr->zbuf;
    if (tid == 0) {
        s_bbox[0] = s_bbox[2] = 1 << 30;
        s_bbox[1] = s_bbox[3] = -1;
    }
    const int gwarps = NA_RC * NA_WARPS;
    const int per_warp = ((T + gwarps * 32 - 1) / (gwarps * 32)) * 32;
    const int t_begin = (rank * NA_WARPS + warp) * per_warp;
    const int t_end = min(T, t_begin + per_warp);
    // the warp's triangles with fragments, ascending (the counts are loaded ahead, eight steps at a time)
    uint16_t *list = s_list[warp];
    int L = 0;
    for (int base = t_begin; base < t_end; base += 32 * 8) {
        uint32_t c[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int idx = base + 32 * u + lane;
            c[u] = idx < t_end ? scr->tri_cnt[idx] : 0u;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const unsigned msk = __ballot_sync(0xffffffffu, c[u] != 0);
            if (c[u]) list[L + __popc(msk & lt_mask)] = (uint16_t)(base + 32 * u + lane - t_begin);
            L += __popc(msk);
        }
    }
    __syncwarp();
    // visit(r, survives, record) for the four slot rows of every listed triangle, whole warps
    auto for_survivors = [&](auto &&visit) {
        for (int e0 = 0; e0 < L; e0 += 32) {
            const int e = e0 + lane;
            bool sv[NTMP] = {false, false, false, false}, own[NTMP] = {false, false, false, false};
            uint32_t pix[NTMP] = {0, 0, 0, 0};
            float al[NTMP] = {0, 0, 0, 0}, be[NTMP] = {0, 0, 0, 0};
            int idx = 0;
            if (e < L) {
                idx = t_begin + list[e];
                const int ib = __ldg(tl + idx), ic = __ldg(tl + T + idx), ia = __ldg(tl + 2 * T + idx);
                const float Z = __ldg(zc + ib);
                const uint32_t zbits = __float_as_uint(Z) & 0x7FFFFFFFu;
                const unsigned long long mykey = zkey(0, Z, idx);
                uint32_t fl2 = 0;
                tri_samples(__ldg(xp + ib), __ldg(yp + ib), __ldg(xp + ic), __ldg(yp + ic), __ldg(xp + ia), __ldg(yp + ia),
                            x0, y0, fl2, [&](int r, uint32_t px, float a, float bb) {
                                const unsigned long long k = __ldcg(zb + px);
#pragma unroll
                                for (int q = 0; q < NTMP; ++q)
                                    if (q == r) {
                                        sv[q] = survives(k, 0, zbits) && !(q == 0 && idx == 0);
                                        own[q] = k == mykey;
                                        pix[q] = px; al[q] = a; be[q] = bb;
                                    }
                            });
            }
#pragma unroll
            for (int r = 0; r < NTMP; ++r)
                visit(r, sv[r], make_int4((int)(pix[r] | (own[r] ? 0x80000000u : 0u)), idx, __float_as_int(al[r]),
                                          __float_as_int(be[r])));
        }
    };
    uint32_t cnt[NTMP] = {0, 0, 0, 0};
    for_survivors([&](int r, bool sv, const int4 &) { cnt[r] += __popc(__ballot_sync(0xffffffffu, sv)); });
    if (lane == 0)
        for (int r = 0; r < NTMP; ++r) s_cnt[warp][r] = cnt[r];
    __syncthreads();
    if (warp < NTMP) {
        // per row: exclusive scan over the block's warps (lane = warp index)
        const uint32_t v = s_cnt[lane][warp];
        uint32_t inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        s_off[lane][warp] = inc - v;
        if (lane == 31) s_blk[warp] = inc;
    }
    cluster.sync();
    uint32_t base[NTMP];
    {
        uint32_t tot[NTMP] = {0, 0, 0, 0}, blkoff[NTMP] = {0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < NA_RC; ++q) {
            const uint32_t *rb = cluster.map_shared_rank(s_blk, q);
#pragma unroll
            for (int r = 0; r < NTMP; ++r) {
                const uint32_t v = rb[r];
                if (q == rank) blkoff[r] = tot[r];
                tot[r] += v;
            }
        }
        uint32_t acc = 0;
#pragma unroll
        for (int r = 0; r < NTMP; ++r) {
            base[r] = acc + blkoff[r] + s_off[warp][r];
            acc += tot[r];
        }
        if (tid == 0 && rank == 0) {
            *count = (int32_t)min(acc, (uint32_t)capacity);
            uint32_t fl = 0;
            if (acc > (uint32_t)capacity) fl |= FLAG_OVERFLOW;
            if (acc < 1000u || acc > 52000u) fl |= FLAG_RENDER_SKIPPED;
            if (acc > 25600u) fl |= FLAG_OUT_OF_DOMAIN;
            if (fl) atomicOr(flags_out, fl);
        }
    }
    int bx0 = 1 << 30, bx1 = -1, by0 = 1 << 30, by1 = -1;
    for_survivors([&](int r, bool sv, const int4 &rec) {
        const unsigned msk = __ballot_sync(0xffffffffu, sv);
        if (sv) {
            const uint32_t pos = base[r] + __popc(msk & lt_mask);
            if (pos < (uint32_t)capacity) {
                int32_t *o = frags + (size_t)pos * 4;
                o[0] = rec.x; o[1] = rec.y; o[2] = rec.z; o[3] = rec.w;
            }
            const int px = (rec.x >> 8) & 255, py = rec.x & 255;
            bx0 = min(bx0, px); bx1 = max(bx1, px);
            by0 = min(by0, py); by1 = max(by1, py);
        }
        base[r] += __popc(msk);
    });
    if (bx1 >= 0) {
        atomicMin(&s_bbox[0], bx0); atomicMax(&s_bbox[1], bx1);
        atomicMin(&s_bbox[2], by0); atomicMax(&s_bbox[3], by1);
    }
    __syncthreads();
    // (a block's survivors on the crop's border flag the frame, whichever block holds them)
    if (tid == 0 && s_bbox[1] >= 0 && (s_bbox[0] < 1 || s_bbox[1] > DIM - 2 || s_bbox[2] < 1 || s_bbox[3] > DIM - 2))
        atomicOr(flags_out, FLAG_OUT_OF_DOMAIN);
    cluster.sync();                                    // no block leaves while its shared memory may be read
}

}  // namespace tdi

extern "C" tdi_status tdi_raster_noalloc(const float *xp, const float *yp, const float *zc,
                                         const int32_t *triangles, int32_t n_vertices,
                                         int32_t n_triangles, int32_t x0, int32_t y0,
                                         int32_t *fragments, int32_t capacity, int32_t *count,
                                         uint32_t *flags, void *stream)
{
    using namespace tdi;
    if (!xp || !yp || !zc || !triangles || !fragments || !count || !flags)
        return fail(TDI_ERR_INVALID, "tdi_raster_noalloc: null pointer");
    if (n_vertices <= 0 || n_triangles <= 0 || capacity <= 0)
        return fail(TDI_ERR_INVALID, "tdi_raster_noalloc: sizes must be positive");
    if (n_triangles > NOALLOC_MAX_TRIANGLES)
        return fail(TDI_ERR_CAPACITY, "tdi_raster_noalloc: at most 131072 triangles (fixed working array)");
    // The array's name is only a host-side stand-in: the kernel needs its address on the
    // current device, looked up on every call (no allocation; valid after a device reset).
    NoAllocScratch *scr = nullptr;
    cudaError_t e0 = cudaGetSymbolAddress((void **)&scr, g_noalloc_scratch);
    if (e0 != cudaSuccess)
        return fail(TDI_ERR_CUDA, std::string("tdi_raster_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(e0));
    cudaStream_t s = (cudaStream_t)stream;
    k_noalloc_reset<<<NPIX / 512, 256, 0, s>>>(scr, flags);
    k_noalloc_depth<<<(n_triangles + 255) / 256, 256, 0, s>>>(xp, yp, zc, triangles, n_vertices, n_triangles, x0, y0, scr,
                                                              flags);
    k_raster_noalloc<<<NA_RC, 1024, 0, s>>>(xp, yp, zc, triangles, n_triangles, x0, y0, scr, fragments, capacity, count,
                                            flags);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(TDI_ERR_CUDA, std::string("tdi_raster_noalloc: launch: ") + cudaGetErrorString(e));
    return TDI_OK;
}
