// Sky view factor: per-patch visibility rays, bit-packed, and the annulus sums.
//
// Visibility (src/kernels/geometry.cu:77-119, src/svf.py:81-106): for every
// pixel and sky patch the shadow sweep toward the patch centre decides whether
// a building blocks the patch (S = 0) and whether vegetation was seen in front
// of the first building hit (V = 1).  The reference stores three float32
// cubes [rows, cols, 153] (7.3 GB at 2000^2); here each (pixel, patch) keeps
// 2 bits, 40 bytes per pixel, in the layout described in solweig_b200.h.
//
// Reduce (geometry.cu:121-159): annulus-weighted sums over bands and the four
// half-sky sectors become per-band popcounts of the packed words, summed in
// the reference's band order so the float64 planes agree to the last bit.
#include "ceiling.cuh"
#include "shadow.cuh"

namespace solweig {

constexpr int kSvfWarps = 8;        // warps per block
constexpr int kSvfPatchGroup = 32;  // patches per packed word

struct SvfRayParams {
    int rows, cols, patches, capacity;
    double hmax;
};

// grid.x: chunks of 32 consecutive pixels; grid.y: patch word (32 patches)
// from word0 on.  geo32: the packed float4 geometry (exact float32 values) or
// null.  With `ceiling` (one launch per word, grid.y = 1): the word's
// ray-ceiling planes [32][pixels], on which the walk stops.
// WALK: 0 float64 rasters, 1 packed geometry.
// 32 registers (8 blocks per SM): the walks are latency-bound and full
// occupancy outweighs the few spills (SVF 5.7 ms faster at 2000^2 than at
// 40 registers).
template <int WALK>
__global__ void __launch_bounds__(32 * kSvfWarps, 8) svf_visibility_kernel(
    const double* __restrict__ dsm, const double* __restrict__ top, const double* __restrict__ bot,
    const float4* __restrict__ geo32, const uint8_t* __restrict__ flags, SvfRayParams prm,
    const int2* __restrict__ ray, const double* __restrict__ dz, const int32_t* __restrict__ lengths,
    uint32_t* __restrict__ masks, int word0, const float2* __restrict__ ceiling) {
    __shared__ uint8_t state[kSvfPatchGroup][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long pixels = (long long)prm.rows * prm.cols;
    // the block's 32 pixels: an 8 x 4 (columns x rows) tile, whose walks are
    // more alike than those of 32 pixels in a row
    const int tiles_x = (prm.cols + 7) / 8;
    const int rr = (blockIdx.x / tiles_x) * 4 + (lane >> 3), cc = (blockIdx.x % tiles_x) * 8 + (lane & 7);
    const int word = word0 + blockIdx.y;
    const bool valid = rr < prm.rows && cc < prm.cols;
    const int r = valid ? rr : 0, c = valid ? cc : 0;
    const long long p = (long long)r * prm.cols + c;
    const double a = valid ? dsm[p] : 0.0;
    const double top_p = valid ? top[p] : 0.0;
    const bool bush = valid && (flags[p] & 2);
    for (int j = warp; j < kSvfPatchGroup; j += kSvfWarps) {
        const int patch = word * kSvfPatchGroup + j;
        uint8_t st = 0;
        if (valid && patch < prm.patches) {
            const long long base = (long long)patch * prm.capacity;
            const int K = lengths[patch];
            const float2* ceil_j = ceiling ? ceiling + (long long)j * pixels : nullptr;
            ShadowResult s;
            if (WALK == 1) {
                s = shadow_walk_geo(GeoF32x4{geo32}, prm.rows, prm.cols, r, c, a, top_p, bush, 0.0, ray + base,
                                    dz + base, K, prm.hmax, true, ceil_j);
            } else {
                s = shadow_walk_geo(GeoF64{dsm, top, bot}, prm.rows, prm.cols, r, c, a, top_p, bush, 0.0,
                                    ray + base, dz + base, K, prm.hmax, true, ceil_j);
            }
            st = (s.shadowed ? 0 : 1) | (s.ever ? 2 : 0);
        }
        state[j][lane] = st;
    }
    __syncthreads();
    if (warp < 2 && valid) {
        uint32_t bits = 0;
#pragma unroll
        for (int j = 0; j < kSvfPatchGroup; ++j) bits |= (uint32_t)((state[j][lane] >> warp) & 1u) << j;
        masks[((long long)warp * SOLWEIG_MASK_WORDS + word) * pixels + p] = bits;
    }
}

// The form on the packed geometry with ceilings, exits and step records, one
// warp per 8 x 4 pixel tile walking all patches of the word in turn (grid.x:
// tiles / 8, one word per launch): the warps of a block carry similar work --
// each walks all 32 patches of its own pixels, so the uneven lengths of single
// walks even out -- and each pixel's two bits are assembled in registers, so no
// warp waits at a barrier.  Same bits as svf_visibility_kernel.
__global__ void __launch_bounds__(32 * kSvfWarps, 8) svf_visibility_warp_kernel(
    const float4* __restrict__ geo32, const float* __restrict__ height, const uint8_t* __restrict__ flags,
    SvfRayParams prm, const double* __restrict__ dz, const int32_t* __restrict__ lengths, uint32_t* __restrict__ masks,
    int word, const float2* __restrict__ ceiling, const int* __restrict__ exits, const int2* __restrict__ rec,
    int kpitch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long pixels = (long long)prm.rows * prm.cols;
    const int tiles_x = (prm.cols + 7) / 8;
    const long long ntiles = (long long)tiles_x * ((prm.rows + 3) / 4);
    const long long tile = (long long)blockIdx.x * kSvfWarps + warp;
    if (tile >= ntiles) return;  // the whole warp
    const int rr = (int)(tile / tiles_x) * 4 + (lane >> 3), cc = (int)(tile % tiles_x) * 8 + (lane & 7);
    if (rr >= prm.rows || cc >= prm.cols) return;
    const long long p = (long long)rr * prm.cols + cc;
    const bool bush = flags[p] & 2;
    const float hmax = __double2float_ru(prm.hmax);
    uint32_t sbits = 0u, vbits = 0u;
    for (int j = 0; j < kSvfPatchGroup; ++j) {
        const int patch = word * kSvfPatchGroup + j;
        if (patch >= prm.patches) break;
        const int K = lengths[patch];
        const int* e = exits + (long long)j * (prm.rows + prm.cols);
        const int kend = min(K, min(__ldg(&e[rr]), __ldg(&e[prm.rows + cc])));
        const ShadowResult s = shadow_walk_packed(geo32, height, ceiling + (long long)j * pixels, (uint32_t)p, bush, 0.0,
                                                  rec + (long long)j * kpitch,
                                                  dz + (long long)patch * prm.capacity, K, kend, hmax);
        sbits |= (s.shadowed ? 0u : 1u) << j;
        vbits |= (s.ever ? 1u : 0u) << j;
    }
    masks[(long long)word * pixels + p] = sbits;
    masks[((long long)SOLWEIG_MASK_WORDS + word) * pixels + p] = vbits;
}

struct SvfReduceParams {
    long long pixels;
    int nbands;
    double trans;
    uint32_t band_mask[SOLWEIG_MAX_BANDS][SOLWEIG_MASK_WORDS];
    uint32_t sector_mask[4][SOLWEIG_MASK_WORDS];
    double wf[SOLWEIG_MAX_BANDS], wa[SOLWEIG_MAX_BANDS];
    double w_cos[SOLWEIG_MAX_BANDS], w_sin[SOLWEIG_MAX_BANDS];  // omega*cos, omega*sin per band
};

__global__ void __launch_bounds__(256) svf_reduce_kernel(const uint32_t* __restrict__ masks,
                                                         const double* __restrict__ bot,
                                                         SvfReduceParams prm,
                                                         double* __restrict__ planes,
                                                         float* __restrict__ veg_sums,
                                                         uint8_t* __restrict__ sky_counts) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= prm.pixels) return;
    const long long n = prm.pixels;
    uint32_t S[SOLWEIG_MASK_WORDS], V[SOLWEIG_MASK_WORDS];
#pragma unroll
    for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
        S[w] = masks[(long long)w * n + p];
        V[w] = masks[(long long)(SOLWEIG_MASK_WORDS + w) * n + p];
    }
    double v[15];
#pragma unroll
    for (int i = 0; i < 15; ++i) v[i] = 0.0;
    double vc = 0.0, vs = 0.0, oc = 0.0, os = 0.0;
    for (int b = 0; b < prm.nbands; ++b) {
        int cnt[15];
#pragma unroll
        for (int i = 0; i < 15; ++i) cnt[i] = 0;
        int nveg = 0, nobst = 0, nsky = 0;
#pragma unroll
        for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
            const uint32_t bm = prm.band_mask[b][w];
            if (bm == 0u) continue;  // a band lies in one or two words: 12 of 40 pairs are left
            const uint32_t sh = S[w] & bm;                // shmat == 1
            const uint32_t vg = ~(S[w] & V[w]) & bm;      // vegmat == 1
            const uint32_t vb = ~(~S[w] & V[w]) & bm;     // vbmat == 1
            cnt[0] += __popc(sh);
            cnt[5] += __popc(vg);
            cnt[10] += __popc(vb);
#pragma unroll
            for (int d = 0; d < 4; ++d) {
                const uint32_t sm = prm.sector_mask[d][w];
                cnt[1 + d] += __popc(sh & sm);
                cnt[6 + d] += __popc(vg & sm);
                cnt[11 + d] += __popc(vb & sm);
            }
            nveg += __popc(V[w] & bm);
            nobst += __popc(~(S[w] & ~V[w]) & bm);
            nsky += __popc(S[w] & ~V[w] & bm);
        }
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            v[g * 5] += prm.wf[b] * cnt[g * 5];
#pragma unroll
            for (int d = 1; d < 5; ++d) v[g * 5 + d] += prm.wa[b] * cnt[g * 5 + d];
        }
        vc += prm.w_cos[b] * nveg;
        vs += prm.w_sin[b] * nveg;
        oc += prm.w_cos[b] * nobst;
        os += prm.w_sin[b] * nobst;
        sky_counts[(long long)b * n + p] = (uint8_t)nsky;
    }
    const double eps = 3.0459e-4;
    v[2] += eps;
    v[3] += eps;
    const double last = bot[p] == 0.0 ? eps : 0.0;
    v[7] += last;
    v[8] += last;
    v[12] += last;
    v[13] += last;
#pragma unroll
    for (int i = 0; i < 15; ++i) {
        if (v[i] > 1.0) v[i] = 1.0;
        planes[(long long)i * n + p] = v[i];
    }
    planes[15 * n + p] = v[0] - (1.0 - v[5]) * (1.0 - prm.trans);
    veg_sums[p] = (float)vc;
    veg_sums[n + p] = (float)vs;
    veg_sums[2 * n + p] = (float)oc;
    veg_sums[3 * n + p] = (float)os;
}

// Packed masks -> the reference's float cubes [pixels][patches].
// VEC consecutive values a thread, 1024 a block; VEC = 4 needs 16-byte aligned
// cubes.  What bounds it is the write of the cubes: with one value a thread and a
// 64-bit division each 142 us for 512 x 448 pixels and 153 patches (421 MB),
// with four 85.
constexpr int kUnpackValues = 1024;
template <int VEC>
__global__ void __launch_bounds__(256) svf_unpack_kernel(const uint32_t* __restrict__ masks,
                                                         long long pixels, int patches,
                                                         float* __restrict__ shm,
                                                         float* __restrict__ vegm,
                                                         float* __restrict__ vbm) {
    const long long first = (long long)blockIdx.x * kUnpackValues, n = pixels * patches;
    const long long p0 = first / patches;
    const int k0 = (int)(first - p0 * patches);
    for (int t = threadIdx.x * VEC; t < kUnpackValues; t += 256 * VEC) {
        const long long i = first + t;
        if (i >= n) return;
        const int ahead = (k0 + t) / patches;
        long long p = p0 + ahead;
        int k = k0 + t - ahead * patches;
        uint32_t S = 0u, V = 0u;
        float sh[VEC], vg[VEC], vb[VEC];
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
            if (e == 0 || (k & 31) == 0) {
                S = V = 0u;
                if (p < pixels) {
                    S = masks[(long long)(k >> 5) * pixels + p];
                    V = masks[(long long)(SOLWEIG_MASK_WORDS + (k >> 5)) * pixels + p];
                }
            }
            const bool s = (S >> (k & 31)) & 1u, v = (V >> (k & 31)) & 1u;
            sh[e] = s ? 1.f : 0.f;
            vg[e] = s && v ? 0.f : 1.f;
            vb[e] = !s && v ? 0.f : 1.f;
            if (++k == patches) {
                k = 0;
                ++p;
            }
        }
        auto put = [&](float* cube, const float (&x)[VEC]) {
            if (!cube) return;
            if (VEC == 4 && i + VEC <= n) {
                *reinterpret_cast<float4*>(cube + i) = make_float4(x[0], x[1 % VEC], x[2 % VEC], x[3 % VEC]);
                return;
            }
#pragma unroll
            for (int e = 0; e < VEC; ++e)
                if (i + e < n) cube[i + e] = x[e];
        };
        put(shm, sh);
        put(vegm, vg);
        put(vbm, vb);
    }
}

// Reference float cubes [pixels][patches] -> packed S/V words.
__global__ void __launch_bounds__(256) svf_pack_kernel(const float* __restrict__ shm,
                                                       const float* __restrict__ vegm,
                                                       const float* __restrict__ vbm,
                                                       long long pixels, int patches,
                                                       uint32_t* __restrict__ masks) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= pixels) return;
    for (int w = 0; w < SOLWEIG_MASK_WORDS; ++w) {
        uint32_t s = 0, v = 0;
        for (int b = 0; b < 32; ++b) {
            const int k = w * 32 + b;
            if (k >= patches) break;
            const long long i = p * patches + k;
            if (shm[i] == 1.0f) s |= 1u << b;
            if (vegm[i] == 0.0f || vbm[i] == 0.0f) v |= 1u << b;
        }
        masks[(long long)w * pixels + p] = s;
        masks[(long long)(SOLWEIG_MASK_WORDS + w) * pixels + p] = v;
    }
}

__global__ void __launch_bounds__(256) diffsh_kernel(const float* __restrict__ sh,
                                                     const float* __restrict__ veg,
                                                     float* __restrict__ out, long long n,
                                                     float trans) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = __fsub_rn(sh[i], __fmul_rn(__fsub_rn(1.0f, veg[i]), __fsub_rn(1.0f, trans)));
}

}  // namespace solweig

using namespace solweig;

extern "C" int solweig_svf_reduce(const uint32_t* masks, const double* vegdem2, int64_t pixels,
                                  const SolweigSkyLayout* layout, const double* band_weights,
                                  const uint8_t* sectors, double transmissivity, double* planes,
                                  float* veg_sums, uint8_t* sky_band_counts, void* stream) {
    SOLWEIG_CHECK_ARG(masks && vegdem2 && layout && band_weights && sectors && planes && veg_sums &&
                          sky_band_counts && pixels > 0,
                      "solweig_svf_reduce: bad arguments");
    SOLWEIG_CHECK_ARG(layout->nbands > 0 && layout->nbands <= SOLWEIG_MAX_BANDS &&
                          layout->patches > 0 && layout->patches <= SOLWEIG_MASK_WORDS * 32,
                      "solweig_svf_reduce: bad layout");
    const int patches = layout->patches;
    cudaStream_t st = as_stream(stream);
    SvfReduceParams q{};
    q.pixels = pixels;
    q.nbands = layout->nbands;
    q.trans = transmissivity;
    for (int k = 0; k < patches; ++k) {
        const int b = layout->band_of_patch[k];
        SOLWEIG_CHECK_ARG(b >= 0 && b < layout->nbands, "solweig_svf: bad band of patch %d", k);
        q.band_mask[b][k >> 5] |= 1u << (k & 31);
        for (int d = 0; d < 4; ++d)
            if (sectors[k] & (1u << d)) q.sector_mask[d][k >> 5] |= 1u << (k & 31);
    }
    for (int b = 0; b < layout->nbands; ++b) {
        q.wf[b] = band_weights[2 * b];
        q.wa[b] = band_weights[2 * b + 1];
        q.w_cos[b] = (double)layout->band_omega[b] * (double)layout->band_cos[b];
        q.w_sin[b] = (double)layout->band_omega[b] * (double)layout->band_sin[b];
    }
    svf_reduce_kernel<<<blocks_for(pixels, 256), 256, 0, st>>>(masks, vegdem2, q, planes, veg_sums,
                                                               sky_band_counts);
    SOLWEIG_CHECK_LAUNCH("svf_reduce_kernel");
    return SOLWEIG_OK;
}

extern "C" int solweig_svf_pack(const float* shmat, const float* vegmat, const float* vbmat,
                                int64_t pixels, int patches, uint32_t* masks, void* stream) {
    SOLWEIG_CHECK_ARG(shmat && vegmat && vbmat && masks && pixels > 0 && patches > 0 &&
                          patches <= SOLWEIG_MASK_WORDS * 32,
                      "solweig_svf_pack: bad arguments");
    svf_pack_kernel<<<blocks_for(pixels, 256), 256, 0, as_stream(stream)>>>(shmat, vegmat, vbmat,
                                                                           pixels, patches, masks);
    SOLWEIG_CHECK_LAUNCH("svf_pack_kernel");
    return SOLWEIG_OK;
}

// Blocks of the visibility kernel: 8 x 4 pixel tiles.
unsigned svf_tiles(int rows, int cols) { return (unsigned)(((cols + 7) / 8) * ((rows + 3) / 4)); }

// first_outside tables of a group of patches: block j = patch0 + j; with
// rec also the patches' step records (kmax >= every length).
__global__ void __launch_bounds__(1024) patch_ray_exits_kernel(int rows, int cols, const int2* __restrict__ rays,
                                                               const double* __restrict__ dz,
                                                               const int32_t* __restrict__ lengths, int capacity,
                                                               int patch0, int count, int* __restrict__ exits,
                                                               int2* __restrict__ rec, int kmax) {
    const int j = blockIdx.x;
    if (j >= count) return;
    const int patch = patch0 + j;
    ray_exits_block(rays + (long long)patch * capacity, lengths[patch], rows, cols,
                    exits + (long long)j * (rows + cols));
    if (rec != nullptr)
        ray_records_block(rays + (long long)patch * capacity, dz + (long long)patch * capacity,
                          min(lengths[patch], kmax), cols, rec + (long long)j * record_pitch(kmax));
}

// Ray tables of the sky patches (src/svf.py:47-75): steps k = 0, 1, ... of the
// digital line towards a patch with the heights dz = (ds k) tan(alt) / scale, up
// to and including the first step above amax or outside the raster.  Quotients
// and products are single float64 roundings and rint rounds half to even, so a
// table equals numpy's bit for bit.  One block per patch; the host's loop over
// the patches took 3.6 ms and its tables up to 5 MB of upload, this kernel 3 us.
struct SvfRayConstants {
    double sin_az[SOLWEIG_MAX_PATCHES], cos_az[SOLWEIG_MAX_PATCHES], tan_az[SOLWEIG_MAX_PATCHES];
    double rise[SOLWEIG_MAX_PATCHES];  // tan(altitude) / scale
    uint8_t ymajor[SOLWEIG_MAX_PATCHES];
};

__global__ void __launch_bounds__(256) svf_ray_tables_kernel(const __grid_constant__ SvfRayConstants q, int rows,
                                                             int cols, double amax, int capacity,
                                                             int2* __restrict__ dxdy, double* __restrict__ dz,
                                                             int32_t* __restrict__ lengths) {
    __shared__ int first;
    const int p = blockIdx.x;
    if (threadIdx.x == 0) first = capacity - 1;
    __syncthreads();
    const double s = q.sin_az[p], c = q.cos_az[p], t = q.tan_az[p];
    const double sx = c > 0 ? -1.0 : c < 0 ? 1.0 : 0.0, sy = s > 0 ? 1.0 : s < 0 ? -1.0 : 0.0;
    const bool ymajor = q.ymajor[p];
    const double ds = fabs(__ddiv_rn(1.0, ymajor ? s : c));
    for (int k = threadIdx.x; k < capacity; k += blockDim.x) {
        const double minor = fabs(rint(ymajor ? __ddiv_rn((double)k, t) : __dmul_rn((double)k, t)));
        const double dx = sx * (ymajor ? minor : (double)k), dy = sy * (ymajor ? (double)k : minor);
        const double z = __dmul_rn(__dmul_rn(ds, (double)k), q.rise[p]);
        dxdy[(long long)p * capacity + k] = make_int2((int)dx, (int)dy);
        dz[(long long)p * capacity + k] = z;
        if (z > amax || fabs(dx) >= rows || fabs(dy) >= cols) {
            atomicMin(&first, k);
            break;  // the later steps are not part of the ray
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) lengths[p] = amax < 0 ? 0 : first + 1;
}

// Work of solweig_svf_ex2: 4 dilated height planes and the plane of H, the 32 ray-ceiling
// planes (ceiling and window maximum per pixel) of one patch word, its 32 first-outside tables and its step
// records (kmax = max(rows, cols) + 2 per patch, >= every ray's length).
struct SvfWork {
    long long dil, height, ceil, exits, rec, total;
    int kmax;
};

SvfWork svf_work_layout(int rows, int cols) {
    const long long px = (long long)rows * cols;
    SvfWork w{};
    w.kmax = (rows > cols ? rows : cols) + 2;
    w.dil = 0;
    w.height = 4LL * 4 * px;
    w.ceil = (5LL * 4 * px + 255) & ~255LL;
    w.exits = (w.ceil + 8LL * kSvfPatchGroup * px + 255) & ~255LL;
    w.rec = (w.exits + 4LL * kSvfPatchGroup * (rows + cols) + 255) & ~255LL;
    w.total = w.rec + 8LL * kSvfPatchGroup * record_pitch(w.kmax);
    return w;
}

extern "C" int solweig_svf_ray_tables(const double* sin_az, const double* cos_az, const double* tan_az,
                                      const double* rise, const uint8_t* ymajor, int patches, int rows, int cols,
                                      double amax, int capacity, int32_t* ray_dxdy, double* ray_dz, int32_t* lengths,
                                      void* stream) {
    SOLWEIG_CHECK_ARG(sin_az && cos_az && tan_az && rise && ymajor && ray_dxdy && ray_dz && lengths,
                      "solweig_svf_ray_tables: null pointer");
    SOLWEIG_CHECK_ARG(patches > 0 && patches <= SOLWEIG_MAX_PATCHES && rows > 0 && cols > 0 && capacity > 0,
                      "solweig_svf_ray_tables: %d patches, %d x %d px, capacity %d", patches, rows, cols, capacity);
    SvfRayConstants q{};
    for (int k = 0; k < patches; ++k) {
        q.sin_az[k] = sin_az[k];
        q.cos_az[k] = cos_az[k];
        q.tan_az[k] = tan_az[k];
        q.rise[k] = rise[k];
        q.ymajor[k] = ymajor[k];
    }
    svf_ray_tables_kernel<<<patches, 256, 0, as_stream(stream)>>>(q, rows, cols, amax, capacity,
                                                                  reinterpret_cast<int2*>(ray_dxdy), ray_dz, lengths);
    SOLWEIG_CHECK_LAUNCH("svf_ray_tables_kernel");
    return SOLWEIG_OK;
}

extern "C" int64_t solweig_svf_work_bytes(int rows, int cols) {
    if (rows <= 0 || cols <= 0) return 0;
    return svf_work_layout(rows, cols).total;
}

int svf_impl(const double* dsm, const double* vegdem, const double* vegdem2, const void* geo32,
             const uint8_t* flags, int rows, int cols, int patches, int capacity, const int32_t* ray_dxdy,
             const double* ray_dz, const int32_t* lengths, double hmax, const SolweigSkyLayout* layout,
             const double* band_weights, const uint8_t* sectors, double transmissivity, uint32_t* masks,
             double* planes, float* veg_sums, uint8_t* sky_band_counts, void* work, int64_t work_bytes,
             void* stream);

extern "C" int solweig_svf_ex(const double* dsm, const double* vegdem, const double* vegdem2,
                              const void* geo32, const uint8_t* flags, int rows, int cols, int patches,
                              int capacity, const int32_t* ray_dxdy, const double* ray_dz,
                              const int32_t* lengths, double hmax, const SolweigSkyLayout* layout,
                              const double* band_weights, const uint8_t* sectors, double transmissivity,
                              uint32_t* masks, double* planes, float* veg_sums, uint8_t* sky_band_counts,
                              void* stream) {
    return svf_impl(dsm, vegdem, vegdem2, geo32, flags, rows, cols, patches, capacity, ray_dxdy, ray_dz, lengths,
                    hmax, layout, band_weights, sectors, transmissivity, masks, planes, veg_sums, sky_band_counts,
                    nullptr, 0, stream);
}

// solweig_svf_ex with a work buffer of solweig_svf_work_bytes (no counterpart
// in the reference): per patch word, ray ceilings and first-outside tables
// let the visibility walks stop early with identical masks.
extern "C" int solweig_svf_ex2(const double* dsm, const double* vegdem, const double* vegdem2,
                               const void* geo32, const uint8_t* flags, int rows, int cols, int patches,
                               int capacity, const int32_t* ray_dxdy, const double* ray_dz,
                               const int32_t* lengths, double hmax, const SolweigSkyLayout* layout,
                               const double* band_weights, const uint8_t* sectors, double transmissivity,
                               uint32_t* masks, double* planes, float* veg_sums, uint8_t* sky_band_counts,
                               void* work, int64_t work_bytes, void* stream) {
    SOLWEIG_CHECK_ARG(work, "solweig_svf_ex2: null work buffer");
    return svf_impl(dsm, vegdem, vegdem2, geo32, flags, rows, cols, patches, capacity, ray_dxdy, ray_dz, lengths,
                    hmax, layout, band_weights, sectors, transmissivity, masks, planes, veg_sums, sky_band_counts,
                    work, work_bytes, stream);
}

int svf_impl(const double* dsm, const double* vegdem, const double* vegdem2, const void* geo32,
             const uint8_t* flags, int rows, int cols, int patches, int capacity, const int32_t* ray_dxdy,
             const double* ray_dz, const int32_t* lengths, double hmax, const SolweigSkyLayout* layout,
             const double* band_weights, const uint8_t* sectors, double transmissivity, uint32_t* masks,
             double* planes, float* veg_sums, uint8_t* sky_band_counts, void* work, int64_t work_bytes,
             void* stream) {
    SOLWEIG_CHECK_ARG(dsm && vegdem && vegdem2 && flags && ray_dxdy && ray_dz && lengths && layout &&
                          band_weights && sectors && masks && planes && veg_sums && sky_band_counts,
                      "solweig_svf: null pointer");
    SOLWEIG_CHECK_ARG(rows > 0 && cols > 0 && capacity > 0, "solweig_svf: bad shape");
    SOLWEIG_CHECK_ARG(patches > 0 && patches <= SOLWEIG_MASK_WORDS * 32 && patches == layout->patches,
                      "solweig_svf: %d patches (max %d, layout %d)", patches,
                      SOLWEIG_MASK_WORDS * 32, layout->patches);
    SOLWEIG_CHECK_ARG(layout->nbands > 0 && layout->nbands <= SOLWEIG_MAX_BANDS,
                      "solweig_svf: bad band count %d", layout->nbands);
    const long long pixels = (long long)rows * cols;
    cudaStream_t st = as_stream(stream);
    cudaError_t e = cudaMemsetAsync(masks, 0, sizeof(uint32_t) * 2 * SOLWEIG_MASK_WORDS * pixels, st);
    if (e != cudaSuccess) {
        set_error("solweig_svf: memset: %s", cudaGetErrorString(e));
        return SOLWEIG_ERR_CUDA;
    }
    SvfRayParams rp{rows, cols, patches, capacity, hmax};
    const int words = (patches + 31) / 32;
    const int2* rays = reinterpret_cast<const int2*>(ray_dxdy);
    const float4* g4 = reinterpret_cast<const float4*>(geo32);
    if (!work) {
        dim3 grid(svf_tiles(rows, cols), words);
        if (g4) svf_visibility_kernel<1><<<grid, 32 * kSvfWarps, 0, st>>>(dsm, vegdem, vegdem2, g4, flags, rp, rays,
                                                                          ray_dz, lengths, masks, 0, nullptr);
        else svf_visibility_kernel<0><<<grid, 32 * kSvfWarps, 0, st>>>(dsm, vegdem, vegdem2, g4, flags, rp, rays,
                                                                       ray_dz, lengths, masks, 0, nullptr);
        SOLWEIG_CHECK_LAUNCH("svf_visibility_kernel");
    } else {
        const SvfWork w = svf_work_layout(rows, cols);
        SOLWEIG_CHECK_ARG(work_bytes >= w.total, "solweig_svf_ex2: work buffer of %lld bytes, need %lld",
                          (long long)work_bytes, w.total);
        SOLWEIG_CHECK_ARG(((uintptr_t)work & 255) == 0, "solweig_svf_ex2: work buffer not 256-byte aligned");
        char* wb = static_cast<char*>(work);
        float* dil = reinterpret_cast<float*>(wb + w.dil);
        float2* ceil = reinterpret_cast<float2*>(wb + w.ceil);
        int* exits = reinterpret_cast<int*>(wb + w.exits);
        // step records when every ray fits kmax (the host's ray tables do)
        int2* rec = (g4 && capacity <= w.kmax && pixels <= kPackedMaxPixels) ? reinterpret_cast<int2*>(wb + w.rec) : nullptr;
        float* height = reinterpret_cast<float*>(wb + w.height);
        SolweigScene S{};
        S.rows = rows;
        S.cols = cols;
        S.dsm = dsm;
        S.vegdem = vegdem;
        S.vegdem2 = vegdem2;
        S.geo32 = geo32;
        dim3 dgrid(blocks_for(cols, kDilTile), blocks_for(rows, kDilTile));
        if (geo32) ceiling_dilate_kernel<true><<<dgrid, dim3(32, 8), 0, st>>>(S, dil, height);
        else ceiling_dilate_kernel<false><<<dgrid, dim3(32, 8), 0, st>>>(S, dil, nullptr);
        SOLWEIG_CHECK_LAUNCH("ceiling_dilate_kernel");
        for (int wd = 0; wd < words; ++wd) {
            const int p0 = wd * kSvfPatchGroup, cnt = std::min(kSvfPatchGroup, patches - p0);
            dim3 cgrid(blocks_for((long long)rows + cols, kCeilLanes), 1, cnt);
            patch_ray_ceiling_kernel<<<cgrid, dim3(kCeilLanes, kCeilWarps), 0, st>>>(S, rays, ray_dz, lengths,
                                                                                     capacity, p0, cnt, dil, ceil);
            SOLWEIG_CHECK_LAUNCH("patch_ray_ceiling_kernel");
            patch_ray_exits_kernel<<<cnt, 1024, 0, st>>>(rows, cols, rays, ray_dz, lengths, capacity, p0, cnt, exits,
                                                          rec, w.kmax);
            SOLWEIG_CHECK_LAUNCH("patch_ray_exits_kernel");
            dim3 grid(svf_tiles(rows, cols), 1);
            if (rec)
                svf_visibility_warp_kernel<<<blocks_for(svf_tiles(rows, cols), kSvfWarps), 32 * kSvfWarps, 0, st>>>(
                    g4, height, flags, rp, ray_dz, lengths, masks, wd, ceil, exits, rec, record_pitch(w.kmax));
            else if (g4)
                svf_visibility_kernel<1><<<grid, 32 * kSvfWarps, 0, st>>>(dsm, vegdem, vegdem2, g4, flags, rp, rays,
                                                                          ray_dz, lengths, masks, wd, ceil);
            else
                svf_visibility_kernel<0><<<grid, 32 * kSvfWarps, 0, st>>>(dsm, vegdem, vegdem2, g4, flags, rp, rays,
                                                                          ray_dz, lengths, masks, wd, ceil);
            SOLWEIG_CHECK_LAUNCH("svf_visibility_kernel");
        }
    }
    return solweig_svf_reduce(masks, vegdem2, pixels, layout, band_weights, sectors, transmissivity,
                              planes, veg_sums, sky_band_counts, stream);
}

extern "C" int solweig_svf(const double* dsm, const double* vegdem, const double* vegdem2,
                           const uint8_t* flags, int rows, int cols, int patches, int capacity,
                           const int32_t* ray_dxdy, const double* ray_dz, const int32_t* lengths,
                           double hmax, const SolweigSkyLayout* layout,
                           const double* band_weights, const uint8_t* sectors,
                           double transmissivity, uint32_t* masks, double* planes,
                           float* veg_sums, uint8_t* sky_band_counts, void* stream) {
    return solweig_svf_ex(dsm, vegdem, vegdem2, nullptr, flags, rows, cols, patches, capacity, ray_dxdy, ray_dz,
                          lengths, hmax, layout, band_weights, sectors, transmissivity, masks, planes, veg_sums,
                          sky_band_counts, stream);
}

extern "C" int solweig_svf_unpack(const uint32_t* masks, int64_t pixels, int patches, float* shmat,
                                  float* vegmat, float* vbmat, void* stream) {
    SOLWEIG_CHECK_ARG(masks && pixels > 0 && patches > 0 && patches <= SOLWEIG_MASK_WORDS * 32,
                      "solweig_svf_unpack: bad arguments");
    const long long n = (long long)pixels * patches;
    // null cubes count as aligned
    const bool aligned = (((uintptr_t)shmat | (uintptr_t)vegmat | (uintptr_t)vbmat) & 15) == 0;
    const unsigned blocks = blocks_for(n, kUnpackValues);
    if (aligned)
        svf_unpack_kernel<4><<<blocks, 256, 0, as_stream(stream)>>>(masks, pixels, patches, shmat, vegmat, vbmat);
    else
        svf_unpack_kernel<1><<<blocks, 256, 0, as_stream(stream)>>>(masks, pixels, patches, shmat, vegmat, vbmat);
    SOLWEIG_CHECK_LAUNCH("svf_unpack_kernel");
    return SOLWEIG_OK;
}

extern "C" int solweig_diffsh(const float* shmat, const float* vegshmat, float* diffsh, int64_t n,
                              float transmissivity, void* stream) {
    SOLWEIG_CHECK_ARG(shmat && vegshmat && diffsh && n >= 0, "solweig_diffsh: bad arguments");
    if (n == 0) return SOLWEIG_OK;
    diffsh_kernel<<<blocks_for(n, 256), 256, 0, as_stream(stream)>>>(shmat, vegshmat, diffsh, n,
                                                                     transmissivity);
    SOLWEIG_CHECK_LAUNCH("diffsh_kernel");
    return SOLWEIG_OK;
}
