// Ray ceilings: per daytime hour, an upper bound at every pixel q of the
// heights that the rest of a sun ray passing through q can still present,
// discounted by the ray's rise.  The shadow sweep uses it to stop walking a
// ray as soon as no later sample can change any of its outputs.
//
// The sweep of pixel p visits q_j = p + o_j (j = 0 .. K-1, o_j the ray table)
// and at step j compares the heights h in {dsm, canopy top, trunk} at q_j
// against the pixel through h - dz_j and h - dz_{j-1}.  Let H = max(dsm,
// vegdem, vegdem2).  If a value C(q_k) satisfies, for every pixel p whose ray
// visits q_k at step k and every later step j >= k,
//        H(q_j) - dz_{j-1}  <=  C(q_k) - dz_{k-1}                        (*)
// then C(q_k) - dz_{k-1} < dsm_p means no later sample reaches above the
// pixel (its shadow height, vegetation flags and, when also <= topmax, the
// canopy top seen by a wall are final).
//
// Construction (all bounds exact, no trigonometry):
//  * frame: the major axis is the one whose offset equals +-j at every step
//    (checked over the whole table); X runs along it in the ray direction and
//    Y along the other axis, oriented so the last offset is >= 0.  Then
//    X(q_j) = X(q_k) + (j - k) and Y(q_j) = Y(p) + m_j with m_j the minor
//    offset.
//  * shear: with v = M / D, M = m_{K-1}, D = K - 1, R(X) = floor(X M / D) in
//    integers and the sheared line N = Y - R(X).  Along one ray
//    N(q_j) - N(q_k) = (e_j - e_k) - (R(X_j) - R(X_k) - (j-k) v) with
//    e_i = m_i - i v, so |N(q_j) - N(q_k)| < spread(e) + 1, i.e. <= W with
//    W = floor(spread) + 1 (spread measured exactly as D * e_i in integers;
//    about 1 for the rounded digital rays, so W = 2).
//  * discount: delta = the smallest increment dz_i - dz_{i-1} of the table
//    (exact in float64 by Sterbenz), rounded down to float32, so
//    dz_{j-1} - dz_{k-1} >= (j - k) delta for j >= k >= 1.
//  * along each sheared line, G(X) = max(Hd(X), G(X+1) - delta) with
//    Hd(X, N) = max over |d| <= W of H(X, N + d + R(X)) and the subtraction
//    rounded up, so G(X, N) >= H(X', N') - (X' - X) delta for X' >= X and
//    |N' - N| <= W: C(q) = G(X(q), N(q)) satisfies (*) for k >= 1.
//
// The dilation runs along the raster's minor axis only, so it is done once
// per day (ceiling_dilate_kernel): H dilated by +-1 and +-2 along the columns
// (row-major planes, for rays whose major axis is the rows) and along the rows
// (stored transposed, for rays whose major axis is the columns).  Either way
// the scan reads plane[a * nb + b] with a the oriented major index and b the
// oriented minor index, so a warp's 32 lanes (consecutive Y) read 32
// consecutive floats.
//
// Window maxima: with the ceiling the scan also writes, per pixel,
// M(X, N) = max over X' in [X, X + kCeilSkip) of Hd(X', N) (no discount).  A
// ray through q_k at step k >= 1 meets q_{k..k+kCeilSkip-1} within +-W lines,
// so H(q_j) - dz_{j-1} <= M(q_k) - dz_{k-1} for those steps: when that is
// <= dsm_p none of their compares is above the pixel and a walk (not of a
// wall pixel) may skip them.  The planes hold (C, M) as float2 per pixel.
//
// Scan layout: a block owns 32 consecutive sheared lines (one per lane) and
// splits the major axis into 16 segments (one per warp; 512 threads, so two
// blocks fit per SM).  Phase 1 scans each
// segment backwards from -inf; phase 2 carries the later segments' maxima in
// and rescans, writing the plane.
#pragma once
#include "common.cuh"

namespace solweig {

constexpr int kCeilLanes = 32;     // sheared lines per block
constexpr int kCeilWarps = 16;     // major-axis segments per block
constexpr int kCeilMaxBand = 3;    // largest dilation W handled
constexpr int kCeilMinSteps = 5;   // the sweep consults the plane from step 4 on

// Upper bound (float32) of max(dsm, vegdem, vegdem2) at pixel p.
template <bool G32>
__device__ __forceinline__ float ceiling_height(const SolweigScene& S, long long p) {
    if (G32) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(S.geo32) + p);
        return fmaxf(v.x, fmaxf(v.y, v.z));
    }
    const double m = fmax(__ldg(&S.dsm[p]), fmax(__ldg(&S.vegdem[p]), __ldg(&S.vegdem2[p])));
    return __double2float_ru(m);
}

struct CeilingFrame {
    int ok;            // 0: the table fits no frame; the plane is +inf
    int rows_major;    // major axis = rows (else columns)
    int s_major, s_minor;
    int nx, nb;        // extents along X (major) and Y (minor)
    int m, d;          // slope v = m / d of the shear
    int band;          // dilation W
    int lines;         // sheared lines: nb + R(nx - 1)
    float delta;       // per-step discount
};

// Frame of one hour's ray, derived by the whole block from the table.
__device__ inline CeilingFrame ceiling_frame(const SolweigScene& S, const int2* __restrict__ ray,
                                      const double* __restrict__ dz, int K) {
    __shared__ long long s_emin, s_emax;
    __shared__ unsigned s_dmin;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x, nt = blockDim.x * blockDim.y;
    const int2 last = ray[K - 1];
    const int sr = last.x < 0 ? -1 : 1, sc = last.y < 0 ? -1 : 1;
    int rows_ok = 1, cols_ok = 1;
    for (int i = tid; i < K; i += nt) {
        const int2 o = __ldg(&ray[i]);
        rows_ok &= (o.x == sr * i);
        cols_ok &= (o.y == sc * i);
    }
    rows_ok = __syncthreads_and(rows_ok);
    cols_ok = __syncthreads_and(cols_ok);
    CeilingFrame f{};
    f.rows_major = rows_ok;
    f.ok = rows_ok || cols_ok;
    if (!f.ok) return f;
    f.s_major = rows_ok ? sr : sc;
    f.s_minor = rows_ok ? sc : sr;
    f.nx = rows_ok ? S.rows : S.cols;
    f.nb = rows_ok ? S.cols : S.rows;
    f.d = K - 1;
    f.m = f.s_minor * (rows_ok ? last.y : last.x);  // >= 0
    if (tid == 0) {
        s_emin = LLONG_MAX;
        s_emax = LLONG_MIN;
        s_dmin = 0x7f800000u;  // +inf
    }
    __syncthreads();
    long long emin = LLONG_MAX, emax = LLONG_MIN;
    float dmin = __int_as_float(0x7f800000);
    int inc_ok = 1;
    for (int i = tid; i < K; i += nt) {
        const int2 o = __ldg(&ray[i]);
        const long long mi = (long long)f.s_minor * (rows_ok ? o.y : o.x);
        const long long e = mi * f.d - (long long)i * f.m;  // D * e_i
        emin = min(emin, e);
        emax = max(emax, e);
        if (i >= 1) {
            const double inc = __ldg(&dz[i]) - __ldg(&dz[i - 1]);  // exact (Sterbenz)
            inc_ok &= (inc >= 0.0);                                 // false for NaN too
            if (inc >= 0.0) dmin = fminf(dmin, __double2float_rd(inc));
        }
    }
    atomicMin(&s_emin, emin);
    atomicMax(&s_emax, emax);
    atomicMin(&s_dmin, __float_as_uint(dmin));  // non-negative floats order as integers
    inc_ok = __syncthreads_and(inc_ok);
    const long long spread = s_emax - s_emin;  // D * spread(e)
    f.band = (int)(spread / f.d) + 1;
    f.delta = __uint_as_float(s_dmin);
    // (nx - 1) * m must fit the 32-bit shear cursor
    if (!inc_ok || f.m > f.d || f.band > kCeilMaxBand || (long long)(f.nx - 1) * f.m > INT_MAX) {
        f.ok = 0;
        return f;
    }
    f.lines = f.nb + (f.nx - 1) * f.m / f.d;
    return f;
}

// Position on a sheared line that steps X down by one: y = line + R(X) with
// R(X) = floor(X m / d), quotient and remainder carried in 32-bit integers
// (X m <= rows * cols), and the offset of (X, y) in the dilated plane carried
// along -- no division and no product per step.  I: int, or for huge rasters
// long long.
template <typename I>
struct ShearCursor {
    int y, rem;
    I at;            // offset as if y were in the raster
    I at_x;          // its change as X goes down by one; as y does: -s_minor
    __device__ __forceinline__ ShearCursor(const CeilingFrame& f, int line, int x) {
        const int num = x * f.m, r = num / f.d;
        rem = num - r * f.d;
        y = line + r;
        at = (I)(f.s_major > 0 ? x : f.nx - 1 - x) * f.nb + (f.s_minor > 0 ? y : f.nb - 1 - y);
        at_x = -f.s_major * (I)f.nb;
    }
    __device__ __forceinline__ bool step_down(const CeilingFrame& f) {  // m <= d; true when y went down
        at += at_x;
        rem -= f.m;
        const bool down = rem < 0;
        if (down) {
            rem += f.d;
            --y;
            at -= f.s_minor;
        }
        return down;
    }
};

constexpr int kCeilBatch = 8;  // samples fetched ahead of the dependent max chain

// H dilated by +-W along the minor axis around Y = y: plane[at] for y in the
// raster.  A line whose centre lies up to W outside it still sees its in-raster
// neighbours: the edge pixel's window covers them.
template <typename I>
__device__ __forceinline__ float ceiling_sample(const float* __restrict__ plane, const CeilingFrame& f, I at, int y) {
    if (y < -f.band || y >= f.nb + f.band) return __int_as_float(0xff800000);
    const int yc = min(max(y, 0), f.nb - 1);
    return __ldg(&plane[at + (I)(f.s_minor * (yc - y))]);
}

// One backward scan of [x0, x1) from g over the lane's sheared line; with OUT,
// writes every pixel of the line: (ceiling, window maximum).  A batch of loads
// is issued before the dependent chain consumes it, without range tests when the
// batch surely lies inside the raster.  ahead[j] is the maximum of Hd at
// x + 1 .. x + 1 + j, so the windows of a batch are running maxima of the batch and
// of `ahead`.  y goes down with x: the part of the segment before the line enters
// the raster is all -inf and skipped, and the scan ends when the line has left
// (both for the whole warp, by its first and last line).
//
// The lanes' lines are neighbours along Y.  Where the rows of the raster run along
// X, a lane's 8-byte stores would each touch a sector of their own, four times
// over: a batch goes through shared memory (`stage`, per warp) and is written row
// by row, 64 bytes at a time.  That was the bound: planes of a 2000^2 day 0.58 ->
// 0.31 ms, of 153 patches at 512 x 448 0.37 -> 0.26 ms; the cheaper steps alone
// gave 0.57 and 0.35.  Now it is the latency of the segments' two passes.
constexpr int kCeilStagePitch = 36;  // float2; 8 banks from one step to the next
template <bool OUT, typename I>
__device__ __forceinline__ float ceiling_run(const float* __restrict__ plane, const CeilingFrame& f, int cols,
                                             int line, int x0, int x1, float g, float2* __restrict__ out,
                                             float2 (*stage)[kCeilStagePitch]) {
    static_assert(kCeilBatch == kCeilSkip, "a batch is a window");
    const float ninf = __int_as_float(0xff800000);
    if (x0 >= x1) return g;
    const int lane = threadIdx.x;  // the block's rows are warps
    const int top = f.nb + f.band - (line - lane);  // the warp is in reach of the raster for R(x) < top
    if (top <= 0) return g;
    if (f.m > 0) x1 = (int)min((long long)x1, ((long long)top * f.d + f.m - 1) / f.m);
    if (x0 >= x1) return g;
    float ahead[kCeilSkip - 1];
#pragma unroll
    for (int i = 0; i < kCeilSkip - 1; ++i) {
        ahead[i] = i > 0 ? ahead[i - 1] : ninf;
        if (OUT && x1 + i < f.nx) {
            const int xx = x1 + i, y = line + (int)(((long long)xx * f.m) / f.d);
            const int a = f.s_major > 0 ? xx : f.nx - 1 - xx, b = f.s_minor > 0 ? y : f.nb - 1 - y;
            ahead[i] = fmaxf(ahead[i], ceiling_sample<I>(plane, f, (I)a * f.nb + b, y));
        }
    }
    int x = x1 - 1;
    ShearCursor<I> cur(f, line, x);
    // the raster offset of the pixel: of a column-major ray another one than the plane's
    const int a1 = f.s_major > 0 ? x : f.nx - 1 - x, b1 = f.s_minor > 0 ? cur.y : f.nb - 1 - cur.y;
    I px = f.rows_major ? (I)a1 * cols + b1 : (I)b1 * cols + a1;
    const I px_x = f.rows_major ? -f.s_major * (I)cols : (I)-f.s_major;
    const I px_y = f.rows_major ? (I)-f.s_minor : -f.s_minor * (I)cols;
    for (; x - (kCeilBatch - 1) >= x0; x -= kCeilBatch) {
        if (cur.y + (kCeilLanes - 1 - lane) < -f.band) return g;
        float v[kCeilBatch];
        int y = cur.y;
        uint32_t down = 0u;  // steps after which y is one lower
        const bool inside = y < f.nb && y >= kCeilBatch;
        if (inside) {
#pragma unroll
            for (int u = 0; u < kCeilBatch; ++u) {
                v[u] = __ldg(&plane[cur.at]);
                if (cur.step_down(f)) down |= 1u << u;
            }
        } else {
#pragma unroll
            for (int u = 0; u < kCeilBatch; ++u) {
                v[u] = ceiling_sample<I>(plane, f, cur.at, cur.y);
                if (cur.step_down(f)) down |= 1u << u;
            }
        }
        float window = ninf;
#pragma unroll
        for (int u = 0; u < kCeilBatch; ++u) {
            g = fmaxf(v[u], __fsub_ru(g, f.delta));
            if (OUT) {
                window = fmaxf(window, v[u]);
                const float2 cell = make_float2(g, u + 1 < kCeilBatch ? fmaxf(window, ahead[kCeilSkip - 2 - u]) : window);
                if (!f.rows_major) stage[u][lane] = cell;
                else if (inside || (y >= 0 && y < f.nb)) out[px] = cell;
                px += px_x;
                if ((down >> u) & 1u) {
                    px += px_y;
                    --y;
                }
            }
        }
        if (OUT && !f.rows_major) {
            // step u of row i (from the lowest) comes from the lane `back` rows below it
            __syncwarp();
            const int u = lane & (kCeilBatch - 1), fell = __popc(down & ((1u << (kCeilBatch - 1)) - 1u));
            const int back = fell - __popc(down & ((1u << u) - 1u));
            const int ylow = cur.y + (int)((down >> (kCeilBatch - 1)) & 1u) - lane;  // of lane 0 at the last step
            const int xu = x - u, a = f.s_major > 0 ? xu : f.nx - 1 - xu;
            for (int i = lane / kCeilBatch; i < kCeilLanes + fell; i += kCeilLanes / kCeilBatch) {
                const int from = i - back, yi = ylow + i;
                if (from < 0 || from >= kCeilLanes || yi < 0 || yi >= f.nb) continue;
                out[(I)(f.s_minor > 0 ? yi : f.nb - 1 - yi) * cols + a] = stage[u][from];
            }
            __syncwarp();
        }
        if (OUT) {
            ahead[0] = v[kCeilBatch - 1];
#pragma unroll
            for (int j = 1; j < kCeilSkip - 1; ++j) ahead[j] = fmaxf(ahead[j - 1], v[kCeilBatch - 1 - j]);
        }
    }
#pragma unroll 1
    for (; x >= x0; --x) {
        const float v = ceiling_sample<I>(plane, f, cur.at, cur.y);
        g = fmaxf(v, __fsub_ru(g, f.delta));
        if (OUT) {
            if (cur.y >= 0 && cur.y < f.nb) out[px] = make_float2(g, fmaxf(v, ahead[kCeilSkip - 2]));
#pragma unroll
            for (int j = kCeilSkip - 2; j > 0; --j) ahead[j] = fmaxf(v, ahead[j - 1]);
            ahead[0] = v;
            px += px_x;
        }
        if (cur.step_down(f)) px += px_y;
    }
    return g;
}

// Both phases for one block of 32 sheared lines (see the file comment).
template <typename I>
__device__ __forceinline__ void ceiling_scan(const float* __restrict__ plane, const CeilingFrame& f, int cols,
                                             int line0, float (*s_seg)[kCeilLanes], float2* __restrict__ out,
                                             float2 (*stage)[kCeilStagePitch]) {
    const int seg = (f.nx + kCeilWarps - 1) / kCeilWarps;
    const int w = threadIdx.y;
    const int x0 = min(f.nx, w * seg), x1 = min(f.nx, x0 + seg);
    const int line = line0 + threadIdx.x;
    const float ninf = __int_as_float(0xff800000);
    // phase 1: segment maxima from -inf
    s_seg[w][threadIdx.x] = ceiling_run<false, I>(plane, f, cols, line, x0, x1, ninf, nullptr, nullptr);
    __syncthreads();
    // phase 2: carry of the later segments, then the rescan that writes
    float carry = ninf;
    for (int s = kCeilWarps - 1; s > w; --s) {
        const int s0 = min(f.nx, s * seg), s1 = min(f.nx, s0 + seg);
        carry = fmaxf(s_seg[s][threadIdx.x], __fsub_ru(carry, __fmul_rd((float)(s1 - s0), f.delta)));
    }
    ceiling_run<true, I>(plane, f, cols, line, x0, x1, carry, out, stage);
}

// The four dilated planes of H (see the file comment), each rows x cols floats:
//   dil[0], dil[1]: +-1, +-2 along the columns, row-major [r][c];
//   dil[2], dil[3]: +-1, +-2 along the rows, transposed [c][r].
// H itself goes to `height` (optional), row-major.
// block (32, 8) over a 32 x 32 tile, H staged with a 2-pixel halo.
constexpr int kDilTile = 32, kDilHalo = 2, kDilPitch = kDilTile + 2 * kDilHalo + 1;

template <bool G32>
__global__ void __launch_bounds__(256) ceiling_dilate_kernel(SolweigScene S, float* __restrict__ dil,
                                                             float* __restrict__ height) {
    __shared__ float tile[kDilTile + 2 * kDilHalo][kDilPitch];
    const int r0 = blockIdx.y * kDilTile, c0 = blockIdx.x * kDilTile;
    const int tid = threadIdx.y * 32 + threadIdx.x;
    const float ninf = __int_as_float(0xff800000);
    constexpr int side = kDilTile + 2 * kDilHalo;
    for (int i = tid; i < side * side; i += 256) {
        const int tr = i / side, tc = i - tr * side;
        const int r = r0 - kDilHalo + tr, c = c0 - kDilHalo + tc;
        tile[tr][tc] = (r >= 0 && r < S.rows && c >= 0 && c < S.cols)
                           ? ceiling_height<G32>(S, (long long)r * S.cols + c) : ninf;
    }
    __syncthreads();
    const long long n = (long long)S.rows * S.cols;
    // along the columns: thread x = column (row-major writes coalesced)
    for (int k = threadIdx.y; k < kDilTile; k += 8) {
        const int r = r0 + k, c = c0 + threadIdx.x;
        if (r >= S.rows || c >= S.cols) continue;
        const float* t = &tile[k + kDilHalo][threadIdx.x + kDilHalo];
        const float d1 = fmaxf(t[0], fmaxf(t[-1], t[1]));
        const float d2 = fmaxf(d1, fmaxf(t[-2], t[2]));
        if (height) height[(long long)r * S.cols + c] = t[0];
        dil[(long long)r * S.cols + c] = d1;
        dil[n + (long long)r * S.cols + c] = d2;
    }
    // along the rows: thread x = row (transposed writes coalesced)
    for (int k = threadIdx.y; k < kDilTile; k += 8) {
        const int r = r0 + threadIdx.x, c = c0 + k;
        if (r >= S.rows || c >= S.cols) continue;
        const int tr = threadIdx.x + kDilHalo, tc = k + kDilHalo;
        const float d1 = fmaxf(tile[tr][tc], fmaxf(tile[tr - 1][tc], tile[tr + 1][tc]));
        const float d2 = fmaxf(d1, fmaxf(tile[tr - 2][tc], tile[tr + 2][tc]));
        dil[2 * n + (long long)c * S.rows + r] = d1;
        dil[3 * n + (long long)c * S.rows + r] = d2;
    }
}

// The ceiling plane of one ray table (K steps) for the raster of S, by one
// block of (32, kCeilWarps) threads owning 32 sheared lines (blockIdx.x); the whole
// block returns together.  Tables the frame does not fit give a +inf plane.
__device__ __forceinline__ void ray_ceiling_block(const SolweigScene& S, const int2* __restrict__ ray,
                                                  const double* __restrict__ dz, int K,
                                                  const float* __restrict__ dil, float2* __restrict__ out,
                                                  float (*s_seg)[kCeilLanes]) {
    __shared__ float2 s_stage[kCeilWarps][kCeilBatch][kCeilStagePitch];
    if (K < kCeilMinSteps) return;
    const long long n = (long long)S.rows * S.cols;
    const CeilingFrame f = ceiling_frame(S, ray, dz, K);
    const int tid = threadIdx.y * kCeilLanes + threadIdx.x;
    if (!f.ok || f.band > 2) {
        for (long long p = (long long)blockIdx.x * blockDim.x * blockDim.y + tid; p < n;
             p += (long long)gridDim.x * blockDim.x * blockDim.y)
            out[p] = make_float2(__int_as_float(0x7f800000), __int_as_float(0x7f800000));
        return;
    }
    const int line_first = blockIdx.x * kCeilLanes;
    if (line_first >= f.lines) return;
    // lane l owns sheared line N = line_first + l - R(nx - 1)
    const int line0 = line_first - (f.lines - f.nb);
    const float* plane = dil + (long long)((f.rows_major ? 0 : 2) + (f.band - 1)) * n;
    // offsets stay within twice (lines + nx) times a side: 32 bits unless the raster is huge
    if ((long long)(f.nb + f.nx) * (f.lines + f.nx) < (1ll << 29))
        ceiling_scan<int>(plane, f, S.cols, line0, s_seg, out, s_stage[threadIdx.y]);
    else
        ceiling_scan<long long>(plane, f, S.cols, line0, s_seg, out, s_stage[threadIdx.y]);
}

// grid (ceil((rows + cols) / 32), 1, hours), block (32, kCeilWarps): the ceiling plane
// of every daytime hour whose ray has at least kCeilMinSteps steps, from the
// dilated planes of ceiling_dilate_kernel.
static __global__ void __launch_bounds__(kCeilLanes * kCeilWarps, 2) day_ray_ceiling_kernel(
    SolweigScene S, const SolweigHour* __restrict__ hours, const float* __restrict__ dil,
    float2* __restrict__ ceiling) {
    __shared__ float s_seg[kCeilWarps][kCeilLanes];
    const SolweigHour& h = hours[blockIdx.z];
    if (!h.daytime) return;
    ray_ceiling_block(S, reinterpret_cast<const int2*>(h.ray_dxdy), h.ray_dz, h.steps, dil,
                      ceiling + (long long)blockIdx.z * S.rows * S.cols, s_seg);
}

// The same for sky-patch rays: grid.z = patch - patch0 of a group of count
// patches; tables [patch][capacity] with lengths[patch] steps.
static __global__ void __launch_bounds__(kCeilLanes * kCeilWarps, 2) patch_ray_ceiling_kernel(
    SolweigScene S, const int2* __restrict__ rays, const double* __restrict__ dz,
    const int32_t* __restrict__ lengths, int capacity, int patch0, int count, const float* __restrict__ dil,
    float2* __restrict__ ceiling) {
    __shared__ float s_seg[kCeilWarps][kCeilLanes];
    const int j = blockIdx.z, patch = patch0 + j;
    if (j >= count) return;
    const long long base = (long long)patch * capacity;
    ray_ceiling_block(S, rays + base, dz + base, lengths[patch], dil,
                      ceiling + (long long)j * S.rows * S.cols, s_seg);
}

}  // namespace solweig
