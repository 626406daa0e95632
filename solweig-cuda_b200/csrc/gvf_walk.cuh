// Ground view factors of a whole day by walk words (walks of up to 22 steps
// with first = 1: pixels of about 1 m and more, scenes without water).
//
// What a walk does apart from its per-hour samples depends only on the scene:
// how many samples it reads before a building, where it meets wall pixels and
// whether the pixel's own wall faces away.  gvf_walks_kernel packs that into
// one word per (pixel, direction) once per scene; day_gvf_walk_kernel then
// only adds the samples of every daytime hour.
//
// A sample is the pair (Lup, albedo * shadow).  Both come from a few land-cover
// classes and shadow values, so within a tile an hour has few distinct pairs
// (five for two ground classes: each in the sun and under trees, and (0, 0) in
// a building's shadow), whatever the rasters hold elsewhere.  With at most kWkValues of them the walk counts
// instead of adding: a sample is one 32-bit word with a one in the 5-bit field
// of its value (a walk has at most 22 samples), four hours are one 16-byte
// load and four integer additions, and the counts meet the values once per
// pixel and hour.  That halves the shared-memory traffic that bounds the walk
// (4 instead of 8 bytes per sample and hour) and leaves nothing to round until
// the end.  A tile with more values (three ground classes give seven) adds the
// pairs, two hours at a time: 2000 x 2000 px with two classes 3.56 ms a day, with
// three 6.50, with an albedo of its own per pixel 7.08, where one thread per pixel
// adding the pairs of four hours took 6.70 whatever the values; 500 x 500 px at
// 2 m 0.24, 0.41 and 0.47 against 1.18 ms.
// gvf_codes_kernel finds each tile's values and writes the number of every
// sample's value once; a tile's walk merges its own and its neighbours' values
// and stages 4 bytes per pixel and pass instead of the four 16-byte quads
// (every pixel is staged 5.3 times, as halo of its neighbours).
//
// The offsets of a step are the same for every pixel: cell offsets of the
// staged tile in the kernel's parameters, read through the uniform datapath.
#pragma once
#include "gvf_fields.cuh"
#include "gvf_words.cuh"

namespace solweig {

namespace {

constexpr int kWkThreads = 512;             // two pixels each, one after the other
constexpr int kWkHours = 4;                 // hours per pass
constexpr int kWkValues = 6;                // distinct samples of an hour that can be counted
constexpr int kWkTileValues = 15;           // ... that one tile can number (4-bit codes, 15: not ground)
constexpr int kWkDictKeys = 64;             // a tile's values of one pass, 16 per hour (16th of hour 0: too many)
constexpr int kWkMaxWidth = kWkTile + 2 * (kWkMaxSteps - 1);  // staged tile side (74)

// Every second 5-bit field of a count word, in 10 bits each (18 walks fit).
constexpr uint32_t kWkFields = 0x01f07c1fu;

// ---------------------------------------------------------- packed float32

typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pack2(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Cell offsets of samples 1 .. second - 1 of a direction, two per pair (an odd
// last one repeats), in a tile of `width` cells per row.
struct WalkOffsets {
    int2 pair[kWkDirs][(kWkMaxSteps + 1) / 2];
};

bool walk_offsets(const int32_t* dxdy, int second, int width, WalkOffsets* out) {
    for (int j = 0; j < kWkDirs; ++j) {
        const int32_t* o = dxdy + 2 * j * second;
        if (o[0] != 0 || o[1] != 0) return false;  // a walk starts at its pixel
        auto cell = [&](int m) { return o[2 * m] * width + o[2 * m + 1]; };
        for (int i = 0; i < (kWkMaxSteps + 1) / 2; ++i) {
            const int m = 2 * i + 1;
            out->pair[j][i] = make_int2(m < second ? cell(m) : 0, m + 1 < second ? cell(m + 1) : 0);
        }
    }
    return true;
}

struct DayWalkArgs {
    int second, halo, width;  // steps, halo and staged tile side (32 + 2 halo)
    uint32_t magic;           // i / width = umulhi(i, magic)
    const uint32_t* walks;
    const uint32_t* codes;    // of gvf_codes_kernel
    const unsigned long long* dict;
    WalkOffsets at;
};

struct WalkTables {                                // of a pass, behind the staged tile
    unsigned long long key[kWkHours][kWkValues];   // distinct samples in order of arrival
    float2 value[kWkHours][kWkValues];             // sorted: the same sums whatever the order
    int shift[kWkHours][kWkValues];                // arrival number of value i
    int count[kWkHours];
    uint32_t word[9][kWkHours][16];                // count word of a code of each of the 3 x 3 tiles
    int day_hour[64];
    int16_t offset[kWkDirs][kWkMaxSteps];          // a.at by step, for lanes at different steps
    int days, over, piece;                         // piece: next 8 x 4 pixel piece to walk
};
constexpr unsigned long long kWkNoKey = ~0ull;

size_t day_walk_smem_bytes(int width) {
    const size_t cells = (size_t)width * width;
    return 16 * cells + sizeof(WalkTables) + cells;
}

// Index of `key` in an insert-only table of n distinct keys, n when it is full.
__device__ __forceinline__ int find_key(unsigned long long* table, int n, unsigned long long key) {
    int slot = 0;
    for (; slot < n; ++slot) {
        unsigned long long at = *(volatile unsigned long long*)(table + slot);
        if (at == kWkNoKey) at = atomicCAS(table + slot, kWkNoKey, key);
        if (at == key || at == kWkNoKey) break;
    }
    return slot;
}

// The daytime hours of the day in order, by one warp; returns their number.
__device__ __forceinline__ int day_hours(const SolweigHour* __restrict__ hours, int nhours, int* out) {
    const int lane = threadIdx.x & 31;
    int k = 0;
    for (int h0 = 0; h0 < nhours && h0 < 64; h0 += 32) {
        const bool day = h0 + lane < nhours && hours[h0 + lane].daytime;
        const uint32_t days = __ballot_sync(0xffffffffu, day);
        if (day) out[k + __popc(days & ((1u << lane) - 1u))] = h0 + lane;
        k += __popc(days);
    }
    return k;
}

// Per 32 x 32 tile and pass of four daytime hours (grid.z): the tile's distinct
// samples (dict) and per pixel the four samples' codes and sunlit-wall bits, 5
// bits each (codes[pass][px]); also the pixels' shadow plane of the GVF and,
// in the first pass, the albedo-without-shadow plane of the scene.
constexpr int kWkCodeThreads = 256;
__global__ void __launch_bounds__(kWkCodeThreads) gvf_codes_kernel(int rows, int cols,
                                                                  const SolweigHour* __restrict__ hours, int nhours,
                                                                  const float4* __restrict__ quads,
                                                                  uint32_t* __restrict__ codes,
                                                                  unsigned long long* __restrict__ dict,
                                                                  float* __restrict__ gvf,
                                                                  const float* __restrict__ nosh_in,
                                                                  float* __restrict__ nosh) {
    __shared__ unsigned long long table[kWkDictKeys];
    __shared__ int day_hour[64], days, over;
    const int tid = threadIdx.x, g0 = blockIdx.z * kWkHours;
    const long long n = (long long)rows * cols;
    if (tid < kWkDictKeys) table[tid] = kWkNoKey;
    if (tid < 32) {
        days = day_hours(hours, nhours, day_hour);
        over = 0;
    }
    __syncthreads();
    const int nd = days;
    if (g0 >= nd) return;
    int hr[kWkHours];  // hours past the last one repeat it and are not written
#pragma unroll
    for (int k = 0; k < kWkHours; ++k) hr[k] = day_hour[min(g0 + k, nd - 1)];
    bool full = false;
#pragma unroll
    for (int i = 0; i < kWkPixels / kWkCodeThreads; ++i) {
        const int t = tid + i * kWkCodeThreads;
        const int r = blockIdx.y * kWkTile + t / kWkTile, c = blockIdx.x * kWkTile + t % kWkTile;
        if (r >= rows || c >= cols) continue;
        const long long p = (long long)r * cols + c;
        uint32_t word = 0u;
#pragma unroll
        for (int k = 0; k < kWkHours; ++k) {
            const float4 q = __ldg(quads + hr[k] * n + p);
            if (g0 + k < nd) gvf[(3LL * hr[k] + 2) * n + p] = q.x;
            uint32_t code = kWkTileValues;
            if ((uint32_t)__float_as_int(q.w) & kQuadGround) {  // walks never add other pixels
                const unsigned long long key = pack2(q.y, q.z * q.x);
                code = find_key(table + 16 * k, kWkTileValues, key);
                full |= code == kWkTileValues || key == kWkNoKey;
                if ((uint32_t)__float_as_int(q.w) & kQuadSunwall) code |= 16u;
            }
            word |= code << (5 * k);
        }
        codes[blockIdx.z * n + p] = word;
        if (g0 == 0 && nosh_in) nosh[p] = nosh_in[p];
    }
    if (full) over = 1;
    __syncthreads();
    if (tid < kWkDictKeys) {
        const long long tile = ((long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
        dict[tile * kWkDictKeys + tid] = tid == kWkTileValues ? (unsigned long long)over : table[tid];
    }
}

// The samples 1 .. lim - 1 of one walk: counts of four hours ...
struct CountWalk {
    typedef uint4 Sample;
    uint32_t acc[4];
    __device__ __forceinline__ void first(uint4 v) { acc[0] = v.x; acc[1] = v.y; acc[2] = v.z; acc[3] = v.w; }
    __device__ __forceinline__ void add(uint4 v) { acc[0] += v.x; acc[1] += v.y; acc[2] += v.z; acc[3] += v.w; }
    __device__ __forceinline__ void add(uint4 u, uint4 v) {
        acc[0] += u.x + v.x; acc[1] += u.y + v.y; acc[2] += u.z + v.z; acc[3] += u.w + v.w;
    }
    __device__ __forceinline__ void repeat(uint4 v, int n) {
        acc[0] += v.x * n; acc[1] += v.y * n; acc[2] += v.z * n; acc[3] += v.w * n;
    }
};
// ... or sums of two hours.
struct SumWalk {
    typedef ulonglong2 Sample;
    f32x2 acc[2];
    __device__ __forceinline__ void first(ulonglong2 v) { acc[0] = v.x; acc[1] = v.y; }
    __device__ __forceinline__ void add(ulonglong2 v) { acc[0] = add2(acc[0], v.x); acc[1] = add2(acc[1], v.y); }
    __device__ __forceinline__ void add(ulonglong2 u, ulonglong2 v) { add(u); add(v); }
    __device__ __forceinline__ void repeat(ulonglong2 v, int n) {
        const f32x2 rest = pack2((float)(n - 1), (float)(n - 1));
        acc[0] = fma2(rest, v.x, add2(acc[0], v.x));
        acc[1] = fma2(rest, v.y, add2(acc[1], v.y));
    }
};

// Samples 1 .. lim - 1 of direction j by pairs: two loads and one three-way
// addition per word.  Kept a loop: unrolled (with compiled-in offsets) it
// stalled on instruction fetch and copied its sums at every exit.
template <typename Walk>
__device__ __forceinline__ void walk_samples(Walk& w, const typename Walk::Sample* own, const WalkOffsets& at,
                                             const int16_t* offset, int j, int lim) {
#pragma unroll 2
    for (int m = 1; m + 1 < lim; m += 2) {
        const int2 o = at.pair[j][m >> 1];
        w.add(own[o.x], own[o.y]);
    }
    if (lim > 1 && !(lim & 1)) w.add(own[offset[lim - 1]]);  // an even number of samples leaves the last one
}

// One pass (four daytime hours, grid.z) of one 32 x 32 tile.  Two blocks per SM,
// so one stages its hours while the other walks.  What bounds it (1000^2 day):
// instruction issue (63 % of the cycles) and shared-memory wavefronts (56 %),
// a sixth of the warps' time at barriers.  The GVF stage per day, against one
// thread per pixel adding float pairs of four hours from 33 bytes of shared
// memory: 6.70 -> 3.59 ms at 2000^2, 1.75 -> 0.90 ms at 1090 x 871, 0.224 ->
// 0.060 ms at 64 x 48 (one block per tile and pass instead of per tile).
//
// Per hour and direction, with f the first step showing a sunlit wall:
//   lup += c1 (e lw + l0) + c2 (w lw + sum),  the albedo with albedo_b for lw,
// where the sum runs over the walk's samples, c2 = 0.4 / 0.9 / (second + 1)
// and w = second - f (0 when f = 0 on a wall facing away) when such a wall was
// met, else c2 = 0.4 / 0.9 / second and w = 0.  The near term (first = 1) is
// the pixel's own sample l0 in every direction, e = 1 and c1 halved when the
// pixel itself is a sunlit wall: it is added once, 18 fold.
__global__ void __launch_bounds__(kWkThreads, 2) day_gvf_walk_kernel(SolweigScene S,
                                                                    const SolweigHour* __restrict__ hours, int nhours,
                                                                    const __grid_constant__ DayWalkArgs a,
                                                                    const float4* __restrict__ quads,
                                                                    float* __restrict__ gvf) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int width = a.width, second = a.second, cells = width * width;
    uint4* plane = reinterpret_cast<uint4*>(smem_raw);
    WalkTables& tb = *reinterpret_cast<WalkTables*>(plane + cells);
    uint8_t* bits = reinterpret_cast<uint8_t*>(&tb + 1);  // sunlit-wall bits of the pass hours
    const int tid = threadIdx.x;
    const int tr = blockIdx.y, tc = blockIdx.x;
    const long long n = (long long)S.rows * S.cols;
    const int row0 = tr * kWkTile - a.halo, col0 = tc * kWkTile - a.halo;
    if (tid < 32) tb.days = day_hours(hours, nhours, tb.day_hour);
    for (int i = tid; i < kWkDirs * kWkMaxSteps; i += kWkThreads) {
        const int j = i / kWkMaxSteps, m = i % kWkMaxSteps;
        const int2 o = a.at.pair[j][m > 0 ? (m - 1) >> 1 : 0];
        tb.offset[j][m] = (int16_t)(m == 0 ? 0 : m & 1 ? o.x : o.y);
    }
    __syncthreads();
    const int nd = tb.days;
    const uint32_t* words = a.walks + (long long)(tr * gridDim.x + tc) * kWkTileWords;
    const float inv_far = (0.4f / 0.9f) / (float)second, inv_far1 = (0.4f / 0.9f) / (float)(second + 1);
    constexpr float albedo_b = 0.2f, inv18 = 1.f / 18.f;

    // the pass's hour of slot k (slots past the last hour repeat it and are not written)
    auto pass_hour = [&](int g0, int k) { return tb.day_hour[min(g0 + k, nd - 1)]; };
    // GVF planes of pixel p and hour hr from its far terms
    auto store = [&](int hr, long long p, bool ground, float far_lup, float far_alb) {
        const SolweigHour& h = hours[hr];
        const float4 q = __ldg(quads + hr * n + p);
        const float l0 = q.y, a0 = q.z * q.x;
        float lup = 18.f * l0, alb = 18.f * a0;
        if (ground) {
            const bool near = (uint32_t)__float_as_int(q.w) & kQuadSunwall;
            const float lw = (float)(kSBC * 0.9 * pow4(h.tgwall + h.ta + 273.15) - kSBC * 0.9 * pow4(h.ta + 273.15));
            const float c1 = near ? 18.f * (0.25f / 0.9f) : 18.f * (0.5f / 0.9f);
            lup = fmaf(c1, near ? lw + l0 : l0, far_lup);
            alb = fmaf(c1, near ? albedo_b + a0 : a0, far_alb);
        }
        gvf[(3LL * hr) * n + p] = (float)((double)(lup * inv18) + kSBC * (double)S.emis[p] * pow4(h.ta + 273.15));
        gvf[(3LL * hr + 1) * n + p] = alb * inv18;
    };
    // first sunlit wall of each slot (byte k) among the wall pixels of a walk
    auto sunlit = [&](uint32_t code, int own, int j, uint32_t& seen, uint32_t& first) {
        uint32_t walls = code & kWkWallBits;
        seen = first = 0u;
        while (walls) {
            const int m = __ffs((int)walls) - 1;
            walls &= walls - 1u;
            const uint32_t b = bits[own + tb.offset[j][m]];
            const uint32_t fresh = ((b * 0x00204081u) & 0x01010101u) & ~seen;  // bit k -> byte k
            seen |= fresh;
            first += fresh * (uint32_t)m;
        }
    };

    // the next 8 x 4 piece's pixel of this thread: warps take pieces as they get
    // free, since walks are of very different lengths
    auto next_piece = [&]() {
        int w = 0;
        if ((tid & 31) == 0) w = atomicAdd(&tb.piece, 1);
        return __shfl_sync(0xffffffffu, w, 0) * 32 + (tid & 31);
    };

    for (int g0 = blockIdx.z * kWkHours; g0 < nd; g0 += gridDim.z * kWkHours) {
        __syncthreads();  // the previous pass no longer reads the tile
        if (tid < kWkHours * kWkValues) (&tb.key[0][0])[tid] = kWkNoKey;
        if (tid == 0) tb.over = tb.piece = 0;
        __syncthreads();
        const int pass = g0 / kWkHours;
        for (int i = tid; i < 9 * kWkDictKeys; i += kWkThreads) {
            // one value of this or a neighbouring tile
            const int nb = i / kWkDictKeys, k = (i % kWkDictKeys) >> 4, s = i & 15;
            const int yt = tr + nb / 3 - 1, xt = tc + nb % 3 - 1;
            uint32_t word = 0u;
            if ((unsigned)yt < gridDim.y && (unsigned)xt < gridDim.x) {
                const unsigned long long key =
                    a.dict[(((long long)pass * gridDim.y + yt) * gridDim.x + xt) * kWkDictKeys + (i % kWkDictKeys)];
                if (s == kWkTileValues) {
                    if (k == 0 && key != 0ull) tb.over = 1;
                } else if (key != kWkNoKey) {
                    const int slot = find_key(tb.key[k], kWkValues, key);
                    if (slot == kWkValues) tb.over = 1;
                    else word = 1u << (5 * slot);
                }
            }
            tb.word[nb][k][s] = word;
        }
        __syncthreads();
#pragma unroll 4
        for (int i = tid; i < cells; i += kWkThreads) {
            const int y = (int)__umulhi((uint32_t)i, a.magic), x = i - y * width;
            const int rr = row0 + y, cc = col0 + x;
            uint32_t code = 0x7bdefu;  // not ground in any hour
            if (in_raster(rr, cc, S.rows, S.cols)) code = __ldg(a.codes + pass * n + (long long)rr * S.cols + cc);
            const uint32_t(*words_of)[16] = tb.word[((y - a.halo + 32) >> 5) * 3 + ((x - a.halo + 32) >> 5)];
            plane[i] = make_uint4(words_of[0][code & 15u], words_of[1][(code >> 5) & 15u],
                                  words_of[2][(code >> 10) & 15u], words_of[3][(code >> 15) & 15u]);
            bits[i] = (uint8_t)(((code >> 4) & 1u) | ((code >> 8) & 2u) | ((code >> 12) & 4u) | ((code >> 16) & 8u));
        }
        if (tid < kWkHours * kWkValues) {  // values in the order of their keys
            const int k = tid / kWkValues, s = tid % kWkValues;
            const unsigned long long key = tb.key[k][s];
            int rank = 0, used = 0;
            for (int o = 0; o < kWkValues; ++o) {
                rank += tb.key[k][o] < key;
                used += tb.key[k][o] != kWkNoKey;
            }
            if (key != kWkNoKey) {
                tb.value[k][rank] = unpack2(key);
                tb.shift[k][rank] = s;
            }
            tb.count[k] = used;
        }
        __syncthreads();

        if (!tb.over) {
#pragma unroll 1
            for (int t = next_piece(); t < kWkPixels; t = next_piece()) {
                int ty, tx;
                walk_pixel(t, ty, tx);
                const int r = tr * kWkTile + ty, c = tc * kWkTile + tx;
                if (r >= S.rows || c >= S.cols) continue;
                const long long p = (long long)r * S.cols + c;
                const int own = (ty + a.halo) * width + tx + a.halo;
                const bool ground = S.flags[p] & 1;
                const uint32_t own_bits = (bits[own] * 0x00204081u) & 0x01010101u;
                // counts of all walks and of those that met a sunlit wall: even and odd fields
                uint32_t all_e[kWkHours], all_o[kWkHours], sun_e[kWkHours], sun_o[kWkHours];
#pragma unroll
                for (int k = 0; k < kWkHours; ++k) all_e[k] = all_o[k] = sun_e[k] = sun_o[k] = 0u;
                uint32_t steps02 = 0u, steps13 = 0u;  // wall steps, 16 bits per hour
                if (ground) {
                    const uint4 v0 = plane[own];
                    uint32_t next = __ldg(words + t);
#pragma unroll 1
                    for (int j = 0; j < kWkDirs; ++j) {
                        const uint32_t code = next;
                        if (j + 1 < kWkDirs) next = __ldg(words + (j + 1) * kWkPixels + t);
                        const int lim = min((int)((code >> kWkLimShift) & 31u), second);
                        CountWalk walk;
                        walk.first(v0);
                        walk_samples(walk, plane + own, a.at, tb.offset[j], j, lim);
                        if (code & kWkFrozen)  // border tiles: step lim and the rest repeat step lim - 1
                            walk.repeat(plane[own + tb.offset[j][lim - 1]], second - lim);
                        uint32_t seen, first;
                        sunlit(code, own, j, seen, first);
                        if (seen) {
                            uint32_t steps = seen * (uint32_t)second - first;
                            if (code & kWkFace) steps &= ~(own_bits * 0xFFu);
                            steps02 += steps & 0x00FF00FFu;
                            steps13 += (steps >> 8) & 0x00FF00FFu;
#pragma unroll
                            for (int k = 0; k < kWkHours; ++k) {
                                if ((seen >> (8 * k)) & 1u) {
                                    sun_e[k] += walk.acc[k] & kWkFields;
                                    sun_o[k] += (walk.acc[k] >> 5) & kWkFields;
                                }
                            }
                        }
#pragma unroll
                        for (int k = 0; k < kWkHours; ++k) {
                            all_e[k] += walk.acc[k] & kWkFields;
                            all_o[k] += (walk.acc[k] >> 5) & kWkFields;
                        }
                    }
                }
#pragma unroll
                for (int k = 0; k < kWkHours; ++k) {
                    if (g0 + k >= nd) continue;
                    const int hr = pass_hour(g0, k);
                    const uint32_t free_e = all_e[k] - sun_e[k], free_o = all_o[k] - sun_o[k];
                    float lup = 0.f, alb = 0.f;
                    for (int i = 0; i < tb.count[k]; ++i) {
                        const int s = tb.shift[k][i], sh = 10 * (s >> 1);
                        const uint32_t nf = ((s & 1 ? free_o : free_e) >> sh) & 1023u;
                        const uint32_t ns = ((s & 1 ? sun_o[k] : sun_e[k]) >> sh) & 1023u;
                        if ((nf | ns) == 0u) continue;  // not read by this pixel: nothing, though it may be NaN or inf
                        const float g = fmaf(inv_far, (float)nf, inv_far1 * (float)ns);
                        const float2 v = tb.value[k][i];
                        lup = fmaf(g, v.x, lup);
                        alb = fmaf(g, v.y, alb);
                    }
                    const uint32_t st = ((k & 1 ? steps13 : steps02) >> (16 * (k >> 1))) & 0xFFFFu;
                    const SolweigHour& h = hours[hr];
                    const float lw =
                        (float)(kSBC * 0.9 * pow4(h.tgwall + h.ta + 273.15) - kSBC * 0.9 * pow4(h.ta + 273.15));
                    store(hr, p, ground, fmaf(inv_far1 * (float)st, lw, lup), fmaf(inv_far1 * (float)st, albedo_b, alb));
                }
            }
            continue;
        }
        // too many distinct samples: the pairs themselves, two hours at a time
        for (int s0 = 0; s0 < kWkHours && g0 + s0 < nd; s0 += 2) {
            const int ha = pass_hour(g0, s0), hb = pass_hour(g0, s0 + 1);
            __syncthreads();
            if (tid == 0) tb.piece = 0;
            for (int i = tid; i < cells; i += kWkThreads) {
                const int y = (int)__umulhi((uint32_t)i, a.magic), x = i - y * width;
                const int rr = row0 + y, cc = col0 + x;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (in_raster(rr, cc, S.rows, S.cols)) {
                    const long long pix = (long long)rr * S.cols + cc;
                    const float4 qa = __ldg(quads + ha * n + pix), qb = __ldg(quads + hb * n + pix);
                    v = make_float4(qa.y, qa.z * qa.x, qb.y, qb.z * qb.x);
                }
                reinterpret_cast<float4*>(plane)[i] = v;
            }
            __syncthreads();
            const ulonglong2* sums = reinterpret_cast<const ulonglong2*>(plane);
#pragma unroll 1
            for (int t = next_piece(); t < kWkPixels; t = next_piece()) {
                int ty, tx;
                walk_pixel(t, ty, tx);
                const int r = tr * kWkTile + ty, c = tc * kWkTile + tx;
                if (r >= S.rows || c >= S.cols) continue;
                const long long p = (long long)r * S.cols + c;
                const int own = (ty + a.halo) * width + tx + a.halo;
                const bool ground = S.flags[p] & 1;
                f32x2 tot[2] = {0ull, 0ull}, wall[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const SolweigHour& h = hours[k ? hb : ha];
                    wall[k] = pack2((float)(kSBC * 0.9 * pow4(h.tgwall + h.ta + 273.15) - kSBC * 0.9 * pow4(h.ta + 273.15)),
                                    albedo_b);
                }
#pragma unroll 1
                for (int j = 0; ground && j < kWkDirs; ++j) {
                    const uint32_t code = __ldg(words + j * kWkPixels + t);
                    const int lim = min((int)((code >> kWkLimShift) & 31u), second);
                    SumWalk walk;
                    walk.first(sums[own]);
                    walk_samples(walk, sums + own, a.at, tb.offset[j], j, lim);
                    if (code & kWkFrozen) walk.repeat(sums[own + tb.offset[j][lim - 1]], second - lim);
                    uint32_t seen, first;
                    sunlit(code, own, j, seen, first);
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const bool sun = (seen >> (8 * (s0 + k))) & 1u;
                        const int f = (int)((first >> (8 * (s0 + k))) & 0xFFu);
                        const float w = sun && !((code & kWkFace) && f == 0) ? (float)(second - f) : 0.f;
                        const float g = sun ? inv_far1 : inv_far;
                        tot[k] = fma2(pack2(g, g), fma2(pack2(w, w), wall[k], walk.acc[k]), tot[k]);
                    }
                }
                const float2 ta = unpack2(tot[0]), tb2 = unpack2(tot[1]);
                store(ha, p, ground, ta.x, ta.y);
                if (g0 + s0 + 1 < nd) store(hb, p, ground, tb2.x, tb2.y);
            }
        }
    }
}

// The scene's walk words and albedo-without-shadow plane (one launch per
// scene), and on request the walk-length codes alone ([4][px], 5 directions
// of 6 bits per word: samples read, frozen tail).  32 x 32 tiles staged with
// a halo of 21 as ground / wall / outside bits and albedo, 1024 threads, two blocks
// per SM (32 registers; one block at 34: 0.28 against 0.34 ms at 1000^2, bound by
// instruction issue).
constexpr int kWkStagedN = kWkMaxWidth * kWkMaxWidth;

size_t gvf_walks_smem_bytes() { return sizeof(float) * kWkStagedN + ((kWkStagedN + 15) & ~15); }

__global__ void __launch_bounds__(kWkPixels, 2) gvf_walks_kernel(SolweigScene S, int second,
                                                                     const __grid_constant__ GvfTable<kWkMaxSteps> tab,
                                                                     uint32_t* __restrict__ hits_out,
                                                                     uint32_t* __restrict__ walks_out,
                                                                     float* __restrict__ nosh_out) {
    constexpr int halo = kWkMaxSteps - 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* albs = reinterpret_cast<float*>(smem_raw);
    uint8_t* bits = reinterpret_cast<uint8_t*>(albs + kWkStagedN);  // 1 ground, 2 wall, 4 outside
    const int tr = blockIdx.y, tc = blockIdx.x;
    const int tid = threadIdx.x;
    const long long n = (long long)S.rows * S.cols;
    const int row0 = tr * kWkTile - halo, col0 = tc * kWkTile - halo;
    for (int i = tid; i < kWkStagedN; i += kWkPixels) {
        const int rr = row0 + i / kWkMaxWidth, cc = col0 + i % kWkMaxWidth;
        const bool in = in_raster(rr, cc, S.rows, S.cols);
        const long long q = in ? (long long)rr * S.cols + cc : 0;
        bits[i] = in ? (uint8_t)((S.flags[q] & 1) | (S.walls && S.walls[q] > 0.0 ? 2 : 0)) : (uint8_t)4;
        albs[i] = in ? S.alb[q] : 0.f;
    }
    __syncthreads();
    int ty, tx;
    walk_pixel(tid, ty, tx);
    const int r = tr * kWkTile + ty, c = tc * kWkTile + tx;
    const bool valid = r < S.rows && c < S.cols;
    const long long p = valid ? (long long)r * S.cols + c : 0;
    const int own = (ty + halo) * kWkMaxWidth + tx + halo;
    const bool own_ground = valid && (bits[own] & 1u);
    const uint32_t face = valid && S.gvf_face ? S.gvf_face[p] : 0u;
    const long long tile = (long long)(tr * gridDim.x + tc) * kWkTileWords;
    constexpr float albedo_b = 0.2f;
    const float inv_second = 1.f / (float)second;
    float nsh = 0.f;
    uint32_t hits[4] = {0u, 0u, 0u, 0u};
#pragma unroll 1
    for (int j = 0; j < kWkDirs; ++j) {
        int hit = 0, lim = 0;
        uint32_t walls = 0u;
        float s_alb = 0.f, n_alb = 0.f;
        if (own_ground) {
            const int* delta = tab.delta + j * second;
            uint32_t b = 1u;
            int m = 0;
#pragma unroll 2
            for (; m < second; ++m) {
                const int at = own + delta[m];
                b = bits[at];
                if (!(b & 1u)) break;
                if (b & 2u) walls |= 1u << m;
                s_alb += albs[at];
            }
            n_alb = m > 0 ? albs[own + delta[0]] : 0.f;
            hit = lim = m;
            if ((b & 4u) && m > 0) {  // frozen tail: step m and the rest repeat step m - 1
                hit = second;
                const float al = albs[own + delta[m - 1]];
                s_alb += al;
                s_alb += (second - 1 - m) * al;
            }
        }
        const bool frozen = hit > lim;
        if (hits_out) hits[j / 5] |= ((uint32_t)lim | (frozen ? 32u : 0u)) << (6 * (j % 5));
        if (walks_out)
            walks_out[tile + j * kWkPixels + tid] =
                walls | ((uint32_t)lim << kWkLimShift) | (frozen ? kWkFrozen : 0u) | (((face >> j) & 1u) ? kWkFace : 0u);
        const int n_wall = second - hit;
        const float nosh1 = hit < 1 ? (albedo_b + n_alb) * 0.5f : n_alb;
        const float nosh2 = n_wall > 0 ? ((float)n_wall * albedo_b + s_alb) * inv_second : s_alb * inv_second;
        nsh += (nosh1 * 0.5f + nosh2 * 0.4f) * (1.f / 0.9f);
    }
    if (!valid) return;
    const float ob = own_ground ? 1.f : 0.f;
    nsh *= ob;
    nsh += 18.f * (albs[own] * (1.f - ob));
    if (hits_out)
        for (int w = 0; w < 4; ++w) hits_out[(long long)w * n + p] = hits[w];
    nosh_out[p] = nsh / 18.f;
}

}  // namespace

}  // namespace solweig
