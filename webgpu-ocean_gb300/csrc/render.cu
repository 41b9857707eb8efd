// render.cu -- headless restatement of WebGPU-Ocean's screen-space fluid
// renderer (render/fluidRender.ts:292-488, fluid path), reading the posvel
// records the simulator writes and producing an image in device memory.
//
// Passes (reference shader in brackets):
//   k_tile_count, k_tile_scan, k_tile_fill   billboards by screen tile
//   k_splat_tiles     depth and thickness splats of every particle's
//                     screen-aligned billboard [depthMap.wgsl:34-79,
//                     thicknessMap.wgsl:27-62]
//   k_resolve         depth map (view z of the nearest fragment) and the
//                     thickness map (r16float)
//   k_filter x 8      separable bilateral filter of the depth map, 4 x (X, Y)
//                     [bilateral.wgsl:18-75], and with its first two passes the
//                     separable gaussian of the thickness map, (X, Y)
//                     [gaussian.wgsl:14-42]
//   k_shade           normals, lighting, fresnel, transmittance, cube-map
//                     reflection [fluid.wgsl:37-98]
// and, for the sphere mode (sphereRenderFl, fluidRender.ts:481-485):
//   the same four     the depth test of every billboard [sphere.wgsl:37-64]
//   k_sphere_shade    the winning particle's lit sphere, coloured by speed
//                     [sphere.wgsl:67-110]
//
// Rasterisation, restated for these billboards: with a perspective matrix
// without skew all four corners of a billboard share their clip w, so the
// quad covers an axis-aligned rectangle [X0, X1) x [Y0, Y1) of the
// framebuffer (x right, y down; pixel centres at +0.5), edges by the
// top-left rule, and the uv varying is linear in screen space.  A quad whose
// plane lies outside the depth range [0, 1] is clipped.  The depth test
// ('less' against a cleared 1.0, first-drawn fragment wins ties) is an
// atomicMin on (depth bits << 32 | particle index); frag_depth is clamped to
// [0, 1].  Thickness is the sum of every fragment's 0.05*sqrt(1 - r^2)
// (additive blending, no depth test), accumulated exactly in 2^-32 fixed
// point and rounded once to r16float, instead of the reference's blend-order
// dependent r16float additions.  Texture loads clamp their coordinates to the
// texture (WGSL's vec2u() saturates negative coordinates at 0; the far edge
// follows the clamping robustness of WebGPU implementations).  Every
// r16float texture write rounds to half precision.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/mpm.h"
#include "f32x2.cuh"
#include "pdl.cuh"
#include "render_math.cuh"

namespace mpm {
void set_last_error(const std::string& msg);  // capi.cu
}

using namespace mpm::x2;
using mpm::launch_pdl;
using mpm::pdl_begin;
using mpm::pdl_wait;
using namespace mpm::rmath;

namespace {

struct Uni {
    float texel[2];
    float sphere_size;
    float pad;
    float invP[16];
    float P[16];
    float V[16];
    float invV[16];
};
static_assert(sizeof(Uni) == 272, "RenderUniforms layout (common.ts:1-9)");

struct Consts {
    int W, H;
    float depth_threshold;   // radius * 10           (fluidRender.ts:38-46)
    float max_filter_size;   // 100
    float ppc;               // projected_particle_constant
};

constexpr uint32_t kOneBits = 0x3f800000u;  // 1.0f
constexpr unsigned long long kClearKey = ((unsigned long long)kOneBits << 32) | 0xffffffffull;

__device__ __forceinline__ float half_round(float x) { return __half2float(__float2half_rn(x)); }

__device__ __forceinline__ float wmax(float a, float b) {
    if (a != a) return b;
    if (b != b) return a;
    return a < b ? b : a;
}
__device__ __forceinline__ float wmin(float a, float b) {
    if (a != a) return b;
    if (b != b) return a;
    return b < a ? b : a;
}

// Screen rectangle and per-fragment quantities of particle i.
struct Billboard {
    V3 view;
    float fxm, fxp, fym, fyp;  // framebuffer x of the uv.x = 0 / 1 edges, y of uv.y = 0 / 1
    int x0, x1, y0, y1;        // covered pixel range, inclusive; empty when x0 > x1
};

__device__ __forceinline__ bool billboard_at(const float4& p, const Uni& u, const Consts& c,
                                             Billboard& b) {
    const float4 vp = mat4_mul(u.V, p.x, p.y, p.z, 1.0f);
    b.view = v3(vp.x, vp.y, vp.z);
    const float s = u.sphere_size;
    const float4 cm = mat4_mul(u.P, add(b.view.x, mul(-0.5f, s)), add(b.view.y, mul(-0.5f, s)), b.view.z, 1.0f);
    const float4 cp = mat4_mul(u.P, add(b.view.x, mul(0.5f, s)), add(b.view.y, mul(0.5f, s)), b.view.z, 1.0f);
    const float4 cc = mat4_mul(u.P, b.view.x, b.view.y, b.view.z, 1.0f);
    if (!(cc.w > 0.0f)) return false;
    const float zq = dvd(cc.z, cc.w);
    if (!(zq >= 0.0f && zq <= 1.0f)) return false;
    const float W = (float)c.W, H = (float)c.H;
    b.fxm = mul(add(dvd(cm.x, cm.w), 1.0f), mul(0.5f, W));
    b.fxp = mul(add(dvd(cp.x, cp.w), 1.0f), mul(0.5f, W));
    b.fym = mul(sub(1.0f, dvd(cm.y, cm.w)), mul(0.5f, H));
    b.fyp = mul(sub(1.0f, dvd(cp.y, cp.w)), mul(0.5f, H));
    const float X0 = fminf(b.fxm, b.fxp), X1 = fmaxf(b.fxm, b.fxp);
    const float Y0 = fminf(b.fym, b.fyp), Y1 = fmaxf(b.fym, b.fyp);
    if (!(X1 > X0) || !(Y1 > Y0)) return false;
    // pixel centres px + 0.5 in [X0, X1), clamped to the image before the
    // conversion to int
    const float lx = ceilf(sub(X0, 0.5f)), hx = sub(ceilf(sub(X1, 0.5f)), 1.0f);
    const float ly = ceilf(sub(Y0, 0.5f)), hy = sub(ceilf(sub(Y1, 0.5f)), 1.0f);
    b.x0 = (int)fminf(fmaxf(lx, 0.0f), W);
    b.x1 = (int)fmaxf(fminf(hx, W - 1.0f), -1.0f);
    b.y0 = (int)fminf(fmaxf(ly, 0.0f), H);
    b.y1 = (int)fmaxf(fminf(hy, H - 1.0f), -1.0f);
    return b.x0 <= b.x1 && b.y0 <= b.y1;
}

__device__ __forceinline__ bool billboard(const float4* posvel, int i, const Uni& u, const Consts& c,
                                          Billboard& b) {
    return billboard_at(posvel[2 * (size_t)i], u, c, b);
}

// Fragment of billboard b at pixel (px, py): false when discarded (r^2 > 1).
struct Frag {
    float depth;  // clamped frag_depth
    float vz;     // colour: view z of the sphere surface
    float nz;     // sqrt(1 - r^2)
};

__device__ __forceinline__ bool fragment(const Billboard& b, int px, int py, const Uni& u, Frag& f) {
    const float cx = add((float)px, 0.5f), cy = add((float)py, 0.5f);
    const float uu = dvd(sub(cx, b.fxm), sub(b.fxp, b.fxm));
    const float vv = dvd(sub(cy, b.fym), sub(b.fyp, b.fym));
    const float nx = sub(mul(uu, 2.0f), 1.0f), ny = sub(mul(vv, 2.0f), 1.0f);
    const float r2 = add(mul(nx, nx), mul(ny, ny));
    if (r2 > 1.0f) return false;
    const float nz = __fsqrt_rn(sub(1.0f, r2));
    const float radius = dvd(u.sphere_size, 2.0f);
    const V3 rv = vadd(b.view, vscale(v3(nx, ny, nz), radius));
    const float4 clip = mat4_mul(u.P, rv.x, rv.y, rv.z, 1.0f);
    f.depth = wmin(wmax(dvd(clip.z, clip.w), 0.0f), 1.0f);
    f.vz = rv.z;
    f.nz = nz;
    return true;
}

// ---------------------------------------------------------------------------
// Splats.  A particle's fragments (50-200) each meet the pixel's depth key
// (64-bit minimum) and thickness (64-bit sum).  Done with global atomics they
// are bound by the L2's atomic rate: one thread per billboard left every lane of
// a warp in a sector of its own, 87e9 atomics/s.  So the billboards are binned
// by 32 x 32-pixel tile first, and a block takes up to kItem of a tile's
// billboards at a time with the tile's pixels in shared memory; each touched
// pixel goes to memory once per block.  Minima and integer sums do not depend
// on the order.  Bound by instruction issue now.  Binning and splats, ncu:
// 70,000 particles at 896x504 127 -> 70 us, a million at 1344x756 417 -> 238 us;
// whole sphere frames 119 -> 64 us (70,000), 344 -> 204 us (a million).
//
// A billboard over more than two tiles along an axis, or one whose edges are
// not ordinary numbers, goes to a list of its own, which warps draw straight
// into memory with the general fragment code; so does every billboard when the
// image has more than kMaxTiles tiles.
// ---------------------------------------------------------------------------
constexpr int kTile = 32;
constexpr int kMaxTiles = 8192;            // counted in shared memory; 3840 x 2160 has 8160
constexpr int kRound = 1 << 20;            // particles binned at a time
constexpr int kItem = 256;                 // billboards per work item
constexpr int kMaxItems = kMaxTiles + 4 * (kRound / 32);
constexpr int kBinBlock = 1024;
constexpr int kTileBlock = 256;
constexpr uint32_t kNoTile = 0xffffffffu, kBig = 0xfffffffeu;

struct Item {
    int tile, first, count;
};

// The binning's buffers, made with the renderer.
struct Bins {
    uint32_t* rect;     // per particle of the round: its tiles, kNoTile or kBig
    uint32_t* count;    // per tile; zero between rounds
    uint32_t* cursor;   // per tile: the next free entry
    uint32_t* entry;    // particle indices by tile
    uint32_t* big;      // particles that are not binned
    Item* item;
    int* state;         // items, big ones, next item to take, next big one
    int tx, ty;         // tiles along x and y
};

// Tiles of billboard b, first tile | second column << 30 | second row << 31.
__device__ __forceinline__ uint32_t tile_rect(const Billboard& b, const Bins& bins) {
    const float most = 1.0e6f;
    const float dx = fabsf(sub(b.fxp, b.fxm)), dy = fabsf(sub(b.fyp, b.fym));
    if (!(fabsf(b.fxm) < most && fabsf(b.fxp) < most && fabsf(b.fym) < most && fabsf(b.fyp) < most &&
          dx > 1.0e-5f && dy > 1.0e-5f))
        return kBig;
    const int x0 = b.x0 / kTile, x1 = b.x1 / kTile, y0 = b.y0 / kTile, y1 = b.y1 / kTile;
    if (x1 - x0 > 1 || y1 - y0 > 1) return kBig;
    return (uint32_t)(y0 * bins.tx + x0) | (uint32_t)(x1 - x0) << 30 | (uint32_t)(y1 - y0) << 31;
}

// Calls f(tile) for each tile of a binned particle.
template <class F>
__device__ __forceinline__ void for_tiles(uint32_t rect, const Bins& bins, F&& f) {
    const int t = (int)(rect & 0x3fffffffu);
    const bool right = (rect >> 30) & 1u, down = rect >> 31;
    f(0, t);
    if (right) f(1, t + 1);
    if (down) f(2, t + bins.tx);
    if (right && down) f(3, t + bins.tx + 1);
}

// Tile counts of particles [first, first + n) and their tile rectangles; also
// clears the image's keys and sums (npix of them, in the first round).
__global__ void __launch_bounds__(kBinBlock)
    k_tile_count(const float4* __restrict__ posvel, int first, int n, Uni u, Consts c, Bins bins,
                 unsigned long long* __restrict__ dkey, unsigned long long* __restrict__ tacc,
                 int npix) {
    pdl_begin();
    extern __shared__ uint32_t s_count[];
    const int tiles = bins.tx * bins.ty;
    const int i = blockIdx.x * kBinBlock + threadIdx.x;
    for (int p = i; p < npix; p += gridDim.x * kBinBlock) {
        dkey[p] = kClearKey;
        if (tacc) tacc[p] = 0ull;
    }
    if (blockIdx.x * kBinBlock >= n) return;
    for (int t = threadIdx.x; t < tiles; t += kBinBlock) s_count[t] = 0u;
    __syncthreads();
    if (i < n) {
        Billboard b;
        const uint32_t rect = billboard(posvel, first + i, u, c, b) ? tile_rect(b, bins) : kNoTile;
        bins.rect[i] = rect;
        if (rect < kBig) for_tiles(rect, bins, [&](int, int t) { atomicAdd(s_count + t, 1u); });
    }
    __syncthreads();
    for (int t = threadIdx.x; t < tiles; t += kBinBlock)
        if (s_count[t]) atomicAdd(bins.count + t, s_count[t]);
}

// First entries of the tiles and the work items, one block.
__global__ void __launch_bounds__(1024) k_tile_scan(Bins bins, uint32_t per) {
    pdl_begin();
    pdl_wait();
    constexpr uint32_t kOwn = 4;  // items of a tile that its thread writes
    __shared__ uint32_t s_w[2][32];
    const int tiles = bins.tx * bins.ty;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t done[2] = {0u, 0u};  // entries and items of the tiles before this pass
    for (int t0 = 0; t0 < tiles; t0 += 1024) {
        const int t = t0 + (int)threadIdx.x;
        const uint32_t c = t < tiles ? bins.count[t] : 0u;
        const uint32_t x[2] = {c, (c + per - 1) / per};
        uint32_t v[2] = {x[0], x[1]};
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, v[k], o);
                if ((int)lane >= o) v[k] += y;
            }
        __syncthreads();  // s_w of the pass before is read
        if (lane == 31) {
            s_w[0][warp] = v[0];
            s_w[1][warp] = v[1];
        }
        __syncthreads();
        uint32_t before[2], all[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            uint32_t w = s_w[k][lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
                if ((int)lane >= o) w += y;
            }
            all[k] = __shfl_sync(0xffffffffu, w, 31);
            before[k] = __shfl_sync(0xffffffffu, w, (int)(warp + 31u) & 31);
            before[k] = done[k] + (warp ? before[k] : 0u) + v[k] - x[k];
            done[k] += all[k];
        }
        if (t < tiles) {
            bins.cursor[t] = before[0];
            if (c) bins.count[t] = 0u;
#pragma unroll
            for (uint32_t k = 0; k < kOwn; ++k)
                if (k < x[1])
                    bins.item[before[1] + k] = Item{t, (int)(before[0] + k * per), (int)min(c - k * per, per)};
        }
        // tiles with more have dozens: their other items by the whole warp
        for (unsigned left = __ballot_sync(0xffffffffu, x[1] > kOwn); left; left &= left - 1u) {
            const int src = __ffs((int)left) - 1;
            const uint32_t count = __shfl_sync(0xffffffffu, c, src);
            const uint32_t first = __shfl_sync(0xffffffffu, before[0], src);
            const uint32_t at = __shfl_sync(0xffffffffu, before[1], src);
            for (uint32_t k = kOwn + lane; k * per < count; k += 32)
                bins.item[at + k] = Item{t - (int)lane + src, (int)(first + k * per), (int)min(count - k * per, per)};
        }
    }
    if (threadIdx.x == 0) {
        bins.state[0] = (int)done[1];
        bins.state[1] = bins.state[2] = bins.state[3] = 0;
    }
}

// The tiles' entries.  A block reserves its share of each tile with one atomic.
__global__ void __launch_bounds__(kBinBlock) k_tile_fill(int first, int n, Bins bins) {
    pdl_begin();
    extern __shared__ uint32_t s_count[];
    const int tiles = bins.tx * bins.ty;
    for (int t = threadIdx.x; t < tiles; t += kBinBlock) s_count[t] = 0u;
    __syncthreads();
    pdl_wait();
    const int i = blockIdx.x * kBinBlock + threadIdx.x;
    const uint32_t rect = i < n ? bins.rect[i] : kNoTile;
    uint32_t rank[4];
    if (rect < kBig)
        for_tiles(rect, bins, [&](int k, int t) { rank[k] = atomicAdd(s_count + t, 1u); });
    else if (rect == kBig)
        bins.big[atomicAdd(bins.state + 1, 1)] = (uint32_t)(first + i);
    __syncthreads();
    for (int t = threadIdx.x; t < tiles; t += kBinBlock)
        if (s_count[t]) s_count[t] = atomicAdd(bins.cursor + t, s_count[t]);
    __syncthreads();
    if (rect < kBig)
        for_tiles(rect, bins, [&](int k, int t) { bins.entry[s_count[t] + rank[k]] = (uint32_t)(first + i); });
}

// Billboard of particle i drawn into memory by one warp.
template <bool THICK>
__device__ __forceinline__ void draw_big(const float4* __restrict__ posvel, int i, const Uni& u,
                                         const Consts& c, unsigned long long* __restrict__ dkey,
                                         unsigned long long* __restrict__ tacc) {
    Billboard b;
    if (!billboard(posvel, i, u, c, b)) return;
    for (int py = b.y0; py <= b.y1; ++py)
        for (int px = b.x0 + (int)(threadIdx.x & 31u); px <= b.x1; px += 32) {
            Frag f;
            if (!fragment(b, px, py, u, f)) continue;
            const size_t p = (size_t)py * c.W + px;
            if (f.depth < 1.0f)
                atomicMin(dkey + p, ((unsigned long long)__float_as_uint(f.depth) << 32) | (unsigned)i);
            if (THICK) {
                const float t = mul(0.05f, f.nz);
                atomicAdd(tacc + p, (unsigned long long)__float2ll_rn(mul(t, 4294967296.0f)));
            }
        }
}

// Every billboard that way (images of more than kMaxTiles tiles).
template <bool THICK>
__global__ void __launch_bounds__(kTileBlock)
    k_splat_direct(const float4* __restrict__ posvel, int n, Uni u, Consts c,
                   unsigned long long* __restrict__ dkey, unsigned long long* __restrict__ tacc) {
    const int i = (int)(blockIdx.x * (kTileBlock / 32) + (threadIdx.x >> 5));
    if (i < n) draw_big<THICK>(posvel, i, u, c, dkey, tacc);
}

__global__ void k_clear(unsigned long long* dkey, unsigned long long* tacc, int npix) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npix) return;
    dkey[p] = kClearKey;
    if (tacc) tacc[p] = 0ull;
}

// a / b from y = RN(1 / b), correctly rounded for 2^-20 <= |b| <= 2^20 and
// quotients of 0 or of magnitudes 2^-60 to 2^20: P. Markstein's final
// correction (IBM J. Res. Dev. 34, 1990) of a quotient within an ulp.
__device__ __forceinline__ float quot(float a, float b, float y) {
    float q = mul(a, y);
    q = __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
    return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}

// A billboard of a work item as the threads read it: uv.x = (x - fxm) / dx,
// uv.y = (y - fym) / dy with the reciprocals; dmin: no fragment is nearer.
struct __align__(16) TileBoard {
    float fxm, dx, rdx, fym;
    float dy, rdy, view_z, dmin;
    uint32_t rect;  // x0 | y0 << 8 | w << 16 | h << 24, from the tile's corner
    int index;
    float view_x, view_y;
};

constexpr int kRowPad = kTile + 1;               // a billboard's rows in different banks
constexpr int kTileCells = kTile * kRowPad;
constexpr int kItemRows = kItem * kTile;

// PERSP: clip z and w depend on view z alone, w = -z, and depth grows away
// from the camera (checked on the host); the terms of x and y are products
// with zero then, which leave the sums as they are for the finite x and y of a
// billboard on the screen.  THICK: thickness too (the sphere mode has none).
//
// A thread takes a row of a billboard at a time: the rows of an item's
// billboards are numbered (s_row), widest billboards first, so that the lanes
// of a warp walk rows of one length and mostly the nearest fragments come first.
// A fragment that is not the nearest costs a shared-memory read when its whole
// billboard lies behind the pixel (dmin), else an approximate quotient; only
// what may be the nearest takes the exact depth and the 64-bit minimum.  The
// pixels start from what other items of the tile have left in memory; the items
// of a tile are taken far apart in time so that there is something.  Measured at
// 70,000 / a million particles: a warp per billboard with a lane per pixel 72 /
// 342 us; rows in arrival order 82 / 270; narrow ones first, with the image's
// depths as the start, 58 / 196; widest first 53 / 192.  Queues of the fragments
// that may be nearest, tested exactly later: 92 / 349.
template <bool THICK, bool PERSP>
__global__ void __launch_bounds__(kTileBlock)
    k_splat_tiles(const float4* __restrict__ posvel, Uni u, Consts c, Bins bins,
                  unsigned long long* __restrict__ dkey, unsigned long long* __restrict__ tacc) {
    __shared__ unsigned long long s_key[kTileCells];
    __shared__ uint32_t s_lo[THICK ? kTileCells : 1], s_hi[THICK ? kTileCells : 1];
    __shared__ TileBoard s_b[kItem];
    __shared__ uint16_t s_row[kItemRows];  // billboard | row << 8
    __shared__ int s_warp[kTileBlock / 32];
    __shared__ int s_wide[kTile];          // billboards by width, then their first places
    __shared__ uint8_t s_h[kItem];         // rows of each, in their order
    __shared__ int s_item;
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const float radius = dvd(u.sphere_size, 2.0f);
    pdl_begin();
    if (THICK)
        for (int p = threadIdx.x; p < kTileCells; p += kTileBlock) s_lo[p] = s_hi[p] = 0u;
    pdl_wait();
    const int items = bins.state[0], big = bins.state[1];
    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(bins.state + 2, 1);
        if (threadIdx.x < kTile) s_wide[threadIdx.x] = 0;
        __syncthreads();
        const int claim = s_item;
        if (claim >= items) break;  // uniform
        // a prime above kMaxItems: every item once, a tile's far apart in time
        const Item item = bins.item[(unsigned long long)claim * 1000003ull % (unsigned)items];
        const int tx = (item.tile % bins.tx) * kTile, ty = (item.tile / bins.tx) * kTile;
        static_assert(kItem == kTileBlock && kItem == 256, "a thread per billboard, numbers of 8 bits");
        for (int p = threadIdx.x; p < kTileCells; p += kTileBlock) {
            const int x = tx + p % kRowPad, y = ty + p / kRowPad;
            s_key[p] = p % kRowPad < kTile && x < c.W && y < c.H ? __ldcg(dkey + (size_t)y * c.W + x) : 0ull;
        }
        const bool mine = (int)threadIdx.x < item.count;
        TileBoard t;
        int w = 0, h = 0, place = 0;
        if (mine) {
            const int i = (int)bins.entry[item.first + threadIdx.x];
            Billboard b;
            billboard(posvel, i, u, c, b);
            const int x0 = max(b.x0 - tx, 0), x1 = min(b.x1 - tx, kTile - 1);
            const int y0 = max(b.y0 - ty, 0), y1 = min(b.y1 - ty, kTile - 1);
            w = x1 - x0 + 1;
            h = y1 - y0 + 1;
            t.fxm = b.fxm;
            t.dx = sub(b.fxp, b.fxm);
            t.rdx = __frcp_rn(t.dx);
            t.fym = b.fym;
            t.dy = sub(b.fyp, b.fym);
            t.rdy = __frcp_rn(t.dy);
            t.view_x = b.view.x;
            t.view_y = b.view.y;
            t.view_z = b.view.z;
            // the depth of the sphere's nearest point, less what rounding
            // (here and in a fragment, both below 5e-7 of depths up to 1) can be
            const float zn = b.view.z + radius;
            t.dmin = PERSP && zn < 0.0f ? __fdividef(u.P[10] * zn + u.P[14], -zn) - 2.0e-6f : -1.0f;
            t.rect = (uint32_t)x0 | (uint32_t)y0 << 8 | (uint32_t)w << 16 | (uint32_t)h << 24;
            t.index = i;
            w = kTile - w;  // widest, and so mostly nearest, first
            place = atomicAdd(s_wide + w, 1);
        }
        __syncthreads();
        if (warp == 0) {  // first places by width
            const int v = s_wide[lane];
            int upto = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, upto, o);
                if ((int)lane >= o) upto += y;
            }
            s_wide[lane] = upto - v;
        }
        __syncthreads();
        if (mine) {
            place += s_wide[w];
            s_b[place] = t;
            s_h[place] = (uint8_t)h;
        }
        __syncthreads();
        h = mine ? s_h[threadIdx.x] : 0;  // of the billboard at this thread's place
        int upto = h;  // rows of the billboards up to this one
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if ((int)lane >= o) upto += v;
        }
        if (lane == 31) s_warp[warp] = upto;
        __syncthreads();
        int before = 0, rows = 0;
#pragma unroll
        for (int k = 0; k < kTileBlock / 32; ++k) {
            const int v = s_warp[k];
            if (k < (int)warp) before += v;
            rows += v;
        }
        before += upto - h;
        for (int k = 0; k < h; ++k) s_row[before + k] = (uint16_t)(threadIdx.x | (unsigned)k << 8);
        __syncthreads();
        for (int k = threadIdx.x; k < rows; k += kTileBlock) {
            const uint32_t m = s_row[k];
            const TileBoard t = s_b[m & 255u];
            const int x0 = (int)(t.rect & 255u), y = (int)(t.rect >> 8 & 255u) + (int)(m >> 8);
            const int wide = (int)(t.rect >> 16 & 255u);
            const float ny = sub(mul(quot(sub(add((float)(ty + y), 0.5f), t.fym), t.dy, t.rdy), 2.0f), 1.0f);
            const float ny2 = mul(ny, ny);
            float cx = add((float)(tx + x0), 0.5f);
            int p = y * kRowPad + x0;
            for (int x = 0; x < wide; ++x, ++p, cx = add(cx, 1.0f)) {
                const float near = __uint_as_float((uint32_t)(s_key[p] >> 32));
                const bool behind = near < t.dmin;
                if (!THICK && behind) continue;
                const float nx = sub(mul(quot(sub(cx, t.fxm), t.dx, t.rdx), 2.0f), 1.0f);
                const float r2 = add(mul(nx, nx), ny2);
                if (r2 > 1.0f) continue;
                const float nz = __fsqrt_rn(sub(1.0f, r2));
                if (THICK) {
                    // below 2^28, in two parts whose sums over an item's
                    // billboards fit 32 bits: additions that return nothing
                    const uint32_t v = __float2uint_rn(mul(mul(0.05f, nz), 4294967296.0f));
                    atomicAdd(s_lo + p, v & 0x3fffu);
                    atomicAdd(s_hi + p, v >> 14);
                    if (behind) continue;
                }
                const float z = add(t.view_z, mul(nz, radius));
                float cz, cw;
                if (PERSP) {
                    cz = add(mul(u.P[10], z), u.P[14]);
                    cw = sub(0.0f, z);
                } else {
                    const float4 clip = mat4_mul(u.P, add(t.view_x, mul(nx, radius)),
                                                 add(t.view_y, mul(ny, radius)), z, 1.0f);
                    cz = clip.z;
                    cw = clip.w;
                }
                // behind the nearest fragment by more than the error of the fast quotient
                if (__fdividef(cz, cw) > near * 1.000004f + 1.0e-30f) continue;
                const float depth = wmin(wmax(dvd(cz, cw), 0.0f), 1.0f);
                const unsigned long long key =
                    ((unsigned long long)__float_as_uint(depth) << 32) | (unsigned)t.index;
                if (depth < 1.0f && key < s_key[p]) atomicMin(s_key + p, key);
            }
        }
        __syncthreads();
        for (int p = threadIdx.x; p < kTileCells; p += kTileBlock) {
            if (p % kRowPad >= kTile || ty + p / kRowPad >= c.H || tx + p % kRowPad >= c.W) continue;
            const size_t q = (size_t)(ty + p / kRowPad) * c.W + tx + p % kRowPad;
            const unsigned long long key = s_key[p];
            if (key < __ldcg(dkey + q)) atomicMin(dkey + q, key);
            if (THICK) {
                const uint32_t lo = s_lo[p], hi = s_hi[p];
                if (lo | hi) {
                    atomicAdd(tacc + q, ((unsigned long long)hi << 14) + lo);
                    s_lo[p] = s_hi[p] = 0u;
                }
            }
        }
    }
    for (;;) {  // a warp per particle that is not binned
        int k = 0;
        if (lane == 0) k = big ? atomicAdd(bins.state + 3, 1) : 0;
        k = __shfl_sync(0xffffffffu, k, 0);
        if (k >= big) break;
        draw_big<THICK>(posvel, (int)bins.big[k], u, c, dkey, tacc);
    }
}

__global__ void k_resolve(const float4* __restrict__ posvel, Uni u, Consts c,
                          const unsigned long long* dkey, const unsigned long long* tacc,
                          float* depth, float* thick) {
    pdl_begin();
    pdl_wait();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= c.W * c.H) return;
    const unsigned long long key = dkey[p];
    float d = 0.0f;  // the depth map's clear colour
    if (key != kClearKey) {
        Billboard b;
        Frag f;
        const int i = (int)(key & 0xffffffffull);
        if (billboard(posvel, i, u, c, b) && fragment(b, p % c.W, p / c.W, u, f)) d = f.vz;
    }
    depth[p] = d;
    const float t = mul(__ll2float_rn((long long)tacc[p]), 2.3283064365386963e-10f);  // 2^-32
    thick[p] = half_round(t);
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// Spatial weights of the two filters, which depend only on the filter
// half-width and the tap offset: bilateral exp(-(x^2 + x^2) / (2 sigma^2)),
// sigma = fs / 3, for fs in [0, kMaxFs] and |x| <= fs (row fs at fs * kWRow);
// gaussian exp(-x^2 / (2 sigma^2)), sigma = 10, |x| <= 30.  Computed once
// with the same operations the filter bodies use, so a table read is
// bit-identical to evaluating the weight in place.
constexpr int kMaxFs = 100;
constexpr int kWRow = kMaxFs + 1;
constexpr int kGaussFs = 30;

__global__ void k_weight_tables(float* __restrict__ wtab, float* __restrict__ gtab) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < kWRow * kWRow) {
        const int fs = e / kWRow, x = e % kWRow;
        const float sigma = dvd((float)fs, 3.0f);
        const float two_sigma = mul(mul(2.0f, sigma), sigma);
        const float xf = (float)x;
        const float rr = add(mul(xf, xf), mul(xf, xf));
        wtab[e] = exp_r(dvd(-rr, two_sigma));
    }
    if (e <= kGaussFs) {
        const float sigma = dvd((float)kGaussFs, 3.0f);
        const float two_sigma = mul(mul(2.0f, sigma), sigma);
        const float xf = (float)e;
        gtab[e] = exp_r(dvd(mul(-xf, xf), two_sigma));
    }
    if (e == 0) {  // the sum of a pixel's gaussian weights, tap by tap
        const float sigma = dvd((float)kGaussFs, 3.0f);
        const float two_sigma = mul(mul(2.0f, sigma), sigma);
        float wsum = 0.0f;
        for (int x = -kGaussFs; x <= kGaussFs; ++x) {
            const float xf = (float)(x < 0 ? -x : x);
            wsum = add(wsum, exp_r(dvd(mul(-xf, xf), two_sigma)));
        }
        gtab[kGaussFs + 1] = wsum;
    }
}

// exp_series() of two numbers.  A packed product that only a packed sum reads
// would become one fused operation of other rounding; a fused one with
// -0 to add rounds as the product does and stays as it is.
__device__ __forceinline__ f2 exp_series2(f2 r, f2 zero) {
    f2 p = dup(2.48015873e-5f);
    p = add2(fma2(p, r, zero), dup(1.98412698e-4f));
    p = add2(fma2(p, r, zero), dup(1.38888889e-3f));
    p = add2(fma2(p, r, zero), dup(8.33333333e-3f));
    p = add2(fma2(p, r, zero), dup(4.16666667e-2f));
    p = add2(fma2(p, r, zero), dup(1.66666667e-1f));
    p = add2(fma2(p, r, zero), dup(0.5f));
    p = add2(fma2(p, r, zero), dup(1.0f));
    p = add2(fma2(p, r, zero), dup(1.0f));
    return p;
}

// exp_r(a / b) for a = -d^2 <= 0 and the filter's b = two_sd, the same bits with
// fewer operations and no branch, so that the taps of a pixel overlap.  The
// quotient: a product with 1 / b where b is a power of two (the application's
// radius: 8), else quot() with RN(1 / b); quotients too small for quot() give
// exp = 1 either way.  The rounding of x / ln 2 by an addition that leaves only
// the integer k, and 2^k as 2^(k + 64) * 2^-64: for k in [-152, 0] the first
// product is exact, so the result is rounded once, as exp_r's is.
struct DepthWeight {
    float b, rb, cut;  // cut: below it a / b < -104 and the weight is 0
    bool range, pow2;  // b fits quot(), is a power of two
    template <bool POW2>
    __device__ __forceinline__ float at(float d) const {
        const float a = mul(-d, d);
        const float x = POW2 ? mul(a, rb) : quot(a, b, rb);
        const float shifted = add(mul(x, 1.44269502f), kMagic);
        const float kf = sub(shifted, kMagic);
        const float r = sub(sub(x, mul(kf, 0.693145751953125f)), mul(kf, 1.42860677e-6f));
        const float e = mul(mul(exp_series(r), scale(shifted)), 0x1p-64f);
        return a < cut ? 0.0f : e;
    }
    // Two of them, in packed operations.
    template <bool POW2>
    __device__ __forceinline__ f2 at2(f2 d, f2 zero) const {
        const f2 a = mul2(d, neg2(d));
        f2 x;
        if (POW2) {
            x = mul2(a, dup(rb));
        } else {
            const f2 nb = dup(-b), y = dup(rb);
            x = mul2(a, y);
            x = fma2(fma2(nb, x, a), y, x);
            x = fma2(fma2(nb, x, a), y, x);
        }
        const f2 shifted = add2(fma2(x, dup(1.44269502f), zero), dup(kMagic));
        const f2 kf = add2(shifted, dup(-kMagic));
        f2 r = add2(x, fma2(kf, dup(-0.693145751953125f), zero));
        r = add2(r, fma2(kf, dup(-1.42860677e-6f), zero));
        const f2 scales = pk(scale(lo(shifted)), scale(hi(shifted)));
        const f2 e = mul2(mul2(exp_series2(r, zero), scales), dup(0x1p-64f));
        return pk(lo(a) < cut ? 0.0f : lo(e), hi(a) < cut ? 0.0f : hi(e));
    }
    static constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23
    // 2^(k + 64) from k + kMagic
    static __device__ __forceinline__ float scale(float shifted) {
        return __int_as_float((__float_as_int(shifted) << 23) + (191 << 23));
    }
};

__device__ __forceinline__ DepthWeight depth_weight(const Consts& c) {
    const float sd = dvd(c.depth_threshold, 3.0f);
    DepthWeight d;
    d.b = mul(mul(2.0f, sd), sd);
    d.rb = __frcp_rn(d.b);
    d.range = d.b >= 0x1p-20f && d.b <= 0x1p20f;
    d.pow2 = (__float_as_uint(d.b) & 0x7fffffu) == 0u;
    d.cut = -105.0f * d.b;
    return d;
}

// One pass of the separable bilateral filter [bilateral.wgsl:18-75], along x
// (X) or y.  Bound by the issue of the taps' exp and, where the filters are
// short, by the start of its launches.  A block holds the depths that its taps
// reach, as far as its widest filter, clamped to the image, in shared memory, so
// that a tap has no index arithmetic, and the taps' weights have no branch and
// are made two at a time.  Per pass (ncu) at 896x504 15.5 -> 12.0 us, at 1344x756
// 20.9 -> 16.8 us before the pairs; shared memory alone 13.3 and 18.3.  A pair's
// packed operations, whole images: 70,000 particles at 896x504 152.5 -> 145.5 us,
// from half as far 566 -> 534, 200,000 at 1200x800 683 -> 639, a million at
// 1344x756 364 -> 355.  One pair at a time: with the loop unrolled to two or four
// 151 / 146, 549 / 531, 652 / 646, 354 / 362.  Loading the first few texels of the
// halo together with the pixels' own, before the filters' widths are known: no
// faster.
constexpr int kFilterThreads = 256;

template <bool X>
struct Bilateral {
    static constexpr int kW = X ? 256 : 32, kH = kFilterThreads / kW;  // pixels of a block
    float d[X ? kW + 2 * kMaxFs : kW * (kH + 2 * kMaxFs)];             // shared memory
    int fs;
};

template <bool X>
__device__ __forceinline__ void bilateral_block(Bilateral<X>& sm, int block,
                                                const float* src,
                                                float* __restrict__ dst, const Consts& c,
                                                const float* __restrict__ wtab) {
    constexpr int kW = Bilateral<X>::kW, kH = Bilateral<X>::kH;
    float* s_d = sm.d;
    int& s_fs = sm.fs;
    const int columns = (c.W + kW - 1) / kW;
    const int bx = block % columns * kW, by = block / columns * kH;
    const int lx = (int)threadIdx.x % kW, ly = (int)threadIdx.x / kW;
    const int px = bx + lx, py = by + ly;
    const bool in = px < c.W && py < c.H;
    const size_t p = (size_t)py * c.W + px;
    const float depth = in ? fabsf(src[p]) : 0.0f;
    int fs = -1;
    if (in) {
        if (depth >= 1e4f || depth <= 0.0f) dst[p] = depth;
        else fs = min(__float2int_rz(c.max_filter_size), __float2int_rz(ceilf(dvd(c.ppc, depth))));
    }
    if (threadIdx.x == 0) s_fs = -1;
    __syncthreads();
    const int warp_fs = __reduce_max_sync(0xffffffffu, fs);
    if ((threadIdx.x & 31u) == 0 && warp_fs >= 0) atomicMax(&s_fs, warp_fs);
    __syncthreads();
    const int halo = s_fs;  // <= max_filter_size = kMaxFs
    if (halo < 0) return;   // uniform
    if (X) {
        for (int k = threadIdx.x; k < kW + 2 * halo; k += kFilterThreads)
            s_d[k] = fabsf(src[(size_t)by * c.W + clampi(bx - halo + k, 0, c.W - 1)]);
    } else {
        for (int k = threadIdx.x; k < kW * (kH + 2 * halo); k += kFilterThreads)
            s_d[k] = fabsf(src[(size_t)clampi(by - halo + k / kW, 0, c.H - 1) * c.W +
                               min(bx + k % kW, c.W - 1)]);
    }
    __syncthreads();
    if (fs < 0) return;
    const float* tap = X ? s_d + lx + halo : s_d + (ly + halo) * kW + lx;
    const float* wrow = wtab + fs * kWRow;
    const DepthWeight weight = depth_weight(c);
    float sum = 0.0f, wsum = 0.0f;
    auto term = [&](float sampled, float w, float wd) {
        sum = add(sum, mul(mul(sampled, w), wd));
        wsum = add(wsum, mul(w, wd));
    };
    auto at = [&](int x) { return tap[X ? x : x * kW]; };
    auto spatial = [&](int x) { return __ldg(wrow + (x < 0 ? -x : x)); };
    auto walk = [&](auto pow2) {
        constexpr bool POW2 = decltype(pow2)::value;
        const f2 nd = dup(-depth), zero = negative_zeros(c.W);
#pragma unroll 1
        for (int x = -fs; x < fs; x += 2) {
            const f2 sampled = pk(at(x), at(x + 1)), w = pk(spatial(x), spatial(x + 1));
            const f2 wd = weight.template at2<POW2>(add2(sampled, nd), zero);
            const f2 sw = mul2(mul2(sampled, w), wd), ww = mul2(w, wd);
            sum = add(add(sum, lo(sw)), hi(sw));
            wsum = add(add(wsum, lo(ww)), hi(ww));
        }
        term(at(fs), spatial(fs), weight.template at<POW2>(sub(at(fs), depth)));
    };
    if (weight.range && weight.pow2) walk(std::true_type{});
    else if (weight.range) walk(std::false_type{});
    else
        for (int x = -fs; x <= fs; ++x) {
            const float rd = sub(at(x), depth);
            term(at(x), spatial(x), exp_r(dvd(mul(-rd, rd), weight.b)));
        }
    dst[p] = dvd(sum, wsum);
}

// One pass of the separable gaussian filter of the thickness
// [gaussian.wgsl:14-42].  A thread filters four neighbouring pixels along the
// filter's axis from one walk through the 64 texels that their taps reach, in
// shared memory, so that a tap costs a product, a sum and half a load.  The
// weights' sum is the same for every pixel and was made with the table.  Per
// pass (ncu) at 896x504 15.8 -> 9.3 us, at 1344x756 26.7 -> 12.5 us.
template <bool X>
struct Gaussian {
    // along x: 4 rows of 256 pixels; along y: 32 rows of 32 pixels
    static constexpr int kW = X ? 256 : 32, kH = X ? 4 : 32;
    static constexpr int kSW = X ? kW + 2 * kGaussFs + 4 : kW, kSH = X ? kH : kH + 2 * kGaussFs;
    alignas(16) float t[kSH * kSW];  // shared memory
    alignas(16) float g[64];
};

template <bool X>
__device__ __forceinline__ void gaussian_block(Gaussian<X>& sm, int block,
                                               const float* src,
                                               float* __restrict__ dst, const Consts& c,
                                               const float* __restrict__ gtab) {
    constexpr int kTaps = 2 * kGaussFs + 1, kOut = 4;
    constexpr int kW = Gaussian<X>::kW, kH = Gaussian<X>::kH, kSW = Gaussian<X>::kSW,
                  kSH = Gaussian<X>::kSH;
    float *s_t = sm.t, *s_g = sm.g;
    const int columns = (c.W + kW - 1) / kW;
    const int bx = block % columns * kW, by = block / columns * kH;
    // this thread's first pixel, from the block's corner
    const int lx = X ? kOut * ((int)threadIdx.x & 63) : (int)threadIdx.x & 31;
    const int ly = X ? (int)threadIdx.x >> 6 : kOut * ((int)threadIdx.x >> 5);
    if (threadIdx.x < 64) {
        const int o = (int)threadIdx.x - kGaussFs;
        s_g[threadIdx.x] = threadIdx.x < kTaps ? gtab[o < 0 ? -o : o] : 0.0f;
    }
    for (int k = threadIdx.x; k < kSH * kSW; k += kFilterThreads) {
        const int x = bx + k % kSW - (X ? kGaussFs : 0), y = by + k / kSW - (X ? 0 : kGaussFs);
        s_t[k] = src[(size_t)clampi(y, 0, c.H - 1) * c.W + clampi(x, 0, c.W - 1)];
    }
    __syncthreads();
    const float* t = s_t + ly * kSW + lx;
    constexpr int kStep = X ? 1 : kSW;
    float centre[kOut];
    bool any = false;
#pragma unroll
    for (int i = 0; i < kOut; ++i) {
        centre[i] = t[(kGaussFs + i) * kStep];
        any |= centre[i] != 0.0f;
    }
    float sum[kOut] = {};
    if (any) {
        float win[kOut + 4];  // texels of the current four taps of all outputs
        auto load4 = [&](int at, float* to) {
            if (X) {
                const float4 v = *reinterpret_cast<const float4*>(t + at);
                to[0] = v.x; to[1] = v.y; to[2] = v.z; to[3] = v.w;
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) to[i] = t[min(at + i, 2 * kGaussFs + 3) * kStep];
            }
        };
        load4(0, win);
#pragma unroll 4
        for (int x = 0; x < 64; x += 4) {  // taps 61 .. 63 do not count
            load4(x + 4, win + 4);
            const float4 g4 = *reinterpret_cast<const float4*>(s_g + x);
            const float g[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (x + q < kTaps) {
#pragma unroll
                    for (int i = 0; i < kOut; ++i) sum[i] = add(sum[i], mul(win[q + i], g[q]));
                }
#pragma unroll
            for (int i = 0; i < kOut; ++i) win[i] = win[4 + i];
        }
    }
    const float wsum = gtab[kGaussFs + 1];
#pragma unroll
    for (int i = 0; i < kOut; ++i) {
        const int px = bx + lx + (X ? i : 0), py = by + ly + (X ? 0 : i);
        if (px < c.W && py < c.H)
            dst[(size_t)py * c.W + px] = centre[i] == 0.0f ? 0.0f : half_round(dvd(sum[i], wsum));
    }
}

// A bilateral pass over `depth` and, in the blocks after its own (if there are
// any), the gaussian pass along the same axis over `thick`.  The two images'
// chains do not depend on each other, and either's launches leave most of the
// GPU's issue slots unused: the gaussian's 16.5 us (ncu, 896x504; 22.8 at
// 1344x756) run in the first two bilateral launches' shadow.
struct FilterPass {
    const float* src;
    float* dst;
};

template <bool X>
__global__ void __launch_bounds__(kFilterThreads)
    k_filter(FilterPass depth, FilterPass thick, int depth_blocks, Consts c,
             const float* __restrict__ wtab, const float* __restrict__ gtab) {
    pdl_begin();
    pdl_wait();
    __shared__ __align__(16) union {
        Bilateral<X> bilateral;
        Gaussian<X> gaussian;
    } sm;
    if ((int)blockIdx.x < depth_blocks)
        bilateral_block<X>(sm.bilateral, (int)blockIdx.x, depth.src, depth.dst, c, wtab);
    else
        gaussian_block<X>(sm.gaussian, (int)blockIdx.x - depth_blocks, thick.src, thick.dst, c, gtab);
}

// fluid.wgsl:19-27: view-space position from a texture coordinate and depth.
__device__ __forceinline__ V3 view_pos(const Uni& u, float tx, float ty, float depth) {
    const float nx = sub(mul(tx, 2.0f), 1.0f);
    const float ny = sub(1.0f, mul(2.0f, ty));
    const float nz = add(-u.P[10], dvd(u.P[14], depth));
    const float4 e = mat4_mul(u.invP, nx, ny, nz, 1.0f);
    return v3(dvd(e.x, e.w), dvd(e.y, e.w), dvd(e.z, e.w));
}

// Bilinear cube-map sample (level 0), faces +x, -x, +y, -y, +z, -z of
// size x size RGBA texels; face selection and (s, t) per the usual cube-map
// table; filtering within the face, clamped to its edge.
__device__ __forceinline__ V3 sample_cube(const float4* __restrict__ env, int size, V3 d) {
    const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    int face;
    float sc, tc, ma;
    if (ax >= ay && ax >= az) {
        ma = ax;
        if (d.x >= 0.0f) { face = 0; sc = -d.z; tc = -d.y; }
        else { face = 1; sc = d.z; tc = -d.y; }
    } else if (ay >= az) {
        ma = ay;
        if (d.y >= 0.0f) { face = 2; sc = d.x; tc = d.z; }
        else { face = 3; sc = d.x; tc = -d.z; }
    } else {
        ma = az;
        if (d.z >= 0.0f) { face = 4; sc = d.x; tc = -d.y; }
        else { face = 5; sc = -d.x; tc = -d.y; }
    }
    if (!(ma > 0.0f) || ma == __int_as_float(0x7f800000)) {
        const float q = __int_as_float(0x7fc00000);
        return v3(q, q, q);
    }
    const float s = mul(0.5f, add(dvd(sc, ma), 1.0f));
    const float t = mul(0.5f, add(dvd(tc, ma), 1.0f));
    const float fu = sub(mul(s, (float)size), 0.5f), fv = sub(mul(t, (float)size), 0.5f);
    const float iu = floorf(fu), iv = floorf(fv);
    const float a = sub(fu, iu), bb = sub(fv, iv);
    const int u0 = clampi((int)iu, 0, size - 1), u1 = clampi((int)iu + 1, 0, size - 1);
    const int v0 = clampi((int)iv, 0, size - 1), v1 = clampi((int)iv + 1, 0, size - 1);
    const float4* f = env + (size_t)face * size * size;
    const float4 c00 = f[v0 * size + u0], c10 = f[v0 * size + u1];
    const float4 c01 = f[v1 * size + u0], c11 = f[v1 * size + u1];
    const float ia = sub(1.0f, a), ib = sub(1.0f, bb);
    auto lerp2 = [&](float p00, float p10, float p01, float p11) {
        const float top = add(mul(p00, ia), mul(p10, a));
        const float bot = add(mul(p01, ia), mul(p11, a));
        return add(mul(top, ib), mul(bot, bb));
    };
    return v3(lerp2(c00.x, c10.x, c01.x, c11.x), lerp2(c00.y, c10.y, c01.y, c11.y),
              lerp2(c00.z, c10.z, c01.z, c11.z));
}

__global__ void k_shade(const float* depth_map, const float* thick_map,
                        const float4* __restrict__ env, int env_size, Uni u, Consts c,
                        float4* __restrict__ out, uchar4* __restrict__ out8) {
    pdl_begin();
    pdl_wait();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= c.W * c.H) return;
    const int px = p % c.W, py = p / c.W;
    const float tx = dvd(add((float)px, 0.5f), (float)c.W);
    const float ty = dvd(add((float)py, 0.5f), (float)c.H);
    const V3 bg = v3(0.8f, 0.8f, 0.8f);
    const float depth = fabsf(depth_map[p]);
    V3 col;
    if (depth >= 1e4f || depth <= 0.0f) {
        col = bg;
    } else {
        const V3 vp = view_pos(u, tx, ty, depth);
        auto at = [&](int qx, int qy, float sx, float sy) {
            const int ix = clampi(qx, 0, c.W - 1), iy = clampi(qy, 0, c.H - 1);
            return view_pos(u, sx, sy, fabsf(depth_map[(size_t)iy * c.W + ix]));
        };
        V3 ddx = vsub(at(px + 1, py, add(tx, u.texel[0]), ty), vp);
        V3 ddy = vsub(at(px, py + 1, tx, add(ty, u.texel[1])), vp);
        const V3 ddx2 = vsub(vp, at(px - 1, py, sub(tx, u.texel[0]), ty));
        const V3 ddy2 = vsub(vp, at(px, py - 1, tx, sub(ty, u.texel[1])));
        if (fabsf(ddx.z) > fabsf(ddx2.z)) ddx = ddx2;
        if (fabsf(ddy.z) > fabsf(ddy2.z)) ddy = ddy2;
        const V3 nn = vnormalize(vcross(ddx, ddy));
        const V3 normal = v3(-nn.x, -nn.y, -nn.z);
        const V3 ray = vnormalize(vp);
        const float4 l4 = mat4_mul(u.V, 0.0f, 0.0f, -1.0f, 0.0f);
        const V3 light = vnormalize(v3(l4.x, l4.y, l4.z));
        const V3 hv = vnormalize(vsub(light, ray));
        const float specular = pow_r(wmax(0.0f, vdot(hv, normal)), 250.0f);
        const float density = 1.5f;
        const float thickness = thick_map[p];
        const V3 dc = v3(0.085f, 0.6375f, 0.9f);
        const float a = mul(-density, thickness);
        const V3 trans = v3(exp_r(mul(a, sub(1.0f, dc.x))), exp_r(mul(a, sub(1.0f, dc.y))),
                            exp_r(mul(a, sub(1.0f, dc.z))));
        const V3 refr = v3(mul(bg.x, trans.x), mul(bg.y, trans.y), mul(bg.z, trans.z));
        const float F0 = 0.02f;
        const float cosv = vdot(normal, v3(-ray.x, -ray.y, -ray.z));
        const float fres = wmin(wmax(add(F0, mul(sub(1.0f, F0), pow_r(sub(1.0f, cosv), 5.0f))), 0.0f), 1.0f);
        const V3 refl = vsub(ray, vscale(normal, mul(2.0f, vdot(normal, ray))));
        const float4 rw = mat4_mul(u.invV, refl.x, refl.y, refl.z, 0.0f);
        const V3 env_col = sample_cube(env, env_size, v3(rw.x, rw.y, rw.z));
        const float omf = sub(1.0f, fres);
        col = v3(add(mul(1.0f, specular), add(mul(refr.x, omf), mul(env_col.x, fres))),
                 add(mul(1.0f, specular), add(mul(refr.y, omf), mul(env_col.y, fres))),
                 add(mul(1.0f, specular), add(mul(refr.z, omf), mul(env_col.z, fres))));
    }
    out[p] = make_float4(col.x, col.y, col.z, 1.0f);
    auto u8 = [](float v) -> unsigned char {
        if (v != v) return 0;
        return (unsigned char)rintf(mul(wmin(wmax(v, 0.0f), 1.0f), 255.0f));
    };
    out8[p] = make_uchar4(u8(col.x), u8(col.y), u8(col.z), 255);
}

// Sphere mode (render/sphere.wgsl, fluidRender.ts:481-485): the depth test
// alone (above), then each pixel shaded from the winning particle.

// sphere.wgsl:67-90 value_to_color: mix(col_k, col_k+1, t) = a*(1-t) + b*t.
__device__ __forceinline__ V3 value_to_color(float value) {
    float a[3], bb[3], t;
    if (0.0f <= value && value < 0.25f) {
        a[0] = 0.0f; a[1] = 0.4f; a[2] = 0.8f;
        bb[0] = 35.0f / 256.0f; bb[1] = 161.0f / 256.0f; bb[2] = 165.0f / 256.0f;
        t = dvd(value, 0.25f);
    } else if (0.25f <= value && value < 0.50f) {
        a[0] = 35.0f / 256.0f; a[1] = 161.0f / 256.0f; a[2] = 165.0f / 256.0f;
        bb[0] = 95.0f / 256.0f; bb[1] = 254.0f / 256.0f; bb[2] = 150.0f / 256.0f;
        t = dvd(sub(value, 0.25f), 0.25f);
    } else if (0.50f <= value && value < 0.75f) {
        a[0] = 95.0f / 256.0f; a[1] = 254.0f / 256.0f; a[2] = 150.0f / 256.0f;
        bb[0] = 243.0f / 256.0f; bb[1] = 250.0f / 256.0f; bb[2] = 49.0f / 256.0f;
        t = dvd(sub(value, 0.50f), 0.25f);
    } else {
        a[0] = 243.0f / 256.0f; a[1] = 250.0f / 256.0f; a[2] = 49.0f / 256.0f;
        bb[0] = 255.0f / 256.0f; bb[1] = 165.0f / 256.0f; bb[2] = 0.0f;
        t = dvd(sub(value, 0.75f), 0.25f);
    }
    const float om = sub(1.0f, t);
    return v3(add(mul(a[0], om), mul(bb[0], t)), add(mul(a[1], om), mul(bb[1], t)),
              add(mul(a[2], om), mul(bb[2], t)));
}

__global__ void k_sphere_shade(const float4* __restrict__ posvel, Uni u, Consts c,
                               const unsigned long long* dkey,
                               float4* __restrict__ out, uchar4* __restrict__ out8,
                               float* __restrict__ depth) {
    pdl_begin();
    pdl_wait();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= c.W * c.H) return;
    const unsigned long long key = dkey[p];
    V3 col = v3(0.8f, 0.8f, 0.8f);  // the sphere pass's clear colour (fluidRender.ts:425)
    float d = 1.0f;
    if (key != kClearKey) {
        Billboard b;
        Frag f;
        const int i = (int)(key & 0xffffffffull);
        const int px = p % c.W, py = p / c.W;
        if (billboard(posvel, i, u, c, b) && fragment(b, px, py, u, f)) {
            const float4 v = posvel[2 * (size_t)i + 1];
            const float speed = __fsqrt_rn(vdot(v3(v.x, v.y, v.z), v3(v.x, v.y, v.z)));
            const float cx = add((float)px, 0.5f), cy = add((float)py, 0.5f);
            const float nx = sub(mul(dvd(sub(cx, b.fxm), sub(b.fxp, b.fxm)), 2.0f), 1.0f);
            const float ny = sub(mul(dvd(sub(cy, b.fym), sub(b.fyp, b.fym)), 2.0f), 1.0f);
            const float inv_len = dvd(1.0f, __fsqrt_rn(3.0f));  // normalize(vec3(1, 1, 1))
            const float diffuse = wmax(0.0f, vdot(v3(nx, ny, f.nz), v3(inv_len, inv_len, inv_len)));
            col = vscale(value_to_color(dvd(speed, 1.5f)), diffuse);
            d = f.depth;
        }
    }
    out[p] = make_float4(col.x, col.y, col.z, 1.0f);
    auto u8 = [](float x) -> unsigned char {
        if (x != x) return 0;
        return (unsigned char)rintf(mul(wmin(wmax(x, 0.0f), 1.0f), 255.0f));
    };
    out8[p] = make_uchar4(u8(col.x), u8(col.y), u8(col.z), 255);
    depth[p] = d;
}

int fail(int code, const std::string& msg) {
    mpm::set_last_error(msg);
    return code;
}

int cuda_fail(cudaError_t e, const char* what) {
    return fail(MPM_E_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

}  // namespace

struct mpm_renderer {
    int device = 0;
    Consts c{};
    unsigned long long* dkey = nullptr;
    unsigned long long* tacc = nullptr;
    float* depth[2] = {nullptr, nullptr};
    float* thick[2] = {nullptr, nullptr};
    float4* color = nullptr;
    uchar4* color8 = nullptr;
    float4* env = nullptr;
    int env_size = 0;
    float* wtab = nullptr;  // bilateral spatial weights, kWRow x kWRow
    float* gtab = nullptr;  // gaussian weights, kGaussFs + 1, and a pixel's sum of them
    Bins bins{};
    int tile_blocks[2][2] = {};  // resident blocks of k_splat_tiles<THICK, PERSP>
};

namespace {

// The image has few enough tiles for the binned splats.
bool binned(const mpm_renderer* r) { return (long long)r->bins.tx * r->bins.ty <= kMaxTiles; }

// Billboards per work item: fewer where there are too few items for the SMs
// (frame of 5,000 particles with items of 32 / 64 / 256: 39 / 42 / 52 us,
// 20,000: 52 / 45 / 53, 70,000: 96 / 83 / 64, a million: 644 / 398 / 204).
uint32_t item_size(int n) { return n < 10000 ? 32u : (n < 40000 ? 64u : (uint32_t)kItem); }

// Clears the image's keys (and sums) and splats n particles into them.  The
// first launch is a plain one, the others of an image are let in early
// (pdl.cuh): the gaps between the fluid view's 14 kernels, 1.5 to 2.5 us each,
// were a tenth of an image's time.  Before and after, us: 70,000 particles as
// spheres at 896x504 64.3 / 54.5, an application's frame of them with two
// substeps 260.5 / 232.6, a million as a fluid at 1344x756 392 / 361.6.
template <bool THICK>
void enqueue_splats(mpm_renderer* r, const float4* pv, int n, const Uni& u, cudaStream_t st) {
    const Consts& c = r->c;
    const int npix = c.W * c.H;
    unsigned long long* tacc = THICK ? r->tacc : nullptr;
    if (n == 0 || !binned(r)) {
        k_clear<<<(npix + 255) / 256, 256, 0, st>>>(r->dkey, tacc, npix);
        if (n) k_splat_direct<THICK><<<n / 8 + 1, kTileBlock, 0, st>>>(pv, n, u, c, r->dkey, tacc);
        return;
    }
    const size_t smem = 4 * (size_t)r->bins.tx * r->bins.ty;
    const bool persp = u.P[2] == 0.0f && u.P[6] == 0.0f && u.P[3] == 0.0f && u.P[7] == 0.0f &&
                       u.P[11] == -1.0f && u.P[15] == 0.0f && u.P[14] < 0.0f &&
                       fabsf(u.P[10]) < 2.0f && u.sphere_size >= 0.0f;
    for (long long at = 0; at < n; at += kRound) {
        const int first = (int)at, m = n - first < kRound ? n - first : kRound;
        const int blocks = (m + kBinBlock - 1) / kBinBlock;
        const int clear = first == 0 ? npix : 0;  // by as many blocks as help
        const int cb = clear ? (clear + 4 * kBinBlock - 1) / (4 * kBinBlock) : 0;
        k_tile_count<<<blocks > cb ? blocks : cb, kBinBlock, smem, st>>>(pv, first, m, u, c, r->bins,
                                                                       r->dkey, tacc, clear);
        launch_pdl(k_tile_scan, 1, 1024, 0, st, r->bins, item_size(n));
        launch_pdl(k_tile_fill, blocks, kBinBlock, smem, st, first, m, r->bins);
        launch_pdl(persp ? k_splat_tiles<THICK, true> : k_splat_tiles<THICK, false>,
                   r->tile_blocks[THICK][persp], kTileBlock, 0, st, pv, u, c, r->bins, r->dkey, tacc);
    }
}

void free_renderer(mpm_renderer* r) {
    cudaFree(r->dkey);
    cudaFree(r->tacc);
    for (int i = 0; i < 2; ++i) {
        cudaFree(r->depth[i]);
        cudaFree(r->thick[i]);
    }
    cudaFree(r->color);
    cudaFree(r->color8);
    cudaFree(r->env);
    cudaFree(r->wtab);
    cudaFree(r->gtab);
    cudaFree(r->bins.rect);
    delete r;
}

// Default environment: a sky gradient (no image decoding here), bright above
// the horizon, darker below, 32 x 32 per face.
std::vector<float> default_env(int size) {
    std::vector<float> px((size_t)6 * size * size * 4);
    for (int f = 0; f < 6; ++f)
        for (int j = 0; j < size; ++j)
            for (int i = 0; i < size; ++i) {
                const float s = 2.0f * ((float)i + 0.5f) / (float)size - 1.0f;
                const float t = 2.0f * ((float)j + 0.5f) / (float)size - 1.0f;
                float d[3];
                switch (f) {  // inverse of the face table used by sample_cube
                    case 0: d[0] = 1; d[1] = -t; d[2] = -s; break;
                    case 1: d[0] = -1; d[1] = -t; d[2] = s; break;
                    case 2: d[0] = s; d[1] = 1; d[2] = t; break;
                    case 3: d[0] = s; d[1] = -1; d[2] = -t; break;
                    case 4: d[0] = s; d[1] = -t; d[2] = 1; break;
                    default: d[0] = -s; d[1] = -t; d[2] = -1; break;
                }
                const float l = std::sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
                const float y = d[1] / l;
                float* q = px.data() + (((size_t)f * size + j) * size + i) * 4;
                const float h = y > 0.0f ? y : 0.0f;
                q[0] = 0.55f + 0.25f * h + (y < 0.0f ? 0.2f * y : 0.0f);
                q[1] = 0.65f + 0.25f * h + (y < 0.0f ? 0.2f * y : 0.0f);
                q[2] = 0.80f + 0.20f * h + (y < 0.0f ? 0.1f * y : 0.0f);
                q[3] = 1.0f;
            }
    return px;
}

int upload_env(mpm_renderer* r, int size, const float* rgba) {
    float4* e = nullptr;
    cudaError_t err = cudaMalloc(&e, sizeof(float4) * 6 * (size_t)size * size);
    if (err == cudaSuccess)
        err = cudaMemcpy(e, rgba, sizeof(float4) * 6 * (size_t)size * size, cudaMemcpyHostToDevice);
    // the copy from pageable memory may outlast its call, and an image on a
    // non-blocking stream would not wait for it
    if (err == cudaSuccess) err = cudaStreamSynchronize(nullptr);
    if (err != cudaSuccess) {
        cudaFree(e);
        return cuda_fail(err, "envmap");
    }
    cudaFree(r->env);
    r->env = e;
    r->env_size = size;
    return MPM_OK;
}

}  // namespace

extern "C" {

int mpm_renderer_create(int width, int height, float radius, float fov, mpm_renderer** out) {
    if (!out) return fail(MPM_E_INVALID, "out is null");
    *out = nullptr;
    if (width < 1 || height < 1 || (long long)width * height > (1LL << 28))
        return fail(MPM_E_INVALID, "image size outside [1, 2^28] pixels");
    if (!(radius > 0.0f) || !(fov > 0.0f) || !(fov < 3.14159f))
        return fail(MPM_E_INVALID, "radius must be positive and fov in (0, pi)");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return fail(MPM_E_NO_DEVICE, "no CUDA device");
    }
    mpm_renderer* r = new mpm_renderer();
    cudaGetDevice(&r->device);
    r->c.W = width;
    r->c.H = height;
    // fluidRender.ts:38-46 (computed in doubles, as JS does, then f32 constants)
    const double diameter = 2.0 * (double)radius;
    r->c.depth_threshold = (float)((double)radius * 10.0);
    r->c.max_filter_size = 100.0f;
    r->c.ppc = (float)((12.0 * diameter * 0.05 * ((double)height / 2.0)) / std::tan((double)fov / 2.0));
    const size_t np = (size_t)width * height;
    cudaError_t e = cudaMalloc(&r->dkey, 8 * np);
    if (e == cudaSuccess) e = cudaMalloc(&r->tacc, 8 * np);
    for (int i = 0; i < 2 && e == cudaSuccess; ++i) {
        e = cudaMalloc(&r->depth[i], 4 * np);
        if (e == cudaSuccess) e = cudaMalloc(&r->thick[i], 4 * np);
    }
    if (e == cudaSuccess) e = cudaMalloc(&r->color, sizeof(float4) * np);
    if (e == cudaSuccess) e = cudaMalloc(&r->color8, sizeof(uchar4) * np);
    if (e == cudaSuccess) e = cudaMalloc(&r->wtab, sizeof(float) * kWRow * kWRow);
    if (e == cudaSuccess) e = cudaMalloc(&r->gtab, sizeof(float) * (kGaussFs + 2));
    r->bins.tx = (width + kTile - 1) / kTile;
    r->bins.ty = (height + kTile - 1) / kTile;
    if (e == cudaSuccess && binned(r)) {
        // one allocation: rectangles, entries, big ones, counts, cursors, items, state
        const size_t tiles = (size_t)r->bins.tx * r->bins.ty;
        const size_t words = (size_t)kRound * 6 + 2 * tiles + 3 * (size_t)kMaxItems + 4;
        e = cudaMalloc(&r->bins.rect, 4 * words);
        if (e == cudaSuccess) {
            r->bins.entry = r->bins.rect + kRound;
            r->bins.big = r->bins.entry + 4 * (size_t)kRound;
            r->bins.count = r->bins.big + kRound;
            r->bins.cursor = r->bins.count + tiles;
            r->bins.item = reinterpret_cast<Item*>(r->bins.cursor + tiles);
            r->bins.state = reinterpret_cast<int*>(r->bins.item + kMaxItems);
            e = cudaMemset(r->bins.count, 0, 4 * tiles);
        }
        int sms = 0;
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, r->device);
        const void* fn[2][2] = {{(const void*)k_splat_tiles<false, false>, (const void*)k_splat_tiles<false, true>},
                                {(const void*)k_splat_tiles<true, false>, (const void*)k_splat_tiles<true, true>}};
        for (int a = 0; a < 2; ++a)
            for (int b = 0; b < 2 && e == cudaSuccess; ++b) {
                int per = 0;
                e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn[a][b], kTileBlock, 0);
                r->tile_blocks[a][b] = sms * (per < 1 ? 1 : per);
            }
    }
    if (e == cudaSuccess) {
        k_weight_tables<<<(kWRow * kWRow + 255) / 256, 256>>>(r->wtab, r->gtab);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        const int rc = cuda_fail(e, "mpm_renderer_create");
        free_renderer(r);
        return rc;
    }
    const std::vector<float> env = default_env(32);
    if (int rc = upload_env(r, 32, env.data())) {
        free_renderer(r);
        return rc;
    }
    *out = r;
    return MPM_OK;
}

int mpm_renderer_destroy(mpm_renderer* r) {
    if (!r) return MPM_OK;
    cudaDeviceSynchronize();
    free_renderer(r);
    return MPM_OK;
}

int mpm_renderer_set_envmap(mpm_renderer* r, int face_size, const float* rgba) {
    if (!r || !rgba || face_size < 1 || face_size > 4096) return fail(MPM_E_INVALID, "bad envmap");
    cudaDeviceSynchronize();
    return upload_env(r, face_size, rgba);
}

int mpm_renderer_execute(mpm_renderer* r, const void* posvel, int n,
                         const mpm_render_uniforms* uniforms, void* stream) {
    if (!r || !uniforms || n < 0 || (n > 0 && !posvel)) return fail(MPM_E_INVALID, "bad arguments");
    Uni u;
    static_assert(sizeof(mpm_render_uniforms) == sizeof(Uni), "uniform layout");
    std::memcpy(&u, uniforms, sizeof(Uni));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const Consts& c = r->c;
    const int npix = c.W * c.H;
    const int pb = (npix + 255) / 256;
    const float4* pv = static_cast<const float4*>(posvel);
    enqueue_splats<true>(r, pv, n, u, st);
    launch_pdl(k_resolve, pb, 256, 0, st, pv, u, c, r->dkey, r->tacc, r->depth[0], r->thick[0]);
    // blocks of w x h pixels, row by row (one grid dimension: images of one column have 2^28 rows)
    const auto grid = [&](int w, int h) { return (unsigned)((c.W + w - 1) / w) * (unsigned)((c.H + h - 1) / h); };
    const unsigned bx = grid(Bilateral<true>::kW, Bilateral<true>::kH);
    const unsigned by = grid(Bilateral<false>::kW, Bilateral<false>::kH);
    for (int it = 0; it < 4; ++it) {  // fluidRender.ts:455-466, and once :474-486
        const unsigned gx = it ? 0u : grid(Gaussian<true>::kW, Gaussian<true>::kH);
        const unsigned gy = it ? 0u : grid(Gaussian<false>::kW, Gaussian<false>::kH);
        launch_pdl(k_filter<true>, bx + gx, kFilterThreads, 0, st, FilterPass{r->depth[0], r->depth[1]},
                   FilterPass{r->thick[0], r->thick[1]}, (int)bx, c, r->wtab, r->gtab);
        launch_pdl(k_filter<false>, by + gy, kFilterThreads, 0, st, FilterPass{r->depth[1], r->depth[0]},
                   FilterPass{r->thick[1], r->thick[0]}, (int)by, c, r->wtab, r->gtab);
    }
    launch_pdl(k_shade, pb, 256, 0, st, r->depth[0], r->thick[0], r->env, r->env_size, u, c, r->color,
               r->color8);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "mpm_renderer_execute");
    return MPM_OK;
}

int mpm_renderer_execute_spheres(mpm_renderer* r, const void* posvel, int n,
                                 const mpm_render_uniforms* uniforms, void* stream) {
    if (!r || !uniforms || n < 0 || (n > 0 && !posvel)) return fail(MPM_E_INVALID, "bad arguments");
    Uni u;
    std::memcpy(&u, uniforms, sizeof(Uni));
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const Consts& c = r->c;
    const int npix = c.W * c.H;
    const int pb = (npix + 255) / 256;
    const float4* pv = static_cast<const float4*>(posvel);
    enqueue_splats<false>(r, pv, n, u, st);
    launch_pdl(k_sphere_shade, pb, 256, 0, st, pv, u, c, r->dkey, r->color, r->color8, r->depth[0]);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "mpm_renderer_execute_spheres");
    return MPM_OK;
}

int mpm_renderer_download(mpm_renderer* r, int what, void* out) {
    if (!r || !out) return fail(MPM_E_INVALID, "bad arguments");
    const size_t np = (size_t)r->c.W * r->c.H;
    const void* src = nullptr;
    size_t bytes = 0;
    switch (what) {
        case MPM_RENDER_COLOR: src = r->color; bytes = sizeof(float4) * np; break;
        case MPM_RENDER_COLOR8: src = r->color8; bytes = 4 * np; break;
        case MPM_RENDER_DEPTH: src = r->depth[0]; bytes = 4 * np; break;
        case MPM_RENDER_THICKNESS: src = r->thick[0]; bytes = 4 * np; break;
        default: return fail(MPM_E_INVALID, "unknown image");
    }
    cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(out, src, bytes, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(e, "mpm_renderer_download");
    return MPM_OK;
}

void* mpm_renderer_color_device_ptr(mpm_renderer* r) { return r ? r->color : nullptr; }

}  // extern "C"
