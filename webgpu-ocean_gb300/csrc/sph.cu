// sph.cu -- the reference's second simulator, SPHSimulator (sph/sph.ts),
// behind the same four-method API: counting-sort grid (sph/grid/*.wgsl),
// density and near density (sph/density.wgsl), pressure / near-pressure /
// viscosity forces (sph/force.wgsl), integration with penalty walls
// (sph/integrate.wgsl) and the posvel copy (sph/copyPosition.wgsl).
//
// Per substep (two per execute(), sph.ts:325-355), six launches:
//   k_sph_bin       cell of every particle (the grid's fixed [-2, 2]^3
//                   domain plus a sentinel), counts per cell and per chunk
//                   of cells
//   k_sph_scan      exclusive prefix sum of the counts
//   k_sph_scatter   particle order by cell
//   k_sph_place     each cell's run in ascending particle index, with sorted
//                   copies of positions and velocities
//   k_sph_density   per sorted slot: density and near density over the
//                   3x3x3 neighbouring cells (x runs merged, as the shader)
//   k_sph_force     per sorted slot: pressure, near pressure, viscosity,
//                   gravity; then walls, velocity and position update, posvel
//
// Arithmetic restates the shaders with every f32 operation explicitly
// rounded (no contraction), in the shaders' operation order.  Two choices
// the reference leaves to its GPU are fixed: neighbours within a cell are
// visited in ascending particle index (the reference's order comes from
// atomic arrival and is arbitrary), and a particle whose flat cell id falls
// outside [0, gridCount) is left out of the grid (the reference indexes the
// count buffer out of bounds).  The reference's particle count uniform is
// written as a float bit pattern (sph.ts:303-306), so its kernels also run
// the ghost threads of the last workgroup; exactly numParticles particles
// are simulated here.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/mpm.h"

namespace mpm {
void set_last_error(const std::string& msg);  // capi.cu
}

namespace {

__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float dvd(float a, float b) { return __fdiv_rn(a, b); }

// Environment (sph.ts:133-152) and SPHParams (sph.ts:154-179), as the
// shaders see them, plus the scale factors the kernel functions compute
// (density.wgsl:37-47, force.wgsl:37-56).
struct Env {
    int X, Y, Z;        // xGrids, yGrids, zGrids
    float cell;         // cellSize
    float half[3];      // xHalf, yHalf, zHalf (the grid's, not the walls')
    float offset;
    float mass, kr, kr2, kr5, kr6, kr9, dt, stiffness, near_stiffness, rest_density, viscosity;
    float s_density, s_near, s_grad, s_near_grad, s_lap;
    int total;          // X * Y * Z
};

__device__ __forceinline__ int f2i(float x) { return __float2int_rz(x); }  // saturating, NaN -> 0

__device__ __forceinline__ void cell_pos(const Env& e, float x, float y, float z, int& xi, int& yi,
                                         int& zi) {
    xi = f2i(floorf(dvd(add(add(x, e.half[0]), e.offset), e.cell)));
    yi = f2i(floorf(dvd(add(add(y, e.half[1]), e.offset), e.cell)));
    zi = f2i(floorf(dvd(add(add(z, e.half[2]), e.offset), e.cell)));
}

// xi + yi * X + zi * X * Y with i32 wraparound.
__device__ __forceinline__ int cell_number(const Env& e, int xi, int yi, int zi) {
    return (int)((unsigned)xi + (unsigned)yi * (unsigned)e.X +
                 (unsigned)zi * (unsigned)e.X * (unsigned)e.Y);
}

// Where a substep's results go, per particle.
struct SphOut {
    float4 *P, *V, *F, *posvel;
};

__device__ __forceinline__ void write_posvel(float4* __restrict__ posvel, size_t i, const float4& p,
                                             const float4& v) {
    posvel[2 * i] = make_float4(p.x, p.y, p.z, 0.0f);
    posvel[2 * i + 1] = make_float4(v.x, v.y, v.z, 0.0f);
}

// The end of force.wgsl:64-128 (gravity), integrate.wgsl:37-64 (penalty walls
// of the real box, velocity and position) and copyPosition.wgsl:27-37 for
// particle i: p = position and density, v = velocity and near density.  Done
// where the forces are summed: the particle is in registers there, and the
// neighbours' copies (DP, DV) are not what is written.
__device__ __forceinline__ void finish_particle(const Env& e, float4 p, float4 v,
                                                const float (&fp)[3], const float (&fv)[3],
                                                const float* __restrict__ box, const SphOut& out,
                                                size_t i) {
    const float dens = p.w;
    const float grv[3] = {mul(dens, 0.0f), mul(dens, -9.8f), mul(dens, 0.0f)};
    float f[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) f[c] = add(add(fp[c], mul(fv[c], e.viscosity)), grv[c]);
    if (dens != 0.0f) {
        float a[3] = {dvd(f[0], dens), dvd(f[1], dens), dvd(f[2], dens)};
        const float ws = 8000.0f;
        const float half[3] = {box[0], box[1], box[2]};
        const float pos[3] = {p.x, p.y, p.z};
        float plus[3][3], minus[3][3];  // [axis][component]
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            const float pd = fminf(sub(half[ax], pos[ax]), 0.0f);
            const float md = fminf(add(half[ax], pos[ax]), 0.0f);
#pragma unroll
            for (int c = 0; c < 3; ++c) {  // vec3f(1., 0., 0.) and vec3f(-1., 0., 0.)
                plus[ax][c] = mul(mul(c == ax ? 1.0f : 0.0f, ws), pd);
                minus[ax][c] = mul(mul(c == ax ? -1.0f : 0.0f, ws), md);
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float xf = add(plus[0][c], minus[0][c]);
            const float yf = add(plus[1][c], minus[1][c]);
            const float zf = add(plus[2][c], minus[2][c]);
            a[c] = add(a[c], add(add(xf, yf), zf));
        }
        v.x = add(v.x, mul(e.dt, a[0]));
        v.y = add(v.y, mul(e.dt, a[1]));
        v.z = add(v.z, mul(e.dt, a[2]));
        p.x = add(p.x, mul(e.dt, v.x));
        p.y = add(p.y, mul(e.dt, v.y));
        p.z = add(p.z, mul(e.dt, v.z));
    }
    out.P[i] = p;
    out.V[i] = v;
    out.F[i] = make_float4(f[0], f[1], f[2], 0.0f);
    write_posvel(out.posvel, i, p, v);
}

// Cells per chunk of the counts' scan, and the chunks the domain can have.
constexpr int kScan = 1024;
constexpr int kMaxChunks = 256;  // 62^3 cells: 233

// Cell of every particle with its rank among the cell's arrivals, and the
// counts per cell and per chunk of cells (through shared memory: the particles
// of a settled pool share a few dozen chunks).  Particles outside the grid
// keep zero densities (density.wgsl:58-59) and so a zero force (force.wgsl) and
// their place; the others' results come from the force kernels.
__global__ void __launch_bounds__(1024)
    k_sph_bin(SphOut out, int n, Env e, int* __restrict__ cell_of, unsigned* __restrict__ count,
              unsigned* __restrict__ chunk, unsigned* __restrict__ rank) {
    __shared__ unsigned s_chunk[kMaxChunks];
    for (int k = threadIdx.x; k < kMaxChunks; k += blockDim.x) s_chunk[k] = 0u;
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        float4 p = out.P[i];
        int xi, yi, zi;
        cell_pos(e, p.x, p.y, p.z, xi, yi, zi);
        const int c = cell_number(e, xi, yi, zi);
        const bool in = c >= 0 && c < e.total;
        cell_of[i] = in ? c : -1;
        if (in) {
            rank[i] = atomicAdd(count + c, 1u);
            atomicAdd(&s_chunk[c / kScan], 1u);
        } else {
            float4 v = out.V[i];
            p.w = v.w = 0.0f;
            out.P[i] = p;
            out.V[i] = v;
            out.F[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            write_posvel(out.posvel, i, p, v);
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < kMaxChunks; k += blockDim.x)
        if (s_chunk[k]) atomicAdd(chunk + k, s_chunk[k]);
}

// Exclusive scan of count[0 .. m) into start[0 .. m]: each CTA adds up the
// chunk counts before its own (at most a few hundred, counted with the cells)
// and scans its chunk; the counts are left zero for the next binning.
__device__ __forceinline__ unsigned block_exclusive(unsigned x, unsigned* s_w, unsigned& total) {
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    unsigned v = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, v, o);
        if ((int)lane >= o) v += y;
    }
    if (lane == 31) s_w[warp] = v;
    __syncthreads();
    if (warp == 0) {
        unsigned w = s_w[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, w, o);
            if ((int)lane >= o) w += y;
        }
        s_w[lane] = w;
    }
    __syncthreads();
    total = s_w[31];
    return v - x + (warp ? s_w[warp - 1] : 0u);
}

__global__ void __launch_bounds__(kScan) k_sph_scan(unsigned* __restrict__ count,
                                                    const unsigned* __restrict__ chunk, int m,
                                                    unsigned* __restrict__ start) {
    __shared__ unsigned s_w[32];
    const int k = blockIdx.x * kScan + threadIdx.x;
    const unsigned c = k < m ? count[k] : 0u;
    unsigned base, tot;
    block_exclusive(threadIdx.x < blockIdx.x ? chunk[threadIdx.x] : 0u, s_w, base);
    __syncthreads();  // s_w reused
    const unsigned ex = block_exclusive(c, s_w, tot);
    if (k < m) {
        start[k] = base + ex;
        if (c) count[k] = 0u;
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) start[m] = base + tot;
}

__global__ void __launch_bounds__(256)
    k_sph_scatter(const int* __restrict__ cell_of, const unsigned* __restrict__ rank,
                  const unsigned* __restrict__ start, int n, unsigned* __restrict__ chunk,
                  unsigned* __restrict__ arrival) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kMaxChunks) chunk[i] = 0u;  // for the next binning
    if (i >= n) return;
    const int c = cell_of[i];
    if (c >= 0) arrival[start[c] + rank[i]] = (unsigned)i;
}

// Each cell's run in ascending particle index: a particle's slot is the
// cell's first one plus the number of smaller indices in the run (a handful at
// SPH densities).  One thread per particle, not per cell: most of the domain's
// cells are empty and a full one's run would be sorted by one thread.
__global__ void __launch_bounds__(256)
    k_sph_place(const float4* __restrict__ P, const float4* __restrict__ V,
                const int* __restrict__ cell_of, const unsigned* __restrict__ start, int total,
                const unsigned* __restrict__ arrival, unsigned* __restrict__ order,
                float4* __restrict__ SP, float4* __restrict__ SV) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= start[total]) return;
    const unsigned i = arrival[t];
    const float4 p = P[i], v = V[i];
    const int c = cell_of[i];
    const unsigned b = start[c], en = start[c + 1];
    unsigned s = b;
    for (unsigned j = b; j < en; ++j) s += arrival[j] < i ? 1u : 0u;
    order[s] = i;
    SP[s] = p;
    SV[s] = v;
}

// density.wgsl:37-47
__device__ __forceinline__ float density_kernel(const Env& e, float r) {
    const float dd = sub(e.kr2, mul(r, r));
    return mul(mul(mul(e.s_density, dd), dd), dd);
}
__device__ __forceinline__ float near_density_kernel(const Env& e, float r) {
    const float d = sub(e.kr, r);
    return mul(mul(mul(e.s_near, d), d), d);
}

__device__ __forceinline__ bool in_grid(const Env& e, int xi, int yi, int zi) {
    return xi < e.X && 0 <= xi && yi < e.Y && 0 <= yi && zi < e.Z && 0 <= zi;
}

// force.wgsl:37-56
__device__ __forceinline__ float grad_kernel(const Env& e, float r) {
    const float d = sub(e.kr, r);
    return mul(mul(e.s_grad, d), d);
}
__device__ __forceinline__ float near_grad_kernel(const Env& e, float r) {
    const float d = sub(e.kr, r);
    return mul(mul(e.s_near_grad, d), d);
}
__device__ __forceinline__ float lap_kernel(const Env& e, float r) {
    return mul(e.s_lap, sub(e.kr, r));
}

// Squared distance, in the shaders' order.
__device__ __forceinline__ float dist2(const float4& a, const float4& b) {
    const float dx = sub(a.x, b.x), dy = sub(a.y, b.y), dz = sub(a.z, b.z);
    return add(add(mul(dx, dx), mul(dy, dy)), mul(dz, dz));
}

// a / b for several a and one b, correctly rounded, from y = RN(1 / b): a
// first quotient, one Newton correction that brings it to within an ulp, and
// Markstein's final one, which rounds correctly because the remainder
// fma(-b, q, a) is exact (P. Markstein, IBM J. Res. Dev. 34, 1990).  Five
// operations instead of a division.  Holds for quotients in [kQuotMin,
// kQuotMax] when b lies in [2^-20, 2^40]: nothing overflows, and the remainder,
// a multiple of 2^-133 there, is exact also where it is subnormal (which the
// build's -ftz=false keeps).  rcp_for_quotients(b) is NaN for other b, so that
// every quotient fails the range test; infinities give NaN too.
constexpr float kQuotMin = 1.0e-20f, kQuotMax = 1.0e20f;

__device__ __forceinline__ float rcp_for_quotients(float b) {
    return b >= 0x1p-20f && b <= 0x1p40f ? __frcp_rn(b) : __int_as_float(0x7fc00000);
}

__device__ __forceinline__ float quot(float a, float b, float y) {
    float q = mul(a, y);
    q = __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
    return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}

// The larger of two, NaN when one is.
__device__ __forceinline__ float fmax_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// The terms that neighbour j (position pj with its density, velocity vj with
// its near density, reciprocals rj of the two) adds to the forces of particle
// i: t[0..2] pressure, t[3..5] near pressure, t[6..8] viscosity
// (force.wgsl:96-120).  A listed particle that is none (the particle itself,
// one without a density) adds nothing: +0, which leaves a sum that started at
// +0 as it is.
__device__ __forceinline__ void force_terms(const Env& e, const float4& pi, const float4& vi,
                                            const float4& pj, const float4& vj, const float2& rj,
                                            float (&t)[9]) {
    const float dens_j = pj.w, near_j = vj.w;
    const float r2 = dist2(pi, pj);
    if (dens_j == 0.0f || near_j == 0.0f || !(0.0f < r2)) {
#pragma unroll
        for (int q = 0; q < 9; ++q) t[q] = 0.0f;
        return;
    }
    // normalize(pos_j - pos_i): the same length as the distance (the
    // differences are exact negatives)
    const float r = __fsqrt_rn(r2);
    const float p_i = mul(e.stiffness, sub(pi.w, e.rest_density));
    const float p_j = mul(e.stiffness, sub(dens_j, e.rest_density));
    const float np_i = mul(e.near_stiffness, vi.w);
    const float np_j = mul(e.near_stiffness, near_j);
    const float sp = mul(add(p_i, p_j), 0.5f);     // / 2, exactly
    const float nsp = mul(add(np_i, np_j), 0.5f);
    const float u[3] = {sub(pj.x, pi.x), sub(pj.y, pi.y), sub(pj.z, pi.z)};
    const float g = grad_kernel(e, r), ng = near_grad_kernel(e, r);
    const float a = mul(-e.mass, sp), an = mul(-e.mass, nsp);
    const float lap = lap_kernel(e, r);
    const float rel[3] = {sub(vj.x, vi.x), sub(vj.y, vi.y), sub(vj.z, vi.z)};
    const float rr = rcp_for_quotients(r);
    float lo = kQuotMax, hi = kQuotMin;
    auto seen = [&](float q) {
        lo = fminf(lo, fabsf(q));
        hi = fmax_nan(hi, fabsf(q));
        return q;
    };
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float dir = seen(quot(u[c], r, rr));
        t[c] = seen(quot(mul(mul(a, dir), g), dens_j, rj.x));
        t[3 + c] = seen(quot(mul(mul(an, dir), ng), near_j, rj.y));
        t[6 + c] = seen(quot(mul(mul(e.mass, rel[c]), lap), dens_j, rj.x));
    }
    if (lo >= kQuotMin && hi <= kQuotMax) return;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float dir = dvd(u[c], r);
        t[c] = dvd(mul(mul(a, dir), g), dens_j);
        t[3 + c] = dvd(mul(mul(an, dir), ng), near_j);
        t[6 + c] = dvd(mul(mul(e.mass, rel[c]), lap), dens_j);
    }
}

// Sorted slots [b, en) of row r (dz = r / 3 - 1, dy = r % 3 - 1, the three
// cells along x merged) of the cells around (vx, vy, vz), in the shaders'
// visiting order for r = 0 .. 8; empty where the row leaves the grid.
__device__ __forceinline__ void neighbour_row(const Env& e, const unsigned* __restrict__ start,
                                              int vx, int vy, int vz, int r, unsigned& b,
                                              unsigned& en) {
    const int z = vz + r / 3 - 1, y = vy + r % 3 - 1;
    b = en = 0u;
    if (z < 0 || z >= e.Z || y < 0 || y >= e.Y) return;
    b = start[cell_number(e, max(vx - 1, 0), y, z)];
    en = start[cell_number(e, min(vx + 1, e.X - 1), y, z) + 1];
}

// ---------------------------------------------------------------------------
// Density and forces.  Bound by instruction issue (densities, 70-78 % of the
// issue slots) and by the latency of the neighbours' gathers (forces).  Of the
// candidates in the 27 cells around a particle one in five is a neighbour, and
// a neighbour's terms cost 2 (density) to 8 times (force) what testing a
// candidate does.  With the terms computed where a candidate passes, some lane
// of a warp passes at nearly every candidate and the others wait (20 % of the
// lanes active in the force).  So the density kernels first collect the
// neighbours that pass, in visiting order, and then compute their terms with
// all lanes busy; they leave the list in memory for the force kernels.  Every
// sum adds its terms in the visiting order, so all variants give the same
// bits.  Per two-substep frame of settled pools, with one warp (10,000
// particles) or one thread per particle testing and computing as it goes, and
// now (the sort's launches included): 10,000 particles 169 -> 55 us, 40,000
// 308 -> 97 us, 400,000 1830 -> 669 us.  Frames 20 to 70 of the fall of 400,000,
// with up to twice the neighbours: 2170 -> 1070 us.
// ---------------------------------------------------------------------------

// Neighbours listed per particle.  Of 400,000 particles at rest each has 36 on
// average and at most 78; while they fall, 70 and at most 193, and in the densest
// frame 3 % have more than 128.  A particle with more than are listed walks its
// rows again for the force (with 64, those at the bottom of the settled pool did:
// 1165 instead of 758 us).  Entry k of sorted particle s is nbr[k * stride + s],
// so that neighbouring particles' entries share sectors.  No lists are kept for capacities above kListedMax, where
// they would take over 4 GB, nor where there is no memory for them.
constexpr int kNeighbours = 128;
constexpr int kListedMax = 1 << 23;

struct NeighbourLists {
    unsigned* nbr;   // null: no lists
    int* n;          // neighbours of each sorted particle, listed or not
    size_t stride;
    __device__ __forceinline__ bool listed(int count) const { return nbr && count <= kNeighbours; }
    __device__ __forceinline__ void put(int s, int k, unsigned j) const {
        if (nbr && k < kNeighbours) nbr[(size_t)k * stride + s] = j;
    }
    __device__ __forceinline__ unsigned get(int s, int k) const { return nbr[(size_t)k * stride + s]; }
};

// G lanes per particle: the lanes test G candidates of a row at a time and a
// ballot gives the ones that pass their places in the list; the lanes compute
// the listed neighbours' terms into shared memory and one lane per accumulator
// adds them in list order.  All control flow is uniform over the warp, whose
// 32 / G particles go through their rows together.
constexpr int kGroupBlock = 256;

template <int G>
struct Group {
    static constexpr int kParticles = kGroupBlock / G;  // particles per block
    static constexpr unsigned kMask = G == 32 ? 0xffffffffu : (1u << (G & 31)) - 1u;
    int p, lane;      // particle of the block, lane of the group
    unsigned shift;   // the group's first lane in the warp
    int m = 0;        // listed neighbours of this round
    int taken = 0;    // and of the rounds before it
    __device__ Group()
        : p((int)threadIdx.x / G), lane((int)threadIdx.x % G), shift(threadIdx.x & 31u & ~(unsigned)(G - 1)) {}
    // This lane's place in the list when its candidate passes (else -1).
    // Every lane of the warp calls it.
    __device__ __forceinline__ int append(bool pass) {
        const unsigned hits = (__ballot_sync(0xffffffffu, pass) >> shift) & kMask;
        const int at = pass ? m + __popc(hits & ((1u << lane) - 1u)) : -1;
        m += __popc(hits);
        return at;
    }
};

// Walks the candidates of this group's particle (none unless `in`), Q per lane
// at a time with all their positions loaded first: put(place, j, r2) for those
// within the kernel radius, take() when the round's list of L has no room for
// G * Q more and at the end.
template <int G, int Q, int L, class Put, class Take>
__device__ __forceinline__ void walk_neighbours(const Env& e, const unsigned* __restrict__ start,
                                                const float4* __restrict__ pos, int pos_stride,
                                                const float4& pi, bool in, Group<G>& g, Put&& put,
                                                Take&& take) {
    static_assert(L >= G * Q, "a batch fits an empty list");
    int vx, vy, vz;
    cell_pos(e, pi.x, pi.y, pi.z, vx, vy, vz);
    in = in && in_grid(e, vx, vy, vz);
#pragma unroll 3
    for (int row = 0; row < 9; ++row) {
        unsigned b = 0u, en = 0u;
        if (in) neighbour_row(e, start, vx, vy, vz, row, b, en);
        for (unsigned j0 = b; __any_sync(0xffffffffu, j0 < en); j0 += G * Q) {
            if (__any_sync(0xffffffffu, g.m > L - G * Q)) take();
            float r2[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const unsigned j = j0 + (unsigned)(q * G + g.lane);
                r2[q] = e.kr2;
                if (j < en) r2[q] = dist2(pi, pos[(size_t)j * pos_stride]);
            }
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const int at = g.append(r2[q] < e.kr2);
                if (at >= 0) put(at, j0 + (unsigned)(q * G + g.lane), r2[q]);
            }
        }
    }
    take();
}

__device__ __forceinline__ void write_density(float4* __restrict__ D, float2* __restrict__ DR,
                                              const float4* __restrict__ SV, int s,
                                              const float4& pi, float dens, float near) {
    const float4 v = SV[s];
    D[2 * (size_t)s] = make_float4(pi.x, pi.y, pi.z, dens);
    D[2 * (size_t)s + 1] = make_float4(v.x, v.y, v.z, near);
    DR[s] = make_float2(rcp_for_quotients(dens), rcp_for_quotients(near));
}

// density.wgsl:58-100, per sorted slot.
template <int G>
__global__ void __launch_bounds__(kGroupBlock)
    k_sph_density(const float4* __restrict__ SP, const float4* __restrict__ SV,
                  float4* __restrict__ D, float2* __restrict__ DR, NeighbourLists nl,
                  const unsigned* __restrict__ start, Env e) {
    using Gr = Group<G>;
    constexpr int kList = 64;
    __shared__ float2 s_t[Gr::kParticles][kList];  // r2 and slot of the listed, then their two terms
    const int nbin = (int)start[e.total];
    if ((int)blockIdx.x * Gr::kParticles >= nbin) return;
    Gr g;
    const int s = (int)blockIdx.x * Gr::kParticles + g.p;
    const bool active = s < nbin;
    const float4 pi = active ? SP[s] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float2* t = s_t[g.p];
    float acc = 0.0f;  // lane 0: density, lane 1: near density
    walk_neighbours<G, 32 / G, kList>(
        e, start, SP, 1, pi, active, g,
        [&](int at, unsigned j, float r2) { t[at] = make_float2(r2, __uint_as_float(j)); },
        [&]() {
            __syncwarp();
            for (int k = g.lane; k < g.m; k += G) {
                const float2 u = t[k];
                const float r = __fsqrt_rn(u.x);
                t[k] = make_float2(mul(e.mass, density_kernel(e, r)),
                                   mul(e.mass, near_density_kernel(e, r)));
                nl.put(s, g.taken + k, __float_as_uint(u.y));
            }
            __syncwarp();
            if (g.lane < 2) {
                const float* u = &t[0].x + g.lane;
#pragma unroll 4
                for (int k = 0; k < g.m; ++k) acc = add(acc, u[2 * k]);
            }
            g.taken += g.m;
            g.m = 0;
            __syncwarp();
        });
    const float near = __shfl_sync(0xffffffffu, acc, (int)g.shift + 1);
    if (active && g.lane == 0) {
        write_density(D, DR, SV, s, pi, acc, near);
        nl.n[s] = g.taken;
    }
}

// The same with one thread per particle, for many particles: a test costs no
// ballot and the terms no trip through shared memory (290 instead of 614
// warp instructions per particle), at a few warps per scheduler.  The list of a
// round is the thread's own column in shared memory; 32 entries, because more
// would cost resident warps (64 entries and one candidate loaded at a time from
// global memory: 264 us at 400,000 particles).  The lanes of a warp
// (neighbouring sorted slots) take their terms together, when some lane's list
// is full and at the end: a lane that took its terms alone would hold up the
// other 31.  They share most of a row's candidates too, so the warp fetches the
// row's run once (four candidates a thread from global memory: 181 us; from the
// run: 171; and four neighbours' positions loaded ahead of their terms: 164).
constexpr int kThreadBlock = 128;
constexpr int kThreadList = 32;
constexpr int kThreadStep = 4;  // candidates between two looks at the lists
constexpr int kRowCache = 96;  // candidates of a row that a warp keeps

__global__ void __launch_bounds__(kThreadBlock)
    k_sph_density_thread(const float4* __restrict__ SP, const float4* __restrict__ SV,
                         float4* __restrict__ D, float2* __restrict__ DR, NeighbourLists nl,
                         const unsigned* __restrict__ start, Env e) {
    __shared__ unsigned s_j[kThreadList][kThreadBlock];
    __shared__ float4 s_row[kThreadBlock / 32][kRowCache];
    const int nbin = (int)start[e.total];
    const int s = blockIdx.x * kThreadBlock + threadIdx.x;
    if ((s & ~31) >= nbin) return;  // uniform per warp
    const bool active = s < nbin;
    const float4 pi = active ? SP[s] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    int vx, vy, vz;
    cell_pos(e, pi.x, pi.y, pi.z, vx, vy, vz);
    const bool in = active && in_grid(e, vx, vy, vz);
    float dens = 0.0f, near = 0.0f;
    int m = 0, taken = 0;
    auto take = [&]() {
        for (int k0 = 0; k0 < m; k0 += 4) {
            unsigned j[4];
            float4 p[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) j[q] = k0 + q < m ? s_j[k0 + q][threadIdx.x] : 0u;
#pragma unroll
            for (int q = 0; q < 4; ++q) p[q] = SP[j[q]];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (k0 + q >= m) break;
                nl.put(s, taken + k0 + q, j[q]);
                const float r = __fsqrt_rn(dist2(pi, p[q]));
                dens = add(dens, mul(e.mass, density_kernel(e, r)));
                near = add(near, mul(e.mass, near_density_kernel(e, r)));
            }
        }
        taken += m;
        m = 0;
        __syncwarp();
    };
    float4* row_p = s_row[threadIdx.x >> 5];
    const unsigned lane = threadIdx.x & 31u;
    for (int row = 0; row < 9; ++row) {
        unsigned b = 0u, en = 0u;
        if (in) neighbour_row(e, start, vx, vy, vz, row, b, en);
        const unsigned lo = __reduce_min_sync(0xffffffffu, b < en ? b : 0xffffffffu);
        const unsigned hi = __reduce_max_sync(0xffffffffu, en);
        if (lo >= hi) continue;  // uniform
        auto walk = [&](auto&& at) {
            while (__any_sync(0xffffffffu, b < en)) {
                if (__any_sync(0xffffffffu, m > kThreadList - kThreadStep)) take();
                float4 p[kThreadStep];
#pragma unroll
                for (int q = 0; q < kThreadStep; ++q) p[q] = at(b + q);
#pragma unroll
                for (int q = 0; q < kThreadStep; ++q)
                    if (b + q < en && dist2(pi, p[q]) < e.kr2) s_j[m++][threadIdx.x] = b + q;
                b += kThreadStep;
            }
        };
        if (hi - lo <= kRowCache) {
            __syncwarp();
            for (unsigned k = lane; k < hi - lo; k += 32) row_p[k] = SP[lo + k];
            __syncwarp();
            walk([&](unsigned j) { return row_p[min(j - lo, (unsigned)kRowCache - 1u)]; });
        } else {
            walk([&](unsigned j) { return SP[min(j, (unsigned)nbin - 1u)]; });
        }
    }
    take();
    if (!active) return;
    write_density(D, DR, SV, s, pi, dens, near);
    nl.n[s] = taken;
}

// force.wgsl:64-128 and the integration, per sorted slot.  D: position and
// density, velocity and near density of each sorted particle (one 32-byte
// sector, for the gathers); DR: the densities' reciprocals.
template <int G>
__global__ void __launch_bounds__(kGroupBlock)
    k_sph_force(const float4* __restrict__ D, const float2* __restrict__ DR,
                NeighbourLists nl, const unsigned* __restrict__ order,
                const unsigned* __restrict__ start, Env e, const float* __restrict__ box,
                SphOut out) {
    using Gr = Group<G>;
    constexpr int kList = 32;  // 36 KB for G = 8: four blocks an SM, as the registers allow
    __shared__ unsigned s_j[Gr::kParticles][kList];
    __shared__ float s_t[Gr::kParticles][9 * kList];
    const int nbin = (int)start[e.total];
    if ((int)blockIdx.x * Gr::kParticles >= nbin) return;
    Gr g;
    const int s = (int)blockIdx.x * Gr::kParticles + g.p;
    const bool active = s < nbin;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int total = active ? nl.n[s] : 0;
    const float4 pi = active ? D[2 * (size_t)s] : zero, vi = active ? D[2 * (size_t)s + 1] : zero;
    float* t = s_t[g.p];
    // lanes 0-2: pressure force component c (two terms per neighbour), lanes
    // 3-5: viscosity force component c
    float acc = 0.0f;
    auto put_terms = [&](int k, unsigned j) {
        float q[9];
        force_terms(e, pi, vi, D[2 * (size_t)j], D[2 * (size_t)j + 1], DR[j], q);
#pragma unroll
        for (int c = 0; c < 9; ++c) t[9 * k + c] = q[c];
    };
    auto add_terms = [&](int m) {
        if (g.lane < 6) {
            const bool pressure = g.lane < 3;
            const float* u = t + (pressure ? g.lane : g.lane + 3);
#pragma unroll 4
            for (int k = 0; k < m; ++k) {
                acc = add(acc, u[9 * k]);
                if (pressure) acc = add(acc, u[9 * k + 3]);
            }
        }
    };
    if (__all_sync(0xffffffffu, nl.listed(total))) {
        // entries of a round are loaded while the round before it computes
        constexpr int kPer = kList / G;
        unsigned j[kPer];
        auto load = [&](int base) {
#pragma unroll
            for (int q = 0; q < kPer; ++q) {
                const int k = base + q * G + g.lane;
                j[q] = k < total ? nl.get(s, k) : 0u;
            }
        };
        load(0);
        for (int base = 0; __any_sync(0xffffffffu, base < total); base += kList) {
            unsigned now[kPer];
#pragma unroll
            for (int q = 0; q < kPer; ++q) now[q] = j[q];
            load(base + kList);
            const int m = min(total - base, kList);
#pragma unroll
            for (int q = 0; q < kPer; ++q)
                if (q * G + g.lane < m) put_terms(q * G + g.lane, now[q]);
            __syncwarp();
            add_terms(m);
            __syncwarp();
        }
    } else {
        unsigned* list = s_j[g.p];
        walk_neighbours<G, 1, kList>(
            e, start, D, 2, pi, active, g, [&](int at, unsigned j, float) { list[at] = j; },
            [&]() {
                __syncwarp();
                for (int k = g.lane; k < g.m; k += G) put_terms(k, list[k]);
                __syncwarp();
                add_terms(g.m);
                g.m = 0;
                __syncwarp();
            });
    }
    float fp[3], fv[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        fp[c] = __shfl_sync(0xffffffffu, acc, (int)g.shift + c);
        fv[c] = __shfl_sync(0xffffffffu, acc, (int)g.shift + 3 + c);
    }
    if (active && g.lane == 0) finish_particle(e, pi, vi, fp, fv, box, out, order[s]);
}


// One thread per particle: the next neighbour's record is gathered while this
// one's terms are computed.
__global__ void __launch_bounds__(kThreadBlock)
    k_sph_force_thread(const float4* __restrict__ D, const float2* __restrict__ DR,
                       NeighbourLists nl, const unsigned* __restrict__ order,
                       const unsigned* __restrict__ start, Env e, const float* __restrict__ box,
                       SphOut out) {
    const int s = blockIdx.x * kThreadBlock + threadIdx.x;
    if (s >= (int)start[e.total]) return;
    const int total = nl.n[s];
    const float4 pi = D[2 * (size_t)s], vi = D[2 * (size_t)s + 1];
    float fp[3] = {0.0f, 0.0f, 0.0f}, fv[3] = {0.0f, 0.0f, 0.0f};
    auto add_terms = [&](const float4& pj, const float4& vj, const float2& rj) {
        float t[9];
        force_terms(e, pi, vi, pj, vj, rj, t);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            fp[c] = add(add(fp[c], t[c]), t[3 + c]);
            fv[c] = add(fv[c], t[6 + c]);
        }
    };
    if (nl.listed(total)) {
        unsigned j = total > 0 ? nl.get(s, 0) : 0u, j2 = total > 1 ? nl.get(s, 1) : 0u;
        float4 pj = D[2 * (size_t)j], vj = D[2 * (size_t)j + 1];
        float2 rj = DR[j];
        for (int k = 0; k < total; ++k) {
            const float4 pc = pj, vc = vj;
            const float2 rc = rj;
            pj = D[2 * (size_t)j2];
            vj = D[2 * (size_t)j2 + 1];
            rj = DR[j2];
            j2 = k + 2 < total ? nl.get(s, k + 2) : 0u;
            add_terms(pc, vc, rc);
        }
    } else {
        int vx, vy, vz;
        cell_pos(e, pi.x, pi.y, pi.z, vx, vy, vz);
        for (int row = 0; row < 9 && in_grid(e, vx, vy, vz); ++row) {
            unsigned b, en;
            neighbour_row(e, start, vx, vy, vz, row, b, en);
            for (unsigned j = b; j < en; ++j)
                if (dist2(pi, D[2 * (size_t)j]) < e.kr2)
                    add_terms(D[2 * (size_t)j], D[2 * (size_t)j + 1], DR[j]);
        }
    }
    finish_particle(e, pi, vi, fp, fv, box, out, order[s]);
}

int fail(int code, const std::string& msg) {
    mpm::set_last_error(msg);
    return code;
}

int cuda_fail(cudaError_t err, const char* what) {
    return fail(MPM_E_CUDA, std::string(what) + ": " + cudaGetErrorString(err));
}

struct SplitMix64 {
    uint64_t s;
    explicit SplitMix64(uint64_t seed) : s(seed) {}
    double random() {
        s += 0x9E3779B97F4A7C15ull;
        uint64_t z = s;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (double)(z >> 11) * (1.0 / 9007199254740992.0);
    }
};

}  // namespace

// Which density and force kernels run at n particles.  Frames in us, settled
// pools (16 lanes / 8 lanes / 8 lanes for the densities and a thread for the
// forces / a thread for both, the last before it shared rows): 8,000 particles
// 51 / 54 / 66 / 101, 12,000 60 / 60 / 69 / 109, 24,000 87 / 83 / 81 / 119,
// 100,000 268 / 222 / 182 / 190, 130,000 330 / 281 / 229 / 225, 400,000 - /
// 1097 / 836 / 758 (696 with them): the fewer the
// particles, the more lanes it takes to hide a particle's chain of loads, and
// the more of them the fewer instructions decide.
constexpr int kSph16Max = 12000;
constexpr int kSphLanesMax = 22000;
constexpr int kSphDensity8Max = 130000;
// The limit on particle counts with lanes, as long as the counts above decide.
constexpr int kSphWarpMaxDefault = 32768;

struct mpm_sph {
    int device = 0;
    int max_particles = 0;
    int n = 0;
    float render_diameter = 0.0f;
    float real_half[3] = {0, 0, 0};
    Env e{};
    char* slab = nullptr;  // the allocation that holds the buffers below, but posvel
    float4 *P = nullptr, *V = nullptr, *F = nullptr;      // by particle
    float4 *SP = nullptr, *SV = nullptr;                  // sorted
    float4* D = nullptr;                                  // sorted, with the densities
    float2* DR = nullptr;                                 // their reciprocals
    NeighbourLists nl{};
    float4* posvel = nullptr;
    bool posvel_owned = false;
    int* cell_of = nullptr;
    unsigned *count = nullptr, *start = nullptr, *rank = nullptr, *order = nullptr;
    unsigned* arrival = nullptr;  // particles by cell, in the order they were counted
    unsigned* chunk = nullptr;    // counts per kScan cells
    // the real box as the kernels read it (a device uniform, so that a
    // captured frame graph survives changeBoxSize)
    float* box_d = nullptr;
    float box_uploaded[3] = {NAN, NAN, NAN};
    bool graph = true;
    int warp_max = -1;  // lanes per particle up to this count, a thread above; -1: see above
    struct FrameGraph {
        int substeps, n;
        cudaGraphExec_t exec;
    };
    std::vector<FrameGraph> graphs;
};

namespace {

void drop_graphs(mpm_sph* s) {
    for (auto& g : s->graphs) cudaGraphExecDestroy(g.exec);
    s->graphs.clear();
}

void free_sph(mpm_sph* s) {
    drop_graphs(s);
    cudaFree(s->slab);
    if (s->posvel_owned) cudaFree(s->posvel);
    delete s;
}

// sph.ts:58-86 and 154-179: grid and kernel constants (JS doubles, stored
// as f32 uniforms) and the scale factors of the kernel functions (f32
// arithmetic on the f32 uniforms; the literals' products are folded in
// double precision first, as WGSL folds abstract constants).
Env make_env() {
    Env e{};
    const double kr = 0.07;
    const double cell = 1.0 * kr;
    const double half = 2.0, len = 2.0 * half, sentinel = 4.0 * cell;
    const int grids = (int)std::ceil((len + sentinel) / cell);
    e.X = e.Y = e.Z = grids;
    e.cell = (float)cell;
    e.half[0] = e.half[1] = e.half[2] = (float)half;
    e.offset = (float)(sentinel / 2.0);
    e.mass = 1.0f;
    e.kr = (float)kr;
    e.kr2 = (float)std::pow(kr, 2);
    e.kr5 = (float)std::pow(kr, 5);
    e.kr6 = (float)std::pow(kr, 6);
    e.kr9 = (float)std::pow(kr, 9);
    e.dt = 0.006f;
    e.stiffness = 20.0f;
    e.near_stiffness = 1.0f;
    e.rest_density = 15000.0f;
    e.viscosity = 100.0f;
    const float pi = (float)3.1415926535;
    e.s_density = 315.0f / ((float)(64.0 * 3.1415926535) * e.kr9);
    e.s_near = 15.0f / (pi * e.kr6);
    e.s_grad = 45.0f / (pi * e.kr6);
    e.s_near_grad = 45.0f / (pi * e.kr5);
    e.s_lap = 45.0f / (pi * e.kr6);
    e.total = e.X * e.Y * e.Z;
    return e;
}

}  // namespace

extern "C" {

int mpm_sph_create(int max_particles, float render_diameter, void* posvel_device,
                   size_t posvel_bytes, mpm_sph** out) {
    if (!out) return fail(MPM_E_INVALID, "out is null");
    *out = nullptr;
    if (max_particles < 0) return fail(MPM_E_INVALID, "negative capacity");
    if (posvel_device && posvel_bytes < (size_t)32 * (size_t)max_particles)
        return fail(MPM_E_INVALID, "posvel buffer smaller than 32 * max_particles bytes");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return fail(MPM_E_NO_DEVICE, "no CUDA device");
    }
    mpm_sph* s = new mpm_sph();
    cudaGetDevice(&s->device);
    s->max_particles = max_particles;
    s->render_diameter = render_diameter;
    s->e = make_env();
    const size_t np = (size_t)(max_particles > 0 ? max_particles : 1);
    const size_t cells = (size_t)s->e.total + 1;
    // one allocation for all of the solver's buffers (an allocation costs as
    // much as a frame), each at a 256-byte boundary; twice through the list:
    // once for the size, once for the places
    size_t bytes = 0;
    bool lists = np <= kListedMax;
    auto place = [&](auto& ptr, size_t count) {
        if (s->slab) ptr = reinterpret_cast<std::remove_reference_t<decltype(ptr)>>(s->slab + bytes);
        bytes += (sizeof(*ptr) * count + 255) / 256 * 256;
    };
    auto place_all = [&]() {
        bytes = 0;
        for (float4** b : {&s->P, &s->V, &s->F, &s->SP, &s->SV}) place(*b, np);
        place(s->D, 2 * np);
        place(s->DR, np);
        place(s->cell_of, np);
        place(s->rank, np);
        place(s->order, np);
        place(s->arrival, np);
        place(s->nl.n, np);
        place(s->count, cells);
        place(s->chunk, kMaxChunks);
        place(s->start, cells);
        place(s->box_d, 3);
        if (lists) place(s->nl.nbr, kNeighbours * np);
    };
    s->nl.stride = np;
    cudaError_t err = cudaSuccess;
    if (posvel_device) {
        s->posvel = static_cast<float4*>(posvel_device);
    } else {
        s->posvel_owned = true;
        err = cudaMalloc(&s->posvel, sizeof(float4) * 2 * np);
    }
    if (err == cudaSuccess) {
        place_all();
        err = cudaMalloc(&s->slab, bytes);
    }
    if (err == cudaErrorMemoryAllocation && s->posvel && lists) {
        // the lists are most of it, and the simulator does without
        cudaGetLastError();
        s->slab = nullptr;
        lists = false;
        place_all();
        err = cudaMalloc(&s->slab, bytes);
    }
    if (err == cudaSuccess) {
        place_all();
        // zero between substeps: the scan and the scatter clear what they have read
        err = cudaMemset(s->count, 0, 4 * cells);
        if (err == cudaSuccess) err = cudaMemset(s->chunk, 0, 4 * kMaxChunks);
    }
    if (err != cudaSuccess) {
        const int rc = cuda_fail(err, "mpm_sph_create");
        free_sph(s);
        return rc;
    }
    *out = s;
    return MPM_OK;
}

int mpm_sph_destroy(mpm_sph* s) {
    if (!s) return MPM_OK;
    cudaDeviceSynchronize();
    free_sph(s);
    return MPM_OK;
}

int mpm_sph_upload(mpm_sph* s, const float* rec64, int n, const float real_half[3]) {
    if (!s || (n > 0 && !rec64) || !real_half) return fail(MPM_E_INVALID, "bad arguments");
    if (n < 0 || n > s->max_particles) return fail(MPM_E_CAPACITY, "numParticles exceeds the particle capacity");
    std::vector<float4> P((size_t)n), V((size_t)n), F((size_t)n);
    for (int i = 0; i < n; ++i) {
        const float* r = rec64 + 16 * (size_t)i;  // particle record, sph.ts:13,205-211
        P[(size_t)i] = make_float4(r[0], r[1], r[2], r[11]);
        V[(size_t)i] = make_float4(r[4], r[5], r[6], r[12]);
        F[(size_t)i] = make_float4(r[8], r[9], r[10], 0.0f);
    }
    cudaError_t err = cudaDeviceSynchronize();
    if (n && err == cudaSuccess) err = cudaMemcpy(s->P, P.data(), sizeof(float4) * n, cudaMemcpyHostToDevice);
    if (n && err == cudaSuccess) err = cudaMemcpy(s->V, V.data(), sizeof(float4) * n, cudaMemcpyHostToDevice);
    if (n && err == cudaSuccess) err = cudaMemcpy(s->F, F.data(), sizeof(float4) * n, cudaMemcpyHostToDevice);
    if (n && err == cudaSuccess) err = cudaMemset(s->posvel, 0, sizeof(float4) * 2 * (size_t)n);
    // copies from pageable memory and memsets may outlast their calls, and a
    // frame on a non-blocking stream would not wait for them
    if (err == cudaSuccess) err = cudaDeviceSynchronize();
    if (err != cudaSuccess) return cuda_fail(err, "mpm_sph_upload");
    s->n = n;
    for (int a = 0; a < 3; ++a) s->real_half[a] = real_half[a];
    return MPM_OK;
}

// SPHSimulator.initDambreak (sph.ts:357-381): y from -0.95 h_y upward without
// bound, x in [-0.95 h_x, 0.95 h_x), z in [-0.95 h_z, 0), step 0.035, one
// jitter 0.001 * Math.random() added to x, y and z (Math.random ->
// SplitMix64(seed)).  Writes 64-byte records; returns the count.
int mpm_sph_scene_dambreak(float* out_rec64, int num_particles, const double half[3], uint64_t seed) {
    if (!out_rec64 || !half || num_particles < 0) return fail(MPM_E_INVALID, "bad arguments");
    SplitMix64 rng(seed);
    const double kr = 0.07, step = 0.5 * kr;
    int n = 0;
    for (double y = -half[1] * 0.95; n < num_particles; y += step) {
        bool any = false;
        for (double x = -0.95 * half[0]; x < 0.95 * half[0] && n < num_particles; x += step)
            for (double z = -0.95 * half[2]; z < 0 * half[2] && n < num_particles; z += step) {
                const double jitter = 0.001 * rng.random();
                float* r = out_rec64 + 16 * (size_t)n;
                std::memset(r, 0, 64);
                r[0] = (float)(x + jitter);
                r[1] = (float)(y + jitter);
                r[2] = (float)(z + jitter);
                ++n;
                any = true;
            }
        if (!any) break;  // an empty layer never fills (degenerate box)
    }
    return n;
}

int mpm_sph_reset_dambreak(mpm_sph* s, int num_particles, const double half[3], uint64_t seed) {
    if (!s || !half) return fail(MPM_E_INVALID, "bad arguments");
    if (num_particles < 0 || num_particles > s->max_particles)
        return fail(MPM_E_CAPACITY, "numParticles exceeds the particle capacity");
    std::vector<float> buf((size_t)16 * (size_t)(num_particles > 0 ? num_particles : 1));
    const int n = mpm_sph_scene_dambreak(buf.data(), num_particles, half, seed);
    if (n < 0) return n;
    const float rh[3] = {(float)half[0], (float)half[1], (float)half[2]};
    return mpm_sph_upload(s, buf.data(), n, rh);
}

int mpm_sph_set_real_box(mpm_sph* s, const float real_half[3]) {
    if (!s || !real_half) return fail(MPM_E_INVALID, "bad arguments");
    for (int a = 0; a < 3; ++a) s->real_half[a] = real_half[a];
    return MPM_OK;
}

}  // extern "C"

namespace {

// G lanes (or one thread) per particle.
template <int G>
void launch_density(mpm_sph* s, cudaStream_t st) {
    if constexpr (G == 1) {
        k_sph_density_thread<<<(s->n + kThreadBlock - 1) / kThreadBlock, kThreadBlock, 0, st>>>(
            s->SP, s->SV, s->D, s->DR, s->nl, s->start, s->e);
    } else {
        const int gb = (s->n + Group<G>::kParticles - 1) / Group<G>::kParticles;
        k_sph_density<G><<<gb, kGroupBlock, 0, st>>>(s->SP, s->SV, s->D, s->DR, s->nl, s->start, s->e);
    }
}

template <int G>
void launch_force(mpm_sph* s, const SphOut& out, cudaStream_t st) {
    if constexpr (G == 1) {
        k_sph_force_thread<<<(s->n + kThreadBlock - 1) / kThreadBlock, kThreadBlock, 0, st>>>(
            s->D, s->DR, s->nl, s->order, s->start, s->e, s->box_d, out);
    } else {
        const int gb = (s->n + Group<G>::kParticles - 1) / Group<G>::kParticles;
        k_sph_force<G><<<gb, kGroupBlock, 0, st>>>(s->D, s->DR, s->nl, s->order, s->start, s->e,
                                                   s->box_d, out);
    }
}

void enqueue_substeps(mpm_sph* s, int substeps, cudaStream_t st) {
    const int n = s->n;
    const Env& e = s->e;
    const SphOut out{s->P, s->V, s->F, s->posvel};
    const int pb = (n + 255) / 256;
    const int chunks = (e.total + kScan - 1) / kScan;
    for (int k = 0; k < substeps; ++k) {
        // big blocks where there are enough of them: fewer blocks add to the few
        // chunk counts (ncu, 400,000 particles: 14.1 -> 11.3 us)
        const int bin_block = n >= 200000 ? 1024 : 256;
        k_sph_bin<<<(n + bin_block - 1) / bin_block, bin_block, 0, st>>>(out, n, e, s->cell_of, s->count, s->chunk, s->rank);
        k_sph_scan<<<chunks, kScan, 0, st>>>(s->count, s->chunk, e.total, s->start);
        k_sph_scatter<<<pb, 256, 0, st>>>(s->cell_of, s->rank, s->start, n, s->chunk, s->arrival);
        // sorted slots: start[total] of them (read on the device); launched
        // over n, the most there can be
        k_sph_place<<<pb, 256, 0, st>>>(s->P, s->V, s->cell_of, s->start, e.total, s->arrival,
                                        s->order, s->SP, s->SV);
        const bool fastest = s->warp_max < 0;
        const bool lanes_f = n <= (fastest ? kSphLanesMax : s->warp_max);
        const bool lanes_d = n <= (fastest ? kSphDensity8Max : s->warp_max);
        if (!lanes_d) launch_density<1>(s, st);
        else if (n <= kSph16Max) launch_density<16>(s, st);
        else launch_density<8>(s, st);
        if (!lanes_f) launch_force<1>(s, out, st);
        else if (n <= kSph16Max) launch_force<16>(s, out, st);
        else launch_force<8>(s, out, st);
    }
}

// The frame's launches as a CUDA graph, captured once per (substeps,
// particle count) and replayed.
cudaError_t launch_graph(mpm_sph* s, int substeps, cudaStream_t st) {
    mpm_sph::FrameGraph* hit = nullptr;
    for (auto& g : s->graphs)
        if (g.substeps == substeps && g.n == s->n) hit = &g;
    if (!hit) {
        cudaStream_t cs = nullptr;
        cudaError_t err = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
        if (err != cudaSuccess) return err;
        cudaGraph_t graph = nullptr;
        err = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
        if (err == cudaSuccess) {
            enqueue_substeps(s, substeps, cs);
            err = cudaStreamEndCapture(cs, &graph);
        }
        cudaGraphExec_t exec = nullptr;
        if (err == cudaSuccess) err = cudaGraphInstantiate(&exec, graph, 0);
        if (graph) cudaGraphDestroy(graph);
        cudaStreamDestroy(cs);
        if (err != cudaSuccess) return err;
        s->graphs.push_back({substeps, s->n, exec});
        hit = &s->graphs.back();
    }
    return cudaGraphLaunch(hit->exec, st);
}

}  // namespace

extern "C" {

// execute (sph.ts:325-355): `substeps` x (grid clear, build, prefix sum,
// reorder, density, reorder, force, integrate, copyPosition).
int mpm_sph_step(mpm_sph* s, int substeps, void* stream) {
    if (!s || substeps < 0) return fail(MPM_E_INVALID, "bad arguments");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (s->n == 0 || substeps == 0) return MPM_OK;
    if (std::memcmp(s->box_uploaded, s->real_half, sizeof(s->real_half)) != 0) {
        // pageable source: staged before the call returns
        const cudaError_t err =
            cudaMemcpyAsync(s->box_d, s->real_half, sizeof(s->real_half), cudaMemcpyHostToDevice, st);
        if (err != cudaSuccess) return cuda_fail(err, "mpm_sph_step");
        std::memcpy(s->box_uploaded, s->real_half, sizeof(s->real_half));
    }
    if (s->graph) {
        const cudaError_t err = launch_graph(s, substeps, st);
        if (err != cudaSuccess) return cuda_fail(err, "mpm_sph_step graph");
    } else {
        enqueue_substeps(s, substeps, st);
    }
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return cuda_fail(err, "mpm_sph_step");
    return MPM_OK;
}

int mpm_sph_set_graph(mpm_sph* s, int enable) {
    if (!s) return fail(MPM_E_INVALID, "bad arguments");
    s->graph = enable != 0;
    return MPM_OK;
}

int mpm_sph_set_warp_per_particle(mpm_sph* s, int max_particles) {
    if (!s || max_particles < -1) return fail(MPM_E_INVALID, "bad arguments");
    const int v = max_particles == kSphWarpMaxDefault ? -1 : max_particles;
    if (v != s->warp_max) drop_graphs(s);  // the captured frames hold the launches
    s->warp_max = v;
    return MPM_OK;
}

int mpm_sph_get_warp_per_particle(const mpm_sph* s) {
    if (!s) return MPM_E_INVALID;
    return s->warp_max < 0 ? kSphWarpMaxDefault : s->warp_max;
}

int mpm_sph_num_particles(const mpm_sph* s) { return s ? s->n : 0; }
int64_t mpm_sph_grid_count(const mpm_sph* s) { return s ? s->e.total : 0; }
void* mpm_sph_posvel_device_ptr(mpm_sph* s) { return s ? s->posvel : nullptr; }

int mpm_sph_download_particles(mpm_sph* s, float* out_rec64) {
    if (!s || (!out_rec64 && s->n)) return fail(MPM_E_INVALID, "bad arguments");
    const int n = s->n;
    std::vector<float4> P((size_t)n), V((size_t)n), F((size_t)n);
    cudaError_t err = cudaDeviceSynchronize();
    if (n && err == cudaSuccess) err = cudaMemcpy(P.data(), s->P, sizeof(float4) * n, cudaMemcpyDeviceToHost);
    if (n && err == cudaSuccess) err = cudaMemcpy(V.data(), s->V, sizeof(float4) * n, cudaMemcpyDeviceToHost);
    if (n && err == cudaSuccess) err = cudaMemcpy(F.data(), s->F, sizeof(float4) * n, cudaMemcpyDeviceToHost);
    if (err != cudaSuccess) return cuda_fail(err, "mpm_sph_download_particles");
    for (int i = 0; i < n; ++i) {
        float* r = out_rec64 + 16 * (size_t)i;
        std::memset(r, 0, 64);
        r[0] = P[(size_t)i].x; r[1] = P[(size_t)i].y; r[2] = P[(size_t)i].z;
        r[4] = V[(size_t)i].x; r[5] = V[(size_t)i].y; r[6] = V[(size_t)i].z;
        r[8] = F[(size_t)i].x; r[9] = F[(size_t)i].y; r[10] = F[(size_t)i].z;
        r[11] = P[(size_t)i].w;   // density
        r[12] = V[(size_t)i].w;   // nearDensity
    }
    return MPM_OK;
}

int mpm_sph_download_posvel(mpm_sph* s, float* out) {
    if (!s || (!out && s->n)) return fail(MPM_E_INVALID, "bad arguments");
    cudaError_t err = cudaDeviceSynchronize();
    if (s->n && err == cudaSuccess)
        err = cudaMemcpy(out, s->posvel, sizeof(float4) * 2 * (size_t)s->n, cudaMemcpyDeviceToHost);
    if (err != cudaSuccess) return cuda_fail(err, "mpm_sph_download_posvel");
    return MPM_OK;
}

}  // extern "C"
