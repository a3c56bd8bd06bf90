// Receptor grid maps (sm_100a): Vina/Vinardo per-ligand-type maps and the fitted function's maps.
//
// The reference launches one thread per grid point that scans every receptor atom (grid.py:24-61,
// gridfit.py:21-57). Here a CTA owns a tile of points: 8 x 8 x 8 (256 threads, two points per thread) or, for grids too
// small to fill the SMs with those, 4 x 4 x 8 (128 threads, one point). The receptor comes as a cell list: atoms sorted by
// cell of a uniform grid, with the start of every cell. A CTA visits only the cells that overlap its tile's bounding box
// grown by the cutoff (columns of cells along z are contiguous in the sorted atoms) and keeps the atoms inside the grown
// box in shared memory (ordered compaction). A warp owns a compact patch of 4 x 4 x 4 points (2 x 4 x 4 with one point per
// thread): its lanes test 32 staged atoms at a time against the patch's box, and only the atoms in reach are evaluated by
// all lanes. Without a cell list (one cell holding every atom in receptor order) this is a scan of the whole receptor per
// CTA, and the summation order per point is the reference's receptor order; with one, it is the cell order.
//
// The distance-dependent parts of the terms depend on the ligand type only through its radius. The Vina kernel keeps
// sums per distinct radius (the Gaussians and the repulsion; the hydrophobic ramp over hydrophobic atoms; the
// hydrogen-bond ramp over donors, acceptors and either) and forms every type's map from them at the end; the fitted
// kernel evaluates the basis once per distinct radius and adds it with each type's weights. Radii (types) are processed
// in groups that fit the registers.
#include "common.cuh"

namespace adock {

#define STAGE_CAP 768       // staged atoms per pass (24 KB for the Vina kernel)
#define RADIUS_GROUP 4
#define FIT_GROUP 8
#define MAX_COLUMNS 64

// Tile of a CTA with PP points per thread: warps own patches of 2 PP x 4 x 4 points.
template <int PP>
struct Tile {
    static constexpr int X = PP == 2 ? 8 : 4, Y = PP == 2 ? 8 : 4, Z = 8;
    static constexpr int WARPS = X * Y * Z / (32 * PP), THREADS = 32 * WARPS;
};

// Sums of one distinct radius that a map needs, without the weights: each term's rounding then stays in proportion to the
// term (everybody's small Gaussians added to a large repulsion would round each time), and the same sums give the
// per-term maps.
enum { SUM_G1, SUM_G2, SUM_REP, SUM_HYD, SUM_DON, SUM_ACC, SUM_EITHER, SUMS };
enum { NEED_HYD = 1, NEED_HB = 2 };

struct VinaPrm {
    float cutoff, rep_off;
    float g1_off, g1_k, g2_off, g2_k;         // Gaussian = 2^-((d - off) k)^2
    float hyd_bad, hyd_inv, hb_bad, hb_inv;   // ramp = saturate((bad - d) inv); a step (good = bad) has inv = infinity
    int falling;                              // a ramp has inv < 0: not 0 far away
    float w[5];
    int n_lt, n_xs, n_rad;
    int per_term;        // write the five unweighted terms
    float rad[24];       // distinct radii, ascending
    int need[24];        // NEED_* of the radius's types
    int rad_of[24];      // each map's radius
    int gate[24];        // each map's sums beside the first three: bit 0 SUM_HYD; bits 1-2 the H-bond sum (0 none)
    float radius[64];
    int flags[64];  // bit0 hydrophobic, bit1 donor, bit2 acceptor
};

struct FitPrm {
    float cutoff, rep_off;
    float g1_off, g1_k, g2_off, g2_k, hyd_bad, hyd_inv, hb_bad, hb_inv;   // as VinaPrm
    int falling;
    float ion_rmin2, ion_cut, rep_cap;                         // ion_rmin2 = minimum distance^2, ion_cut = 1 / cutoff^2
    int n_lt, n_rt;
    float rad_lig[64];   // in order of radius
    int out_slot[64];    // output map (and W column) of each (radius-ordered) type
};

// Uniform cell grid over the receptor: cell (cx, cy, cz) holds sorted atoms [start[c], start[c + 1]) with
// c = (cx * ny + cy) * nz + cz. start == NULL: one cell holding all n atoms in receptor order.
struct Cells {
    const int* start;
    int nx, ny, nz;
    float ox, oy, oz, size;
};

// The columns of cells (fixed cx, cy; the cz range of the box) that overlap [lo, hi]: begin of each column's atom range
// and prefix sums of the lengths in off[0..ncol]. Called by all threads; returns the number of columns.
__device__ __forceinline__ int tile_columns(const Cells& C, int n_rec, const float* lo, const float* hi, int* begin, int* off) {
    if (!C.start) {
        if (threadIdx.x == 0) {
            begin[0] = 0;
            off[0] = 0;
            off[1] = n_rec;
        }
        __syncthreads();
        return 1;
    }
    auto cell = [&](float v, float o, int n) { return min(max((int)floorf((v - o) / C.size), 0), n - 1); };
    const int x0 = cell(lo[0], C.ox, C.nx), x1 = cell(hi[0], C.ox, C.nx);
    const int y0 = cell(lo[1], C.oy, C.ny), y1 = cell(hi[1], C.oy, C.ny);
    const int z0 = cell(lo[2], C.oz, C.nz), z1 = cell(hi[2], C.oz, C.nz);
    const int rows = y1 - y0 + 1, ncol = min((x1 - x0 + 1) * rows, MAX_COLUMNS);
    if (threadIdx.x < 32) {   // two columns per lane
        int carry = 0;
        for (int h = 0; h < MAX_COLUMNS; h += 32) {
            const int i = h + threadIdx.x;
            int len = 0;
            if (i < ncol) {
                const int c = ((x0 + i / rows) * C.ny + y0 + i % rows) * C.nz;
                const int b = C.start[c + z0];
                begin[i] = b;
                len = C.start[c + z1 + 1] - b;
            }
            int incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)threadIdx.x >= o) incl += t;
            }
            off[i + 1] = carry + incl;
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (threadIdx.x == 0) off[0] = 0;
    }
    __syncthreads();
    return ncol;
}

// Stage the atoms inside [lo, hi] (per axis) from position `start` of the concatenated columns, at most STAGE_CAP, through
// put(slot, xyz, type); returns the position where staging stopped (the total when all atoms were seen). Staged order =
// column order.
template <int THREADS, typename PUT>
__device__ __forceinline__ int stage_atoms(const float* __restrict__ rxyz, const int* __restrict__ rtype, const int* begin,
                                           const int* off, int ncol, int start, const float* lo, const float* hi, int* count,
                                           int* wsum, PUT put) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int total = off[ncol];
    int n = 0;
    int v0 = start;
    for (; v0 < total && n + THREADS <= STAGE_CAP; v0 += THREADS) {
        const int v = v0 + tid;
        bool in = false;
        float x = 0.f, y = 0.f, z = 0.f;
        int a = 0;
        if (v < total) {
            int c = 0;   // the column of position v: off[c] <= v < off[c + 1]
#pragma unroll
            for (int o = MAX_COLUMNS / 2; o > 0; o >>= 1)
                if (c + o < ncol && off[c + o] <= v) c += o;
            a = begin[c] + (v - off[c]);
            x = rxyz[3 * a]; y = rxyz[3 * a + 1]; z = rxyz[3 * a + 2];
            in = !(x < lo[0] || x > hi[0] || y < lo[1] || y > hi[1] || z < lo[2] || z > hi[2]);
        }
        const unsigned bal = __ballot_sync(0xffffffffu, in);
        if (lane == 0) wsum[wid] = __popc(bal);
        __syncthreads();
        int o = n, tot = 0;
#pragma unroll
        for (int w = 0; w < THREADS / 32; ++w) {
            if (w < wid) o += wsum[w];
            tot += wsum[w];
        }
        if (in) put(o + __popc(bal & ((1u << lane) - 1u)), x, y, z, rtype[a]);
        n += tot;
        __syncthreads();
    }
    *count = n;
    return min(v0, total);
}

// The tile, patch and points of a thread, and the atom columns of its CTA.
template <int PP>
struct TileSetup {
    float x[PP], y, z;              // points (the second one 2 further along x)
    long long p[PP];                // output index, -1 outside the grid
    float plo[3], phi[3];           // the warp's patch grown by the cutoff
    float lo[3], hi[3];             // the tile grown by the cutoff
    __device__ __forceinline__ TileSetup(float ox, float oy, float oz, float spacing, int nx, int ny, int nz, float cutoff) {
        using T = Tile<PP>;
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        const int t0[3] = {(int)blockIdx.x * T::X, (int)blockIdx.y * T::Y, (int)blockIdx.z * T::Z};
        const int px = 2 * PP, wx = T::X / px, wy = T::Y / 4;
        const int w0[3] = {t0[0] + (wid % wx) * px, t0[1] + (wid / wx % wy) * 4, t0[2] + wid / (wx * wy) * 4};
        const float o[3] = {ox, oy, oz};
        const int n[3] = {nx, ny, nz}, tile[3] = {T::X, T::Y, T::Z}, patch[3] = {px, 4, 4};
        for (int d = 0; d < 3; ++d) {
            lo[d] = o[d] + t0[d] * spacing - cutoff;
            hi[d] = o[d] + (min(t0[d] + tile[d], n[d]) - 1) * spacing + cutoff;
            plo[d] = o[d] + w0[d] * spacing;
            phi[d] = o[d] + (min(w0[d] + patch[d], n[d]) - 1) * spacing;
        }
        const int j = w0[1] + (lane >> 2 & 3), k = w0[2] + (lane & 3);
        y = oy + j * spacing;
        z = oz + k * spacing;
        for (int h = 0; h < PP; ++h) {
            const int i = w0[0] + (lane >> 4) + 2 * h;
            x[h] = ox + i * spacing;
            p[h] = i < nx && j < ny && k < nz ? ((long long)i * ny + j) * nz + k : -1;
        }
    }
    // whether an atom can be within the cutoff of a point of the patch (reach2: cutoff^2, widened for rounding)
    __device__ __forceinline__ bool in_reach(float ax, float ay, float az, float reach2) const {
        const float dx = fmaxf(fmaxf(plo[0] - ax, ax - phi[0]), 0.f), dy = fmaxf(fmaxf(plo[1] - ay, ay - phi[1]), 0.f),
                    dz = fmaxf(fmaxf(plo[2] - az, az - phi[2]), 0.f);
        return dx * dx + dy * dy + dz * dz <= reach2;
    }
};

// 2^x; results below 2^-126 are 0
__device__ __forceinline__ float exp2_ftz(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// A pair beyond the cutoff is moved to this surface distance, where the Gaussians, the repulsion and rising ramps are
// exactly 0 (falling ramps, bad < good, are gated separately): no branch, so a thread's two points stay in flight.
#define FAR_AWAY 1e4f

// 1 / x to 1 ulp; subnormal x counts as 0
__device__ __forceinline__ float rcp_ftz(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Distances of an atom at offsets (dx, dy, dz) from the thread's points; far: beyond the cutoff. r = r2 / sqrt(r2) with one
// Newton step, so it is as exact as sqrtf.
template <int PP>
struct Distances {
    float r[PP], r2[PP];
    bool far[PP];
    __device__ __forceinline__ Distances(float ax, const float (&x)[PP], float dy, float dz, float cut2) {
#pragma unroll
        for (int h = 0; h < PP; ++h) {
            const float dx = ax - x[h];
            r2[h] = __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
            far[h] = r2[h] >= cut2;
            const float rinv = rsqrt_ftz(fmaxf(r2[h], 1e-20f)), y = r2[h] * rinv;
            r[h] = __fmaf_rn(__fmaf_rn(-y, y, r2[h]), 0.5f * rinv, y);
        }
    }
};

// Vina maps. Bound by instruction issue and the two exponentials per (atom, point, radius). A thread per point that
// added five sums per ligand type and tested every staged atom took 687 us for 8,000 receptor atoms, 81^3 points and 8
// types (4 radii), this 294 us, the per-term maps 304 us.
template <int PP>
__global__ void __launch_bounds__(Tile<PP>::THREADS, PP == 2 ? 3 : 8) grid_vina_kernel(const float* __restrict__ rxyz,
                                                                      const int* __restrict__ rtype, int n_rec,
                                                                      const __grid_constant__ Cells C, float ox, float oy,
                                                                      float oz, float spacing, int nx, int ny, int nz,
                                                                      const __grid_constant__ VinaPrm P,
                                                                      float* __restrict__ out) {
    __shared__ float4 S[STAGE_CAP];   // xyz, radius
    __shared__ float4 G[STAGE_CAP];   // 1 or 0: hydrophobic, donor, acceptor, donor or acceptor
    __shared__ int wsum[Tile<PP>::WARPS], col_begin[MAX_COLUMNS], col_off[MAX_COLUMNS + 1];
    const TileSetup<PP> t(ox, oy, oz, spacing, nx, ny, nz, P.cutoff);
    const int ncol = tile_columns(C, n_rec, t.lo, t.hi, col_begin, col_off);
    const int lane = threadIdx.x & 31, total = col_off[ncol];
    const float cut2 = P.cutoff * P.cutoff, reach2 = cut2 * 1.0001f + 1e-3f;
    const long long npts = (long long)nx * ny * nz;
    for (int r0 = 0; r0 < P.n_rad; r0 += RADIUS_GROUP) {
        float sum[PP][RADIUS_GROUP][SUMS];
#pragma unroll
        for (int h = 0; h < PP; ++h)
#pragma unroll
            for (int q = 0; q < RADIUS_GROUP; ++q)
#pragma unroll
                for (int m = 0; m < SUMS; ++m) sum[h][q][m] = 0.f;
        int start = 0;
        while (start < total) {
            int cnt;
            start = stage_atoms<Tile<PP>::THREADS>(rxyz, rtype, col_begin, col_off, ncol, start, t.lo, t.hi, &cnt, wsum,
                                                   [&](int s, float ax, float ay, float az, int ta) {
                                                       const int f = P.flags[ta];
                                                       S[s] = make_float4(ax, ay, az, P.radius[ta]);
                                                       G[s] = make_float4(f & 1 ? 1.f : 0.f, f & 2 ? 1.f : 0.f,
                                                                          f & 4 ? 1.f : 0.f, f & 6 ? 1.f : 0.f);
                                                   });
            for (int s0 = 0; s0 < cnt; s0 += 32) {
                const int s = s0 + lane;
                bool near = false;
                if (s < cnt) {
                    const float4 A = S[s];
                    near = t.in_reach(A.x, A.y, A.z, reach2);
                }
                unsigned todo = __ballot_sync(0xffffffffu, near);
                while (todo) {
                    const int at = s0 + __ffs(todo) - 1;
                    todo &= todo - 1;
                    const float4 A = S[at], g = G[at];
                    const Distances<PP> D(A.x, t.x, A.y - t.y, A.z - t.z, cut2);
                    float r[PP], on[PP];
#pragma unroll
                    for (int h = 0; h < PP; ++h) {
                        r[h] = D.far[h] ? FAR_AWAY : D.r[h] - A.w;
                        on[h] = D.far[h] ? 0.f : 1.f;
                    }
#pragma unroll
                    for (int q = 0; q < RADIUS_GROUP; ++q) {
                        if (r0 + q >= P.n_rad) break;
                        const int need = P.need[r0 + q];
#pragma unroll
                        for (int h = 0; h < PP; ++h) {
                            const float d = r[h] - P.rad[r0 + q];
                            const float u1 = (d - P.g1_off) * P.g1_k, u2 = (d - P.g2_off) * P.g2_k;
                            const float dr = fminf(d - P.rep_off, 0.f);
                            float* a = sum[h][q];
                            a[SUM_G1] += exp2_ftz(-u1 * u1);
                            a[SUM_G2] += exp2_ftz(-u2 * u2);
                            a[SUM_REP] += dr * dr;
                            if (need & NEED_HYD) {
                                float hyd = __saturatef((P.hyd_bad - d) * P.hyd_inv);
                                if (P.falling) hyd *= on[h];
                                a[SUM_HYD] += hyd * g.x;
                            }
                            if (need & NEED_HB) {
                                float hb = __saturatef((P.hb_bad - d) * P.hb_inv);
                                if (P.falling) hb *= on[h];
                                a[SUM_DON] += hb * g.y;
                                a[SUM_ACC] += hb * g.z;
                                a[SUM_EITHER] += hb * g.w;
                            }
                        }
                    }
                }
            }
            __syncthreads();
        }
        // the maps of these radii
        for (int o = 0; o < P.n_lt; ++o) {
#pragma unroll
            for (int q = 0; q < RADIUS_GROUP; ++q) {
                if (P.rad_of[o] != r0 + q) continue;
                const int hb = P.gate[o] >> 1;
#pragma unroll
                for (int h = 0; h < PP; ++h) {
                    if (t.p[h] < 0) continue;
                    const float* a = sum[h][q];
                    const float e_hyd = P.gate[o] & 1 ? a[SUM_HYD] : 0.f;
                    const float e_hb = hb == 0 ? 0.f : (hb == 1 ? a[SUM_DON] : (hb == 2 ? a[SUM_ACC] : a[SUM_EITHER]));
                    const float e[5] = {a[SUM_G1], a[SUM_G2], a[SUM_REP], e_hyd, e_hb};
                    float* dst = out + (long long)o * npts + t.p[h];
                    if (P.per_term) {
#pragma unroll
                        for (int m = 0; m < 5; ++m) dst[(long long)m * P.n_lt * npts] = e[m];
                    } else {
                        float v = 0.f;
#pragma unroll
                        for (int m = 0; m < 5; ++m) v += P.w[m] * e[m];
                        *dst = v;
                    }
                }
            }
        }
    }
}

// Fitted maps. Bound by instruction issue: six multiply-adds per (atom, point, type) beside the basis per radius; the
// weights come from shared memory, once for a thread's two points. One point per thread with every staged atom tested took
// 732 us for 8,000 receptor atoms, 81^3 points and 8 types, this 452 us.
// Packed FP32 pairs for the two points (fma.rn.f32x2) were slower in both kernels (287 and 432 us): the exponentials, minima
// and ramps stay scalar, so the registers and moves of the pairs cost more than the issue slots they save.
template <int PP>
__global__ void __launch_bounds__(Tile<PP>::THREADS, PP == 2 ? 3 : 6) grid_fit_kernel(const float* __restrict__ rxyz,
                                                                     const int* __restrict__ rext, int n_rec,
                                                                     const __grid_constant__ Cells C, float ox, float oy,
                                                                     float oz, float spacing, int nx, int ny, int nz,
                                                                     const __grid_constant__ FitPrm P,
                                                                     const float* __restrict__ W,
                                                                     const float* __restrict__ rad_rec,
                                                                     float* __restrict__ out) {
    __shared__ float4 S[STAGE_CAP];   // xyz, ext type
    __shared__ int wsum[Tile<PP>::WARPS], col_begin[MAX_COLUMNS], col_off[MAX_COLUMNS + 1];
    extern __shared__ float2 Wsh[];   // [n_rt, FIT_GROUP, 3] slice of W (radius-ordered types), then rad_rec [n_rt]
    float* Rsh = (float*)(Wsh + (size_t)P.n_rt * FIT_GROUP * 3);
    const TileSetup<PP> t(ox, oy, oz, spacing, nx, ny, nz, P.cutoff);
    const int ncol = tile_columns(C, n_rec, t.lo, t.hi, col_begin, col_off);
    const int lane = threadIdx.x & 31, total = col_off[ncol];
    const float cut2 = P.cutoff * P.cutoff, reach2 = cut2 * 1.0001f + 1e-3f;
    const long long npts = (long long)nx * ny * nz;
    for (int i = threadIdx.x; i < P.n_rt; i += Tile<PP>::THREADS) Rsh[i] = rad_rec[i];

    for (int q0 = 0; q0 < P.n_lt; q0 += FIT_GROUP) {
        const int gq = min(FIT_GROUP, P.n_lt - q0);
        __syncthreads();
        for (int e = threadIdx.x; e < P.n_rt * FIT_GROUP * 6; e += Tile<PP>::THREADS) {
            const int rt = e / (FIT_GROUP * 6), q = (e / 6) % FIT_GROUP, b = e % 6;
            ((float*)Wsh)[e] = q < gq ? W[((long long)rt * P.n_lt + P.out_slot[q0 + q]) * 6 + b] : 0.f;
        }
        __syncthreads();
        float acc[PP][FIT_GROUP], acc_rep[PP][FIT_GROUP];   // the repulsion apart: see SUM_REP
#pragma unroll
        for (int h = 0; h < PP; ++h)
#pragma unroll
            for (int q = 0; q < FIT_GROUP; ++q) acc[h][q] = acc_rep[h][q] = 0.f;
        int start = 0;
        while (start < total) {
            int cnt;
            start = stage_atoms<Tile<PP>::THREADS>(rxyz, rext, col_begin, col_off, ncol, start, t.lo, t.hi, &cnt, wsum,
                                                   [&](int s, float ax, float ay, float az, int ta) {
                                                       S[s] = make_float4(ax, ay, az, __int_as_float(ta));
                                                   });
            for (int s0 = 0; s0 < cnt; s0 += 32) {
                const int s = s0 + lane;
                bool near = false;
                if (s < cnt) {
                    const float4 A = S[s];
                    near = t.in_reach(A.x, A.y, A.z, reach2);
                }
                unsigned todo = __ballot_sync(0xffffffffu, near);
                while (todo) {
                    const int at = s0 + __ffs(todo) - 1;
                    todo &= todo - 1;
                    const float4 A = S[at];
                    const int ta = __float_as_int(A.w);
                    const float ra = Rsh[ta];
                    const float2* Wa = Wsh + (size_t)ta * FIT_GROUP * 3;
                    const Distances<PP> D(A.x, t.x, A.y - t.y, A.z - t.z, cut2);
                    float r[PP], on[PP], ion[PP], g1[PP], g2[PP], rep[PP], hyd[PP], hb[PP];
#pragma unroll
                    for (int h = 0; h < PP; ++h) {
                        on[h] = D.far[h] ? 0.f : 1.f;
                        r[h] = D.far[h] ? FAR_AWAY : D.r[h] - ra;
                        // 1 / max(r, minimum)^2 straight from r^2: one rounding less than by way of r
                        ion[h] = D.far[h] ? 0.f : rcp_ftz(fmaxf(D.r2[h], P.ion_rmin2)) - P.ion_cut;
                    }
#pragma unroll
                    for (int q = 0; q < FIT_GROUP; ++q) {
                        if (q >= gq) break;
                        if (q == 0 || P.rad_lig[q0 + q] != P.rad_lig[q0 + q - 1]) {   // next radius
#pragma unroll
                            for (int h = 0; h < PP; ++h) {
                                const float d = r[h] - P.rad_lig[q0 + q];
                                const float u1 = (d - P.g1_off) * P.g1_k, u2 = (d - P.g2_off) * P.g2_k;
                                const float dr = fminf(d - P.rep_off, 0.f);
                                g1[h] = exp2_ftz(-u1 * u1);
                                g2[h] = exp2_ftz(-u2 * u2);
                                rep[h] = fminf(dr * dr, P.rep_cap);
                                hyd[h] = __saturatef((P.hyd_bad - d) * P.hyd_inv);
                                hb[h] = __saturatef((P.hb_bad - d) * P.hb_inv);
                                if (P.falling) { hyd[h] *= on[h]; hb[h] *= on[h]; }
                            }
                        }
                        const float2 w0 = Wa[q * 3], w1 = Wa[q * 3 + 1], w2 = Wa[q * 3 + 2];
#pragma unroll
                        for (int h = 0; h < PP; ++h) {
                            acc[h][q] += w0.x * g1[h];
                            acc[h][q] += w0.y * g2[h];
                            acc[h][q] += w1.y * hyd[h];
                            acc[h][q] += w2.x * hb[h];
                            acc[h][q] += w2.y * ion[h];
                            acc_rep[h][q] += w1.x * rep[h];
                        }
                    }
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int h = 0; h < PP; ++h)
            if (t.p[h] >= 0)
#pragma unroll
                for (int q = 0; q < FIT_GROUP; ++q)
                    if (q < gq) out[(long long)P.out_slot[q0 + q] * npts + t.p[h]] = acc[h][q] + acc_rep[h][q];
    }
}

template <typename T>
__global__ void convert_kernel(const float* __restrict__ src, T* __restrict__ dst, long long n);
// FP16 saturates at +-65504 (map values inside receptor atoms can exceed the FP16 range; a clamped value keeps
// such points repulsive instead of turning the interpolation into inf/NaN)
template <>
__global__ void convert_kernel<__half>(const float* __restrict__ src, __half* __restrict__ dst, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = __float2half_rn(fminf(fmaxf(src[i], -65504.f), 65504.f));
}
template <>
__global__ void convert_kernel<__nv_bfloat16>(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = __float2bfloat16_rn(src[i]);
}

// Order of a launch's ligand types by radius (stable): positions order[0..n) into the caller's type list.
static void order_by_radius(const float* rad, int n, int* order) {
    for (int q = 0; q < n; ++q) order[q] = q;
    for (int a = 1; a < n; ++a) {   // insertion sort, n <= 64
        const int v = order[a];
        int b = a - 1;
        while (b >= 0 && rad[order[b]] > rad[v]) {
            order[b + 1] = order[b];
            --b;
        }
        order[b + 1] = v;
    }
}

// columns of cells that a tile of `points` x `points` points can touch: ceil(extent / size) + 1 per axis
static int tile_reach(const Cells& C, int points, float cutoff, float spacing) {
    const int per = (int)ceilf((points * spacing + 2.f * cutoff) / C.size) + 1;
    return per * per;
}

static int check_cells(const Cells& C, float cutoff, float spacing) {
    if (!C.start) return ADOCK_OK;
    ADOCK_CHECK_ARG(C.nx >= 1 && C.ny >= 1 && C.nz >= 1 && C.size > 0.f, "bad cell grid");
    ADOCK_CHECK_ARG(tile_reach(C, 4, cutoff, spacing) <= MAX_COLUMNS,
                    "cell size %.3f too small for the cutoff (at most %d columns per tile)", C.size, MAX_COLUMNS);
    return ADOCK_OK;
}

template <int PP>
static dim3 tiles(int nx, int ny, int nz) {
    using T = Tile<PP>;
    return dim3((nx + T::X - 1) / T::X, (ny + T::Y - 1) / T::Y, (nz + T::Z - 1) / T::Z);
}

// Two points per thread need a quarter of the CTAs: taken where those fill the SMs twice (and a tile's columns fit). 61^3
// points are 512 such CTAs (124 us for 1,500 atoms); 28^3 points only 64, where one point per thread gives 196.
static bool two_points(const Cells& C, float cutoff, float spacing, int nx, int ny, int nz) {
    const dim3 g = tiles<2>(nx, ny, nz);
    return (long long)g.x * g.y * g.z >= 2LL * sm_count() && (!C.start || tile_reach(C, 8, cutoff, spacing) <= MAX_COLUMNS);
}

// exp(-((d - off) / w)^2) = 2^-((d - off) k)^2 and the ramp's slope 1 / (bad - good). The offsets stay apart from the
// products: folded into one multiply-add (k d - c) a step's or a zero width's infinite k would meet an infinite c and give
// NaN. The extra instruction per term costs 3 % (8,000 atoms, 81^3 points, 8 types: 295 us folded, 303 us so).
static float gauss_k(float w) { return (float)(sqrt(1.4426950408889634) / (double)w); }
static float ramp_inv(float good, float bad) { return (float)(1.0 / ((double)bad - (double)good)); }

static int grid_vina_launch(const float* rec_xyz, const int* rec_types, int n_rec, const Cells& C, const float* radius,
                            const int* hyd, const int* don, const int* acc, int n_xs, const int* lig_types, int n_lt,
                            float ox, float oy, float oz, float spacing, int nx, int ny, int nz, const float* prm,
                            int per_term, float* out, void* stream) {
    ADOCK_CHECK_ARG(n_rec >= 0 && (n_rec == 0 || (rec_xyz && rec_types)), "bad receptor arrays");
    ADOCK_CHECK_ARG(radius && hyd && don && acc && lig_types && prm && out, "null argument");
    ADOCK_CHECK_ARG(n_xs >= 1 && n_xs <= 64, "n_xs must be in [1, 64] (got %d)", n_xs);
    ADOCK_CHECK_ARG(n_lt >= 1 && n_lt <= 24, "n_lt must be in [1, 24] (got %d)", n_lt);
    ADOCK_CHECK_ARG(nx >= 1 && ny >= 1 && nz >= 1, "grid dimensions must be >= 1");
    ADOCK_CHECK_ARG(spacing > 0.f, "spacing must be > 0");
    int rc = check_cells(C, prm[0], spacing);
    if (rc) return rc;
    VinaPrm P;
    P.cutoff = prm[0];
    P.g1_off = prm[1]; P.g1_k = gauss_k(prm[2]);
    P.g2_off = prm[3]; P.g2_k = gauss_k(prm[4]);
    P.rep_off = prm[5];
    P.hyd_bad = prm[7]; P.hyd_inv = ramp_inv(prm[6], prm[7]);
    P.hb_bad = prm[9]; P.hb_inv = ramp_inv(prm[8], prm[9]);
    P.falling = !(P.hyd_inv > 0.f && P.hb_inv > 0.f);
    for (int m = 0; m < 5; ++m) P.w[m] = prm[10 + m];
    P.n_lt = n_lt; P.n_xs = n_xs; P.per_term = per_term;
    for (int q = 0; q < n_lt; ++q) ADOCK_CHECK_ARG(lig_types[q] >= 0 && lig_types[q] < n_xs, "ligand type out of range");
    float rl[24];
    int order[24];
    for (int q = 0; q < n_lt; ++q) rl[q] = radius[lig_types[q]];
    order_by_radius(rl, n_lt, order);
    P.n_rad = 0;
    for (int q = 0; q < n_lt; ++q) {
        const int o = order[q], lt = lig_types[o];
        if (q == 0 || rl[o] != P.rad[P.n_rad - 1]) P.rad[P.n_rad++] = rl[o];
        if (q == 0 || P.rad_of[order[q - 1]] != P.n_rad - 1) P.need[P.n_rad - 1] = 0;
        P.rad_of[o] = P.n_rad - 1;
        // a donor type bonds with acceptor atoms, an acceptor type with donor atoms
        const int hb = don[lt] ? (acc[lt] ? 3 : 2) : (acc[lt] ? 1 : 0);
        P.gate[o] = (hyd[lt] ? 1 : 0) | (hb << 1);
        P.need[P.n_rad - 1] |= (hyd[lt] ? NEED_HYD : 0) | (hb ? NEED_HB : 0);
    }
    for (int q = P.n_rad; q < 24; ++q) {
        P.rad[q] = 0.f;
        P.need[q] = 0;
    }
    for (int q = n_lt; q < 24; ++q) P.rad_of[q] = P.gate[q] = 0;
    for (int t = 0; t < 64; ++t) {
        P.radius[t] = t < n_xs ? radius[t] : 0.f;
        P.flags[t] = t < n_xs ? ((hyd[t] ? 1 : 0) | (don[t] ? 2 : 0) | (acc[t] ? 4 : 0)) : 0;
    }
    const dim3 small = tiles<1>(nx, ny, nz);
    ADOCK_CHECK_ARG(small.y < 65536 && small.z < 65536, "grid too large");
    cudaStream_t st = (cudaStream_t)stream;
    if (two_points(C, prm[0], spacing, nx, ny, nz))
        grid_vina_kernel<2><<<tiles<2>(nx, ny, nz), Tile<2>::THREADS, 0, st>>>(rec_xyz, rec_types, n_rec, C, ox, oy, oz,
                                                                                      spacing, nx, ny, nz, P, out);
    else
        grid_vina_kernel<1><<<small, Tile<1>::THREADS, 0, st>>>(rec_xyz, rec_types, n_rec, C, ox, oy, oz, spacing, nx,
                                                                       ny, nz, P, out);
    ADOCK_CUDA(cudaGetLastError());
    return ADOCK_OK;
}

template <int PP>
static int launch_fit(const float* rec_xyz, const int* rec_ext, int n_rec, const Cells& C, float ox, float oy, float oz,
                      float spacing, int nx, int ny, int nz, const FitPrm& P, const float* W, const float* rad_rec, float* out,
                      cudaStream_t st) {
    const size_t smem = ((size_t)P.n_rt * FIT_GROUP * 6 + P.n_rt) * sizeof(float);
    ADOCK_CUDA(cudaFuncSetAttribute(grid_fit_kernel<PP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    grid_fit_kernel<PP><<<tiles<PP>(nx, ny, nz), Tile<PP>::THREADS, smem, st>>>(rec_xyz, rec_ext, n_rec, C, ox, oy, oz, spacing,
                                                                                nx, ny, nz, P, W, rad_rec, out);
    ADOCK_CUDA(cudaGetLastError());
    return ADOCK_OK;
}

static int grid_fit_launch(const float* rec_xyz, const int* rec_ext, int n_rec, const Cells& C, const float* rad_rec,
                           int n_rt, const float* rad_lig, int n_lt, const float* W, float ox, float oy, float oz,
                           float spacing, int nx, int ny, int nz, const float* prm, float* out, void* stream) {
    ADOCK_CHECK_ARG(n_rec >= 0 && (n_rec == 0 || (rec_xyz && rec_ext)), "bad receptor arrays");
    ADOCK_CHECK_ARG(rad_rec && rad_lig && W && prm && out, "null argument");
    ADOCK_CHECK_ARG(n_lt >= 1 && n_lt <= 64, "n_lt must be in [1, 64] (got %d)", n_lt);
    ADOCK_CHECK_ARG(n_rt >= 1 && n_rt <= 1024, "n_rt must be in [1, 1024] (got %d)", n_rt);
    ADOCK_CHECK_ARG(nx >= 1 && ny >= 1 && nz >= 1, "grid dimensions must be >= 1");
    ADOCK_CHECK_ARG(spacing > 0.f, "spacing must be > 0");
    int rc = check_cells(C, prm[0], spacing);
    if (rc) return rc;
    FitPrm P;
    P.cutoff = prm[0];
    P.g1_off = prm[1]; P.g1_k = gauss_k(prm[2]);
    P.g2_off = prm[3]; P.g2_k = gauss_k(prm[4]);
    P.rep_off = prm[5];
    P.hyd_bad = prm[7]; P.hyd_inv = ramp_inv(prm[6], prm[7]);
    P.hb_bad = prm[9]; P.hb_inv = ramp_inv(prm[8], prm[9]);
    P.falling = !(P.hyd_inv > 0.f && P.hb_inv > 0.f);
    P.ion_rmin2 = prm[10] > 0.f ? prm[10] * prm[10] : 0.f; P.ion_cut = 1.f / (prm[0] * prm[0]); P.rep_cap = prm[11];
    P.n_lt = n_lt; P.n_rt = n_rt;
    int order[64];
    order_by_radius(rad_lig, n_lt, order);
    for (int q = 0; q < 64; ++q) {
        P.rad_lig[q] = q < n_lt ? rad_lig[order[q]] : 0.f;
        P.out_slot[q] = q < n_lt ? order[q] : 0;
    }
    const dim3 small = tiles<1>(nx, ny, nz);
    ADOCK_CHECK_ARG(small.y < 65536 && small.z < 65536, "grid too large");
    cudaStream_t st = (cudaStream_t)stream;
    return two_points(C, prm[0], spacing, nx, ny, nz)
               ? launch_fit<2>(rec_xyz, rec_ext, n_rec, C, ox, oy, oz, spacing, nx, ny, nz, P, W, rad_rec, out, st)
               : launch_fit<1>(rec_xyz, rec_ext, n_rec, C, ox, oy, oz, spacing, nx, ny, nz, P, W, rad_rec, out, st);
}

static Cells whole_receptor() {
    Cells C{};
    C.start = nullptr;
    return C;
}

static Cells make_cells(const int* cell_start, const int* cell_dims, const float* cell_origin, float cell_size) {
    Cells C;
    C.start = cell_start;
    C.nx = cell_dims[0]; C.ny = cell_dims[1]; C.nz = cell_dims[2];
    C.ox = cell_origin[0]; C.oy = cell_origin[1]; C.oz = cell_origin[2];
    C.size = cell_size;
    return C;
}

}  // namespace adock

using namespace adock;

extern "C" int adock_grid_vina(const float* rec_xyz, const int* rec_types, int n_rec, const float* radius,
                               const int* hyd, const int* don, const int* acc, int n_xs, const int* lig_types,
                               int n_lt, float ox, float oy, float oz, float spacing, int nx, int ny, int nz,
                               const float* prm, int per_term, float* out, void* stream) {
    return grid_vina_launch(rec_xyz, rec_types, n_rec, whole_receptor(), radius, hyd, don, acc, n_xs, lig_types, n_lt,
                            ox, oy, oz, spacing, nx, ny, nz, prm, per_term, out, stream);
}

extern "C" int adock_grid_vina_cells(const float* rec_xyz, const int* rec_types, int n_rec, const int* cell_start,
                                     const int* cell_dims, const float* cell_origin, float cell_size,
                                     const float* radius, const int* hyd, const int* don, const int* acc, int n_xs,
                                     const int* lig_types, int n_lt, float ox, float oy, float oz, float spacing,
                                     int nx, int ny, int nz, const float* prm, int per_term, float* out, void* stream) {
    ADOCK_CHECK_ARG(cell_start && cell_dims && cell_origin, "null cell-list argument");
    return grid_vina_launch(rec_xyz, rec_types, n_rec, make_cells(cell_start, cell_dims, cell_origin, cell_size),
                            radius, hyd, don, acc, n_xs, lig_types, n_lt, ox, oy, oz, spacing, nx, ny, nz, prm,
                            per_term, out, stream);
}

extern "C" int adock_grid_fit(const float* rec_xyz, const int* rec_ext, int n_rec, const float* rad_rec, int n_rt,
                              const float* rad_lig, int n_lt, const float* W, float ox, float oy, float oz,
                              float spacing, int nx, int ny, int nz, const float* prm, float* out, void* stream) {
    return grid_fit_launch(rec_xyz, rec_ext, n_rec, whole_receptor(), rad_rec, n_rt, rad_lig, n_lt, W, ox, oy, oz,
                           spacing, nx, ny, nz, prm, out, stream);
}

extern "C" int adock_grid_fit_cells(const float* rec_xyz, const int* rec_ext, int n_rec, const int* cell_start,
                                    const int* cell_dims, const float* cell_origin, float cell_size,
                                    const float* rad_rec, int n_rt, const float* rad_lig, int n_lt, const float* W,
                                    float ox, float oy, float oz, float spacing, int nx, int ny, int nz,
                                    const float* prm, float* out, void* stream) {
    ADOCK_CHECK_ARG(cell_start && cell_dims && cell_origin, "null cell-list argument");
    return grid_fit_launch(rec_xyz, rec_ext, n_rec, make_cells(cell_start, cell_dims, cell_origin, cell_size), rad_rec,
                           n_rt, rad_lig, n_lt, W, ox, oy, oz, spacing, nx, ny, nz, prm, out, stream);
}

extern "C" int adock_grid_convert(const float* src, void* dst, long long n, int dtype, void* stream) {
    ADOCK_CHECK_ARG(src && dst && n >= 0, "bad argument");
    if (n == 0) return ADOCK_OK;
    const unsigned blocks = (unsigned)std::min<long long>((n + 255) / 256, 148LL * 32);
    if (dtype == ADOCK_GRID_F16)
        convert_kernel<__half><<<blocks, 256, 0, (cudaStream_t)stream>>>(src, (__half*)dst, n);
    else if (dtype == ADOCK_GRID_BF16)
        convert_kernel<__nv_bfloat16><<<blocks, 256, 0, (cudaStream_t)stream>>>(src, (__nv_bfloat16*)dst, n);
    else
        ADOCK_CHECK_ARG(false, "dtype must be ADOCK_GRID_F16 or ADOCK_GRID_BF16");
    ADOCK_CUDA(cudaGetLastError());
    return ADOCK_OK;
}
