// Device code of the search kernels (sm_100a), included by the per-grid-dtype translation units
// (search_f32.cu, search_f16.cu, search_bf16.cu) that instantiate the launchers, and by search.cu.
//
// Execution model: one warp owns one chain (pose). Lanes own heavy atoms a = lane + 32*i (i < APL, AM = 32*APL),
// whose ligand-frame coordinates, grid slot and torsion bitmask are read from the working layout (L1, L2) in each
// evaluation. Per-warp shared memory holds world coordinates, radii, forces, torsion axes, the BFGS inverse Hessian and
// the state vectors.
// The Monte-Carlo kernel is persistent: warps pull chains from a device work counter (longest ligands first),
// so uneven ligands do not leave SMs idle at the tail.
#pragma once
#include "common.cuh"

namespace adock {

#define EPSF 1.1920929e-07f

// Code-size knobs of the MC kernel (instruction-cache footprint vs register allocation across calls).
#ifdef ADOCK_COLD_NOINLINE
#define ADOCK_COLD_ATTR __noinline__
#else
#define ADOCK_COLD_ATTR __forceinline__
#endif
#define PAIR_ROUNDS_MAX 256   // pair schedule: at most 256 rounds of 32 (8,192 pairs) are reordered
// Intra-pair records: a ligand's pairs are scheduled in rounds of 32 slots, one per lane. x: first atom (bits 0-7),
// second atom (8-15), flags (16-17), and how the slots of a round share atoms: the next higher lane with the same first
// atom (18-22; the lane itself if none) and with the same second atom (23-27), and whether the slot is the first with
// its first atom (28) and with its second atom (29). Empty slots are -1. y: how many more slots the round's most
// repeated first atom (bits 0-4) and second atom (5-9) have.
#define PR_NEXT 18    // + 5 * side
#define PR_LEAD 28    // + side

#define EX_TILE 64   // receptor atoms that the exact energy stages at a time (one bit each in a 64-bit mask)

struct SearchParams {
    // B200 working layout
    const float4* atoms;   // [L, AM]
    const uint32_t* masks; // [L, AM]
    const float4* tors;    // [L, KM, 2]
    const int2* pairs;     // [L, P_pad] records (PR_NEXT), scheduled in rounds of 32
    const int4* info;      // [L] na, nt, np, rec_idx
    const float* rg;       // [L]
    int AM, KM, P, P_pad;
    // grids
    const void* flat;
    const long long* offs;
    const long long* dims;
    const float* origin;
    const float* lo;
    const float* hi;
    const int* nmaps;      // [R] maps built per receptor (may be NULL)
    float inv_s, pen;
    // receptor atoms for exact mode
    const float* rxyz;
    const int* rtyp;
    const int* rn;
    int RN;
    PairPrm pp;
    int n_types;
};

// type tables for exact mode, staged in shared memory by every block that may need them
struct TypeTables {
    float radius[64];
    int flags[64];  // bit0 hydrophobic, bit1 donor, bit2 acceptor
};

struct McParams {
    const int* chain_lig;
    const int* chain_id;
    int n_chains;
    const int* nbr;
    const int* nbr_n;
    int nb_max;
    float* cur;
    float* cur_e;
    float* best;
    float* best_e;
    int init_opt, mc_steps, bfgs_iters;
    float temp, amp_pos, amp_rot;
    unsigned long long seed;
    int step_offset;
    int exact;
    const int* order;
    int* queue;
    unsigned long long* evals;
    // learned proposal: moves [N, prop_k, 32] for steps 0..prop_k-1 of this launch (NULL: plain MC only)
    const float* prop;
    int prop_k;
    float prop_frac;                 // fraction of steps that take the learned move (the rest: plain MC)
    unsigned long long* prop_stats;  // [4] proposals made, proposals accepted, plain steps, plain accepted
    // training-data log of accepted improving moves: features [cap, 320] BF16, moves [cap, 32]
    __nv_bfloat16* log_x;
    float* log_y;
    int* log_n;
    int log_cap;
    const int* lig_active;           // [L] or NULL: chains of a ligand with flag 0 are left unchanged
    int prop_tries;                  // learned steps: candidate targets per step (the lowest-energy one is optimised)
    const float* hint;               // [L, PROP_HINT] ligand-best rows for the logged features, or NULL
};

#define PROP_IN 320
#define PROP_HINT 32
#define PROP_MOVE 32
#define PROP_FAIL_MAX 8

__device__ __forceinline__ int hb_pair(int fa, int fb) {
    return (((fa & 2) && (fb & 4)) || ((fa & 4) && (fb & 2))) ? PF_HB : 0;
}
__device__ __forceinline__ int hyd_pair(int fa, int fb) { return ((fa & 1) && (fb & 1)) ? PF_HYD : 0; }

__device__ __forceinline__ void stage_tables(TypeTables& dst, const TypeTables& src) {
    for (int i = threadIdx.x; i < 64; i += blockDim.x) {
        dst.radius[i] = src.radius[i];
        dst.flags[i] = src.flags[i];
    }
    __syncthreads();
}

// ------------------------------------------------------------------------------------------ per-warp workspace
// Float offsets of the per-warp shared workspace for a given AM / KM (float4 arrays first).
struct WSLayout {
    int X, FT, RT, V, ap, au, tp, tu, ax, cs, sn, H, x, xn, xo, cur, best, g, gn, go, total;
    __host__ __device__ WSLayout(int AM, int KM, bool exact) {
        const int DM = 6 + KM, SD = 7 + KM;
        int o = 0;
        X = o; o += 4 * AM;    // world coordinates and radii, [4][AM] (x, y, z, radius arrays)
        FT = o; o += 8 * AM;   // forces [3][AM] (and the exact energy [AM]); then float4 (force, torsion bitmask) and
                               // float4 (torque, 0) per atom
        RT = o; o += exact ? 4 * EX_TILE : 0;   // a tile of receptor atoms, float4 (xyz, type | flags << 8)
        V = o; o += 4 * DM;    // BFGS vectors, float4 (p, -H y, y, g) per component
        ap = o; o += 4 * KM;
        au = o; o += 4 * KM;
        tp = o; o += 4 * KM;
        tu = o; o += 4 * KM;
        ax = o; o += KM;      // packed axis atom indices (a0 | a1 << 16)
        cs = o; o += KM;
        sn = o; o += KM;
        H = o; o += DM * DM;
        x = o; o += SD;
        xn = o; o += SD;
        xo = o; o += SD;
        cur = o; o += SD;
        best = o; o += SD;
        g = o; o += DM;
        gn = o; o += DM;
        go = o; o += DM;
        total = (o + 3) & ~3;  // keep 16-byte alignment of the next warp
    }
};

// Per-chain context (registers).
template <int APL>
struct Chain {
    int na, nt, nrounds;
    float rg;
    const int2* pairs;
    const char* grid;
    long long n3;
    int ny, nz;
    float o[3], lo[3], hi[3], fmx[3];
    const float* rx;
    const int* rt;
    int rn;
    const int* nb;
    int nbn;
    const float4* atoms;     // this ligand's rows of the working layout
    const uint32_t* masks;
};

template <int APL, typename GT>
__device__ __forceinline__ void load_chain(Chain<APL>& c, const SearchParams& P, const TypeTables& tt, int l, float* ws,
                                           const WSLayout& L, int lane, const int* nb, int nbn) {
    const int4 inf = P.info[l];
    c.na = inf.x; c.nt = inf.y;
    c.nrounds = (inf.z + 31) >> 5;
    const int ri = inf.w;
    c.rg = P.rg[l];
    c.pairs = P.pairs + (long long)l * P.P_pad;
    const long long nx = P.dims[3 * ri], ny = P.dims[3 * ri + 1], nz = P.dims[3 * ri + 2];
    c.n3 = nx * ny * nz;
    c.ny = (int)ny; c.nz = (int)nz;
    c.grid = (const char*)((const GT*)P.flat + P.offs[ri]);
    for (int d = 0; d < 3; ++d) {
        c.o[d] = P.origin[3 * ri + d]; c.lo[d] = P.lo[3 * ri + d]; c.hi[d] = P.hi[3 * ri + d];
    }
    c.fmx[0] = (float)(nx - 1) - 1e-4f; c.fmx[1] = (float)(ny - 1) - 1e-4f; c.fmx[2] = (float)(nz - 1) - 1e-4f;
    c.rx = P.rxyz ? P.rxyz + (long long)ri * P.RN * 3 : nullptr;
    c.rt = P.rtyp ? P.rtyp + (long long)ri * P.RN : nullptr;
    c.rn = P.rn ? P.rn[ri] : 0;
    c.nb = nb; c.nbn = nbn;
    c.atoms = P.atoms + (long long)l * P.AM;
    c.masks = P.masks + (long long)l * P.AM;
#pragma unroll 1
    for (int a = lane; a < 32 * APL; a += 32) {
        const int typ = __float_as_int(c.atoms[a].w) >> 16;
        ws[L.X + 3 * 32 * APL + a] = tt.radius[typ < 0 ? 0 : typ & 63];
    }
    const float4* tr = P.tors + (long long)l * P.KM * 2;
    float4* ap = (float4*)(ws + L.ap);
    float4* au = (float4*)(ws + L.au);
    int* axs = (int*)(ws + L.ax);
    for (int k = lane; k < P.KM; k += 32) {
        const float4 p = tr[2 * k], u = tr[2 * k + 1];
        ap[k] = p;
        au[k] = u;
        axs[k] = (__float_as_int(p.w) & 0xffff) | (__float_as_int(u.w) << 16);
    }
    __syncwarp();
}

// trilinear lookup + analytic gradient of one atom (mckernel.py:140-149, :176-195)
template <typename GT>
__device__ __forceinline__ float trilinear(const GT* G, int ny, int nz, const float* o, const float* fmx, float inv_s,
                                           float X0, float X1, float X2, float& gx, float& gy, float& gz) {
    const float xx[3] = {X0, X1, X2};
    float fw[3], inside[3];
    int i0[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float f = (xx[d] - o[d]) * inv_s;
        const float fc = fminf(fmaxf(f, 0.f), fmx[d]);
        inside[d] = (f > 0.f && f < fmx[d]) ? 1.f : 0.f;
        const int ii = (int)floorf(fc);
        i0[d] = ii;
        fw[d] = fc - ii;
    }
    const long long b000 = ((long long)i0[0] * ny + i0[1]) * nz + i0[2];
    const long long sx = (long long)ny * nz;
    const float v000 = gload(G + b000), v001 = gload(G + b000 + 1), v010 = gload(G + b000 + nz),
                v011 = gload(G + b000 + nz + 1);
    const float v100 = gload(G + b000 + sx), v101 = gload(G + b000 + sx + 1), v110 = gload(G + b000 + sx + nz),
                v111 = gload(G + b000 + sx + nz + 1);
    const float wx = fw[0], wy = fw[1], wz = fw[2];
    const float c00 = v000 * (1 - wz) + v001 * wz, c01 = v010 * (1 - wz) + v011 * wz;
    const float c10 = v100 * (1 - wz) + v101 * wz, c11 = v110 * (1 - wz) + v111 * wz;
    const float c0 = c00 * (1 - wy) + c01 * wy, c1 = c10 * (1 - wy) + c11 * wy;
    const float e = c0 * (1 - wx) + c1 * wx;
    gx = (c1 - c0) * inv_s * inside[0];
    gy = ((c01 - c00) * (1 - wx) + (c11 - c10) * wx) * inv_s * inside[1];
    gz = (((v001 - v000) * (1 - wy) + (v011 - v010) * wy) * (1 - wx) +
          ((v101 - v100) * (1 - wy) + (v111 - v110) * wy) * wx) * inv_s * inside[2];
    return e;
}

// Intra-ligand pair term of one scheduled slot: energy and the force on the first atom, 0 for an empty slot and beyond
// the cutoff. Positions and radii are four arrays of AM floats, so that 32 lanes touching 32 different atoms hit 32
// different shared-memory banks (a float4 per atom would put the x components of 32 atoms on 8 banks). Branch-free, so
// that the slots a lane has in flight overlap.
template <int AM, bool GRAD>
__device__ __forceinline__ float pair_slot(int w, bool valid, const float* X, const PairPrm& pp, float3& f) {
    const float *Xi = X + (w & 0xff), *Xj = X + ((w >> 8) & 0xff);
    const float rx = Xi[0] - Xj[0], ry = Xi[AM] - Xj[AM], rz = Xi[2 * AM] - Xj[2 * AM];
    // r and 1/r from one reciprocal square root; clamping r^2 at 1e-12 is the reference's max(r, 1e-6)
    const float r2 = rx * rx + ry * ry + rz * rz;
    const float rinv = rsqrt_ftz(fmaxf(r2, 1e-12f));
    const float r = r2 * rinv;
    const bool on = valid && !(r >= pp.cutoff);
    float de;
    const float e = pair_energy(r, Xi[3 * AM] + Xj[3 * AM], w >> 16, pp, de);
    if (GRAD) {
        const float sc = on ? de * rinv : 0.f;
        f.x = __fmul_rn(sc, rx); f.y = __fmul_rn(sc, ry); f.z = __fmul_rn(sc, rz);
    }
    return on ? e : 0.f;
}

// Adds one side of a round's pair forces to the forces F [3][AM]. Lanes that share an atom on the side form a chain in
// lane order (see PR_NEXT); its first lane adds the members' forces, fetched by shuffles, and alone updates the entry.
// Shared float atomics give the same sums (lanes that meet on an atom add in lane order) but serialise there.
template <int AM, int SIDE>
__device__ __forceinline__ void push_forces(int w, int repeats, float3 f, float* F) {
    const int next = (w >> (PR_NEXT + 5 * SIDE)) & 31;
    float* Fa = F + ((w >> (8 * SIDE)) & 0xff);
    float sx, sy, sz;
    if (SIDE) {
        sx = __fsub_rn(Fa[0], f.x); sy = __fsub_rn(Fa[AM], f.y); sz = __fsub_rn(Fa[2 * AM], f.z);
    } else {
        sx = __fadd_rn(Fa[0], f.x); sy = __fadd_rn(Fa[AM], f.y); sz = __fadd_rn(Fa[2 * AM], f.z);
    }
    int src = next;
    bool ok = src != (threadIdx.x & 31);
#pragma unroll 1
    for (int k = repeats; k > 0; --k) {
        const float vx = __shfl_sync(0xffffffffu, f.x, src), vy = __shfl_sync(0xffffffffu, f.y, src),
                    vz = __shfl_sync(0xffffffffu, f.z, src);
        const int n = __shfl_sync(0xffffffffu, next, src);
        if (ok) {
            sx = SIDE ? __fsub_rn(sx, vx) : __fadd_rn(sx, vx);
            sy = SIDE ? __fsub_rn(sy, vy) : __fadd_rn(sy, vy);
            sz = SIDE ? __fsub_rn(sz, vz) : __fadd_rn(sz, vz);
        }
        ok = ok && n != src;
        src = n;
    }
    if ((w >> (PR_LEAD + SIDE)) & 1) {
        Fa[0] = sx;
        Fa[AM] = sy;
        Fa[2 * AM] = sz;
    }
    __syncwarp();
}

// Intra-ligand pairs: adds the lane's slots to its share e of the energy (returned) and, with GRAD, the forces to the
// atoms' entries of [3][AM] in shared memory. An atom's contributions are added in the order round, first atoms before second atoms, lane.
// Bound by instruction issue and the latency of the rounds' shared-memory updates (about 95 instructions per slot for
// the pair term, 66 per round for the two sides). With shared float atomics for the forces and the pair parameters read
// through a generic pointer this loop took 10.3 k of a single warp's 19 k cycles per evaluation (24 atoms, 7 rounds);
// now 2.9 k (averaged over evaluations with and without the gradient). Summing in registers instead was slower: owners pulling by shuffles (132 instructions per round), or
// per-atom slot lists over forces left in shared memory (12 wavefronts per entry from bank conflicts).
template <int APL, bool GRAD>
__device__ __forceinline__ float pair_terms(float* ws, const WSLayout& L, const Chain<APL>& c, const PairPrm& pp, float e,
                                            int lane) {
    constexpr int AM = 32 * APL;
    const float* X = ws + L.X;
    float* FF = ws + L.FT;
    // two rounds in flight; the next two rounds' records are loaded while these are evaluated
    const int empty = lane * (33 << PR_NEXT);   // atom 0 twice, linked to itself, first of nothing
    const int2 none = make_int2(-1, 0);
    int2 pa = c.nrounds > 0 ? c.pairs[lane] : none;
    int2 pb = c.nrounds > 1 ? c.pairs[32 + lane] : none;
#pragma unroll 1
    for (int r = 0; r < c.nrounds; r += 2) {
        const int2 qa = (r + 2 < c.nrounds) ? c.pairs[(r + 2) * 32 + lane] : none;
        const int2 qb = (r + 3 < c.nrounds) ? c.pairs[(r + 3) * 32 + lane] : none;
        const int wa = pa.x < 0 ? empty : pa.x, wb = pb.x < 0 ? empty : pb.x;
        float3 fa, fb;
        e += pair_slot<AM, GRAD>(wa, pa.x >= 0, X, pp, fa);
        e += pair_slot<AM, GRAD>(wb, pb.x >= 0, X, pp, fb);
        if (GRAD) {
            push_forces<AM, 0>(wa, pa.y & 31, fa, FF);
            push_forces<AM, 1>(wa, pa.y >> 5, fa, FF);
            if (r + 1 < c.nrounds) {
                push_forces<AM, 0>(wb, pb.y & 31, fb, FF);
                push_forces<AM, 1>(wb, pb.y >> 5, fb, FF);
            }
        }
        pa = qa;
        pb = qb;
    }
    return e;
}

// Exact inter energy of the lane's atoms (positions in shared memory) with the receptor atoms, or the chain's
// neighbour list, into inter [AM], and the forces, into [3][AM], summed in list order. A tile of receptor atoms is staged in shared
// memory; each lane first collects the tile's atoms inside the cutoff of its atom as a bit mask (a few instructions per
// pair, no branches), then evaluates the pair terms of its set bits, two in flight, so that the terms run with most
// lanes busy: some 50 of a pose's 300 neighbours are inside the 8 A cutoff of one atom. Bound by instruction issue.
// Walking the list with dependent loads and evaluating the terms wherever any lane's pair was inside took 190 k cycles
// per evaluation (300 neighbours, 14 warps per SM), this about 31 k.
template <int APL>
__device__ __forceinline__ void exact_terms(float* ws, const WSLayout& L, const Chain<APL>& c, const SearchParams& P,
                                            const TypeTables& tt, int lane) {
    constexpr int AM = 32 * APL;
    const float* X = ws + L.X;
    float4* RT = (float4*)(ws + L.RT);
    const float cut2 = P.pp.cutoff * P.pp.cutoff;
    const int n = c.nb ? c.nbn : c.rn;
    auto fetch = [&](int k) {
        if (k >= n) return make_float4(0.f, 0.f, 0.f, 0.f);
        const int b = c.nb ? c.nb[k] : k;
        const int tb = c.rt[b] & 63;   // index kept inside the 64-entry type tables
        return make_float4(c.rx[3 * b], c.rx[3 * b + 1], c.rx[3 * b + 2], __int_as_float(tb | (tt.flags[tb] << 8)));
    };
    float* FF = ws + L.FT;
    float* inter = FF + 3 * AM;
#pragma unroll
    for (int i = 0; i < 4 * APL; ++i) FF[lane + 32 * i] = 0.f;
    float4 n0 = fetch(lane), n1 = fetch(32 + lane);
#pragma unroll 1
    for (int t0 = 0; t0 < n; t0 += EX_TILE) {
        __syncwarp();
        RT[lane] = n0;
        RT[32 + lane] = n1;
        __syncwarp();
        n0 = fetch(t0 + EX_TILE + lane);
        n1 = fetch(t0 + EX_TILE + 32 + lane);
        const unsigned long long valid = n - t0 >= 64 ? ~0ull : (1ull << (n - t0)) - 1ull;
#pragma unroll 1
        for (int a = lane; a - lane < c.na; a += 32) {
            const float X0 = X[a], X1 = X[AM + a], X2 = X[2 * AM + a];
            unsigned m0 = 0, m1 = 0;
#pragma unroll 8
            for (int b = 0; b < 32; ++b) {
                const float4 B = RT[b], C = RT[32 + b];
                float rx = X0 - B.x, ry = X1 - B.y, rz = X2 - B.z;
                float r2 = rx * rx + ry * ry + rz * rz;
                m0 |= (r2 >= cut2 ? 0u : 1u) << b;
                rx = X0 - C.x; ry = X1 - C.y; rz = X2 - C.z;
                r2 = rx * rx + ry * ry + rz * rz;
                m1 |= (r2 >= cut2 ? 0u : 1u) << b;
            }
            unsigned long long m = a < c.na ? (((unsigned long long)m1 << 32) | m0) & valid : 0ull;
            const int ta = (__float_as_int(c.atoms[a].w) >> 16) & 63;
            const float ra = tt.radius[ta];
            const int fa = tt.flags[ta];
            float ea = inter[a];
            float3 f = make_float3(FF[a], FF[AM + a], FF[2 * AM + a]);
            const int most = __reduce_max_sync(0xffffffffu, __popcll(m));
#pragma unroll 1
            for (int t = 0; t < most; t += 2) {
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const bool on = m != 0ull;
                    const float4 B = RT[on ? __ffsll((long long)m) - 1 : 0];
                    m &= m - 1ull;
                    const float rx = X0 - B.x, ry = X1 - B.y, rz = X2 - B.z;
                    const float r2 = rx * rx + ry * ry + rz * rz;
                    const int tb = __float_as_int(B.w) & 63, fb = __float_as_int(B.w) >> 8;
                    const float rinv = rsqrt_ftz(fmaxf(r2, 1e-12f));
                    const float r = r2 * rinv;
                    float de;
                    const float ep = pair_energy(r, ra + tt.radius[tb], hyd_pair(fa, fb) | hb_pair(fa, fb), P.pp, de);
                    if (on) {
                        ea += ep;
                        const float sc = de * rinv;
                        f.x += sc * rx; f.y += sc * ry; f.z += sc * rz;
                    }
                }
            }
            inter[a] = ea;
            FF[a] = f.x; FF[AM + a] = f.y; FF[2 * AM + a] = f.z;
        }
    }
}

// Energy + analytic pose gradient of state s (shared, SD floats) into g (shared, DM floats); E on all lanes.
// Same energy as mckernel.py:108-244: torsions applied leaf -> root on reference coordinates, rotation,
// translation; trilinear grid (or exact pairwise) inter energy with the quadratic out-of-box penalty; intra
// pairs. Gradient: dE/dt = sum F, torque = sum (X - t) x F, dE/dtheta_k = u_k . sum_{a moved by k} (X_a - p_k) x F_a,
// evaluated as u_k . (sum X' x F - p'_k x sum F) over the subtree of k (X' = X - t).
// EX selects the inter energy at compile time: exact pairwise over receptor atoms (or the chain's neighbour list),
// else the trilinear grid, so the grid-mode kernels carry no receptor loop. Without `grad` only the energy is
// evaluated (the same value) and g is left alone: a rejected line-search point needs no gradient.
template <int APL, typename GT, bool EX>
__device__ __forceinline__ float eval_eg(float* ws, const WSLayout& L, const float* s, float* g, const Chain<APL>& c,
                         const SearchParams& P, const TypeTables& tt, int lane, bool grad) {
    constexpr int AM = 32 * APL;
    float* X = ws + L.X;     // [3][AM] world coordinates (radii behind them)
    const float4* ap = (const float4*)(ws + L.ap);
    const float4* au = (const float4*)(ws + L.au);
    float4* tp = (float4*)(ws + L.tp);
    float4* tu = (float4*)(ws + L.tu);
    const int* axs = (const int*)(ws + L.ax);
    float* cs = ws + L.cs;
    float* sn = ws + L.sn;

    const float t0 = s[0], t1 = s[1], t2 = s[2];
    float qw = s[3], qx = s[4], qy = s[5], qz = s[6];
    const float nq = rsqrtf(qw * qw + qx * qx + qy * qy + qz * qz);
    qw *= nq; qx *= nq; qy *= nq; qz *= nq;
    const float R00 = 1 - 2 * (qy * qy + qz * qz), R01 = 2 * (qx * qy - qz * qw), R02 = 2 * (qx * qz + qy * qw);
    const float R10 = 2 * (qx * qy + qz * qw), R11 = 1 - 2 * (qx * qx + qz * qz), R12 = 2 * (qy * qz - qx * qw);
    const float R20 = 2 * (qx * qz - qy * qw), R21 = 2 * (qy * qz + qx * qw), R22 = 1 - 2 * (qx * qx + qy * qy);
#pragma unroll 1
    for (int k = lane; k < c.nt; k += 32) {
        float sv, cv;
        __sincosf(s[7 + k], &sv, &cv);
        cs[k] = cv;
        sn[k] = sv;
    }
    __syncwarp();
    float e = 0.f;
    float* FF = ws + L.FT;   // forces dE/dX, [3][AM]
    const GT* grid = (const GT*)c.grid;
    // The lane's atoms; rolled, and the ligand rows read again each time: the loop saves code, and instruction-cache misses
    // were the kernel's largest stall (1.95 of 6.9 cycles per issue). With the other rolled loops and the one line-search
    // step: 256 ligands x 32 chains, start + 8 steps 17.6 -> 14.0 ms.
    auto place = [&](int a, float4 v) {
        float px = v.x, py = v.y, pz = v.z;
        uint32_t m = c.masks[a];
        while (m) {
            const int k = __ffs(m) - 1;
            m &= m - 1;
            const float4 A = ap[k], U = au[k];
            const float cv = cs[k], sv = sn[k];
            const float vx = px - A.x, vy = py - A.y, vz = pz - A.z;
            const float d = U.x * vx + U.y * vy + U.z * vz;
            const float cx = U.y * vz - U.z * vy, cy = U.z * vx - U.x * vz, cz = U.x * vy - U.y * vx;
            px = A.x + vx * cv + cx * sv + U.x * d * (1 - cv);
            py = A.y + vy * cv + cy * sv + U.y * d * (1 - cv);
            pz = A.z + vz * cv + cz * sv + U.z * d * (1 - cv);
        }
        // spelled out: poses round the same whatever code surrounds them
        X[a] = __fmaf_rn(R02, pz, __fmaf_rn(R00, px, __fmul_rn(R01, py))) + t0;
        X[AM + a] = __fmaf_rn(R12, pz, __fmaf_rn(R10, px, __fmul_rn(R11, py))) + t1;
        X[2 * AM + a] = __fmaf_rn(R22, pz, __fmaf_rn(R20, px, __fmul_rn(R21, py))) + t2;
    };
    if constexpr (EX) {
#pragma unroll 1
        for (int a = lane; a < c.na; a += 32) place(a, c.atoms[a]);
        __syncwarp();
        exact_terms<APL>(ws, L, c, P, tt, lane);
    }
#pragma unroll 1
    for (int a = lane; a < c.na; a += 32) {
        float ea, gg[3];
        if constexpr (EX) {
            ea = FF[3 * AM + a];
            gg[0] = FF[a]; gg[1] = FF[AM + a]; gg[2] = FF[2 * AM + a];
        } else {
            const float4 v = c.atoms[a];
            place(a, v);
            ea = trilinear<GT>(grid + (long long)(__float_as_int(v.w) & 0xffff) * c.n3, c.ny, c.nz, c.o, c.fmx, P.inv_s, X[a],
                               X[AM + a], X[2 * AM + a], gg[0], gg[1], gg[2]);
        }
        const float xx[3] = {X[a], X[AM + a], X[2 * AM + a]};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float lo = fmaxf(c.lo[d] - xx[d], 0.f), hi = fmaxf(xx[d] - c.hi[d], 0.f);
            ea += P.pen * (lo * lo + hi * hi);
            gg[d] += P.pen * (-2.f * lo + 2.f * hi);
        }
        e += ea;
        FF[a] = gg[0];
        FF[AM + a] = gg[1];
        FF[2 * AM + a] = gg[2];
    }
    __syncwarp();
    if (!grad) {
        e = warp_sum(pair_terms<APL, false>(ws, L, c, P.pp, e, lane));
        __syncwarp();
        return e;
    }
    e = pair_terms<APL, true>(ws, L, c, P.pp, e, lane);
    // world torsion axes (axis atoms' current positions)
#pragma unroll 1
    for (int k = lane; k < c.nt; k += 32) {
        const int a0 = axs[k] & 0xffff, a1 = axs[k] >> 16;
        const float Ax = X[a0], Ay = X[AM + a0], Az = X[2 * AM + a0];
        const float ux = X[a1] - Ax, uy = X[AM + a1] - Ay, uz = X[2 * AM + a1] - Az;
        const float nn = rsqrtf(fmaxf(ux * ux + uy * uy + uz * uz, 1e-12f));
        tp[k] = make_float4(Ax - t0, Ay - t1, Az - t2, 0.f);
        tu[k] = make_float4(ux * nn, uy * nn, uz * nn, 0.f);
    }
    // each atom's force with its torsion bitmask, and its torque (X - t) x F (in place of the forces)
    float4* FA = (float4*)(ws + L.FT);
    float4* TA = FA + AM;
    float3 F[APL];
#pragma unroll
    for (int i = 0; i < APL; ++i) {
        const int a = lane + 32 * i;
        F[i] = make_float3(FF[a], FF[AM + a], FF[2 * AM + a]);
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < APL; ++i) {
        const int a = lane + 32 * i;
        if (a < c.na) {
            const float Fx = F[i].x, Fy = F[i].y, Fz = F[i].z;
            const float dx = X[a] - t0, dy = X[AM + a] - t1, dz = X[2 * AM + a] - t2;
            FA[a] = make_float4(Fx, Fy, Fz, __uint_as_float(c.masks[a]));
            TA[a] = make_float4(dy * Fz - dz * Fy, dz * Fx - dx * Fz, dx * Fy - dy * Fx, 0.f);
        }
    }
    __syncwarp();
    // subtree sums of F and (X - t) x F: sum k < nt is torsion k's subtree, sum k == nt is the whole ligand.
    // The nt + 1 sums are spread over all 32 lanes: G lanes per atom chunk (G = next power of two >= nt + 1),
    // 32 / G chunks, combined by shuffles.
    if (c.nt < 32) {
        const int G = c.nt < 1 ? 1 : (c.nt < 3 ? 4 : (c.nt < 7 ? 8 : (c.nt < 15 ? 16 : 32)));
        const int k = lane & (G - 1), chunk = lane / G, C = 32 / G;
        float S0 = 0.f, S1 = 0.f, S2 = 0.f, T0 = 0.f, T1 = 0.f, T2 = 0.f;
        const uint32_t bit = k < c.nt ? 1u << k : 0u;
        const bool all = k == c.nt;
#pragma unroll 4
        for (int a = chunk; a < c.na; a += C) {
            const float4 f = FA[a], t = TA[a];
            if (all || (__float_as_uint(f.w) & bit)) {
                S0 += f.x; S1 += f.y; S2 += f.z;
                T0 += t.x; T1 += t.y; T2 += t.z;
            }
        }
        for (int o = G; o < 32; o <<= 1) {
            S0 += __shfl_xor_sync(0xffffffffu, S0, o); S1 += __shfl_xor_sync(0xffffffffu, S1, o);
            S2 += __shfl_xor_sync(0xffffffffu, S2, o); T0 += __shfl_xor_sync(0xffffffffu, T0, o);
            T1 += __shfl_xor_sync(0xffffffffu, T1, o); T2 += __shfl_xor_sync(0xffffffffu, T2, o);
        }
        if (chunk == 0 && k <= c.nt) {
            if (k == c.nt) {
                g[0] = S0; g[1] = S1; g[2] = S2; g[3] = T0; g[4] = T1; g[5] = T2;
            } else {
                const float4 Pk = tp[k], Uk = tu[k];
                const float cx = T0 - (Pk.y * S2 - Pk.z * S1);
                const float cy = T1 - (Pk.z * S0 - Pk.x * S2);
                const float cz = T2 - (Pk.x * S1 - Pk.y * S0);
                g[6 + k] = cx * Uk.x + cy * Uk.y + cz * Uk.z;
            }
        }
    } else {
#pragma unroll 1
        for (int k = lane; k <= c.nt; k += 32) {
            float S0 = 0.f, S1 = 0.f, S2 = 0.f, T0 = 0.f, T1 = 0.f, T2 = 0.f;
            const bool all = (k == c.nt);
            const uint32_t bit = all ? 0u : (1u << k);
            for (int a = 0; a < c.na; ++a) {
                const float4 f = FA[a], t = TA[a];
                if (all || (__float_as_uint(f.w) & bit)) {
                    S0 += f.x; S1 += f.y; S2 += f.z;
                    T0 += t.x; T1 += t.y; T2 += t.z;
                }
            }
            if (all) {
                g[0] = S0; g[1] = S1; g[2] = S2; g[3] = T0; g[4] = T1; g[5] = T2;
            } else {
                const float4 Pk = tp[k], Uk = tu[k];
                g[6 + k] = (T0 - (Pk.y * S2 - Pk.z * S1)) * Uk.x + (T1 - (Pk.z * S0 - Pk.x * S2)) * Uk.y +
                           (T2 - (Pk.x * S1 - Pk.y * S0)) * Uk.z;
            }
        }
    }
    e = warp_sum(e);
    __syncwarp();
    return e;
}

__device__ __forceinline__ void wcopy(float* dst, const float* src, int D, int lane) {
#pragma unroll 1
    for (int i = lane; i < D; i += 32) dst[i] = src[i];
    __syncwarp();
}
// xn = x (+) alpha p (p = V[].x): translation add, rotation-vector increment of the quaternion, torsion add (mckernel.py:256-265)
__device__ __forceinline__ void conf_step(float* xn, const float* x, const float4* V, float alpha, int nt, int lane) {
    if (lane == 0) {
        xn[0] = x[0] + alpha * V[0].x; xn[1] = x[1] + alpha * V[1].x; xn[2] = x[2] + alpha * V[2].x;
        xn[3] = x[3]; xn[4] = x[4]; xn[5] = x[5]; xn[6] = x[6];
        quat_apply_rotvec(xn + 3, alpha * V[3].x, alpha * V[4].x, alpha * V[5].x);
    }
#pragma unroll 1
    for (int k = lane; k < nt; k += 32) xn[7 + k] = x[7 + k] + alpha * V[6 + k].x;
    __syncwarp();
}
// -sum_j H_ij v_j of component i (component `v` of the vectors V); H symmetric, stored with lane i owning column i
// (conflict-free); two accumulators
template <int v>
__device__ __forceinline__ float neg_hv(const float* H, const float4* V, int i, int D) {
    float a0 = 0.f, a1 = 0.f;
    int j = 0;
#pragma unroll 2
    for (; j + 1 < D; j += 2) {
        a0 += H[j * D + i] * (v == 2 ? V[j].z : V[j].w);
        a1 += H[(j + 1) * D + i] * (v == 2 ? V[j + 1].z : V[j + 1].w);
    }
    if (j < D) a0 += H[j * D + i] * (v == 2 ? V[j].z : V[j].w);
    return -(a0 + a1);
}

// Vina-1.2-style BFGS on state x (shared, in/out); returns the final energy (mckernel.py:267-326).
// The curvature scalar y.p and the update guard alpha * y.p >= eps are evaluated in float64.
// Inlined at the MC kernel's one call site, with one inlined eval_eg: one copy keeps the kernel small enough for the
// instruction cache, and the pair parameters stay constant-bank operands. (As a function of its own it read them
// through a generic pointer, again after every shared-memory store of the pair loop.)
template <int APL, typename GT, bool EX>
__device__ __forceinline__ float bfgs(float* ws, const WSLayout& L, float* x, int iters, const Chain<APL>& c,
                                      const SearchParams& P, const TypeTables& tt, int lane, unsigned& n_eval) {
    const int D = 6 + c.nt, S = 7 + c.nt;
    float* H = ws + L.H;
    float* g = ws + L.g;
    float* gn = ws + L.gn;
    float* go = ws + L.go;
    float4* V = (float4*)(ws + L.V);
    float* xn = ws + L.xn;
    float* xo = ws + L.xo;
    // One evaluation per pass of this loop: the start point on the first pass, then the line-search trial points.
    // Keeping a single call site keeps a single inlined copy of eval_eg in the kernel. About 70 % of the first trials
    // are accepted, but only a third of the later ones: those are evaluated without the gradient first, and once more
    // with it (`again`, the same energy) when they are accepted. The 10th point is taken in any case.
    float f0 = 0.f, f_orig = 0.f, pg = 0.f, alpha = 1.f;
    int step = 0, trial = 0;
    bool first = true, again = false;
    while (true) {
        if (!first && !again) conf_step(xn, x, V, alpha, c.nt, lane);
        const bool grad = first || again || trial == 0 || trial == 9;
        const float f = eval_eg<APL, GT, EX>(ws, L, first ? x : xn, first ? g : gn, c, P, tt, lane, grad);
        if (!again) ++n_eval;
        if (first) {
            first = false;
            f0 = f_orig = f;
            wcopy(xo, x, S, lane);
            float s = 0.f;
#pragma unroll 1
            for (int i = lane; i < D; i += 32) {
                go[i] = g[i];
                float a0 = 0.f, a1 = 0.f;   // p = -H g with H the identity
#pragma unroll 1
                for (int j = 0; j < D; j += 2) {
                    a0 += (i == j ? 1.f : 0.f) * g[j];
                    if (j + 1 < D) a1 += (i == j + 1 ? 1.f : 0.f) * g[j + 1];
                }
                const float pi = -(a0 + a1);
                V[i].x = pi;
                s += pi * g[i];
            }
            __syncwarp();
            if (iters <= 0) break;
            pg = warp_sum(s);
            continue;
        }
        // Armijo test (c = 1e-4); up to 10 trials halving alpha. After a 10th failed trial the last point is taken
        // with alpha already halved, as in the reference's loop.
        bool stuck = false;
        if (!again) {
            if (!(f - f0 < 1e-4f * alpha * pg)) {
                alpha *= 0.5f;
                if (++trial < 10) continue;
                stuck = true;
#pragma unroll 1
                for (int i = lane; i < S; i += 32) stuck = stuck && __float_as_int(x[i]) == __float_as_int(xn[i]);
                stuck = __all_sync(0xffffffffu, stuck);
            } else if (!grad) {
                again = true;
                continue;
            }
        }
        again = false;
        // The 10th point is the iteration's own start: its gradient step is 0, H stays, and every further iteration
        // would repeat this one.
        if (stuck) break;
        f0 = f;
#pragma unroll 1
        for (int i = lane; i < S; i += 32) x[i] = xn[i];
        float gg = 0.f, yy = 0.f;
        double yp = 0.0;
#pragma unroll 1
        for (int i = lane; i < D; i += 32) {
            const float gi = gn[i], yi = gi - g[i];
            gg += gi * gi;
            yy += yi * yi;
            yp += (double)yi * (double)V[i].x;
            g[i] = gi;
            V[i].z = yi;
            V[i].w = gi;
        }
        __syncwarp();
        gg = warp_sum(gg);
        yy = warp_sum(yy);
        yp = warp_sum_d(yp);
        if (!(sqrtf(gg) >= 1e-5f)) break;
        if (step == 0) {   // H: the identity, rescaled from the first step's curvature
            const float dg = fabsf(yy) > EPSF ? (float)((double)alpha * yp / (double)yy) : 1.f;
#pragma unroll 1
            for (int i = lane; i < D; i += 32)
#pragma unroll 2
                for (int j = 0; j < D; ++j) H[j * D + i] = (i == j) ? dg : 0.f;
            __syncwarp();
        }
        const double ayp = (double)alpha * yp;
        float s = 0.f;
        if (ayp >= (double)EPSF) {
#pragma unroll 1
            for (int i = lane; i < D; i += 32) {
                const float mi = neg_hv<2>(H, V, i, D);
                V[i].y = mi;
                s += V[i].z * mi;
            }
            __syncwarp();
            const float yhy = -warp_sum(s);
            const float r = (float)(1.0 / ayp);
            const float c2 = alpha * alpha * (r * r * yhy + r);
            const float ar = alpha * r;
            // the update and the new direction -H g in one sweep over H
            s = 0.f;
            float pn[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = lane + 32 * h;
                pn[h] = 0.f;
                if (i < D) {
                    const float mi = V[i].y, pi = V[i].x;
                    float a0 = 0.f, a1 = 0.f;
#pragma unroll 2
                    for (int j = 0; j < D; ++j) {
                        const float4 v = V[j];
                        float hij = H[j * D + i];
                        hij += ar * (mi * v.x + v.y * pi) + c2 * pi * v.x;
                        H[j * D + i] = hij;
                        if (j & 1) a1 += hij * v.w; else a0 += hij * v.w;
                    }
                    pn[h] = -(a0 + a1);
                    s += pn[h] * V[i].w;
                }
            }
            __syncwarp();
            if (lane < D) V[lane].x = pn[0];
            if (lane + 32 < D) V[lane + 32].x = pn[1];
        } else {
#pragma unroll 1
            for (int i = lane; i < D; i += 32) {
                const float pi = neg_hv<3>(H, V, i, D);
                s += pi * V[i].w;
                V[i].x = pi;
            }
        }
        __syncwarp();
        if (++step >= iters) break;
        pg = warp_sum(s);
        alpha = 1.f;
        trial = 0;
    }
    if (!(f0 <= f_orig)) {
        f0 = f_orig;
        wcopy(x, xo, S, lane);
        wcopy(g, go, D, lane);
    }
    return f0;
}

// ------------------------------------------------------------------------------------------ proposal features
// sign(v) log(1 + |v|): energies and map values of any magnitude in a range the network handles
__device__ __forceinline__ float slog(float v) { return copysignf(log1pf(fabsf(v)), v); }

// Feature row (PROP_IN = 320 values, BF16) of state s (energy e) of ligand l, computed by one warp:
//   [0, 216)   27 samples x 8 maps: nearest-grid map values at the centroid + {-2, 0, 2} A per axis, as
//              sign(v) log(1 + |v|) (maps beyond the receptor's count are 0)
//   [216, 219) translation relative to the box centre / 10 A
//   [219, 223) orientation quaternion, sign chosen so that w >= 0
//   [223, 263) sin, cos of torsions 0..19 (0 beyond the ligand's torsion count)
//   [263, 275) heavy atoms / 64, torsions / 20, radius of gyration / 10, intra pairs / 2000, fraction of atoms
//              per map slot 0..7
//   ligand-best hint (hint: the lowest-energy state over the ligand's chains, PROP_HINT floats = t, q, torsions
//   0..19, energy at 27, valid flag at 28; all 0 when hint is NULL or not valid):
//   [275, 278) (t_hint - t) / 10 A
//   [278, 281) rotation vector of q_hint q^-1 (w >= 0) / pi
//   [281]      slog(e - e_hint)
//   [282]      slog(e) (0 when e is not finite)
//   [283]      1
//   [284, 288) 0
//   [288, 308) torsion differences theta_hint - theta wrapped to [-pi, pi), / pi (0 beyond the torsion count)
//   [308, 320) 0
template <typename GT>
__device__ ADOCK_COLD_ATTR void prop_features(const SearchParams& P, int l, const float* s, float e, const float* hint,
                                              __nv_bfloat16* out, int lane) {
    const int4 inf = P.info[l];
    const int na = inf.x, nt = inf.y, np = inf.z, ri = inf.w;
    const int nx = (int)P.dims[3 * ri], ny = (int)P.dims[3 * ri + 1], nz = (int)P.dims[3 * ri + 2];
    const long long n3 = (long long)nx * ny * nz;
    const int nm = P.nmaps ? min(P.nmaps[ri], 8) : 8;
    const GT* G = (const GT*)P.flat + P.offs[ri];
    if (lane < 27) {
        const float px = s[0] + 2.f * (float)(lane % 3 - 1), py = s[1] + 2.f * (float)((lane / 3) % 3 - 1),
                    pz = s[2] + 2.f * (float)(lane / 9 - 1);
        const int i = min(max(__float2int_rn((px - P.origin[3 * ri]) * P.inv_s), 0), nx - 1);
        const int j = min(max(__float2int_rn((py - P.origin[3 * ri + 1]) * P.inv_s), 0), ny - 1);
        const int k = min(max(__float2int_rn((pz - P.origin[3 * ri + 2]) * P.inv_s), 0), nz - 1);
        const long long idx = ((long long)i * ny + j) * nz + k;
        for (int q = 0; q < 8; ++q) {
            const float v = q < nm ? gload(G + q * n3 + idx) : 0.f;
            out[lane * 8 + q] = __float2bfloat16(slog(v));
        }
    }
    if (lane == 27) {
        for (int d = 0; d < 3; ++d)
            out[216 + d] = __float2bfloat16((s[d] - 0.5f * (P.lo[3 * ri + d] + P.hi[3 * ri + d])) * 0.1f);
        float qw = s[3], qx = s[4], qy = s[5], qz = s[6];
        const float nq = rsqrtf(qw * qw + qx * qx + qy * qy + qz * qz) * (qw < 0.f ? -1.f : 1.f);
        out[219] = __float2bfloat16(qw * nq); out[220] = __float2bfloat16(qx * nq);
        out[221] = __float2bfloat16(qy * nq); out[222] = __float2bfloat16(qz * nq);
        out[263] = __float2bfloat16(na / 64.f); out[264] = __float2bfloat16(nt / 20.f);
        out[265] = __float2bfloat16(P.rg[l] / 10.f); out[266] = __float2bfloat16(np / 2000.f);
    }
    if (lane < 20) {
        float sv = 0.f, cv = 0.f;
        if (lane < nt) __sincosf(s[7 + lane], &sv, &cv);
        out[223 + 2 * lane] = __float2bfloat16(sv);
        out[224 + 2 * lane] = __float2bfloat16(cv);
    }
    if (lane >= 24 && lane < 32) {   // fraction of atoms per map slot
        const int q = lane - 24;
        int cnt = 0;
        for (int a = 0; a < na; ++a) cnt += ((__float_as_int(P.atoms[(long long)l * P.AM + a].w) & 0xffff) == q);
        out[267 + q] = __float2bfloat16(na ? (float)cnt / na : 0.f);
    }
    // ligand-best hint
    const bool hv = hint != nullptr && hint[28] > 0.5f;
    if (lane == 0) {
        float f[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (hv) {
            for (int d = 0; d < 3; ++d) f[d] = (hint[d] - s[d]) * 0.1f;
            // r = q_hint * conj(q), both normalised; rotation vector 2 atan2(|v|, w) v / |v|
            const float na = rsqrtf(s[3] * s[3] + s[4] * s[4] + s[5] * s[5] + s[6] * s[6]);
            const float nb = rsqrtf(hint[3] * hint[3] + hint[4] * hint[4] + hint[5] * hint[5] + hint[6] * hint[6]);
            const float aw = s[3] * na, ax = -s[4] * na, ay = -s[5] * na, az = -s[6] * na;
            const float bw = hint[3] * nb, bx = hint[4] * nb, by = hint[5] * nb, bz = hint[6] * nb;
            float rw = bw * aw - bx * ax - by * ay - bz * az;
            float rx = bw * ax + bx * aw + by * az - bz * ay;
            float ry = bw * ay - bx * az + by * aw + bz * ax;
            float rz = bw * az + bx * ay - by * ax + bz * aw;
            if (rw < 0.f) { rw = -rw; rx = -rx; ry = -ry; rz = -rz; }
            const float sn = sqrtf(rx * rx + ry * ry + rz * rz);
            const float sc = sn > 1e-7f ? 2.f * atan2f(sn, rw) / sn : 2.f;
            f[3] = rx * sc * 0.31830988f; f[4] = ry * sc * 0.31830988f; f[5] = rz * sc * 0.31830988f;
            f[6] = isfinite(e) ? slog(e - hint[27]) : 0.f;
            f[8] = 1.f;
        }
        f[7] = (hv && isfinite(e)) ? slog(e) : 0.f;
        for (int i = 0; i < 9; ++i) out[275 + i] = __float2bfloat16(isfinite(f[i]) ? f[i] : 0.f);
        for (int i = 284; i < 288; ++i) out[i] = __float2bfloat16(0.f);
    }
    if (lane < 20) {
        float d = 0.f;
        if (hv && lane < nt) {
            d = hint[7 + lane] - s[7 + lane];
            d = d - 6.2831853f * floorf((d + 3.14159265f) * 0.15915494f);
            d = isfinite(d) ? d * 0.31830988f : 0.f;
        }
        out[288 + lane] = __float2bfloat16(d);
    }
    if (lane < 12) out[308 + lane] = __float2bfloat16(0.f);
    __syncwarp();
}

// True on all lanes when a learned target state (t, q and the ligand's first 20 torsions in x) is finite. A non-finite
// target is never optimised: clamped map lookups and ramps can give non-finite coordinates a finite energy.
__device__ __forceinline__ bool target_finite(const float* x, int nt, int lane) {
    bool ok = true;
    if (lane < 7) ok = isfinite(x[lane]);
    for (int k = lane; k < nt && k < 20; k += 32) ok = ok && isfinite(x[7 + k]);
    return __all_sync(0xffffffffu, ok);
}

// Training-log row of a state (lane 0 writes): t (3), q (4), theta 0..19 (0 past the torsion count), torsion
// count at 27, chain index at 28; the training target (the move to a later state of the same chain) is computed
// after the run.
static __device__ ADOCK_COLD_ATTR void log_state(const float* s, int nt, int ch, float* y) {
    for (int i = 0; i < 7; ++i) y[i] = s[i];
    for (int t = 0; t < 20; ++t) y[7 + t] = t < nt ? s[7 + t] : 0.f;
    y[27] = (float)nt;
    y[28] = (float)ch;
    for (int t = 29; t < 32; ++t) y[t] = 0.f;
}

template <int APL, typename GT, int MINB, bool EX>
__global__ void __launch_bounds__(128, MINB) mc_kernel(const __grid_constant__ SearchParams P,
                                                       const __grid_constant__ McParams M,
                                                       const __grid_constant__ TypeTables ttg) {
    extern __shared__ float4 smem4[];
    __shared__ TypeTables tt;
    stage_tables(tt, ttg);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const WSLayout L(P.AM, P.KM, EX);
    float* ws = (float*)smem4 + (size_t)wid * L.total;
    const int SDM = 7 + P.KM;
    unsigned n_eval = 0;
    unsigned long long n_atom_eval = 0;
    while (true) {
        int idx = 0;
        if (lane == 0) idx = atomicAdd(M.queue, 1);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= M.n_chains) break;
        const int ch = M.order ? M.order[idx] : idx;
        const int l = M.chain_lig[ch];
        if (M.lig_active && M.lig_active[l] == 0) continue;
        const int cid = M.chain_id[ch];
        const unsigned n_eval_start = n_eval;
        Chain<APL> c;
        const int* nb = M.nbr ? M.nbr + (long long)ch * M.nb_max : nullptr;
        const int nbn = M.nbr ? M.nbr_n[ch] : 0;
        load_chain<APL, GT>(c, P, tt, l, ws, L, lane, nb, nbn);
        const int S = 7 + c.nt;
        const int iters = M.bfgs_iters > 0 ? M.bfgs_iters : (25 + c.na) / 3;
        float* cur = ws + L.cur;
        float* best = ws + L.best;
        float* x = ws + L.x;
        float* gcur = M.cur + (long long)ch * SDM;
        float* gbest = M.best + (long long)ch * SDM;
        for (int i = lane; i < S; i += 32) {
            cur[i] = gcur[i];
            best[i] = gbest[i];
        }
        __syncwarp();
        float ec = M.cur_e[ch], eb = M.best_e[ch];
        int prop_fail = 0;
        unsigned long long n_prop = 0, n_prop_acc = 0, n_plain = 0, n_plain_acc = 0;
        if (!M.init_opt && ec < eb) {
            eb = ec;
            wcopy(best, cur, S, lane);
        }
        // step -1 is the start optimisation: BFGS from the current state, taken without a test
        for (int st = M.init_opt ? -1 : 0; st < M.mc_steps; ++st) {
            const bool init = st < 0;
            const int sg = M.step_offset + st;
            wcopy(x, cur, S, lane);
            // learned move while the proposal has not failed PROP_FAIL_MAX times in a row, else plain MC
            const bool use_prop = !init && M.prop && prop_fail < PROP_FAIL_MAX &&
                                  (M.prop_frac >= 1.f || uniform01(M.seed, cid, sg, 3) < M.prop_frac);
            // The proposed target state (drawn around the state the network read at the segment start). With T > 1
            // tries per step, passes 0..T-1 of the loop below evaluate one candidate each and the last pass
            // optimises the lowest-energy one; all other steps take the last pass only.
            const int T = use_prop && M.prop_tries > 1 ? M.prop_tries : 0;
            const float* mv0 = use_prop ? M.prop + ((long long)ch * M.prop_k +
                                                    (long long)(st % (M.prop_k / M.prop_tries)) * M.prop_tries) * PROP_MOVE
                                        : nullptr;
            int pick = 0;
            float e_min = 3.4e38f, en = 3.4e38f;   // a non-finite learned target keeps en: rejected without optimisation
            for (int tr = 0; tr <= T; ++tr) {
                const bool last = tr == T;
                if (use_prop) {
                    if (tr > 0) wcopy(x, cur, S, lane);
                    const float* mv = mv0 + (long long)(last ? pick : tr) * PROP_MOVE;
                    if (lane < 7) x[lane] = mv[lane];
                    for (int k = lane; k < c.nt && k < 20; k += 32) x[7 + k] = mv[7 + k];
                    __syncwarp();
                    if (!target_finite(x, c.nt, lane)) continue;
                } else if (!init) {
                    const int nm = 2 + c.nt;
                    const int which = min((int)(uniform01(M.seed, cid, sg, 0) * nm), nm - 1);
                    if (lane == 0) {
                        float v[3];
                        if (which == 0) {
                            unit_ball(M.seed, cid, sg, 10, v);
                            x[0] += M.amp_pos * v[0]; x[1] += M.amp_pos * v[1]; x[2] += M.amp_pos * v[2];
                        } else if (which == 1) {
                            unit_ball(M.seed, cid, sg, 10, v);
                            const float sc = M.amp_rot / fmaxf(c.rg, 1.0f);
                            quat_apply_rotvec(x + 3, sc * v[0], sc * v[1], sc * v[2]);
                        } else {
                            x[7 + which - 2] = (2.f * uniform01(M.seed, cid, sg, 1) - 1.f) * 3.14159265f;
                        }
                    }
                    __syncwarp();
                }
                const float et = bfgs<APL, GT, EX>(ws, L, x, last ? iters : 0, c, P, tt, lane, n_eval);
                if (last) en = et;
                else if (et < e_min) { e_min = et; pick = tr; }
            }
            if (init) {
                ec = en;
                wcopy(cur, x, S, lane);
                if (ec < eb) {
                    eb = ec;
                    wcopy(best, x, S, lane);
                }
                continue;
            }
            const bool accept =
                isfinite(en) && ((en < ec) || (uniform01(M.seed, cid, sg, 2) < __expf((ec - en) / M.temp)));
            if (use_prop) { ++n_prop; n_prop_acc += accept; } else { ++n_plain; n_plain_acc += accept; }
            prop_fail = accept ? 0 : (use_prop ? prop_fail + 1 : prop_fail);
            if (accept && en < ec && M.log_x) {   // training data: features of the pre-move state + the move
                int row = 0;
                if (lane == 0) row = atomicAdd(M.log_n, 1);
                row = __shfl_sync(0xffffffffu, row, 0);
                if (row < M.log_cap) {
                    prop_features<GT>(P, l, cur, ec, M.hint ? M.hint + (long long)l * PROP_HINT : nullptr,
                                      M.log_x + (long long)row * PROP_IN, lane);
                    if (lane == 0) log_state(cur, c.nt, ch, M.log_y + (long long)row * PROP_MOVE);
                }
                __syncwarp();
            }
            if (accept) {
                ec = en;
                wcopy(cur, x, S, lane);
                if (en < eb) {
                    eb = en;
                    wcopy(best, x, S, lane);
                }
            }
        }
        if (M.prop_stats && lane == 0 && M.mc_steps > 0) {
            atomicAdd(&M.prop_stats[0], n_prop); atomicAdd(&M.prop_stats[1], n_prop_acc);
            atomicAdd(&M.prop_stats[2], n_plain); atomicAdd(&M.prop_stats[3], n_plain_acc);
        }
        for (int i = lane; i < S; i += 32) {
            gcur[i] = cur[i];
            gbest[i] = best[i];
        }
        if (lane == 0) {
            M.cur_e[ch] = ec;
            M.best_e[ch] = eb;
        }
        n_atom_eval += (unsigned long long)(n_eval - n_eval_start) * c.na;
        __syncwarp();
    }
    if (M.evals && lane == 0 && n_eval) {
        atomicAdd(&M.evals[0], (unsigned long long)n_eval);
        atomicAdd(&M.evals[1], n_atom_eval);
    }
}

template <int APL, typename GT, bool EX>
__global__ void __launch_bounds__(128) eg_kernel(const __grid_constant__ SearchParams P, const int* chain_lig, int n,
                                                 const float* state, float* e_out, float* g_out,
                                                 const __grid_constant__ TypeTables ttg) {
    extern __shared__ float4 smem4[];
    __shared__ TypeTables tt;
    stage_tables(tt, ttg);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const WSLayout L(P.AM, P.KM, EX);
    float* ws = (float*)smem4 + (size_t)wid * L.total;
    const int SDM = 7 + P.KM, DMM = 6 + P.KM;
    const int warps = (blockDim.x >> 5) * gridDim.x;
    for (int ch = blockIdx.x * (blockDim.x >> 5) + wid; ch < n; ch += warps) {
        const int l = chain_lig[ch];
        Chain<APL> c;
        load_chain<APL, GT>(c, P, tt, l, ws, L, lane, nullptr, 0);
        float* x = ws + L.x;
        float* g = ws + L.g;
        for (int i = lane; i < SDM; i += 32) x[i] = state[(long long)ch * SDM + i];
        __syncwarp();
        const float e = eval_eg<APL, GT, EX>(ws, L, x, g, c, P, tt, lane, true);
        for (int i = lane; i < DMM; i += 32) g_out[(long long)ch * DMM + i] = i < 6 + c.nt ? g[i] : 0.f;
        if (lane == 0) e_out[ch] = e;
        __syncwarp();
    }
}

// ------------------------------------------------------------------------------------------ Stage A
// e(T) = sum_a min(cap, nearest-grid energy + out-of-box penalty) of every (ligand, conformer, rotation) over the lattice
// translations T; minimum and argmin (ties -> lowest index), mckernel.py:451-521.
// A CTA takes one conformer and SA_ROT (or fewer) of its rotations. A warp works on 32 / W rotations at a time, W lanes
// striding over the translations of each, with W the power of two (8 to 32) that covers them: a probe-filtered lattice
// holds from a handful of points in a packed pocket to thousands in an open box. (A CTA of 256 threads per rotation ran
// with 8 of them busy on 8 points: 196,608 rotations 2,764 us, now 230 us.) Where a CTA has fewer rotations than warps (few
// ligands) and the lattice has more than 32 points, its warps share a rotation's translations, else a rotation has one warp.
// An open lattice of 1,000 points, 3,072 rotations of a ligand of 24 atoms: 256 threads per rotation 200 us, one warp per
// rotation on 384 CTAs 370 us, now 167 us; 64 ligands 16.8, 13.0 and 13.3 ms.
// Bound by the latency of the map gathers (L2; a rotation's positions share few sectors), hence 48 warps per SM and
// eight gathers in flight per lane. Positions round to grid points by adding 1.5 * 2^23 (round to nearest even, like the
// float-to-int conversion it replaces, which runs at a quarter of the rate), and one of the two penalty terms per axis is
// 0, so the larger is squared.
#define SA_WARPS 4
#define SA_ROT 32

// The launch's CTAs are sized for a lattice of many points. With few, a CTA's own start (a chain of dependent loads) is most
// of its time, so every f-th CTA takes its successors' rotations too and those end at once. One ligand, 3,072 rotations on
// 3,072 CTAs or folded: 8 points 38 or 25 us, 1,000 points 167 or 370 us.
__device__ __forceinline__ int stage_a_fold(int nT, int fold) { return nT <= 16 ? fold : (nT <= 32 ? (fold + 1) / 2 : 1); }

template <typename GT>
__global__ void __launch_bounds__(32 * SA_WARPS) stage_a_kernel(const __grid_constant__ SearchParams P, const float* conf, int C,
                                                                const float* quats, int Q, int q_chunk, int fold, const float* trans,
                                                                const int* ntrans, int NT_MAX, const int* lig_box,
                                                                float cap, float* best_e, int* best_i) {
    extern __shared__ float4 smem4[];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int chunks = (Q + q_chunk - 1) / q_chunk;
    const int lc = (int)(blockIdx.x / chunks), l = lc / C, chunk = (int)(blockIdx.x % chunks);
    const int box = lig_box ? lig_box[l] : l;   // translations per ligand, or per box shared by ligands
    const int nT = ntrans[box], f = stage_a_fold(nT, fold);
    if (chunk % f) return;   // its rotations belong to an earlier CTA
    const int q0 = chunk * q_chunk, q1 = min(q0 + q_chunk * f, Q);
    const int4 inf = P.info[l];
    const int n_at = inf.x, ri = inf.w;
    const int nx = (int)P.dims[3 * ri], ny = (int)P.dims[3 * ri + 1], nz = (int)P.dims[3 * ri + 2];
    const long long n3 = (long long)nx * ny * nz;
    const GT* G = (const GT*)P.flat + P.offs[ri];
    const float ox = P.origin[3 * ri], oy = P.origin[3 * ri + 1], oz = P.origin[3 * ri + 2];
    const float lx = P.lo[3 * ri], ly = P.lo[3 * ri + 1], lz = P.lo[3 * ri + 2];
    const float hx = P.hi[3 * ri], hy = P.hi[3 * ri + 1], hz = P.hi[3 * ri + 2];
    const float mx = (float)(nx - 1), my = (float)(ny - 1), mz = (float)(nz - 1);
    const float inv = P.inv_s, pen = P.pen;
    // element indices fit 32 bits (else the slot stays in w and the index is formed in 64); grids of 2^22 points along an
    // axis or more do not fit either
    bool wide = max(nx, max(ny, nz)) >= 1 << 22;
    for (int a = tid; a < n_at; a += blockDim.x)
        wide = wide || ((__float_as_int(P.atoms[(long long)l * P.AM + a].w) & 0xffff) + 1) * n3 > 0x7fffffffLL;
    wide = __syncthreads_or(wide);
    const float magic = 12582912.f;   // 1.5 * 2^23
    const unsigned bits = 0x4B400000u, sy = (unsigned)nz, sx = (unsigned)(ny * nz);
    const int W = nT <= 8 ? 8 : (nT <= 16 ? 16 : 32), groups = 32 / W, row = P.AM + 1;
    float4* X = smem4 + (size_t)wid * 4 * row;   // [32 / W][AM + 1] rotated conformer + slot offset
    const float* p = conf + (long long)lc * P.AM * 3;
    const float* Tb = trans + (long long)box * NT_MAX * 3;
    // warps per rotation: with more than one, each team of warps takes exactly one rotation
    const int team = nT > 32 ? max(1, SA_WARPS / (q1 - q0)) : 1, member = wid % team;
    __shared__ float team_e[SA_WARPS];
    __shared__ int team_i[SA_WARPS];
    for (int qb = q0 + wid / team * groups; qb < q1; qb += SA_WARPS / team * groups) {
        for (int t = lane; t < groups * n_at; t += 32) {
            const int h = t / n_at, a = t - h * n_at, q = min(qb + h, q1 - 1);
            float qw = quats[4 * q], qx = quats[4 * q + 1], qy = quats[4 * q + 2], qz = quats[4 * q + 3];
            const float nq = rsqrtf(qw * qw + qx * qx + qy * qy + qz * qz);
            qw *= nq; qx *= nq; qy *= nq; qz *= nq;
            const float px = p[3 * a], py = p[3 * a + 1], pz = p[3 * a + 2];
            const int slot = __float_as_int(P.atoms[(long long)l * P.AM + a].w) & 0xffff;
            const unsigned w = wide ? (unsigned)slot : (unsigned)(slot * n3) - bits * (sx + sy + 1u);
            X[h * row + a] = make_float4(
                (1 - 2 * (qy * qy + qz * qz)) * px + 2 * (qx * qy - qz * qw) * py + 2 * (qx * qz + qy * qw) * pz,
                2 * (qx * qy + qz * qw) * px + (1 - 2 * (qx * qx + qz * qz)) * py + 2 * (qy * qz - qx * qw) * pz,
                2 * (qx * qz - qy * qw) * px + 2 * (qy * qz + qx * qw) * py + (1 - 2 * (qx * qx + qy * qy)) * pz,
                __uint_as_float(w));
        }
        __syncwarp();
        const int h = lane / W;
        const float4* Xq = X + h * row;
        float be = 3.4e38f;
        int bi = 0;
        for (int ti = (lane & (W - 1)) + W * member; ti < nT; ti += W * team) {
            const float T0 = Tb[3 * ti], T1 = Tb[3 * ti + 1], T2 = Tb[3 * ti + 2];
            float e = 0.f;
#pragma unroll 8
            for (int a = 0; a < n_at; ++a) {
                const float4 v = Xq[a];
                const float x = v.x + T0, y = v.y + T1, z = v.z + T2;
                float ea;
                if (!wide) {
                    const float fx = fminf(fmaxf(__fmul_rn(x - ox, inv), 0.f), mx), fy = fminf(fmaxf(__fmul_rn(y - oy, inv), 0.f), my),
                                fz = fminf(fmaxf(__fmul_rn(z - oz, inv), 0.f), mz);
                    const unsigned at = __float_as_uint(__fadd_rn(fx, magic)) * sx + __float_as_uint(__fadd_rn(fy, magic)) * sy +
                                        __float_as_uint(__fadd_rn(fz, magic)) + __float_as_uint(v.w);
                    ea = gload(G + at);
                } else {
                    const int i = min(max(__float2int_rn((x - ox) * inv), 0), nx - 1);
                    const int j = min(max(__float2int_rn((y - oy) * inv), 0), ny - 1);
                    const int k = min(max(__float2int_rn((z - oz) * inv), 0), nz - 1);
                    ea = gload(G + (long long)__float_as_uint(v.w) * n3 + ((long long)i * ny + j) * nz + k);
                }
                const float dx = fmaxf(fmaxf(lx - x, x - hx), 0.f), dy = fmaxf(fmaxf(ly - y, y - hy), 0.f),
                            dz = fmaxf(fmaxf(lz - z, z - hz), 0.f);
                ea += pen * (dx * dx + dy * dy + dz * dz);
                e += fminf(ea, cap);
            }
            if (e < be) { be = e; bi = ti; }
        }
        for (int o = W / 2; o > 0; o >>= 1) {
            const float oe = __shfl_xor_sync(0xffffffffu, be, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (oe < be || (oe == be && oi < bi)) { be = oe; bi = oi; }
        }
        if (team > 1) {
            if (lane == 0) {
                team_e[wid] = be;
                team_i[wid] = bi;
            }
        } else if ((lane & (W - 1)) == 0 && qb + h < q1) {
            best_e[(long long)lc * Q + qb + h] = be;
            best_i[(long long)lc * Q + qb + h] = bi;
        }
        __syncwarp();
    }
    if (team > 1) {
        __syncthreads();
        if (lane == 0 && member == 0) {
            const int q = q0 + wid / team;
            float be = team_e[wid];
            int bi = team_i[wid];
            for (int w = wid + 1; w < wid + team; ++w)
                if (team_e[w] < be || (team_e[w] == be && team_i[w] < bi)) { be = team_e[w]; bi = team_i[w]; }
            if (q < q1) {
                best_e[(long long)lc * Q + q] = be;
                best_i[(long long)lc * Q + q] = bi;
            }
        }
    }
}

// ------------------------------------------------------------------------------------------ float64 re-score
// One CTA of RS_WARPS warps per state: float64 forward kinematics, exact pairwise inter energy over all receptor atoms
// (or the grid interpolated in float64 when no receptor atoms are given), out-of-box penalty, intra pairs.
// Bound by the float64 pair terms (two exponentials each). Receptor atoms outside the pose's bounding box grown by the
// cutoff are dropped, the rest staged in shared memory; warps take batches of 32 of them, find the pairs inside the
// cutoff with a float32 distance (widened by its rounding) and queue them, so that the exact distance and the terms run
// 32 pairs at a time. A warp per pose that tested every receptor atom in float64 for each of its atoms and evaluated
// the terms wherever one lane was inside took 1,945 us for 8,192 poses x 1,500 receptor atoms, this
// 407 us.
#define RS_WARPS 4
#define RS_LIST 1024   // staged receptor atoms

struct RescoreSmem {   // after the coordinates [3][AM] (double)
    float4 rec[RS_LIST];               // receptor atoms: xyz, type | flags << 8
    unsigned short queue[RS_WARPS][64], with[RS_WARPS][64];   // pairs to evaluate: pose atom, staged receptor atom
    int count[RS_WARPS];
    float box[6];
    double inter[RS_WARPS], intra[RS_WARPS];
};

template <typename GT>
__global__ void __launch_bounds__(32 * RS_WARPS) rescore64_kernel(const __grid_constant__ SearchParams P, const int* chain_lig,
                                                                  const float* state, double* e_total, double* e_intra,
                                                                  float* Xout, const __grid_constant__ TypeTables ttg,
                                                                  const __grid_constant__ PairPrm64 pp) {
    extern __shared__ double smemd[];
    __shared__ TypeTables tt;
    __shared__ RescoreSmem S;
    stage_tables(tt, ttg);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    double *X = smemd, *Y = smemd + P.AM, *Z = smemd + 2 * P.AM;
    const int SDM = 7 + P.KM;
    const long long ch = blockIdx.x;
    const int l = chain_lig[ch];
    const int4 inf = P.info[l];
    const int na = inf.x, nt = inf.y, np = inf.z, ri = inf.w;
    const float4* atoms = P.atoms + (long long)l * P.AM;
    const float* s = state + ch * SDM;
    double qw = s[3], qx = s[4], qy = s[5], qz = s[6];
    const double nq = 1.0 / sqrt(qw * qw + qx * qx + qy * qy + qz * qz);
    qw *= nq; qx *= nq; qy *= nq; qz *= nq;
    const double R00 = 1 - 2 * (qy * qy + qz * qz), R01 = 2 * (qx * qy - qz * qw), R02 = 2 * (qx * qz + qy * qw);
    const double R10 = 2 * (qx * qy + qz * qw), R11 = 1 - 2 * (qx * qx + qz * qz), R12 = 2 * (qy * qz - qx * qw);
    const double R20 = 2 * (qx * qz - qy * qw), R21 = 2 * (qy * qz + qx * qw), R22 = 1 - 2 * (qx * qx + qy * qy);
    const float4* tr = P.tors + (long long)l * P.KM * 2;
    double einter = 0.0, eintra = 0.0;
    const double cut = pp.cutoff;
    double* trig = smemd + 3 * P.AM;   // [KM][2] cos, sin
    float* xf = (float*)(trig + 2 * P.KM);   // [3][AM] float32 coordinates
    for (int k = tid; k < nt; k += 32 * RS_WARPS) sincos((double)s[7 + k], &trig[2 * k + 1], &trig[2 * k]);
    __syncthreads();
    for (int a = tid; a < na; a += 32 * RS_WARPS) {
        const float4 v = atoms[a];
        double px = v.x, py = v.y, pz = v.z;
        uint32_t m = P.masks[(long long)l * P.AM + a];
        while (m) {
            const int k = __ffs(m) - 1;
            m &= m - 1;
            if (k >= nt) break;
            const float4 A = tr[2 * k], U = tr[2 * k + 1];
            const double cv = trig[2 * k], sv = trig[2 * k + 1];
            const double vx = px - A.x, vy = py - A.y, vz = pz - A.z;
            const double d = U.x * vx + U.y * vy + U.z * vz;
            const double cx = U.y * vz - U.z * vy, cy = U.z * vx - U.x * vz, cz = U.x * vy - U.y * vx;
            px = A.x + vx * cv + cx * sv + U.x * d * (1 - cv);
            py = A.y + vy * cv + cy * sv + U.y * d * (1 - cv);
            pz = A.z + vz * cv + cz * sv + U.z * d * (1 - cv);
        }
        const double X0 = R00 * px + R01 * py + R02 * pz + s[0];
        const double X1 = R10 * px + R11 * py + R12 * pz + s[1];
        const double X2 = R20 * px + R21 * py + R22 * pz + s[2];
        X[a] = X0; Y[a] = X1; Z[a] = X2;
        xf[a] = (float)X0; xf[P.AM + a] = (float)X1; xf[2 * P.AM + a] = (float)X2;
        Xout[(ch * P.AM + a) * 3] = (float)X0;
        Xout[(ch * P.AM + a) * 3 + 1] = (float)X1;
        Xout[(ch * P.AM + a) * 3 + 2] = (float)X2;
        if (!P.rxyz) {
            const int slot = __float_as_int(v.w) & 0xffff;
            const GT* G = (const GT*)P.flat + P.offs[ri];
            const long long nx = P.dims[3 * ri], ny = P.dims[3 * ri + 1], nz = P.dims[3 * ri + 2];
            const double xx[3] = {X0, X1, X2};
            const double nn[3] = {(double)nx, (double)ny, (double)nz};
            double fw[3];
            long long i0[3];
            for (int d = 0; d < 3; ++d) {
                const double f = (xx[d] - P.origin[3 * ri + d]) / (double)(1.0f / P.inv_s);
                const double fc = fmin(fmax(f, 0.0), nn[d] - 1.0 - 1e-4);
                i0[d] = (long long)floor(fc);
                fw[d] = fc - (double)i0[d];
            }
            const GT* Gs = G + (long long)slot * nx * ny * nz;
            double ea = 0.0;
            for (int dx = 0; dx < 2; ++dx)
                for (int dy = 0; dy < 2; ++dy)
                    for (int dz = 0; dz < 2; ++dz) {
                        const double w = (dx ? fw[0] : 1 - fw[0]) * (dy ? fw[1] : 1 - fw[1]) * (dz ? fw[2] : 1 - fw[2]);
                        ea += w * (double)gload(Gs + ((i0[0] + dx) * ny + (i0[1] + dy)) * nz + (i0[2] + dz));
                    }
            einter += ea;
        }
        const double xx[3] = {X0, X1, X2};
        for (int d = 0; d < 3; ++d) {
            const double lo = fmax((double)P.lo[3 * ri + d] - xx[d], 0.0), hi = fmax(xx[d] - (double)P.hi[3 * ri + d], 0.0);
            einter += (double)P.pen * (lo * lo + hi * hi);
        }
    }
    __syncthreads();
    if (P.rxyz) {
        // bounding box of the pose (everything when a coordinate is not finite)
        float reach = 0.f;   // largest coordinate: scales the float32 rounding of the distances
        if (wid == 0) {
            float lo[3] = {3.4e38f, 3.4e38f, 3.4e38f}, hi[3] = {-3.4e38f, -3.4e38f, -3.4e38f};
            bool fine = true;
            for (int a = lane; a < na; a += 32) {
                const float x[3] = {xf[a], xf[P.AM + a], xf[2 * P.AM + a]};
                for (int d = 0; d < 3; ++d) {
                    fine = fine && isfinite(x[d]);
                    lo[d] = fminf(lo[d], x[d]);
                    hi[d] = fmaxf(hi[d], x[d]);
                }
            }
            fine = __all_sync(0xffffffffu, fine);
            for (int d = 0; d < 3; ++d)
                for (int o = 16; o > 0; o >>= 1) {
                    lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
                    hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
                }
            if (lane == 0)
                for (int d = 0; d < 3; ++d) {
                    S.box[d] = fine ? lo[d] : -INFINITY;
                    S.box[3 + d] = fine ? hi[d] : INFINITY;
                }
        }
        __syncthreads();
        for (int d = 0; d < 6; ++d) reach = fmaxf(reach, fabsf(S.box[d]));
        // a float32 distance below the cutoff differs from the exact one by less than 4e-6 of the coordinates
        const float wide = P.pp.cutoff + 1e-3f + 1e-5f * reach, cut2w = wide * wide;
        const float lx = S.box[0] - wide, ly = S.box[1] - wide, lz = S.box[2] - wide;
        const float hx = S.box[3] + wide, hy = S.box[4] + wide, hz = S.box[5] + wide;
        const float* rx = P.rxyz + (long long)ri * P.RN * 3;
        const int* rt = P.rtyp + (long long)ri * P.RN;
        const int rn = P.rn[ri];
        auto evaluate = [&](int q) {   // queue entry q of this warp
            const int a = S.queue[wid][q];
            const float4 B = S.rec[S.with[wid][q]];
            const double dx = X[a] - B.x, dy = Y[a] - B.y, dz = Z[a] - B.z;
            const double r2 = dx * dx + dy * dy + dz * dz;
            if (r2 >= cut * cut) return;
            const int ta = (__float_as_int(atoms[a].w) >> 16) & 63, fa = tt.flags[ta];
            const int tb = __float_as_int(B.w) & 63, fb = __float_as_int(B.w) >> 8;
            einter += pair_energy64(sqrt(r2), (double)tt.radius[ta] + (double)tt.radius[tb], hyd_pair(fa, fb) | hb_pair(fa, fb),
                                    pp);
        };
        int listed = 0;
        for (int r0 = 0; r0 < rn; r0 += 32 * RS_WARPS) {
            // stage the next 128 receptor atoms that lie in the box, in receptor order
            const int r = r0 + tid;
            bool in = false;
            float x = 0.f, y = 0.f, z = 0.f;
            if (r < rn) {
                x = rx[3 * r]; y = rx[3 * r + 1]; z = rx[3 * r + 2];
                in = !(x < lx || x > hx || y < ly || y > hy || z < lz || z > hz);
            }
            const unsigned bal = __ballot_sync(0xffffffffu, in);
            if (lane == 0) S.count[wid] = __popc(bal);
            __syncthreads();
            int at = listed + __popc(bal & ((1u << lane) - 1u));
            for (int w = 0; w < RS_WARPS; ++w) {
                if (w < wid) at += S.count[w];
                listed += S.count[w];
            }
            if (in) {
                const int tb = rt[r] & 63;   // index kept inside the 64-entry type tables
                S.rec[at] = make_float4(x, y, z, __int_as_float(tb | (tt.flags[tb] << 8)));
            }
            __syncthreads();
            if (listed + 32 * RS_WARPS <= RS_LIST && r0 + 32 * RS_WARPS < rn) continue;
            // batches of 32 staged atoms per warp against every atom of the pose
            int queued = 0;
            for (int b0 = 32 * wid; b0 < listed; b0 += 32 * RS_WARPS) {
                const int bi = b0 + lane;
                const bool have = bi < listed;
                const float4 B = S.rec[have ? bi : 0];
                for (int a = 0; a < na; ++a) {
                    const float dx = xf[a] - B.x, dy = xf[P.AM + a] - B.y, dz = xf[2 * P.AM + a] - B.z;
                    const bool near = have && !(dx * dx + dy * dy + dz * dz > cut2w);
                    const unsigned m = __ballot_sync(0xffffffffu, near);
                    if (near) {
                        const int q = queued + __popc(m & ((1u << lane) - 1u));
                        S.queue[wid][q] = (unsigned short)a;
                        S.with[wid][q] = (unsigned short)bi;
                    }
                    queued += __popc(m);
                    if (queued >= 32) {   // at most 63 queued: evaluate the last 32
                        __syncwarp();
                        queued -= 32;
                        evaluate(queued + lane);
                        __syncwarp();
                    }
                }
            }
            __syncwarp();
            if (lane < queued) evaluate(lane);
            listed = 0;
            __syncthreads();
        }
    }
    const int2* pairs = P.pairs + (long long)l * P.P_pad;
    const int nslot = ((np + 31) >> 5) << 5;
    for (int q = tid; q < nslot; q += 32 * RS_WARPS) {
        const int2 pr = pairs[q];
        if (pr.x < 0) continue;
        const int i = pr.x & 0xff, j = (pr.x >> 8) & 0xff, fl = pr.x >> 16;
        const double dx = X[i] - X[j], dy = Y[i] - Y[j], dz = Z[i] - Z[j];
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        if (r >= cut) continue;
        const int ti = (__float_as_int(atoms[i].w) >> 16) & 63;
        const int tj = (__float_as_int(atoms[j].w) >> 16) & 63;
        eintra += pair_energy64(r, (double)tt.radius[ti] + (double)tt.radius[tj], fl, pp);
    }
    einter = warp_sum_d(einter);
    eintra = warp_sum_d(eintra);
    if (lane == 0) {
        S.inter[wid] = einter;
        S.intra[wid] = eintra;
    }
    __syncthreads();
    if (tid == 0) {
        double ei = 0.0, ea = 0.0;
        for (int w = 0; w < RS_WARPS; ++w) {
            ei += S.inter[w];
            ea += S.intra[w];
        }
        e_total[ch] = ei + ea;
        e_intra[ch] = ea;
    }
}

// feature rows of n states (one warp per state); cur_e [n] and hint [L, PROP_HINT] may be NULL
template <typename GT>
__global__ void __launch_bounds__(128) prop_features_kernel(const __grid_constant__ SearchParams P, const int* chain_lig,
                                                            int n, const float* state, const float* cur_e,
                                                            const float* hint, __nv_bfloat16* out) {
    __shared__ float s[4][7 + 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int ch = blockIdx.x * 4 + wid;
    if (ch >= n) return;
    const int SDM = 7 + P.KM;
    for (int i = lane; i < SDM && i < 7 + 32; i += 32) s[wid][i] = state[(long long)ch * SDM + i];
    __syncwarp();
    const int l = chain_lig[ch];
    prop_features<GT>(P, l, s[wid], cur_e ? cur_e[ch] : 0.f, hint ? hint + (long long)l * PROP_HINT : nullptr,
                      out + (long long)ch * PROP_IN, lane);
}

// ------------------------------------------------------------------------------------------ launchers
// Launch variants of the persistent MC kernel (128 threads per block): minimum resident blocks per SM, which
// caps registers per thread (4 -> 128, 6 -> 80, 8 -> 64). Variant 0 is the default.
static const int MC_VARIANT_MINB[4] = {4, 4, 6, 8};

template <int APL, typename GT, int MINB>
static int launch_mc_v(const SearchParams& P, const McParams& M, const TypeTables& tt, cudaStream_t st) {
    const int wpb = 4;
    const WSLayout L(P.AM, P.KM, M.exact);
    const size_t smem = (size_t)wpb * L.total * sizeof(float);
    auto kern = M.exact ? mc_kernel<APL, GT, MINB, true> : mc_kernel<APL, GT, MINB, false>;
    ADOCK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    ADOCK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * wpb, smem));
    if (per_sm < 1) per_sm = 1;
    long long blocks = (long long)sm_count() * per_sm;
    const long long need = (M.n_chains + wpb - 1) / wpb;
    if (blocks > need) blocks = need;
    if (blocks < 1) blocks = 1;
    ADOCK_CUDA(cudaMemsetAsync(M.queue, 0, sizeof(int), st));
    kern<<<(unsigned)blocks, 32 * wpb, smem, st>>>(P, M, tt);
    ADOCK_CUDA(cudaGetLastError());
    return ADOCK_OK;
}

template <int APL, typename GT>
static int launch_mc_apl(const SearchParams& P, const McParams& M, const TypeTables& tt, cudaStream_t st, int variant) {
    switch (MC_VARIANT_MINB[(variant >= 0 && variant < 4) ? variant : 0]) {
        case 6: return launch_mc_v<APL, GT, 6>(P, M, tt, st);
        case 8: return launch_mc_v<APL, GT, 8>(P, M, tt, st);
        default: return launch_mc_v<APL, GT, 4>(P, M, tt, st);
    }
}

template <typename GT>
int launch_mc(const SearchParams& P, const McParams& M, const TypeTables& tt, cudaStream_t st, int variant) {
    switch (P.AM / 32) {
        case 1: return launch_mc_apl<1, GT>(P, M, tt, st, variant);
        case 2: return launch_mc_apl<2, GT>(P, M, tt, st, variant);
        case 3: return launch_mc_apl<3, GT>(P, M, tt, st, variant);
        default: return launch_mc_apl<4, GT>(P, M, tt, st, variant);
    }
}

template <int APL, typename GT>
static int launch_eg_t(const SearchParams& P, const int* cl, int n, const float* state, float* e, float* g, int exact,
                       const TypeTables& tt, cudaStream_t st) {
    const int wpb = 4;
    const WSLayout L(P.AM, P.KM, exact);
    const size_t smem = (size_t)wpb * L.total * sizeof(float);
    auto kern = exact ? eg_kernel<APL, GT, true> : eg_kernel<APL, GT, false>;
    ADOCK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    long long blocks = (n + wpb - 1) / wpb;
    const long long cap = (long long)sm_count() * 16;
    if (blocks > cap) blocks = cap;
    kern<<<(unsigned)blocks, 32 * wpb, smem, st>>>(P, cl, n, state, e, g, tt);
    ADOCK_CUDA(cudaGetLastError());
    return ADOCK_OK;
}

template <typename GT>
int launch_eg(const SearchParams& P, const int* cl, int n, const float* state, float* e, float* g, int exact,
              const TypeTables& tt, cudaStream_t st) {
    switch (P.AM / 32) {
        case 1: return launch_eg_t<1, GT>(P, cl, n, state, e, g, exact, tt, st);
        case 2: return launch_eg_t<2, GT>(P, cl, n, state, e, g, exact, tt, st);
        case 3: return launch_eg_t<3, GT>(P, cl, n, state, e, g, exact, tt, st);
        default: return launch_eg_t<4, GT>(P, cl, n, state, e, g, exact, tt, st);
    }
}

template <typename GT>
int launch_stage_a(const SearchParams& P, long long blocks, const float* conf, int C, const float* quats, int Q,
                   const float* trans, const int* ntrans, int nt_max, const int* lig_box, float cap, float* best_e,
                   int* best_i, cudaStream_t st) {
    const size_t smem = (size_t)SA_WARPS * 4 * (P.AM + 1) * sizeof(float4);
    ADOCK_CUDA(cudaFuncSetAttribute(stage_a_kernel<GT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const long long lc = blocks / Q;   // (ligand, conformer) pairs
    // 32 rotations per CTA share the conformer; fewer where that leaves an SM less than the 12 CTAs (48 warps) that hide the
    // gathers' latency. A packed pocket's few points are too little work for so many CTAs: see stage_a_fold.
    auto ctas = [&](int q) { return lc * ((Q + q - 1) / q); };
    int q_chunk = SA_ROT, q_packed = SA_ROT;
    while (q_packed > 8 && ctas(q_packed) < 4LL * sm_count()) q_packed /= 2;
    while (q_chunk > 1 && ctas(q_chunk) < 12LL * sm_count()) q_chunk /= 2;
    const int fold = max(1, q_packed / q_chunk);
    stage_a_kernel<GT><<<(unsigned)ctas(q_chunk), 32 * SA_WARPS, smem, st>>>(P, conf, C, quats, Q, q_chunk, fold, trans, ntrans,
                                                                             nt_max, lig_box, cap, best_e, best_i);
    ADOCK_CUDA(cudaGetLastError());
    return ADOCK_OK;
}

template <typename GT>
int launch_rescore64(const SearchParams& P, const int* cl, int n, const float* state, double* et, double* ei, float* X,
                     const TypeTables& tt, const adock_sf_t& sf, cudaStream_t st) {
    const size_t smem = (3 * (size_t)P.AM + 2 * (size_t)P.KM) * sizeof(double) + 3 * (size_t)P.AM * sizeof(float);
    rescore64_kernel<GT><<<n, 32 * RS_WARPS, smem, st>>>(P, cl, state, et, ei, X, tt, make_pair_prm64(sf.prm));
    ADOCK_CUDA(cudaGetLastError());
    return ADOCK_OK;
}

template <typename GT>
int launch_prop_features(const SearchParams& P, const int* cl, int n, const float* state, const float* cur_e,
                         const float* hint, __nv_bfloat16* out, cudaStream_t st) {
    prop_features_kernel<GT><<<(unsigned)((n + 3) / 4), 128, 0, st>>>(P, cl, n, state, cur_e, hint, out);
    ADOCK_CUDA(cudaGetLastError());
    return ADOCK_OK;
}

#define ADOCK_SEARCH_INSTANTIATE(GT)                                                                              \
    template int launch_prop_features<GT>(const SearchParams&, const int*, int, const float*, const float*,       \
                                          const float*, __nv_bfloat16*, cudaStream_t);                            \
    template int launch_mc<GT>(const SearchParams&, const McParams&, const TypeTables&, cudaStream_t, int);       \
    template int launch_eg<GT>(const SearchParams&, const int*, int, const float*, float*, float*, int,           \
                               const TypeTables&, cudaStream_t);                                                  \
    template int launch_stage_a<GT>(const SearchParams&, long long, const float*, int, const float*, int,         \
                                    const float*, const int*, int, const int*, float, float*, int*,              \
                                    cudaStream_t);                                                                \
    template int launch_rescore64<GT>(const SearchParams&, const int*, int, const float*, double*, double*,       \
                                      float*, const TypeTables&, const adock_sf_t&, cudaStream_t);

#define ADOCK_SEARCH_EXTERN(GT)                                                                                   \
    extern template int launch_prop_features<GT>(const SearchParams&, const int*, int, const float*, const float*, \
                                                 const float*, __nv_bfloat16*, cudaStream_t);                     \
    extern template int launch_mc<GT>(const SearchParams&, const McParams&, const TypeTables&, cudaStream_t, int); \
    extern template int launch_eg<GT>(const SearchParams&, const int*, int, const float*, float*, float*, int,    \
                                      const TypeTables&, cudaStream_t);                                           \
    extern template int launch_stage_a<GT>(const SearchParams&, long long, const float*, int, const float*, int,  \
                                           const float*, const int*, int, const int*, float, float*, int*,       \
                                           cudaStream_t);                                                         \
    extern template int launch_rescore64<GT>(const SearchParams&, const int*, int, const float*, double*,         \
                                             double*, float*, const TypeTables&, const adock_sf_t&, cudaStream_t);

// host helpers shared by the translation units of the search (defined in search.cu)
TypeTables make_tables(const adock_sf_t* sf);
int make_params(SearchParams& P, const adock_ligands_t* lig, const adock_work_t* work, const adock_grids_t* grids,
                const adock_sf_t* sf, const adock_receptors_t* rec);

}  // namespace adock
