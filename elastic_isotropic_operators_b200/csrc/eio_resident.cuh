// Resident time loop of the nonlinear operators: a whole propagation of one or
// several shots in one cooperative launch, both levels of every wavefield (the
// adjoint: the products its stencils read) held in shared memory throughout.
//
// Bound of the per-step launches on small grids: latency.  A step of k_step
// takes 6.5 us at 312 x 520 and 5.2 at 72 x 104, whatever its size: launch,
// loads, barrier, stencils, tail, one after the other in one wave.  Here a CTA
// owns a rectangle of the grid (one CTA per SM, the rectangles tile the grid)
// and only the edges of the rectangles travel.  Measured (B200, a fine step, from
// calls of two record lengths): 72 x 104 5.2 -> 2.65 us (adjoint 5.6 -> 2.8), 312 x
// 520 6.5 -> 4.0 (6.75 -> 4.3), three shots of 312 x 424 8.8 -> 6.4, 408 x 1016 8.5
// -> 6.0; what is left is the exchange of edges, about 1 us a phase from store to
// arrival (at 312 x 520 L2 moves 9 % of what it can, shared memory 49 %).
//
// Leapfrog in two phases.  n = d (d o + D(c)) updates the velocities from the
// stresses and the stresses from the velocities, so a step is two independent
// phases: V (new velocities from the current stresses) and G (new stresses
// from the current velocities).  Even steps run V then G, odd steps G then V.
// Every phase then depends on the phase before the previous one, and the
// exchange of one phase's edges overlaps the whole next phase.
//
// Two roles.  Compute warps run the phases.  Service warps do the rest of the
// phase before, meanwhile: fetch the neighbours' edges of it (the next phase
// reads them), record the receivers, bring in the next phase's sources, and
// publish the edges where the compute threads have several units each (with
// one unit each they publish their own, half a phase earlier).  One barrier per
// phase joins them.  (Done by the compute warps, that work was two thirds of
// their instructions.)
//
// Edges.  The 8th-order star needs the four cells next to a rectangle's sides,
// no corners: two fields per direction and phase.  Edge cells travel as
// (value, step) pairs, 64-bit stores a reader sees whole, and the reader polls
// the data itself: no flag and no fence.  Slots alternate with the step's
// parity; a slot is rewritten two steps later, after its reader's own edges of
// the step between have arrived.  Waits are bounded: a thread that runs out of
// polls raises the error flag, its CTA returns at the next barrier and the
// others follow.
//
// A unit is CB adjacent columns of one float4 of z; at two columns the x
// windows overlap in registers (27 LDS.128 per four cells against 41).  The code
// of a phase exists once and a thread loops over its units: unrolled over
// units, or copied per phase order, it outgrew the instruction cache (26 us a
// step of 312 x 520).
//
// The arithmetic of a cell (stencils, taper, sources) is that of k_step in the
// same order, so the traces are the same bits.
#pragma once
#include "eio_kernels.cuh"

namespace eio {

// One fine step's time weights, uploaded per launch.
struct __align__(16) ResStep {
    int inj_t; float iw0, iw1;          // source rows inj_t, inj_t + 1
    int ext_t; float ew0, ew1;          // recorded rows ext_t, ext_t + 1
    int ext_op;                         // RES_* below
    int pad;
};
static_assert(sizeof(ResStep) == 32, "eight words");
// recorded rows live in shared memory: the first step reads them, a step on a
// new sample first puts out the row that is complete, the last puts out both
enum { RES_LOAD = 1, RES_UP = 2, RES_DOWN = 4, RES_STORE = 8 };

// A point cell of a CTA: column of the signal matrix per field and z cell, -1 none
struct ResPoint {
    int col[5][4];
    int q, x, pad[2];                   // float4 row and column in the rectangle
};

struct ResShot {
    float* lev[2][5];                   // adjoint: the fields themselves (old levels are read, new ones written); zero at first
    const float* par[5];
    const float* dampz; const float* dampx;
    int nz, nx;
    int Pz, Px;                         // rectangles along z and x (z fastest)
    // sources and receivers (nullptr: none): points of CTA c from first[c] to first[c + 1];
    // inj_map: column of a unit -> source point of its CTA (CB entries per unit, -1 none)
    const short* inj_map; const int* inj_first; const ResPoint* inj_pt;
    const int* ext_first; const ResPoint* ext_pt;
    const float* inj_sig[5]; float* ext_sig[5];
    int inj_ld[5], ext_ld[5];
    uint4* xbuf;                        // edge slots of this shot
};

struct ResArgs {
    const ResShot* shot;
    const ResStep* step;
    int nsteps;
    int nserv;                          // threads of the service warps (the first ones)
    int pub;                            // the compute threads publish their edges themselves
    int per_shot;                       // CTAs per shot
    int mq, mx;                         // largest rectangle: float4 rows, columns
    int map_stride;                     // entries of a CTA in the point maps
    int inj_cap, ext_cap;               // most points of a CTA
    float cz[4], cx[4];
    int* err;
    long long wait_limit;
};

// edge slots of one CTA, phase kind and parity, in float4: x sides [side][field][4][mq], z sides [side][field][mx]
__host__ __device__ constexpr int res_edge(int mq, int mx) { return 16 * mq + 4 * mx; }
// float4 rows of the thread grid: eight lanes read eight float4s of one column, no bank conflict
__host__ __device__ constexpr int res_rows(int mq) { return (mq + 7) / 8 * 8; }
__host__ __device__ constexpr int res_pitch(int mq) { return 4 * (mq + 2); }
__host__ __device__ constexpr int res_field(int mq, int mx) { return res_pitch(mq) * (mx + 2 * FAT); }
constexpr int RES_INJ = 80 + 24, RES_EXT = 40 + 24;   // floats per point: raw source rows of two steps / recorded rows; ResPoint
// shared memory in floats: both levels of five fields, taper, edge tables, points
constexpr size_t res_smem(int mq, int mx, int inj_cap, int ext_cap) {
    return sizeof(float) * ((size_t)10 * res_field(mq, mx) + 4 * mq + (mx + 3) / 4 * 4 + 4 * res_edge(mq, mx) +
                            (inj_cap ? res_rows(mq) * mx / 2 : 0) + (size_t)RES_INJ * inj_cap + (size_t)RES_EXT * ext_cap);
}
// Most threads of a CTA: 128 registers each, of which the phases spill 8 bytes a thread (adjoint 12, two columns
// 48).  At 768 (80 registers) they spilt 200 to 600 and a step of 312 x 520 took 6.7 us (adjoint 7.4) instead of
// 4.0 (4.3).
constexpr int RES_THREADS = 512;

__device__ __forceinline__ void ll_store(uint4* p, float4 v, unsigned tag)
{
    const unsigned long long t = (unsigned long long)tag << 32;
    const unsigned long long a = t | __float_as_uint(v.x), b = t | __float_as_uint(v.y), c = t | __float_as_uint(v.z),
                             d = t | __float_as_uint(v.w);
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p + 1), "l"(c), "l"(d) : "memory");
}
struct LLRaw {
    unsigned long long a, b, c, d;
    __device__ __forceinline__ void load(const uint4* p)
    {
        asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
        asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(c), "=l"(d) : "l"(p + 1) : "memory");
    }
    __device__ __forceinline__ bool ready(unsigned tag) const
    {
        return (unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag && (unsigned)(c >> 32) == tag &&
               (unsigned)(d >> 32) == tag;
    }
    __device__ __forceinline__ float4 value() const
    {
        return make_float4(__uint_as_float((unsigned)a), __uint_as_float((unsigned)b), __uint_as_float((unsigned)c),
                           __uint_as_float((unsigned)d));
    }
};

// a load the compiler keeps where it is written (issued early, its latency behind the stencils)
__device__ __forceinline__ float4 ldg4_early(const float* p)
{
    float4 v;
    asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// the same for data this thread wrote in this launch
__device__ __forceinline__ float4 ld4_early(const float* p)
{
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void cp_async4(float* s, const float* g)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(s);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(a), "l"(g) : "memory");
}

// z window of the unit at s (own value given)
__device__ __forceinline__ void zwin_own(const float* s, float4 b, float* w)
{
    const float4 a = ld4(s - 4), c = ld4(s + 4);
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
    w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
    w[8] = c.x; w[9] = c.y; w[10] = c.z; w[11] = c.w;
}

// shared-memory slots: velocities (adjoint: rhox vx, rhoz vz), stresses (adjoint: A, B, mu sxz of adj_products)
enum { SV0 = 0, SV1 = 1, SG0 = 2, SG1 = 3, SG2 = 4 };

template <int DIR, int CB>
__global__ void __launch_bounds__(RES_THREADS, 1) k_resident(const __grid_constant__ ResArgs g)
{
    extern __shared__ __align__(16) float res_sm[];
    float* const sm = res_sm;
    __shared__ ResShot sh;
    __shared__ __align__(16) int stw[3][8];         // weights of the last, this and the next step
    __shared__ int bad;

    const int tid = threadIdx.x, nthr = blockDim.x;
    const int cta = blockIdx.x % g.per_shot;
    {
        const int* src = reinterpret_cast<const int*>(g.shot + blockIdx.x / g.per_shot);
        int* dst = reinterpret_cast<int*>(&sh);
        for (int i = tid; i < (int)(sizeof(ResShot) / 4); i += nthr) dst[i] = src[i];
        if (tid < 8) stw[0][tid] = reinterpret_cast<const int*>(g.step)[tid];
        if (tid == 0) bad = 0;
    }
    __syncthreads();

    const int RZ = res_pitch(g.mq), FS = res_field(g.mq, g.mx);
    float* const sdz = sm + 10 * FS;                 // taper of my rows and columns
    float* const sdx = sdz + 4 * g.mq;
    int2* const etab = reinterpret_cast<int2*>(sdx + (g.mx + 3) / 4 * 4);
    int2* const ptab = etab + res_edge(g.mq, g.mx);
    short* const imap = reinterpret_cast<short*>(ptab + res_edge(g.mq, g.mx));  // column of a unit -> source point, -1 none
    float* const pin = reinterpret_cast<float*>(imap) + (g.inj_cap ? res_rows(g.mq) * g.mx / 2 : 0);
    ResPoint* const ipt = reinterpret_cast<ResPoint*>(pin + 80 * g.inj_cap);    // [points][2 steps][5][2][4], then the points
    float* const pex = reinterpret_cast<float*>(ipt + g.inj_cap);
    ResPoint* const ept = reinterpret_cast<ResPoint*>(pex + 40 * g.ext_cap);    // [points][5][2][4], then the points
    const int nz = sh.nz, nx = sh.nx;
    const int pz = cta % sh.Pz, px = cta / sh.Pz;
    const int nq = (nz - 2 * FAT) / 4, ng = (nx - 2 * FAT) / CB;
    const int q0 = pz * nq / sh.Pz, nqr = (pz + 1) * nq / sh.Pz - q0;
    const int g0 = px * ng / sh.Px, ngr = (px + 1) * ng / sh.Px - g0, ncr = ngr * CB;
    const int zb = FAT + 4 * q0, xb = FAT + g0 * CB;     // the rectangle's first cell
    const int rows = res_rows(g.mq), units = rows * ngr;   // units of the thread grid
    const bool left = px > 0, right = px < sh.Px - 1, top = pz > 0, bottom = pz < sh.Pz - 1;

    // ---- both levels start at zero, and so do the halos at the grid's frame, for good
    for (int i = tid; i < 10 * FS; i += nthr) sm[i] = 0.f;
    for (int i = tid; i < 4 * nqr; i += nthr) sdz[i] = sh.dampz[zb + i];
    for (int i = tid; i < ncr; i += nthr) sdx[i] = sh.dampx[xb + i];

    // ---- the edges this CTA fetches (etab) and publishes (ptab): place in the slots of the neighbour or
    // of this CTA; cell | field << 28 | z side << 29
    const int edge = res_edge(g.mq, g.mx);
    const int plane = 2 * edge * g.per_shot;                    // uint4 per (kind, parity)
    const int nxs = 8 * nqr, nzs = 2 * ncr;                     // per side: 2 fields x 4 columns x nqr; 2 fields x ncr
    const int nl = left ? nxs : 0, nr = nl + (right ? nxs : 0), nt = nr + (top ? nzs : 0), nit = nt + (bottom ? nzs : 0);
    for (int i = tid; i < nit; i += nthr) {
        if (i < nr) {
            const int side = i >= nl, k = i - (side ? nl : 0);
            const int fi = k / (4 * nqr), col = k / nqr % 4, qq = k % nqr, z = FAT + 4 * qq;
            const int nb = cta + (side ? sh.Pz : -sh.Pz), e = fi * 4 * g.mq + col * g.mq + qq;
            etab[i] = make_int2(2 * (nb * edge + (side ^ 1) * 8 * g.mq + e),
                                ((side ? FAT + ncr + col : col) * RZ + z) | fi << 28);
            ptab[i] = make_int2(2 * (cta * edge + side * 8 * g.mq + e), ((side ? ncr + col : FAT + col) * RZ + z) | fi << 28);
        } else {
            const int side = i >= nt, k = i - (side ? nt : nr);
            const int fi = k / ncr, col = k % ncr;
            const int nb = cta + (side ? 1 : -1), e = 16 * g.mq + fi * g.mx + col, x = (FAT + col) * RZ;
            etab[i] = make_int2(2 * (nb * edge + (side ^ 1) * 2 * g.mx + e),
                                (x + (side ? FAT + 4 * nqr : 0)) | fi << 28 | 1 << 29);
            ptab[i] = make_int2(2 * (cta * edge + side * 2 * g.mx + e), (x + (side ? 4 * nqr : FAT)) | fi << 28 | 1 << 29);
        }
    }
    // ---- my CTA's points
    const int ninj = sh.inj_map ? sh.inj_first[cta + 1] - sh.inj_first[cta] : 0;
    const int next = sh.ext_first ? sh.ext_first[cta + 1] - sh.ext_first[cta] : 0;
    for (int i = tid; i < 24 * ninj; i += nthr)
        reinterpret_cast<int*>(ipt)[i] = reinterpret_cast<const int*>(sh.inj_pt + sh.inj_first[cta])[i];
    for (int i = tid; i < 24 * next; i += nthr)
        reinterpret_cast<int*>(ept)[i] = reinterpret_cast<const int*>(sh.ext_pt + sh.ext_first[cta])[i];
    for (int i = tid; i < 80 * ninj; i += nthr) pin[i] = 0.f;   // cells without a source stay zero
    if (ninj)
        for (int i = tid; i < units * CB; i += nthr) imap[i] = sh.inj_map[(long long)cta * g.map_stride + i];
    __syncthreads();

    // ---- service warps
    const int ns = g.nserv;
    const bool service = tid < ns;
    // raw source rows of phase kind (0: velocities, 1: stresses) of a step, asynchronously into its half of pin
    auto sources = [&](const ResStep& w, int kind, int par) {
        const int F0 = kind ? 2 : 0, n4 = kind ? 12 : 8;
        for (int i = tid; i < ninj * n4; i += ns) {
            const int pt = i / n4, r = i % n4, f = F0 + r / 4, j = r % 4;
            const int col = ipt[pt].col[f][j];
            if (col < 0) continue;
            float* d = pin + pt * 80 + par * 40 + f * 8 + j;
            const float* s = sh.inj_sig[f] + (long long)w.inj_t * sh.inj_ld[f] + col;
            cp_async4(d, s);
            cp_async4(d + 4, s + sh.inj_ld[f]);      // inj_t is at most the last row but one
        }
    };
    auto slot = [](int kind, int code) {             // shared field of an edge entry
        const int fi = code >> 28 & 1, zs = code >> 29 & 1;
        return kind == 0 ? fi : (fi ? SG2 : zs ? SG1 : SG0);
    };
    // my edges of a phase (its values in buffer buf) to the slots
    auto publish = [&](int kind, int par, unsigned tag, const float* buf) {
        uint4* base = sh.xbuf + (long long)(kind * 2 + par) * plane;
        for (int i = tid; i < nit; i += ns) {
            const int2 e = ptab[i];
            ll_store(base + e.x, ld4(buf + slot(kind, e.y) * FS + (e.y & 0x0fffffff)), tag);
        }
    };
    // the same from a compute thread, for its unit: one field on the sides it borders on
    auto edge_x = [&](uint4* base, unsigned tag, int fi, int x, int q, float4 v) {
        if (left && x < 4) ll_store(base + 2 * (cta * edge + fi * 4 * g.mq + x * g.mq + q), v, tag);
        if (right && x >= ncr - 4) ll_store(base + 2 * (cta * edge + (2 + fi) * 4 * g.mq + (x - ncr + 4) * g.mq + q), v, tag);
    };
    auto edge_z = [&](uint4* base, unsigned tag, int fi, int x, int q, float4 v) {
        if (top && q == 0) ll_store(base + 2 * (cta * edge + 16 * g.mq + fi * g.mx + x), v, tag);
        if (bottom && q == nqr - 1) ll_store(base + 2 * (cta * edge + 16 * g.mq + (2 + fi) * g.mx + x), v, tag);
    };
    // the neighbours' edges of a phase into the halo of buffer buf
    auto fetch = [&](int kind, int par, unsigned tag, float* buf) {
        const uint4* base = sh.xbuf + (long long)(kind * 2 + par) * plane;
        for (int i0 = tid; i0 < nit; i0 += 4 * ns) {
            unsigned todo = 0;
            int2 e[4];
#pragma unroll
            for (int r = 0; r < 4; r++)
                if (i0 + r * ns < nit) {
                    e[r] = etab[i0 + r * ns];
                    todo |= 1u << r;
                }
            long long polls = 0;
            while (todo) {
                LLRaw x[4];
#pragma unroll
                for (int r = 0; r < 4; r++)
                    if (todo >> r & 1) x[r].load(base + e[r].x);
#pragma unroll
                for (int r = 0; r < 4; r++)
                    if ((todo >> r & 1) && x[r].ready(tag)) {
                        st4(buf + slot(kind, e[r].y) * FS + (e[r].y & 0x0fffffff), x[r].value());
                        todo &= ~(1u << r);
                    }
                if (todo && (++polls > g.wait_limit || ((polls & 1023) == 0 && *reinterpret_cast<volatile int*>(g.err)))) {
                    bad = 1;
                    atomicExch(g.err, 1);
                    return;
                }
            }
        }
    };
    // receivers of a phase: the new values in shared memory (buf) or global memory (N)
    auto record = [&](const ResStep& w, int kind, const float* buf, float* const* N) {
        const int F0 = kind ? 2 : 0, n4 = kind ? 12 : 8;
        for (int i = tid; i < next * n4; i += ns) {
            const int pt = i / n4, r = i % n4, f = F0 + r / 4, j = r % 4;
            const int col = ept[pt].col[f][j];
            if (col < 0) continue;
            const int q = ept[pt].q, x = ept[pt].x;
            const float n = DIR == 0 ? buf[f * FS + (FAT + x) * RZ + FAT + 4 * q + j]
                                           : N[f][(xb + x) * nz + zb + 4 * q + j];
            float* const p = pex + pt * 40 + f * 8 + j;
            float* const row = sh.ext_sig[f] + (long long)w.ext_t * sh.ext_ld[f] + col;
            const long long ld = sh.ext_ld[f];
            float a = p[0], b = p[4];
            if (w.ext_op & RES_LOAD) {
                a = row[0];
                b = row[ld];
            } else if (w.ext_op & RES_UP) {
                row[-ld] = a;
                a = b;
                b = 0.f;
            } else if (w.ext_op & RES_DOWN) {
                row[2 * ld] = b;
                b = a;
                a = 0.f;
            }
            a += n * w.ew0;
            b += n * w.ew1;
            if (w.ext_op & RES_STORE) {
                row[0] = a;
                row[ld] = b;
            }
            p[0] = a;
            p[4] = b;
        }
    };

    const int ct = tid - ns, nct = nthr - ns;            // compute threads
    const int dq = nct % rows, dg = nct / rows;
    if (service && ninj) {
        sources(*reinterpret_cast<const ResStep*>(stw[0]), 0, 0);
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();

#pragma unroll 1
    for (int s = 0; s < g.nsteps; s++) {
        const ResStep& w = *reinterpret_cast<const ResStep*>(stw[s % 3]);
        const int odd = s & 1;                           // even steps: velocities first
        // the current level is read from cb; a new value goes to nb, where its old level is
        float* const cb = sm + (odd ? 5 * FS : 0);
        float* const nb = sm + (odd ? 0 : 5 * FS);
        float* const* const O = sh.lev[odd];             // adjoint: old level, replaced by the new one

#pragma unroll 1
        for (int ph = 0; ph < 2; ph++) {
            const int kind = ph ^ odd;                   // 0: new velocities from the stresses, 1: the other way
            if (service) {
                // the phase before this one, of step ps
                const int ps = ph ? s : s - 1, pk = ph ? kind ^ 1 : kind, po = ps & 1;
                // the longest latencies first: the next step's weights, the next phase's sources
                int nw = 0;
                if (ph == 0 && tid < 8 && s + 1 < g.nsteps) nw = __ldg(reinterpret_cast<const int*>(g.step + s + 1) + tid);
                if (ninj) {
                    if (ph == 0) sources(w, kind ^ 1, odd);
                    else if (s + 1 < g.nsteps) sources(*reinterpret_cast<const ResStep*>(stw[(s + 1) % 3]), kind, odd ^ 1);
                }
                if (ps >= 0) {
                    const ResStep& pw = *reinterpret_cast<const ResStep*>(stw[ps % 3]);
                    float* const pb = sm + (po ? 0 : 5 * FS);
                    const bool more = !(s + 1 == g.nsteps && ph == 1);
                    if (more && !g.pub) publish(pk, po, (unsigned)ps + 1, pb);
                    record(pw, pk, pb, sh.lev[po]);
                    // into the level the next step reads
                    if (more) fetch(pk, po, (unsigned)ps + 1, pb);
                }
                if (ph == 0 && tid < 8 && s + 1 < g.nsteps) stw[(s + 1) % 3][tid] = nw;
                if (ninj) asm volatile("cp.async.wait_all;" ::: "memory");
            } else {
            const bool pub = g.pub && !(s + 1 == g.nsteps);
            uint4* const pbase = sh.xbuf + (long long)(kind * 2 + odd) * plane;
            const unsigned tag = (unsigned)s + 1;

            int q = ct % rows, gr = ct / rows;
#pragma unroll 1
            for (int u = ct; u < units; u += nct) {
                if (q < nqr) {
                const int xl = gr * CB;
                const int so = (FAT + xl) * RZ + FAT + 4 * q;
                const int gi = (xb + xl) * nz + zb + 4 * q;
                const float4 dz4 = ld4(sdz + 4 * q);
                int pts[CB];
#pragma unroll
                for (int c = 0; c < CB; c++) pts[c] = ninj ? imap[u * CB + c] : -1;

                // the value t of field f (the update) of column c to the new level
                float4 old[3][CB];                       // adjoint: the phase's old levels
                auto finish = [&](int f, int c, float4 t) -> float4 {
                    const int k = gi + c * nz;
                    const float4 o = DIR == 0 ? ld4(nb + f * FS + so + c * RZ) : old[f < 2 ? f : f - 2][c];
                    float dd[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) dd[j] = fminf(at(dz4, j), sdx[xl + c]);
#pragma unroll
                    for (int j = 0; j < 4; j++) at(t, j) = dd[j] * at(o, j) + at(t, j);
                    if (pts[c] >= 0) {
                        const float* p = pin + pts[c] * 80 + odd * 40 + f * 8;
                        const float4 a = ld4(p), b = ld4(p + 4);
#pragma unroll
                        for (int j = 0; j < 4; j++) at(t, j) += at(a, j) * w.iw0 + at(b, j) * w.iw1;
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) at(t, j) *= dd[j];
                    if (DIR == 1) st4(O[f] + k, t);
                    return t;
                };

                if (kind == 0) {
                    float4 a[CB], b[CB], med[2][CB];
#pragma unroll
                    for (int c = 0; c < CB; c++)
#pragma unroll
                        for (int k = 0; k < 2; k++) {
                            med[k][c] = ldg4_early(sh.par[k] + gi + c * nz);
                            if (DIR == 1) old[k][c] = ld4_early(O[k] + gi + c * nz);
                        }
                    {
                        float4 x[CB + 7];
                        const float* p = cb + SG0 * FS + so;
#pragma unroll
                        for (int m = 0; m < CB + 7; m++) x[m] = ld4(p + (m - 4) * RZ);
#pragma unroll
                        for (int c = 0; c < CB; c++) a[c] = dmx(x, c + 4, g.cx);
                    }
                    {
                        float4 x[CB + 7];
                        const float* p = cb + SG2 * FS + so;
#pragma unroll
                        for (int m = 0; m < CB + 7; m++) x[m] = ld4(p + (m - 3) * RZ);
#pragma unroll
                        for (int c = 0; c < CB; c++) {
                            b[c] = dpx(x, c + 3, g.cx);
                            float z[12];
                            zwin_own(p + c * RZ, x[c + 3], z);
                            const float4 d = dpz(z, g.cz);
#pragma unroll
                            for (int j = 0; j < 4; j++) at(a[c], j) = at(a[c], j) + at(d, j);
                        }
                    }
                    const float* p = cb + SG1 * FS + so;
#pragma unroll
                    for (int c = 0; c < CB; c++) {
                        float z[12];
                        zwin_own(p + c * RZ, ld4(p + c * RZ), z);
                        const float4 d = dmz(z, g.cz);
                        const float4 m0 = med[0][c], m1 = med[1][c];
                        float4 t0, t1;
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            at(t0, j) = DIR == 0 ? at(m0, j) * at(a[c], j) : -at(a[c], j);
                            const float e = at(d, j) + at(b[c], j);
                            at(t1, j) = DIR == 0 ? at(m1, j) * e : -e;
                        }
                        t0 = finish(0, c, t0);
                        t1 = finish(1, c, t1);
                        if (DIR == 1) {
#pragma unroll
                            for (int j = 0; j < 4; j++) {
                                at(t0, j) = at(m0, j) * at(t0, j);
                                at(t1, j) = at(m1, j) * at(t1, j);
                            }
                        }
                        if (pub) {
                            edge_x(pbase, tag, 0, xl + c, q, t0);
                            edge_z(pbase, tag, 0, xl + c, q, t0);
                            edge_x(pbase, tag, 1, xl + c, q, t1);
                            edge_z(pbase, tag, 1, xl + c, q, t1);
                        }
                        st4(nb + SV0 * FS + so + c * RZ, t0);
                        st4(nb + SV1 * FS + so + c * RZ, t1);
                    }
                } else {
                    float4 dx[CB], dz[CB], sz[CB], med[3][CB];
#pragma unroll
                    for (int c = 0; c < CB; c++)
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            med[k][c] = ldg4_early(sh.par[2 + k] + gi + c * nz);
                            if (DIR == 1) old[k][c] = ld4_early(O[2 + k] + gi + c * nz);
                        }
                    {
                        float4 x[CB + 7];
                        const float* p = cb + SV0 * FS + so;
#pragma unroll
                        for (int m = 0; m < CB + 7; m++) x[m] = ld4(p + (m - 3) * RZ);
#pragma unroll
                        for (int c = 0; c < CB; c++) {
                            dx[c] = dpx(x, c + 3, g.cx);
                            float z[12];
                            zwin_own(p + c * RZ, x[c + 3], z);
                            sz[c] = dmz(z, g.cz);
                        }
                    }
                    {
                        float4 x[CB + 7];
                        const float* p = cb + SV1 * FS + so;
#pragma unroll
                        for (int m = 0; m < CB + 7; m++) x[m] = ld4(p + (m - 4) * RZ);
#pragma unroll
                        for (int c = 0; c < CB; c++) {
                            const float4 d = dmx(x, c + 4, g.cx);
#pragma unroll
                            for (int j = 0; j < 4; j++) at(sz[c], j) = at(sz[c], j) + at(d, j);
                            float z[12];
                            zwin_own(p + c * RZ, x[c + 4], z);
                            dz[c] = dpz(z, g.cz);
                        }
                    }
#pragma unroll
                    for (int c = 0; c < CB; c++) {
                        const float4 l2m = med[0][c], lam = med[1][c], mu = med[2][c];
                        float4 t2, t3, t4;
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            if (DIR == 0) {
                                at(t2, j) = at(l2m, j) * at(dx[c], j) + at(lam, j) * at(dz[c], j);
                                at(t3, j) = at(lam, j) * at(dx[c], j) + at(l2m, j) * at(dz[c], j);
                                at(t4, j) = at(mu, j) * at(sz[c], j);
                            } else {
                                at(t2, j) = -at(dx[c], j);
                                at(t3, j) = -at(dz[c], j);
                                at(t4, j) = -at(sz[c], j);
                            }
                        }
                        const float4 n2 = finish(2, c, t2), n3 = finish(3, c, t3), n4 = finish(4, c, t4);
                        float4 v0 = n2, v1 = n3, v2 = n4;
                        if (DIR == 1) {
#pragma unroll
                            for (int j = 0; j < 4; j++) {
                                at(v0, j) = at(l2m, j) * at(n2, j) + at(lam, j) * at(n3, j);
                                at(v1, j) = at(lam, j) * at(n2, j) + at(l2m, j) * at(n3, j);
                                at(v2, j) = at(mu, j) * at(n4, j);
                            }
                        }
                        if (pub) {
                            edge_x(pbase, tag, 0, xl + c, q, v0);
                            edge_z(pbase, tag, 0, xl + c, q, v1);
                            edge_x(pbase, tag, 1, xl + c, q, v2);
                            edge_z(pbase, tag, 1, xl + c, q, v2);
                        }
                        st4(nb + SG0 * FS + so + c * RZ, v0);
                        st4(nb + SG1 * FS + so + c * RZ, v1);
                        st4(nb + SG2 * FS + so + c * RZ, v2);
                    }
                }

                }
                q += dq;
                gr += dg;
                if (q >= rows) { q -= rows; gr++; }
            }

            }
            __syncthreads();
            if (bad) return;
        }
    }
    // receivers of the last phase
    if (service) {
        const int ps = g.nsteps - 1, po = ps & 1;
        record(*reinterpret_cast<const ResStep*>(stw[ps % 3]), 1 ^ po, sm + (po ? 0 : 5 * FS), sh.lev[po]);
    }
}

}  // namespace eio
