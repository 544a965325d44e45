// fwi_resident.cuh -- whole time loops in one launch, wavefields in shared memory.
//
// Same arithmetic as the TMA-staged passes (fwi_tma.cuh; every cell's result
// is bit-identical), another schedule: the padded grid of each shot of a launch
// is cut into ntx x ntz tiles, one per CTA (at most one CTA per SM), and the
// five fields, the CPML memories and the materials of a tile stay in that CTA's
// shared memory for a whole program of time steps.  Per step and cell nothing
// of the state moves through L2 or HBM; only the energy sums and, in the
// adjoint, ux/uz, the gradients and a stored wavefield are read and written
// there, each by the one thread that owns the cell (no synchronisation).
//
// What bounds the launch-per-pass schedule on small grids is not bandwidth: a
// pass of the 244 x 244 grid takes ~4.5 us (launch, descriptor and tensor-map
// fetches, one tile's copy latency), two launches per step.  Here a pass
// costs its shared-memory stencil and one halo exchange.  Measured, us per
// forward step, launches -> resident: 200x200 order 4 9.5 -> 3.1, 600x380
// order 8 13.7 -> 5.7, 800x400 order 8 17.6 -> 8.7; adjoint steps over a stored
// wavefield 200x200 15.8 -> 4.6.  What bounds it now: about 1.1 us of exchange
// latency per pass, and above two rows per thread the shared-memory loads of the
// stencil (31 per pair of cells) at 16 warps per SM.
//
// Halo exchange: a thread that has updated a pair in the outer FP rows or E
// columns of its tile writes it straight into the neighbour's inbox.  Each float
// travels with a 32-bit tag in one 8-byte word (a single relaxed GPU-scope
// store), the tag counting the passes; the reader polls the words themselves, so
// an exchange is one store and one load of latency, with no fence, flag or grid
// barrier, and a pass has one CTA barrier (after the halos are in).  A word is
// overwritten only after the reader's answer to it has arrived: a tile writes
// its next velocities only after it has read the stresses its neighbours made
// from the previous ones.  Corners are not needed (the stencils are axis-aligned).
//
// The launch is cooperative (the CTAs wait on one another).  Polls are bounded
// as the TMA waits are: one that runs out sets bit 2 of the error word, every
// CTA then leaves at its next poll.
#pragma once

#include "fwi_resident.h"
#include "fwi_tma.cuh"

namespace fwi {

// Shared memory of a CTA (floats): the stencil weights (each twice) and 1.0, the
// CPML coefficients [tp][6], the fields [rows][5][PW] and strip memories of one
// or two simulations, the materials [tzm][5][kResTX].  The rows of the fields are
// interleaved, so every operand of a cell lies at a compile-time distance from
// one address.
extern __shared__ __align__(128) float res_smem[];
constexpr int kResOne = 24, kResCpml = 32;
enum { RF_VX = 0, RF_VZ = 1, RF_SZX = 2, RF_SZZ = 3, RF_SXX = 4 };  // order within a row

template <int FP>
struct ResGeom {
    static constexpr int E = 2 * ((FP + 1) / 2);  // column halo
    static constexpr int PW = kResTX + 2 * E;     // pitch of a field's row
    static constexpr int RW = 5 * PW;             // a row of all fields
    static constexpr int CELL0 = FP * RW + E;     // cell (0, 0) of the tile, first field
    // one row more than the halos need: the second row of an odd last pair is
    // loaded and dropped
    __host__ __device__ static constexpr int field_floats(int tzm) { return (tzm + 2 * FP + 3) * RW; }
    __host__ __device__ static constexpr int sim_floats(const ResTiling& t) {
        return (field_floats(t.tzm) + 3) / 4 * 4 + 8 * t.tzm * t.sxp + 8 * t.szr * (kResTX / 2);
    }
    __host__ __device__ static constexpr int fields_at(int tp) { return (kResCpml + 6 * tp + 31) / 32 * 32; }
    __host__ __device__ static constexpr int inbox_words(int tzm) { return 4 * (FP * kResTX + E * tzm); }
    __host__ __device__ static constexpr size_t smem(const ResTiling& t, int tp, int mode) {
        return sizeof(float) * ((size_t)sim_floats(t) * (mode == RES_BOTH ? 2 : 1) + fields_at(tp) +
                                (size_t)5 * t.tzm * kResTX);
    }
};

__device__ __forceinline__ ulonglong2 ll_load(const unsigned long long* p) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void ll_store(unsigned long long* p, float2 v, unsigned tag) {
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(t | __float_as_uint(v.x)),
                 "l"(t | __float_as_uint(v.y))
                 : "memory");
}
__device__ __forceinline__ float ll_value(unsigned long long w) { return __uint_as_float((unsigned)w); }

// Bounded poll: checks the clock and the error word every 64 tries.
// res_poll_check: the poll's start time (t0, or now when 0), or ~0 to give up.
static __device__ __noinline__ unsigned long long res_poll_check(unsigned long long t0, unsigned long long lim, int* err) {
    const unsigned long long t = global_ns();
    if (t0 == 0) return t;
    if (t - t0 > lim) {
        atomicOr(err, 4);
        return ~0ull;
    }
    return *(volatile int*)err != 0 ? ~0ull : t0;
}

// A thread's cells -- column pair pi of the tile (first column cp = 2 pi),
// rows [ra, rb) -- and what is special about them.  The tile's pairs lie in one
// group of 8, 16 or 32 lanes (the least that holds them); the rows of a group
// are the same for all its lanes.
enum : unsigned {
    RT_ON0 = 1u, RT_ON1 = 2u,          // the lane's column is updated (not a border column)
    RT_LEFT = 4u, RT_RIGHT = 8u,       // the tile has a left / right neighbour
    RT_X0 = 16u, RT_X1 = 32u,          // the lane's column is sampled for the FWI window
    RT_PX0 = 64u, RT_PX1 = 128u,       // the lane lies in an x strip
    RT_PLEFT = 256u,                   // the left one
};
struct ResThread {
    int b, x0, z0, np, nr;  // shot, first column and row (padded grid), column pairs, rows of the tile
    int pi, ra, rb;
    int gw;                 // lanes of a group
    int up, down;           // rows < up go to the tile above, rows >= down to the one below
    int ztop, zbot;         // rows < ztop and >= zbot lie in a z strip
    int xslot;              // strip pair
    unsigned fl;
    // rows (bit row - ra) that are not plain: sent to a neighbour, in a strip, next
    // to the border or (spec_s, the stress passes) the free surface
    unsigned spec, spec_s;
};

// Events of a thread's own cells: one injection (row * 2 + lane, -1: none; row
// of the signals) and recordings in one row.  Tiles whose events do not fit
// this form run them between barriers (defer).
struct ResEvents {
    int ir, ic;        // injection
    int rr, rc0, rc1;  // recordings (row; trace rows of the two lanes, -1: none)
    unsigned spec;     // rows (bit row - ra) with an event
    bool defer;
};

// Halos out.  An inbox: [from above][2][FP][kResTX], [from below], [from the
// left][2][tzm][E], [from the right]; two fields are sent along each axis.
// Rows: a pair of updated values, by the lanes of its row as they have it.
template <int FP>
__device__ __forceinline__ void res_send_z(const ResArgs& A, const ResThread& T, int box, int row, unsigned tag, float2 za,
                                           float2 zb) {
    const int cp = 2 * T.pi;
    if (row < T.up) {
        unsigned long long* p = A.inbox + ((int)(blockIdx.x - A.t.ntx) * 4 + box) * A.iw + 2 * FP * kResTX + row * kResTX + cp;
        ll_store(p, za, tag);
        ll_store(p + FP * kResTX, zb, tag);
    }
    if (row >= T.down) {
        unsigned long long* p = A.inbox + ((int)(blockIdx.x + A.t.ntx) * 4 + box) * A.iw + (row - T.nr + FP) * kResTX + cp;
        ll_store(p, za, tag);
        ll_store(p + FP * kResTX, zb, tag);
    }
}
// Columns: the outer E columns of the group's rows (fields fa, fb), spread over
// its lanes once the rows are done; sent by the few lanes that own them, every
// row would take a warp through the same stores for two or three lanes.
template <int FP>
__device__ __forceinline__ void res_send_x(const ResArgs& A, const ResThread& T, int sim, int box, unsigned tag, int fa,
                                           int fb) {
    using G = ResGeom<FP>;
    constexpr int E = G::E, per = 2 * E;
    __syncwarp();
    if (!(T.fl & (RT_LEFT | RT_RIGHT))) return;
    const int n = (T.rb - T.ra) * per;
    for (int i = (int)threadIdx.x & (T.gw - 1); i < n; i += T.gw) {
        const int row = T.ra + i / per, q = i % per, right = q >= E, f = (q / (E / 2)) & 1, j = 2 * (q % (E / 2));
        if (!(T.fl & (right ? RT_RIGHT : RT_LEFT))) continue;
        const float2 v = ld2(res_smem + A.fields + sim * A.sim + G::CELL0 + row * G::RW + (f ? fb : fa) * G::PW + j +
                             (right ? 2 * T.np - E : 0));
        ll_store(A.inbox + ((int)(blockIdx.x + (right ? 1 : -1)) * 4 + box) * A.iw + 4 * FP * kResTX +
                     ((right ? 0 : 2 * A.t.tzm) + f * A.t.tzm + row) * E + j,
                 v, tag);
    }
}

// The velocities of this thread's group (after a restore, or events between barriers).
template <int FP>
__device__ __forceinline__ void res_send_velocities(const ResArgs& A, const ResThread& T, int sim, unsigned tag) {
    using G = ResGeom<FP>;
    if (T.pi < T.np) {
#pragma unroll 1
        for (int row = T.ra; row < T.rb; row++) {
            const float* p = res_smem + A.fields + sim * A.sim + G::CELL0 + row * G::RW + 2 * T.pi;
            res_send_z<FP>(A, T, sim * 2, row, tag, ld2(p + RF_VX * G::PW), ld2(p + RF_VZ * G::PW));
        }
    }
    res_send_x<FP>(A, T, sim, sim * 2, tag, RF_VX, RF_VZ);
}

// What a thread reads of an inbox: rows from above or below (a warp takes one
// row of one field), columns from the left or right (a thread takes one row of
// one field).  Offsets of words in the inbox and of the halo cells they go to,
// for the velocities; the stresses' cells lie 2 PW / xd1 further.
template <int FP>
struct ResHalo {
    static constexpr int NZ = (4 * FP + 15) / 16, NX = ResGeom<FP>::E / 2, N = NZ + NX;
    int zsrc[NZ], zdst[NZ], xsrc, xdst, xd1;
    unsigned want;  // bit per word pair
    __device__ __forceinline__ ResHalo(const ResArgs& A, const ResThread& T, int tx, int tz) {
        using G = ResGeom<FP>;
        constexpr int PW = G::PW, E = G::E;
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int c0 = A.fields + G::CELL0;
        const int in = (int)blockIdx.x * 4 * A.iw;
        want = 0;
#pragma unroll
        for (int q = 0; q < NZ; q++) {
            const int line = warp + 16 * q;
            const int bot = line >= 2 * FP, l = line - bot * 2 * FP, f = l >= FP, r = l - f * FP;
            zsrc[q] = in + (bot ? 2 * FP * kResTX : 0) + (f * FP + r) * kResTX + 2 * lane;
            zdst[q] = c0 + (bot ? T.nr + r : r - FP) * G::RW + f * PW + 2 * lane;
            if (line < 4 * FP && lane < T.np && (bot ? tz + 1 < A.t.ntz : tz > 0)) want |= 1u << q;
        }
        const int row = threadIdx.x >> 2, right = (threadIdx.x >> 1) & 1, f = threadIdx.x & 1;
        xsrc = in + 4 * FP * kResTX + ((right ? 2 * A.t.tzm : 0) + f * A.t.tzm + row) * E;
        xdst = c0 + row * G::RW + f * PW + (right ? 2 * T.np : -E);
        // velocities: vx, vz along x; stresses: sxx, szx
        xd1 = (f ? RF_SZX - RF_VZ : RF_SXX - RF_VX) * PW;
        if (row < T.nr && (right ? tx + 1 < A.t.ntx : tx > 0)) want |= ((1u << NX) - 1) << NZ;
    }
    // The neighbours' words of tag `tag` into the halos of simulation sim; false
    // when a poll ran out or another CTA gave up.  A thread's words are polled
    // together: one at a time, each word that was not there at the first look
    // would cost another round trip to L2.
    __device__ __forceinline__ bool fill(const ResArgs& A, int sim, int pass, unsigned tag) const {
        const unsigned long long* in = A.inbox + (sim * 2 + pass) * A.iw;
        const int so = sim * A.sim, zd = so + (pass ? 2 * ResGeom<FP>::PW : 0), xd = so + (pass ? xd1 : 0);
        unsigned todo = want, n = 0;
        unsigned long long t0 = 0;
        while (todo) {
            ulonglong2 v[N];
#pragma unroll
            for (int q = 0; q < N; q++)
                if (todo >> q & 1) v[q] = ll_load(in + (q < NZ ? zsrc[q < NZ ? q : 0] : xsrc + 2 * (q - NZ)));
#pragma unroll
            for (int q = 0; q < N; q++)
                if ((todo >> q & 1) && (unsigned)(v[q].x >> 32) == tag && (unsigned)(v[q].y >> 32) == tag) {
                    const int d = q < NZ ? zdst[q < NZ ? q : 0] + zd : xdst + 2 * (q - NZ) + xd;
                    *reinterpret_cast<float2*>(res_smem + d) = make_float2(ll_value(v[q].x), ll_value(v[q].y));
                    todo &= ~(1u << q);
                }
            if (todo && (++n & 63u) == 0) {
                t0 = res_poll_check(t0, A.wait_ns, A.err);
                if (t0 == ~0ull) return false;
            }
        }
        return true;
    }
};

__device__ __forceinline__ Cpml res_coeff(int p) {
    const float2* q = reinterpret_cast<const float2*>(res_smem + kResCpml) + 3 * p;
    const float2 u = q[0], v = q[1], w = q[2];
    return {u.x, u.y, v.x, v.y, w.x, w.y};
}

// CPML of the derivatives of one row: (dx1, dz1) with the integer-grid
// coefficients, (dx2, dz2) with the half-grid ones; roundings of the TMA
// passes.  pass: 0 stress, 1 velocity (their memories).
template <int FP>
__device__ __forceinline__ void res_cpml(const ResArgs& A, const ResThread& T, int sim, int pass, int row, float2& dx1,
                                         float2& dx2, float2& dz1, float2& dz2) {
    float* const strips = res_smem + A.fields + sim * A.sim;
    if (T.fl & (RT_PX0 | RT_PX1)) {
        float4* m = reinterpret_cast<float4*>(strips + A.xs) + (pass * A.t.tzm + row) * A.t.sxp + T.xslot;
        const int px = T.x0 + 2 * T.pi - ((T.fl & RT_PLEFT) ? FP : A.f.pnx);
        float4 v = *m;
#pragma unroll
        for (int l = 0; l < 2; l++) {
            if (!(T.fl & (l ? RT_PX1 : RT_PX0))) continue;
            const Cpml c = res_coeff(px + l);
            float& e1 = l ? dx1.y : dx1.x;
            float& e2 = l ? dx2.y : dx2.x;
            float& o1 = l ? v.y : v.x;
            float& o2 = l ? v.w : v.z;
            o1 = __fmaf_rn(c.b, o1, __fmul_rn(c.a, e1));
            o2 = __fmaf_rn(c.bh, o2, __fmul_rn(c.ah, e2));
            e1 = __fmaf_rn(e1, c.iK, o1);
            e2 = __fmaf_rn(e2, c.iKh, o2);
        }
        *m = v;
    }
    if (row < T.ztop || row >= T.zbot) {
        const int iz = T.z0 + row;
        const Cpml cz = res_coeff(row < T.ztop ? iz - FP : iz - A.f.pnz);
        const int slot = row < T.ztop ? row : row - T.zbot + T.ztop;
        float4* m = reinterpret_cast<float4*>(strips + A.zs) + (pass * A.t.szr + slot) * (kResTX / 2) + T.pi;
        const float4 v = *m;
        const float2 m1 = fma2(bc2(cz.b), make_float2(v.x, v.y), mul2(bc2(cz.a), dz1));
        const float2 m2 = fma2(bc2(cz.bh), make_float2(v.z, v.w), mul2(bc2(cz.ah), dz2));
        *m = make_float4(m1.x, m1.y, m2.x, m2.y);
        dz1 = fma2(dz1, bc2(cz.iK), m1);
        dz2 = fma2(dz2, bc2(cz.iKh), m2);
    }
}

__device__ __forceinline__ void res_put(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }
// Border columns stay zero.
__device__ __forceinline__ float2 res_keep(float2 v, unsigned fl) {
    return make_float2((fl & RT_ON0) ? v.x : 0.f, (fl & RT_ON1) ? v.y : 0.f);
}
// The stencil weights, in registers.
template <int FP>
__device__ __forceinline__ void res_weights(float2 (&hx)[FP], float2 (&hz)[FP]) {
#pragma unroll
    for (int k = 0; k < FP; k++) {
        hx[k] = ld2(res_smem + 2 * k);
        hz[k] = ld2(res_smem + 2 * kMaxHalf + 2 * k);
    }
}
// A pair into global memory; border columns are left alone.
__device__ __forceinline__ void res_out(float* p, float2 v, unsigned fl) { st2(p, v, fl & RT_ON0, fl & RT_ON1); }

// Row of the FWI window's samples that grid row iz is (-1: none), and the
// sample column of a lane whose flag is set.
__device__ __forceinline__ int res_zf(const ItemDesc& D, int iz) {
    if (iz < D.wz1 || iz >= D.wz2) return -1;
    const int d = iz - D.wz1;
    if (D.fwi_dz == 1) return d;
    return d % D.fwi_dz == 0 ? d / D.fwi_dz : -1;
}
__device__ __forceinline__ int res_xf(const ItemDesc& D, int ix) {
    return D.fwi_dx == 1 ? ix - D.wx1 : (ix - D.wx1) / D.fwi_dx;
}

// Gradient samples and displacement integrals of one row (adjoint).
struct ResGrad {
    float2 ux, uz;
    float g[6], sv[10];
    int zf;
};
template <bool TWO>
__device__ __forceinline__ void res_grad_load(ResGrad& q, const ResArgs& A, const ResThread& T, int row, int it,
                                              unsigned flags) {
    const ItemDesc& D = A.a;
    const int iz = T.z0 + row, ix = T.x0 + 2 * T.pi;
    const long long c = T.b * A.field + (long long)iz * D.pitch + ix;
    q.zf = -1;
    if (!inb(c - T.b * A.field + 1, FWI_NFIELD(D), 54)) return;
    q.ux = ld2(D.ux + c);
    q.uz = ld2(D.uz + c);
    if (!(flags & FL_GRAD) || !(T.fl & (RT_X0 | RT_X1))) return;
    q.zf = res_zf(D, iz);
    if (q.zf < 0) return;
#pragma unroll
    for (int l = 0; l < 2; l++) {
        if (!(T.fl & (l ? RT_X1 : RT_X0))) continue;
        const int o = q.zf * D.nfx + res_xf(D, ix + l);
        if (!inb(o, FWI_NGRAD(D), 55)) continue;
        const long long og = T.b * 3 * A.nf + o;
        q.g[l] = D.glam[og];
        q.g[2 + l] = D.gmu[og];
        q.g[4 + l] = D.grho[og];
        if constexpr (!TWO) {
            const float* w = D.fwd + ((long long)T.b * A.nft + it / D.fwi_dt) * 5 * A.nf + o;
#pragma unroll
            for (int f = 0; f < 5; f++) q.sv[2 * f + l] = w[f * A.nf];
        }
    }
}

// Stress pass of one simulation.  ADJ: with the ux/uz integration and, on a
// sampled step, the gradient (TWO: from the forward simulation's fields,
// otherwise from the stored wavefield).
template <int FP, int R, bool ADJ, bool TWO>
__device__ __forceinline__ bool res_stress(const ResArgs& A, const ResThread& T, const ResHalo<FP>& H, bool wait_v,
                                           unsigned tag_v, unsigned tag_s, int it, unsigned flags) {
    using G = ResGeom<FP>;
    constexpr int PW = G::PW, RW = G::RW;
    constexpr int NW = 2 * FP + R - 1;
    constexpr int sim = ADJ && TWO ? 1 : 0;  // place of the simulation in shared memory
    const ItemDesc& D = ADJ ? A.a : A.f;
    const int cp = 2 * T.pi, rb = T.pi < T.np ? T.rb : T.ra;
    ResGrad q;
    if constexpr (ADJ)
        if (T.ra < rb) res_grad_load<TWO>(q, A, T, T.ra, it, flags);
    bool ok = true;
    if (wait_v) ok = H.fill(A, sim, 0, tag_v);
    if (__syncthreads_or(!ok)) return false;
    float2 hx[FP], hz[FP];
    res_weights<FP>(hx, hz);
    const float2 one = ld2(res_smem + kResOne);
    for (int r = T.ra; r < rb; r += R) {
        float* const f0 = res_smem + A.fields + sim * A.sim + G::CELL0 + r * RW + cp;
        float2 wvx[NW], wvz[NW];
#pragma unroll
        for (int j = 0; j < NW; j++) {
            wvx[j] = ld2(f0 + (j - FP + 1) * RW + RF_VX * PW);
            wvz[j] = ld2(f0 + (j - FP) * RW + RF_VZ * PW);
        }
#pragma unroll
        for (int rr = 0; rr < R; rr++) {
            const int row = r + rr;
            if (row >= rb) break;
            float* const f = f0 + rr * RW;
            RowPairs<FP> tvx, tvz;
            tvx.load(f + RF_VX * PW, wvx[rr + FP - 1]);
            tvz.load(f + RF_VZ * PW, wvz[rr + FP]);
            float2 vx_x = tvx.dminus(hx);
            float2 vz_x = tvz.dplus(hx);
            float2 vx_z = make_float2(0.f, 0.f), vz_z = make_float2(0.f, 0.f);
#pragma unroll
            for (int k = 1; k <= FP; k++) {
                vx_z = fma2(hz[k - 1], sub2(wvx[rr + k + FP - 1], wvx[rr - k + FP]), vx_z);
                vz_z = fma2(hz[k - 1], sub2(wvz[rr + k - 1 + FP], wvz[rr - k + FP]), vz_z);
            }
            const bool special = (T.spec_s >> (row - T.ra)) & 1u;
            if (special) res_cpml<FP>(A, T, sim, 0, row, vx_x, vz_x, vz_z, vx_z);
            const float* m = res_smem + A.mat + row * (5 * kResTX) + cp;
            const float2 L = ld2(m), M2 = ld2(m + kResTX), MZ = ld2(m + 2 * kResTX);
            const float2 pxx = ld2(f + RF_SXX * PW), pzx = ld2(f + RF_SZX * PW), pzz = ld2(f + RF_SZZ * PW);
            float2 sxx, szx, szz;
            // the increments are added as the two-pass kernels add them: the forward
            // ones with a multiplier of one that the compiler cannot see (no
            // contraction with the product), the adjoint ones by a plain sum
            const float2 tr = mul2(L, add2(vx_x, vz_z));
            if constexpr (ADJ) {
                szx = add2(pzx, mul2(MZ, add2(vz_x, vx_z)));
                sxx = add2(pxx, fma2(M2, vx_x, tr));
                szz = add2(pzz, fma2(M2, vz_z, tr));
            } else {
                szx = fma2(one, mul2(MZ, add2(vz_x, vx_z)), pzx);
                sxx = fma2(one, fma2(M2, vx_x, tr), pxx);
                szz = fma2(one, fma2(M2, vz_z, tr), pzz);
            }
            if (special) {
                if (D.fsurf && T.z0 + row <= 2 * FP) {
                    if (T.z0 + row == FP) {
                        szz = make_float2(0.f, 0.f);
                        szx = make_float2(0.f, 0.f);
                        sxx.x = fsurf_sxx(vx_x.x, L.x, M2.x);
                        sxx.y = fsurf_sxx(vx_x.y, L.y, M2.y);
                    } else {  // images above the free surface (the first tile's rows are the grid's)
                        float* const i = f - 2 * row * RW;
                        res_put(i + RF_SZX * PW, res_keep(make_float2(-szx.x, -szx.y), T.fl));
                        res_put(i + RF_SZZ * PW, res_keep(make_float2(-szz.x, -szz.y), T.fl));
                    }
                }
                res_send_z<FP>(A, T, sim * 2 + 1, row, tag_s, szx, szz);
                sxx = res_keep(sxx, T.fl);
                szx = res_keep(szx, T.fl);
                szz = res_keep(szz, T.fl);
            }
            res_put(f + RF_SXX * PW, sxx);
            res_put(f + RF_SZX * PW, szx);
            res_put(f + RF_SZZ * PW, szz);
            // the rest is off the neighbours' path: storage, or integrals and gradient, of
            // the fields as they were before the update
            if constexpr (!ADJ) {
                if ((flags & FL_STORE) && (T.fl & (RT_X0 | RT_X1))) {
                    const int zs = res_zf(D, T.z0 + row);
#pragma unroll
                    for (int l = 0; l < 2; l++) {
                        const long long o = (long long)zs * D.nfx + res_xf(D, T.x0 + cp + l);
                        if (zs < 0 || !(T.fl & (l ? RT_X1 : RT_X0)) || !inb(o, FWI_NGRAD(D), 56)) continue;
                        float* w = D.store + ((long long)T.b * A.nft + it / D.fwi_dt) * 5 * A.nf + o;
                        w[F_VX * A.nf] = __fdiv_rn(lane(wvx[rr + FP - 1], l), D.dt);
                        w[F_VZ * A.nf] = __fdiv_rn(lane(wvz[rr + FP], l), D.dt);
                        w[F_SXX * A.nf] = lane(pxx, l);
                        w[F_SZX * A.nf] = lane(pzx, l);
                        w[F_SZZ * A.nf] = lane(pzz, l);
                    }
                }
            } else {
                const long long c = T.b * A.field + (long long)(T.z0 + row) * D.pitch + T.x0 + cp;
                const float2 dt2 = bc2(D.dt);
                const float2 ux = fma2(dt2, wvx[rr + FP - 1], q.ux);
                const float2 uz = fma2(dt2, wvz[rr + FP], q.uz);
                if (inb(c - T.b * A.field + 1, FWI_NFIELD(D), 57)) {
                    res_out(D.ux + c, ux, T.fl);
                    res_out(D.uz + c, uz, T.fl);
                }
                if (q.zf >= 0) {
                    const float2 idt = bc2(D.inv_dt), gs = bc2(D.gscale);
                    const float2 lpm = mul2(fma2(bc2(0.5f), M2, L), idt);
                    const float2 mu = mul2(mul2(bc2(0.5f), M2), idt);
                    const float2 lpm2 = mul2(lpm, lpm), mu2 = mul2(mu, mu);
                    float2 fvx, fvz, fsxx, fszx, fszz, s1, s23;
                    if constexpr (TWO) {  // the forward state of the step, as the TMA adjoint pass reads it
                        const float* w = f - A.sim;
                        fvx = mul2(ld2(w + RF_VX * PW), idt);
                        fvz = mul2(ld2(w + RF_VZ * PW), idt);
                        fsxx = ld2(w + RF_SXX * PW);
                        fszx = ld2(w + RF_SZX * PW);
                        fszz = ld2(w + RF_SZZ * PW);
                        const float2 il = make_float2(0.25f * rcp_approx(lpm2.x), 0.25f * rcp_approx(lpm2.y));
                        const float2 im = make_float2(rcp_approx(mu2.x), rcp_approx(mu2.y));
                        s1 = mul2(mul2(add2(fsxx, fszz), add2(pxx, pzz)), il);
                        const float2 s2 = mul2(mul2(sub2(fsxx, fszz), sub2(pxx, pzz)), im);
                        s23 = add2(add2(mul2(mul2(fszx, pzx), im), s1), s2);
                    } else {  // the stored wavefield (velocities over dt); rounded quotients
                        fvx = make_float2(q.sv[0], q.sv[1]);
                        fvz = make_float2(q.sv[2], q.sv[3]);
                        fsxx = make_float2(q.sv[4], q.sv[5]);
                        fszx = make_float2(q.sv[6], q.sv[7]);
                        fszz = make_float2(q.sv[8], q.sv[9]);
                        const float2 n1 = mul2(mul2(add2(fsxx, fszz), add2(pxx, pzz)), bc2(0.25f));
                        const float2 n2 = fma2(fszx, pzx, mul2(sub2(fsxx, fszz), sub2(pxx, pzz)));
                        s1 = make_float2(__fdiv_rn(n1.x, lpm2.x), __fdiv_rn(n1.y, lpm2.y));
                        s23 = add2(s1, make_float2(__fdiv_rn(n2.x, mu2.x), __fdiv_rn(n2.y, mu2.y)));
                    }
                    const float2 s4 = fma2(ux, fvx, mul2(uz, fvz));
                    const float2 nl = fma2(gs, s1, make_float2(q.g[0], q.g[1]));
                    const float2 nm = fma2(gs, s23, make_float2(q.g[2], q.g[3]));
                    const float2 nr = fma2(make_float2(-D.gscale, -D.gscale), s4, make_float2(q.g[4], q.g[5]));
#pragma unroll
                    for (int l = 0; l < 2; l++) {
                        const int o = q.zf * D.nfx + res_xf(D, T.x0 + cp + l);
                        if (!(T.fl & (l ? RT_X1 : RT_X0)) || !inb(o, FWI_NGRAD(D), 58)) continue;
                        const long long og = T.b * 3 * A.nf + o;
                        D.glam[og] = lane(nl, l);
                        D.gmu[og] = lane(nm, l);
                        D.grho[og] = lane(nr, l);
                    }
                }
                if (row + 1 < rb) res_grad_load<TWO>(q, A, T, row + 1, it, flags);
            }
        }
    }
    res_send_x<FP>(A, T, sim, sim * 2 + 1, tag_s, RF_SXX, RF_SZX);
    return true;
}

// Events of a tile between barriers: the injections of a cell are added in
// order by the thread of its first event, then the recordings read vz.
static __device__ __noinline__ void res_events(float* vz, const float* inj, float* rec, const int2* ev, int nev, int nt,
                                               int it, bool record) {
    __syncthreads();
    for (int i = threadIdx.x; i < nev; i += kResThreads) {
        const int2 e = ev[i];
        if (e.y < 0 || (e.x & kResMore)) continue;
        float val = vz[e.x] + inj[(size_t)e.y * nt + it];
        for (int k = i + 1; k < nev && (ev[k].x & kResMore) && ev[k].y >= 0; k++)
            val = val + inj[(size_t)ev[k].y * nt + it];
        vz[e.x] = val;
    }
    __syncthreads();
    if (record)
        for (int i = threadIdx.x; i < nev; i += kResThreads) {
            const int2 e = ev[i];
            if (e.y < 0) rec[(size_t)(~e.y) * nt + it] = vz[e.x & (kResMore - 1)];
        }
}

// Velocity pass (FL_WE: energy sum) with the injections and (FL_RECORD)
// recordings.  sim: place in shared memory.
template <int FP, int R, bool ADJ>
__device__ __forceinline__ bool res_velocity(const ResArgs& A, const ResThread& T, const ResHalo<FP>& H,
                                             const ResEvents& ev, int sim, unsigned tag_v, unsigned tag_s, int it,
                                             unsigned flags, const int2* list, int nev) {
    using G = ResGeom<FP>;
    constexpr int PW = G::PW, RW = G::RW;
    constexpr int NW = 2 * FP + R - 1;
    const ItemDesc& D = ADJ ? A.a : A.f;
    const bool we = (flags & FL_WE) != 0;
    const int cp = 2 * T.pi, rb = T.pi < T.np ? T.rb : T.ra;
    const long long c0 = T.b * A.field + (long long)T.z0 * D.pitch + T.x0 + cp;
    float2 e[R];
    auto load_we = [&](int r) {
#pragma unroll
        for (int rr = 0; rr < R; rr++)
            if (we && r + rr < rb && inb(c0 - T.b * A.field + (r + rr) * D.pitch + 1, FWI_NFIELD(D), 59))
                e[rr] = ld2(D.We + c0 + (r + rr) * D.pitch);
    };
    if (T.ra < rb) load_we(T.ra);
    float inj = 0.f;
    if (ev.ir >= 0) inj = D.inj[(size_t)ev.ic * D.nt + it];
    const bool ok = H.fill(A, sim, 1, tag_s);
    if (__syncthreads_or(!ok)) return false;
    float2 hx[FP], hz[FP];
    res_weights<FP>(hx, hz);
    const float2 one = ld2(res_smem + kResOne);
    const unsigned spec = T.spec | ev.spec;
    for (int r = T.ra; r < rb; r += R) {
        float* const f0 = res_smem + A.fields + sim * A.sim + G::CELL0 + r * RW + cp;
        float2 wsx[NW], wsz[NW];
#pragma unroll
        for (int j = 0; j < NW; j++) {
            wsx[j] = ld2(f0 + (j - FP) * RW + RF_SZX * PW);
            wsz[j] = ld2(f0 + (j - FP + 1) * RW + RF_SZZ * PW);
        }
#pragma unroll
        for (int rr = 0; rr < R; rr++) {
            const int row = r + rr;
            if (row >= rb) break;
            float* const f = f0 + rr * RW;
            RowPairs<FP> tsx, tzx;
            tsx.load(f + RF_SXX * PW, ld2(f + RF_SXX * PW));
            tzx.load(f + RF_SZX * PW, wsx[rr + FP]);
            float2 sxx_x = tsx.dplus(hx);
            float2 szx_x = tzx.dminus(hx);
            float2 szx_z = make_float2(0.f, 0.f), szz_z = make_float2(0.f, 0.f);
#pragma unroll
            for (int k = 1; k <= FP; k++) {
                szx_z = fma2(hz[k - 1], sub2(wsx[rr + k - 1 + FP], wsx[rr - k + FP]), szx_z);
                szz_z = fma2(hz[k - 1], sub2(wsz[rr + k + FP - 1], wsz[rr - k + FP]), szz_z);
            }
            const bool special = (spec >> (row - T.ra)) & 1u;
            if (special) res_cpml<FP>(A, T, sim, 1, row, sxx_x, szx_x, szz_z, szx_z);
            const float* m = res_smem + A.mat + row * (5 * kResTX) + cp;
            float2 vxn = fma2(one, mul2(ld2(m + 3 * kResTX), add2(sxx_x, szx_z)), ld2(f + RF_VX * PW));
            const float2 vze = fma2(one, mul2(ld2(m + 4 * kResTX), add2(szx_x, szz_z)), ld2(f + RF_VZ * PW));
            float2 vzn = vze;
            if (special) {
                if (ev.ir >= 0 && (ev.ir >> 1) == row) {
                    if (ev.ir & 1) vzn.y += inj;
                    else vzn.x += inj;
                }
                if (!ev.defer) res_send_z<FP>(A, T, sim * 2, row, tag_v, vxn, vzn);
                if ((flags & FL_RECORD) && ev.rr == row) {
                    if (ev.rc0 >= 0) D.rec[(size_t)ev.rc0 * D.nt + it] = vzn.x;
                    if (ev.rc1 >= 0) D.rec[(size_t)ev.rc1 * D.nt + it] = vzn.y;
                }
                vxn = res_keep(vxn, T.fl);
                vzn = res_keep(vzn, T.fl);
            }
            res_put(f + RF_VX * PW, vxn);
            res_put(f + RF_VZ * PW, vzn);
            // energy of the velocities before the injection
            if (we && inb(c0 - T.b * A.field + row * D.pitch + 1, FWI_NFIELD(D), 60))
                res_out(D.We + c0 + row * D.pitch, add2(e[rr], fma2(vxn, vxn, mul2(vze, vze))), T.fl);
        }
        if (r + R < rb) load_we(r + R);
    }
    if (ev.defer) {
        res_events(res_smem + A.fields + sim * A.sim + G::CELL0 + RF_VZ * PW, D.inj, D.rec, list, nev, D.nt, it, (flags & FL_RECORD) != 0);
        res_send_velocities<FP>(A, T, sim, tag_v);
    } else {
        res_send_x<FP>(A, T, sim, sim * 2, tag_v, RF_VX, RF_VZ);
    }
    return true;
}

// A simulation's tile to (save) or from the state at `st` (a batch state's
// layout: five fields, then the CPML memories).  st null: zeros.  The values of
// a row are all on their way before the first is needed.
template <int FP>
__device__ __noinline__ void res_state_io(const ResArgs& A, const ResThread T, int sim, float* st, bool save, bool images) {
    using G = ResGeom<FP>;
    if (T.pi >= T.np) return;
    const ItemDesc& D = A.f;  // geometry (the same for both simulations)
    const int fo[5] = {RF_VX, RF_VZ, RF_SXX, RF_SZX, RF_SZZ};  // in the order of Field
    float* const base = res_smem + A.fields + sim * A.sim;
    const int cp = 2 * T.pi, ix = T.x0 + cp;
    const int px = ix - ((T.fl & RT_PLEFT) ? FP : D.pnx);
    float* const sx = st + 5 * A.field;
    float* const sz = sx + 4 * A.xstrip;
    const float2 zero = make_float2(0.f, 0.f);
    // with a free surface the first tile also writes the images above it
    const int first = images && T.z0 == FP && D.fsurf && T.ra == 0 && T.rb > 0 ? -FP : T.ra;
    for (int row = first; row < T.rb; row++) {
        const int iz = T.z0 + row;
        const long long c = (long long)iz * D.pitch + ix;
        if (!inb(c + 1, FWI_NFIELD(D), 61)) continue;
        float* const f = base + G::CELL0 + row * G::RW + cp;
        if (row < 0) {
            res_out(st + F_SZX * A.field + c, ld2(f + RF_SZX * G::PW), T.fl);
            res_out(st + F_SZZ * A.field + c, ld2(f + RF_SZZ * G::PW), T.fl);
            continue;
        }
        // x strips: mem_vx_x, mem_vz_x of the stress pass, mem_sxx_x, mem_szx_x of the
        // velocity pass, each of the two lanes
        float* const vx = base + A.xs + 4 * (row * A.t.sxp + T.xslot);
        const int vx1 = 4 * A.t.tzm * A.t.sxp;
        const long long m = (long long)iz * D.tp + px;
        const bool l0 = (T.fl & RT_PX0) && inb(m, FWI_NXS(D), 62), l1 = (T.fl & RT_PX1) && inb(m + 1, FWI_NXS(D), 62);
        // z strips: global order mem_vx_z, mem_vz_z, mem_szz_z, mem_szx_z; in shared memory
        // the integer-grid one first: stress (vz_z, vx_z), velocity (szz_z, szx_z)
        const int pz = row < T.ztop ? iz - FP : iz - D.pnz, slot = row < T.ztop ? row : row - T.zbot + T.ztop;
        float* const vz = base + A.zs + 4 * (slot * (kResTX / 2) + T.pi);
        const int vz1 = 4 * A.t.szr * (kResTX / 2);
        const long long mz = (long long)pz * D.pitch + ix;
        const bool zs = (row < T.ztop || row >= T.zbot) && inb(mz + 1, FWI_NZS(D), 63);
        if (save) {
#pragma unroll
            for (int k = 0; k < 5; k++) res_out(st + k * A.field + c, ld2(f + fo[k] * G::PW), T.fl);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float* v = vx + (k >> 1) * vx1 + 2 * (k & 1);
                if (l0) sx[k * A.xstrip + m] = v[0];
                if (l1) sx[k * A.xstrip + m + 1] = v[1];
            }
            if (zs) {
                res_out(sz + mz, ld2(vz + 2), T.fl);
                res_out(sz + A.zstrip + mz, ld2(vz), T.fl);
                res_out(sz + 2 * A.zstrip + mz, ld2(vz + vz1), T.fl);
                res_out(sz + 3 * A.zstrip + mz, ld2(vz + vz1 + 2), T.fl);
            }
        } else {
            float2 v[5], z[4];
            float x[8];
#pragma unroll
            for (int k = 0; k < 5; k++) v[k] = st ? ld2(st + k * A.field + c) : zero;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                x[2 * k] = l0 && st ? sx[k * A.xstrip + m] : 0.f;
                x[2 * k + 1] = l1 && st ? sx[k * A.xstrip + m + 1] : 0.f;
                z[k] = zs && st ? ld2(sz + k * A.zstrip + mz) : zero;
            }
#pragma unroll
            for (int k = 0; k < 5; k++) res_put(f + fo[k] * G::PW, res_keep(v[k], T.fl));
            if (l0 || l1) {
                *reinterpret_cast<float4*>(vx) = make_float4(x[0], x[1], x[2], x[3]);
                *reinterpret_cast<float4*>(vx + vx1) = make_float4(x[4], x[5], x[6], x[7]);
            }
            if (zs) {
                *reinterpret_cast<float4*>(vz) = make_float4(z[1].x, z[1].y, z[0].x, z[0].y);
                *reinterpret_cast<float4*>(vz + vz1) = make_float4(z[2].x, z[2].y, z[3].x, z[3].y);
            }
        }
    }
}

// Events of this thread's cells; false where they do not fit ResEvents.
__device__ __forceinline__ bool res_own_events(ResEvents& e, const ResThread& T, const int2* ev, int nev, int pw,
                                               bool record) {
    bool fits = true;
    for (int i = 0; i < nev; i++) {
        const int2 v = ev[i];
        const int cell = v.x & (kResMore - 1), row = cell / pw, col = cell - row * pw;
        if (row < T.ra || row >= T.rb || (col >> 1) != T.pi) continue;  // (col >> 1 < np)
        if (v.y >= 0) {
            fits &= e.ir < 0;
            e.ir = row * 2 + (col & 1);
            e.ic = v.y;
            e.spec |= 1u << (row - T.ra);
        } else if (record) {
            int& rc = (col & 1) ? e.rc1 : e.rc0;
            fits &= rc < 0 && (e.rr < 0 || e.rr == row);
            e.rr = row;
            rc = ~v.y;
            e.spec |= 1u << (row - T.ra);
        }
    }
    return fits;
}

template <int FP, int MODE>
__global__ void __launch_bounds__(kResThreads, 1) resident_kernel(const __grid_constant__ ResArgs A) {
    // rows a thread takes at once (four rows share more of a window's loads but
    // spill: 860x460 order 8 8.5 us a step against 6.7)
    constexpr int R = 2;
    using G = ResGeom<FP>;
    constexpr bool TWO = MODE == RES_BOTH;
    if (__syncthreads_or(*(volatile int*)A.err != 0)) return;  // an earlier launch gave up
    if (A.stall && blockIdx.x == 0) return;
    const ItemDesc& D = A.f;
    // CPML coefficients into shared memory, fields and memories to zero
    for (int i = threadIdx.x; i < 6 * D.tp; i += kResThreads) res_smem[kResCpml + i] = D.cpml[6 * D.tp + i];
    if (threadIdx.x < 2 * kMaxHalf) {
        res_smem[threadIdx.x] = D.hx[threadIdx.x >> 1];
        res_smem[2 * kMaxHalf + threadIdx.x] = D.hz[threadIdx.x >> 1];
    } else if (threadIdx.x < 2 * kMaxHalf + 2) {
        res_smem[kResOne + threadIdx.x - 2 * kMaxHalf] = A.one;
    }
    for (int i = threadIdx.x; i < A.sim * (TWO ? 2 : 1); i += kResThreads) res_smem[A.fields + i] = 0.f;
    ResThread T;
    const int per_shot = A.t.ntx * A.t.ntz;
    T.b = blockIdx.x / per_shot;
    const int t = blockIdx.x - T.b * per_shot, tx = t % A.t.ntx, tz = t / A.t.ntx;
    {
        const int pairs = res_pairs(D.nxt, FP), nz = D.nzt - 2 * FP;
        const int p0 = res_cut(pairs, A.t.ntx, tx), r0 = res_cut(nz, A.t.ntz, tz);
        T.np = res_cut(pairs, A.t.ntx, tx + 1) - p0;
        T.nr = res_cut(nz, A.t.ntz, tz + 1) - r0;
        T.x0 = res_xb(FP) + 2 * p0;
        T.z0 = FP + r0;
        T.up = tz > 0 ? FP : 0;
        T.down = tz + 1 < A.t.ntz ? T.nr - FP : T.nr;
        const ResStrips st = res_strips(D.nzt, D.nxt, D.ppad, D.npml, D.fsurf);
        T.ztop = min(max(st.top - T.z0, 0), T.nr);
        T.zbot = min(max(st.bottom - T.z0, 0), T.nr);
        T.gw = T.np > 16 ? 32 : T.np > 8 ? 16 : 8;
        const int groups = min(T.nr, kResThreads / T.gw);
        const int gi = (int)threadIdx.x / T.gw;
        T.pi = (int)threadIdx.x & (T.gw - 1);
        T.ra = gi < groups ? res_cut(T.nr, groups, gi) : 0;
        T.rb = gi < groups ? res_cut(T.nr, groups, gi + 1) : 0;
        const int ix = T.x0 + 2 * T.pi;
        const PairCols pc = pair_cols<FP>(D, ix, true);
        T.fl = (pc.on0 ? RT_ON0 : 0u) | (pc.on1 ? RT_ON1 : 0u) | (pc.px[0] >= 0 ? RT_PX0 : 0u) |
               (pc.px[1] >= 0 ? RT_PX1 : 0u) | (ix < st.left ? RT_PLEFT : 0u);
        if (tx > 0) T.fl |= RT_LEFT;
        if (tx + 1 < A.t.ntx) T.fl |= RT_RIGHT;
        // left strip pairs of the tile, then its right strip pairs
        const int nl = min(max((st.left - T.x0 + 1) / 2, 0), T.np);
        const int fr = max((st.right - T.x0) / 2, 0);  // first pair with a column >= right
        T.xslot = ix < st.left ? T.pi : nl + T.pi - fr;
#pragma unroll
        for (int l = 0; l < 2; l++) {
            const int i = ix + l;
            if ((l ? pc.on1 : pc.on0) && i >= D.wx1 && i < D.wx2 && (i - D.wx1) % D.fwi_dx == 0)
                T.fl |= l ? RT_X1 : RT_X0;
        }
        // materials of this thread's cells
        const float* const mat[5] = {D.L, D.M2, D.MZX, D.BX, D.BZ};
        for (int row = T.ra; row < T.rb && T.pi < T.np; row++) {
            const size_t c = (size_t)(T.z0 + row) * D.pitch + ix;
            if (!inb((long long)c + 1, FWI_NFIELD(D), 51)) continue;
#pragma unroll
            for (int k = 0; k < 5; k++)
                res_put(res_smem + A.mat + (row * 5 + k) * kResTX + 2 * T.pi, ld2(mat[k] + c));
        }
        T.spec = T.spec_s = 0u;
        const bool edge = (T.fl & (RT_PX0 | RT_PX1)) || (T.fl & (RT_ON0 | RT_ON1)) != (RT_ON0 | RT_ON1);
        for (int row = T.ra; row < T.rb; row++) {
            const unsigned bit = 1u << (row - T.ra);
            if (edge || row < T.up || row >= T.down || row < T.ztop || row >= T.zbot) T.spec |= bit;
            if (D.fsurf && T.z0 + row <= 2 * FP) T.spec_s |= bit;
        }
        T.spec_s |= T.spec;
    }
    const ResHalo<FP> H(A, T, tx, tz);
    ResEvents ef = {-1, 0, -1, -1, -1, 0u, false}, ea = ef;
    const int2 *lf = nullptr, *la = nullptr;
    int nf = 0, na = 0;
    if (MODE != RES_STORED) {
        lf = A.ev_f + A.evo_f[blockIdx.x];
        nf = A.evo_f[blockIdx.x + 1] - A.evo_f[blockIdx.x];
        const bool fits = res_own_events(ef, T, lf, nf, G::RW, MODE == RES_FORWARD);
        ef.defer = __syncthreads_or(!fits);
        if (ef.defer) ef.ir = ef.rr = -1;
    }
    if (MODE != RES_FORWARD) {
        la = A.ev_a + A.evo_a[blockIdx.x];
        na = A.evo_a[blockIdx.x + 1] - A.evo_a[blockIdx.x];
        const bool fits = res_own_events(ea, T, la, na, G::RW, false);
        ea.defer = __syncthreads_or(!fits);
        if (ea.defer) ea.ir = -1;
    }
    // last tags sent after a velocity / stress pass, per simulation, and
    // whether the velocity halos are yet to be read
    unsigned tvf = A.tag0, tva = A.tag0, tsf = A.tag0, tsa = A.tag0;
    bool pend_f = false, pend_a = false;
    ResOp next = A.ops[0];
    for (int k = 0; k < A.nops; k++) {
        const ResOp op = next;
        if (k + 1 < A.nops) next = A.ops[k + 1];
        if (MODE != RES_STORED && op.kind == RES_ADV) {
            for (int it = op.a; it < op.b; it++) {
                const unsigned sf = MODE == RES_FORWARD && (op.flags & FL_STORE) && it % D.fwi_dt == 0 ? FL_STORE : 0u;
                if (!res_stress<FP, R, false, TWO>(A, T, H, pend_f, tvf, ++tsf, it, sf)) return;
                const unsigned vf = MODE == RES_FORWARD ? (unsigned)op.flags & (FL_WE | FL_RECORD) : 0u;
                if (!res_velocity<FP, R, false>(A, T, H, ef, 0, ++tvf, tsf, it, vf, lf, nf)) return;
                pend_f = true;
            }
        } else if (MODE != RES_FORWARD && op.kind == RES_ADJ) {
            for (int it = op.b - 1; it >= op.a; it--) {
                const unsigned sf = (op.flags & FL_GRAD) && it % D.fwi_dt == 0 ? FL_GRAD : 0u;
                if (!res_stress<FP, R, true, TWO>(A, T, H, pend_a, tva, ++tsa, it, sf)) return;
                if (!res_velocity<FP, R, true>(A, T, H, ea, TWO ? 1 : 0, ++tva, tsa, it, FL_WE, la, na)) return;
                pend_a = true;
            }
        } else if (MODE != RES_STORED && op.kind == RES_SAVE) {
            // (each thread writes and later reads its own cells only)
            res_state_io<FP>(A, T, 0, A.snap + T.b * A.state + op.a * A.slot_stride, true, false);
        } else if (MODE == RES_BOTH && op.kind == RES_RESTORE) {
            // other threads may still differentiate the old state; the halos of the
            // restored one come from the neighbours, as after a pass
            __syncthreads();
            res_state_io<FP>(A, T, 0, op.a < 0 ? nullptr : A.snap + T.b * A.state + op.a * A.slot_stride, false, false);
            res_send_velocities<FP>(A, T, 0, ++tvf);
            pend_f = true;
        } else if (op.kind == RES_FINAL) {
            res_state_io<FP>(A, T, TWO ? op.a : 0, (op.a ? A.a.vx : A.f.vx) + T.b * A.state, true, true);
        }
    }
}

}  // namespace fwi
