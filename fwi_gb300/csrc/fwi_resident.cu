// The resident kernel: the whole time loop of a few shots in one launch, with
// their state in shared memory.
//
// A time step streams 16-20 bytes per cell through HBM when the state lives
// there, and its kernels start and end once per step.  Here a shot's grid is
// cut into tiles (fwi_resident.h), one thread block each; a block keeps its
// tile's two pressure levels and CPML memory variables in shared memory from
// the first step to the last, so a step touches global memory only for the
// tile edges, c2 (which stays in L2), the sources, the receivers and -- every
// store_snap steps -- the snapshots and the imaging accumulator.
//
// Tile edges travel as (value, step) pairs in 8-byte words, each stored and
// read whole: a block stores the R rows and four columns along each common edge
// into its outbox, and the neighbour polls the word until it carries the step
// it waits for, so that no fence and no separate flag stand between the two.
// Outboxes are double-buffered by step parity: a block overwrites the words
// of step k with those of step k+2 only after its neighbours have sent step
// k+1, which they do after they have read step k.  All blocks of a launch are
// resident together (cooperative launch); every wait has an iteration limit,
// after which the block sets *err and the launch ends.
//
// A block has twelve computing warps and four that exchange the edges, record
// the receivers and fetch the sources.  In a step the computing warps first
// update the cells that neighbours read (phase 0), announce that, and go on with
// the rest (phase 1); meanwhile the others send the edges of the new level and
// take in the neighbours' (of the new level too: its halo is read from the next
// step on).  One barrier ends the step.  With the exchange done by the computing
// threads -- two barriers a step, polling, sending -- a step of three 400 x
// 2000 shots took 6.2 us instead of 5.6, one of twelve 163 x 384 shots 4.3
// instead of 3.5, and one of 200 x 400 2.36 instead of 2.11 (now 5.0, 3.2 and
// 1.85: the row loops and the exchange have become shorter since).
//
// The arithmetic is that of fwi_step.cu, expression by expression (rounded
// multiplies and adds in the reference's order, no contraction): results are
// bit-identical to the streaming kernels and to the reference arithmetic.
#include "fwi_div.cuh"
#include "fwi_resident.cuh"
#include "fwi_stencil.cuh"

namespace fwi {

namespace {

constexpr int RES_ROWS = 3;  // rows that c2 of the interior quads is fetched ahead
constexpr int RES_WORDS = 4;  // pairs of edge words a thread sends or polls at a time
// Polls of one word: seconds, where a neighbour is at most microseconds behind.
// A constant of the build (the test of the error path builds a short one): as a
// launch parameter it cost the smallest grids 2.5 % of a step.
#ifndef FWI_RESIDENT_POLLS
#define FWI_RESIDENT_POLLS (1 << 22)
#endif
constexpr int SPIN_LIMIT = FWI_RESIDENT_POLLS;

// Edge words, one 64-bit access each.  The statements name no memory: nothing
// else of the launch is ordered against them but through the words themselves
// and the step's barriers.
__device__ __forceinline__ unsigned long long edge_word(float v, unsigned tag) {
    return (unsigned long long)tag << 32 | __float_as_uint(v);
}
__device__ __forceinline__ void put2(uint2* dst, float2 v, unsigned tag) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(dst), "l"(edge_word(v.x, tag)),
                 "l"(edge_word(v.y, tag)));
}
__device__ __forceinline__ uint4 get2(const uint2* src) {
    unsigned long long a, b;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(src));
    return make_uint4((unsigned)a, (unsigned)(a >> 32), (unsigned)b, (unsigned)(b >> 32));
}

// The block's barriers: all threads at the end of a step (true if any thread
// brought `bad`), and the first phase's end, which the computing threads only
// announce.
__device__ __forceinline__ bool step_done(bool bad) {
    unsigned r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 0, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((unsigned)bad)
        : "memory");
    return r != 0;
}
__device__ __forceinline__ void edges_done() {
    asm volatile("barrier.cta.arrive 1, %0;" ::"n"(RES_BLOCK) : "memory");
}
__device__ __forceinline__ void edges_wait() {
    asm volatile("barrier.cta.sync 1, %0;" ::"n"(RES_BLOCK) : "memory");
}

// A thread's work in one phase, packed: its quad's first column or its column
// (16 bits), its kind + 1 (3 bits; 0: none), its rows [ya, yb) (16 bits each).
struct ResWork {
    unsigned xk, rows, smask;
};
struct ResThread {
    const ResTile* t;      // in shared memory
    float* sm;             // the block's shared memory
    int kind, x, ya, yb;   // its quad's first column or its column; its rows
    unsigned smask;        // bit r: row ya + r has a source line
};

// c2 of the tile's quads: in shared memory, or in global memory (L2) where the
// pressure levels need the room.
__device__ __forceinline__ const float* tile_c2(const ResParams& P, const ResThread& h) {
    return h.t->o_c2 >= 0 ? h.sm + h.t->o_c2 : P.c2g + h.t->c2;
}

// The source values of row y of a thread's quad.
template <int MODE>
__device__ __forceinline__ void source_row(const ResThread& h, int y, int par, float* sv) {
    const ResTile& t = *h.t;
    const int line = reinterpret_cast<const int*>(h.sm + t.o_row)[y - t.y0];
    to_arr(ld4(h.sm + t.o_line + (par * t.lines[MODE] + line) * t.cp + h.x - t.x0), sv);
}

// Interior quads of the model rows.  The 2R+1 rows of p around the current one
// stay in registers, row r in slot r mod 9 of an unrolled loop of nine rows, so
// that none moves: a row takes five shared loads and a store of a quad, 24
// wavefronts a warp beside 48 (R = 3) packed-FP32 cycles.  c2, which may come
// from L2, is fetched three rows ahead; fetching the other values a row ahead
// was slower (5.26 instead of 5.04 us a step of three 400 x 2000 shots), as
// were three rows at a time with their 2R+3 rows loaded anew (5.6) and 16
// computing warps of 104 registers (7.1: spills).
template <int R, int MODE>
__device__ __forceinline__ void quads_interior(const ResParams& P, const ResThread& h, const float* cur, float* nxt,
                                               float4 (&c4)[RES_ROWS], int par) {
    constexpr int N = 9;
    static_assert(2 * R + 1 <= N && N % RES_ROWS == 0, "slots");
    const ResTile& t = *h.t;
    const int pitch = t.pitch, cp_ = t.cp, o = (h.ya - t.y0 + R) * pitch + h.x - t.x0 + 4;
    const float* pc = cur + o;
    float* pn = nxt + o;
    const float* cc = tile_c2(P, h) + (h.ya - t.y0) * cp_ + h.x - t.x0;
    int left = h.yb - h.ya;  // rows to go
    if (left <= 0) return;
    float2 cp[R + 1];
#pragma unroll
    for (int i = 0; i <= R; ++i) cp[i] = make_float2(P.c2[i], P.c2[i]);
    float4 q[N];
#pragma unroll
    for (int i = 0; i <= 2 * R; ++i) q[i] = ld4(pc + (i - R) * pitch);
    unsigned sm = h.smask;
    while (true) {
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const float4 L = ld4(pc - 4), Rt = ld4(pc + 4), pm = ld4(pn);
            float sv[4] = {0.f, 0.f, 0.f, 0.f};
            const bool src = sm & 1u;
            if (src) source_row<MODE>(h, h.yb - left, par, sv);
            float r[4];
            interior_update2f<R, true>([&](int i) { return q[(j + i) % N]; }, L, Rt, pm, c4[j % RES_ROWS], sv, cp, r, src);
            st4(pn, from_arr(r));
            if (left > RES_ROWS) c4[j % RES_ROWS] = ld4(cc + RES_ROWS * cp_);
            if (--left == 0) return;
            q[(j + 2 * R + 1) % N] = ld4(pc + (R + 1) * pitch);
            sm >>= 1;
            pc += pitch;
            pn += pitch;
            cc += cp_;
        }
    }
}

// The same rows one at a time on the steps that store a snapshot (MODE 0) or
// image (MODE 1: the next row's snapshot and accumulator values are fetched
// while a row is computed; blocks of two or three rows, their values loaded
// together, and an L2 prefetch a step ahead were not faster).
template <int R, int MODE>
__device__ __forceinline__ void quads_snapshot(const ResParams& P, const ResShot& S, const ResThread& h,
                                               const float* cur, float* nxt, int par, int snap) {
    constexpr bool IMG = MODE == 1;
    const ResTile& t = *h.t;
    const int pitch = t.pitch, o = (h.ya - t.y0 + R) * pitch + h.x - t.x0 + 4;
    const float* pc = cur + o;
    float* pn = nxt + o;
    const float* cc = tile_c2(P, h) + (h.ya - t.y0) * t.cp + h.x - t.x0;
    const size_t g0 = (size_t)h.ya * S.pitch + S.off + h.x;
    float* F = S.snaps + (size_t)snap * S.ny * S.pitch + g0;
    double* K = P.grad_form ? S.k64 + g0 : reinterpret_cast<double*>(S.k32 + g0);
    const size_t kp = P.grad_form ? S.pitch : S.pitch / 2;
    float4 c, f;
    double2 ka, kb;
    auto fetch = [&](int r, float4& cv, float4& fv, double2& a, double2& b) {
        cv = ld4(cc + r * t.cp);
        if (!IMG) return;
        fv = ldg4(F + (size_t)r * S.pitch);
        if (P.grad_form) ld_d4(K + r * kp, a, b);
        else a = *reinterpret_cast<const double2*>(K + r * kp);  // FP32 form: the row's four values
    };
    float2 cp[R + 1];
#pragma unroll
    for (int i = 0; i <= R; ++i) cp[i] = make_float2(P.c2[i], P.c2[i]);
    if (h.ya < h.yb) fetch(0, c, f, ka, kb);
#pragma unroll 1
    for (int y = h.ya, r = 0; y < h.yb; ++y, ++r) {
        float4 cn = c, fn = f;
        double2 kan = ka, kbn = kb;
        if (y + 1 < h.yb) fetch(r + 1, cn, fn, kan, kbn);
        float4 q[2 * R + 1];
#pragma unroll
        for (int i = 0; i <= 2 * R; ++i) q[i] = ld4(pc + (i - R) * pitch);
        const float4 pmv = ld4(pn);
        float p3[4], pm1[4], sv[4] = {0.f, 0.f, 0.f, 0.f};
        const bool src = (h.smask >> r) & 1u;
        if (src) source_row<MODE>(h, y, par, sv);
        interior_update2f<R, true>([&](int i) { return q[i]; }, ld4(pc - 4), ld4(pc + 4), pmv, c, sv, cp, p3, src);
        st4(pn, from_arr(p3));
        to_arr(pmv, pm1);
        if (MODE == 0) {
            // Fields = (p_3 - p_1)*0.5/dt  (solver_acoustic_SS.f90:447)
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = (p3[e] - pm1[e]) * 0.5f;
            div4_by_const(v, P.dt, P.rdt);
            st4(F + (size_t)r * S.pitch, from_arr(v));
        } else {
            // kernel += -0.5*(p_3-p_1)*Fields*store_snap  (:465-466)
            float fv[4], k2[4];
            to_arr(f, fv);
#pragma unroll
            for (int e = 0; e < 4; ++e) k2[e] = -(((0.5f * (p3[e] - pm1[e])) * fv[e]) * P.ss);
            if (P.grad_form == 0) {
                float4 kv;
                kv.x = __int_as_float(__double2loint(ka.x)) + k2[0];
                kv.y = __int_as_float(__double2hiint(ka.x)) + k2[1];
                kv.z = __int_as_float(__double2loint(ka.y)) + k2[2];
                kv.w = __int_as_float(__double2hiint(ka.y)) + k2[3];
                *reinterpret_cast<float4*>(K + r * kp) = kv;
            } else {
                ka.x += (double)k2[0];
                ka.y += (double)k2[1];
                kb.x += (double)k2[2];
                kb.y += (double)k2[3];
                st_d4(K + r * kp, ka, kb);
            }
        }
        c = cn;
        f = fn;
        ka = kan;
        kb = kbn;
        pc += pitch;
        pn += pitch;
    }
}

// Quads of the bottom pad rows: the bottom CPML strip (pml_matrices_y,
// solver_PML_matrices.f90:42-81).  The derivatives of the clamped rows are
// evaluated at the row they copy: p rows below nyt-1-R at row nyt-1-R, phi
// rows outside [R, dn-1-R] of the strip at its nearest end
// (solver_space_derivs.f90:38-53, :109-128).
template <int R>
__device__ __forceinline__ void quads_bottom(const ResParams& P, const ResShot& S, const ResThread& h,
                                             const float* cur, float* nxt, int k) {
    const ResTile& t = *h.t;
    const int pitch = t.pitch, cp_ = t.cp, dn = S.dn, ny = S.ny, last = ny + dn - 1 - R, par = k & 1;
    const int xo = h.x - t.x0;
    const float* phy = h.sm + t.o_y + (par ? dn * cp_ : 0) + xo;  // old y-phi, then the new one's place
    float* phn = h.sm + t.o_y + (par ? 0 : dn * cp_) + xo;
    float* chy = h.sm + t.o_y + 2 * dn * cp_ + xo;
    const float* fac = h.sm + t.o_fac;
    float2 c1p[R + 1], c2p[R + 1];
#pragma unroll
    for (int i = 0; i <= R; ++i) {
        c1p[i] = make_float2(P.c1[i], P.c1[i]);
        c2p[i] = make_float2(P.c2[i], P.c2[i]);
    }
#pragma unroll 1
    for (int y = h.ya; y < h.yb; ++y) {
        const int jl = y - ny, yc = min(y, last), jc = min(max(jl, R), dn - 1 - R);
        const float* pc = cur + (y - t.y0 + R) * pitch + xo + 4;
        const float* pd = cur + (yc - t.y0 + R) * pitch + xo + 4;
        const float4 C = ld4(pc), L = ld4(pc - 4), Rt = ld4(pc + 4);
        const float w[12] = {L.x, L.y, L.z, L.w, C.x, C.y, C.z, C.w, Rt.x, Rt.y, Rt.z, Rt.w};
        float* pn = nxt + (y - t.y0 + R) * pitch + xo + 4;
        const float4 PM = ld4(pn), CC = ld4(h.sm + t.o_cb + jl * cp_ + xo);
        const float4 PHY = ld4(phy + jl * cp_), CHY = ld4(chy + jl * cp_);
        const float2 Ap = make_float2(fac[jl], fac[jl]), Bp = make_float2(fac[dn + jl], fac[dn + jl]);
        float2 d2y[2], dy[2], dph[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) d2y[e] = dy[e] = dph[e] = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i <= R; ++i) {
            const float4 a = ld4(pd + i * pitch), b = ld4(pd - i * pitch);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float2 u = pr(a, e), d = pr(b, e);
                d2y[e] = __fadd2_rn(d2y[e], mul0(__fadd2_rn(u, d), c2p[i]));
                if (i) dy[e] = __fadd2_rn(dy[e], mul0(__fadd2_rn(u, make_float2(-d.x, -d.y)), c1p[i]));
            }
        }
#pragma unroll
        for (int i = 1; i <= R; ++i) {
            const float4 a = ld4(phy + (jc + i) * cp_), b = ld4(phy + (jc - i) * cp_);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float2 u = pr(a, e), d = pr(b, e);
                dph[e] = __fadd2_rn(dph[e], mul0(__fadd2_rn(u, make_float2(-d.x, -d.y)), c1p[i]));
            }
        }
        float phv[4], chv[4], p3[4];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float2 d2x = make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i <= R; ++i) {
                const int ia = 4 + 2 * e + i, ib = 4 + 2 * e - i;
                d2x = __fadd2_rn(d2x, mul0(c2p[i], make_float2(w[ia] + w[ib], w[ia + 1] + w[ib + 1])));
            }
            const float2 phyn = __fadd2_rn(mul0(Ap, pr(PHY, e)), mul0(Bp, dy[e]));
            const float2 chyn = __fadd2_rn(mul0(Ap, pr(CHY, e)), mul0(Bp, __fadd2_rn(d2y[e], dph[e])));
            const float2 prop = __fadd2_rn(dph[e], chyn);
            const float2 p = pr(C, e), pm = pr(PM, e);
            const float2 base = __fadd2_rn(make_float2(-pm.x, -pm.y), __fadd2_rn(p, p));
            const float2 r = __fadd2_rn(base, mul0(pr(CC, e), __fadd2_rn(__fadd2_rn(d2x, d2y[e]), prop)));
            phv[2 * e] = phyn.x;
            phv[2 * e + 1] = phyn.y;
            chv[2 * e] = chyn.x;
            chv[2 * e + 1] = chyn.y;
            p3[2 * e] = r.x;
            p3[2 * e + 1] = r.y;
        }
        st4(phn + jl * cp_, from_arr(phv));
        st4(chy + jl * cp_, from_arr(chv));
        st4(pn, from_arr(p3));
    }
}

// Side-strip columns, one per thread: the x-CPML strips with the grid-edge
// clamps and the interior columns next to them (model rows), the corners and
// the y-CPML columns next to them (bottom pad rows).  A clamped derivative is
// evaluated at the column or row it copies.
template <int R, int MODE, bool SNAP, bool BOT>
__device__ __forceinline__ void strip_columns(const ResParams& P, const ResShot& S, const ResThread& h,
                                              const float* cur, float* nxt, int k, int snap) {
    const ResTile& t = *h.t;
    const int pitch = t.pitch, cp_ = t.cp, dn = S.dn, ny = S.ny, nx = S.nx, nxt_ = nx + 2 * dn, par = k & 1;
    const int H = t.y1 - t.y0, col = h.x, xo = col - t.x0;
    const bool right = col >= dn + nx, xc = col < dn || right;  // x-CPML column
    const int il = right ? col - dn - nx : col;                 // its index in the dn-wide strip
    const int cfi = right ? il : dn - 1 - col;                  // its factor (solver_PML_matrices.f90:296-312)
    const int dcx = min(max(col, R), nxt_ - 1 - R) - col;       // column the p derivatives are taken at
    const int dci = min(max(il, R), dn - 1 - R);                // strip column the phi derivative is taken at
    const int ic = xc ? il : R;  // an index inside the strip arrays for every lane
    float* xb = h.sm + (right ? t.o_xr : t.o_xl);
    const float* phx = xb + (par ? H * dn : 0);
    float* phxn = xb + (par ? 0 : H * dn);
    float* chx = xb + 2 * H * dn;
    const float* phy = h.sm + t.o_y + (par ? dn * cp_ : 0) + xo;
    float* phyn_ = h.sm + t.o_y + (par ? 0 : dn * cp_) + xo;
    float* chy = h.sm + t.o_y + 2 * dn * cp_ + xo;
    const float* fac = h.sm + t.o_fac;
    const bool left = xo < t.nl;
    const float* c2 = h.sm + (left ? t.o_cl + xo : t.o_cr + col - (t.x1 - t.nr));
    const int c2p = left ? t.nl : t.nr;
    const bool src = !BOT && h.smask != 0;
    // the column's rows around the current one (model rows; a third of the loads
    // of a row would be theirs)
    float qy[2 * R + 1];
    if (!BOT) {
        const float* p0 = cur + (h.ya - t.y0) * pitch + xo + 4;
#pragma unroll
        for (int i = 0; i < 2 * R; ++i) qy[i + 1] = p0[i * pitch];
    }
    // lanes outside the x-CPML columns run the same row with phi = chi = 0
    // derivatives of their own (not used): no branch but the source line's
#pragma unroll 1
    for (int y = h.ya; y < h.yb; ++y) {
        const int row = y - t.y0, jl = y - ny;
        const float* pc = cur + (row + R) * pitch + xo + 4;
        if (!BOT) {
#pragma unroll
            for (int i = 0; i < 2 * R; ++i) qy[i] = qy[i + 1];
            qy[2 * R] = pc[R * pitch];
        }
        const float* px = pc + dcx;
        const float* py = BOT ? cur + (min(y, ny + dn - 1 - R) - t.y0 + R) * pitch + xo + 4 : pc;
        float* pn = nxt + (row + R) * pitch + xo + 4;
        const float* fx = phx + row * dn + dci;
        float2 a2 = make_float2(0.f, 0.f), a1 = make_float2(0.f, 0.f);  // (d2x, d2y), (dx, dy)
        float2 ap = make_float2(0.f, 0.f);                              // derivatives of the old (x-phi, y-phi)
        const float* fy = BOT ? phy + min(max(jl, R), dn - 1 - R) * cp_ : fx;
#pragma unroll
        for (int i = 0; i <= R; ++i) {
            const float2 hi = make_float2(px[i], BOT ? py[i * pitch] : qy[R + i]);
            const float2 lo = make_float2(px[-i], BOT ? py[-i * pitch] : qy[R - i]);
            const float2 t1 = make_float2(P.c1[i], P.c1[i]);
            a2 = __fadd2_rn(a2, mul0(__fadd2_rn(hi, lo), make_float2(P.c2[i], P.c2[i])));
            if (i) {
                a1 = __fadd2_rn(a1, mul0(__fadd2_rn(hi, make_float2(-lo.x, -lo.y)), t1));
                const float2 fh = make_float2(fx[i], BOT ? fy[i * cp_] : 0.f);
                const float2 fl = make_float2(fx[-i], BOT ? fy[-i * cp_] : 0.f);
                ap = __fadd2_rn(ap, mul0(__fadd2_rn(fh, make_float2(-fl.x, -fl.y)), t1));
            }
        }
        const float p = BOT ? pc[0] : qy[R], pm1 = *pn, c = c2[row * c2p];
        const float base = (-pm1) + 2.f * p, d2 = a2.x + a2.y;
        // corners: factor(max(i, j)) in both directions (solver_PML_coeffs.f90:240-267)
        const int fi = BOT ? (xc ? max(jl, cfi) : jl) : (xc ? cfi : 0);
        const float A = fac[fi], B = fac[dn + fi];
        const float phn = A * phx[row * dn + ic] + B * a1.x;
        const float chn = A * chx[row * dn + ic] + B * (a2.x + ap.x);
        const float propx = ap.x + chn;
        float p3;
        if (!BOT) {
            float sv = 0.f;
            if (src && ((h.smask >> (y - h.ya)) & 1u))
                sv = h.sm[t.o_line + (par * t.lines[MODE] + reinterpret_cast<const int*>(h.sm + t.o_row)[row]) * cp_ + xo];
            p3 = base + c * (d2 + (xc ? propx : sv));
        } else {
            const float pyn = A * phy[jl * cp_] + B * a1.y;
            const float cyn = A * chy[jl * cp_] + B * (a2.y + ap.y);
            const float propy = ap.y + cyn;
            // corners in two stages (solver_acoustic_SS.f90:395-411)
            p3 = xc ? (base + c * (d2 + propx)) + c * propy : base + c * (d2 + propy);
            phyn_[jl * cp_] = pyn;
            chy[jl * cp_] = cyn;
        }
        if (xc) {
            phxn[row * dn + il] = phn;
            chx[row * dn + il] = chn;
        }
        if (SNAP && !BOT && !xc) {
            const size_t g = (size_t)y * S.pitch + S.off + col;
            float* F = S.snaps + (size_t)snap * S.ny * S.pitch + g;
            if (MODE == 0) {
                *F = div_by_const((p3 - pm1) * 0.5f, P.dt, P.rdt);
            } else {
                const float k2 = -(((0.5f * (p3 - pm1)) * __ldg(F)) * P.ss);
                if (P.grad_form == 0) S.k32[g] = S.k32[g] + k2;
                else S.k64[g] += (double)k2;
            }
        }
        *pn = p3;
    }
}

// A pair of edge words: its first float in a pressure level's halo (bits
// 0-15), the side (bits 16-17), whether the second word exists (bit 18).
__device__ __forceinline__ unsigned edge_pair(int side, int dst, bool two) {
    return (unsigned)dst | (unsigned)side << 16 | (two ? 1u << 18 : 0u);
}

// Edge words of a communicating thread: edge_pair of each (0: none), the tile's
// own cell that it sends, the neighbour's word that it takes in.  W of them at
// a time: as many as the tile has for a thread, for the instructions of a pass
// are fetched anew in every step (tiny tiles with one or two: 1.66 -> 1.52 us).
struct EdgeWords {
    unsigned e[RES_WORDS];
    int cell[RES_WORDS], at[RES_WORDS];
};

// The tile's edges to its neighbours.
template <int W>
__device__ __forceinline__ void send_words(const float* p, uint2* own, unsigned k, const EdgeWords& w) {
    float2 v[W];
#pragma unroll
    for (int i = 0; i < W; ++i)
        if (w.e[i]) v[i] = *reinterpret_cast<const float2*>(p + w.cell[i]);
#pragma unroll
    for (int i = 0; i < W; ++i)
        if (w.e[i]) put2(own + 2 * i * RES_COMM, v[i], k);
}

// The neighbours' edges into the halo: all words that are not there yet are
// asked for together.  False when the wait runs out.
template <int W>
__device__ __forceinline__ bool receive_words(float* p, const uint2* out, unsigned k, const EdgeWords& w, int* err) {
    unsigned need = 0;
#pragma unroll
    for (int i = 0; i < W; ++i)
        if (w.e[i]) need |= 1u << i;
    for (int n = 0; need; ++n) {
        if (n > SPIN_LIMIT || ((n & 0xfff) == 0xfff && *(volatile int*)err)) return false;
        uint4 v[W];
#pragma unroll
        for (int i = 0; i < W; ++i)
            if (need >> i & 1) v[i] = get2(out + w.at[i]);
#pragma unroll
        for (int i = 0; i < W; ++i) {
            if (!(need >> i & 1) || v[i].y != k || ((w.e[i] >> 18) && v[i].w != k)) continue;
            *reinterpret_cast<float2*>(p + (w.e[i] & 0xffff)) =
                make_float2(__uint_as_float(v[i].x), __uint_as_float(v[i].z));
            need &= ~(1u << i);
        }
    }
    return true;
}

template <int R, int MODE>
__global__ void __launch_bounds__(RES_BLOCK, 1) k_resident(const __grid_constant__ ResParams P) {
    extern __shared__ float4 smem4[];
    // per-block constants live in shared memory: the row loops need the registers
    __shared__ ResTile tile;
    __shared__ ResShot shot;
    __shared__ int in[4];           // by side: pair b of this tile is word in + 2*b of its parity's plane
    float* sm = reinterpret_cast<float*>(smem4);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    {
        const int* src = reinterpret_cast<const int*>(P.tiles + blockIdx.x);
        int* dst = reinterpret_cast<int*>(&tile);
        for (int i = tid; i < (int)(sizeof(ResTile) / sizeof(int)); i += RES_BLOCK) dst[i] = src[i];
    }
    __syncthreads();
    const ResTile& t = tile;
    if (tid == 0) {
        shot = P.shots[t.shot];
        for (int s = 0; s < 4; ++s) {
            if (t.nbr[s] < 0) continue;
            const ResTile& n = P.tiles[t.nbr[s]];
            in[s] = n.out / 2 + 2 * (n.pair0[s ^ 1] - t.pair0[s]);
        }
    }
    __syncthreads();
    const ResShot& S = shot;
    const int H = t.y1 - t.y0, W = t.x1 - t.x0, dn = S.dn;
    for (int i = tid; i < t.floats / 4; i += RES_BLOCK) smem4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    // c2 = c**2*dt**2/d**2 with the nearest model cell in the pads
    // (solver_acoustic_SS.f90:271-292), Vp = sqrt(lambda/1000.)
    for (int i = tid; i < H * t.cp; i += RES_BLOCK) {
        const int x = i / H, y = i - x * H;
        const int my = min(t.y0 + y, S.ny - 1), mx = min(max(t.x0 + x - dn, 0), S.nx - 1);
        float v = __ldg(S.model + (size_t)my + (size_t)(S.x0 + mx) * S.ldv);
        if (P.from_lambda) v = __fsqrt_rn(__fdiv_rn(v, 1000.f));
        v = __fdiv_rn(__fmul_rn(__fmul_rn(v, v), P.dt2), P.d2);
        if (t.o_c2 >= 0) sm[t.o_c2 + y * t.cp + x] = v;
        else P.c2g[(size_t)t.c2 + y * t.cp + x] = v;
        if (x < t.nl) sm[t.o_cl + y * t.nl + x] = v;
        if (x < W && x >= W - t.nr) sm[t.o_cr + y * t.nr + x - (W - t.nr)] = v;
        if (t.y0 + y >= S.ny) sm[t.o_cb + (t.y0 + y - S.ny) * t.cp + x] = v;
    }
    for (int i = tid; i < H; i += RES_BLOCK) reinterpret_cast<int*>(sm + t.o_row)[i] = P.rows[t.rows[MODE] + i];
    for (int i = tid; i < dn; i += RES_BLOCK) {
        sm[t.o_fac + i] = P.fA[i];
        sm[t.o_fac + dn + i] = P.fB[i];
    }
    ResWork work[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        work[p] = ResWork{0, 0, 0};
        for (int g = p ? t.ngroups[0] : 0; g < t.ngroups[0] + (p ? t.ngroups[1] : 0); ++g) {
            const ResGroup& G = t.g[g];
            if (warp < G.warp0 || warp >= G.warp0 + G.nwarps) continue;
            const int i = (warp - G.warp0) * 32 + lane, b = i / G.np, c = i - b * G.np;
            if (c >= G.n) continue;
            const int ya = min(G.y0 + b * G.h, G.y1), yb = min(ya + G.h, G.y1);
            work[p].xk = (unsigned)(G.x0 + (G.kind < 2 ? 4 * c : c)) | (unsigned)(G.kind + 1) << 16;
            work[p].rows = (unsigned)ya | (unsigned)yb << 16;
            for (int y = ya; y < yb; ++y)
                if (P.rows[t.rows[MODE] + y - t.y0] >= 0) work[p].smask |= 1u << (y - ya);
        }
    }
    auto unpack = [&](const ResWork& w) {
        ResThread h;
        h.t = &tile;
        h.sm = sm;
        h.kind = (int)(w.xk >> 16) - 1;
        h.x = (int)(w.xk & 0xffff);
        h.ya = (int)(w.rows & 0xffff);
        h.yb = (int)(w.rows >> 16);
        h.smask = w.smask;
        return h;
    };
    // c2 of the first rows of a phase's interior quads, on its way while the
    // threads poll or wait
    float4 c4[RES_ROWS];
    auto load_c2 = [&](const ResWork& w) {
        const ResThread h = unpack(w);
        if (h.kind != 0) return;
        const float* cc = tile_c2(P, h) + (h.ya - t.y0) * t.cp + h.x - t.x0;
#pragma unroll
        for (int j = 0; j < RES_ROWS; ++j)
            if (h.ya + j < h.yb) c4[j] = ld4(cc + j * t.cp);
    };
    // the pairs of edge words this tile reads
    unsigned* const pairs = reinterpret_cast<unsigned*>(sm + t.o_pair);
    const int npair = t.npair;
    {
        int at = 0;
        for (int s = 0; s < 4; ++s) {
            if (t.nbr[s] < 0) continue;
            const int w2 = (W + 1) / 2, n = s < 2 ? 2 * H : R * w2;
            for (int i = tid; i < n; i += RES_BLOCK) {
                if (s < 2) {
                    const int y = i >> 1, x = 2 * (i & 1);
                    pairs[at + i] = edge_pair(s, (R + y) * t.pitch + (s ? 4 + W : 0) + x, true);
                } else {
                    const int y = i / w2, x = 2 * (i - y * w2);
                    pairs[at + i] = edge_pair(s, (s == 2 ? y : R + H + y) * t.pitch + 4 + x, x + 1 < W);
                }
            }
            at += n;
        }
    }
    // the tile's receivers and sources; the value of a thread's first source is fetched a step ahead
    const int nrec = MODE == 0 && P.record ? t.rec1 - t.rec0 : 0, nsrc = t.src1[MODE] - t.src0[MODE];
    ResRec* const recs = reinterpret_cast<ResRec*>(sm + t.o_rec);
    ResSrc* const srcs = reinterpret_cast<ResSrc*>(sm + t.o_src);
    for (int i = tid; i < nrec; i += RES_BLOCK) recs[i] = P.rec[t.rec0 + i];
    for (int i = tid; i < nsrc; i += RES_BLOCK) srcs[i] = P.src[t.src0[MODE] + i];
    const bool comm = tid >= RES_THREADS;
    if (comm) {
        // source values of step k, S(k-1, j), into the lines of its parity
        const int ct = tid - RES_THREADS;
        auto sources = [&](int k) {
#pragma unroll 1
            for (int e = ct; e < nsrc; e += RES_COMM) {
                const ResSrc en = srcs[e];
                sm[t.o_line + (k & 1) * t.lines[MODE] * t.cp + en.pos] =
                    __ldg(S.srcv + (size_t)en.vidx * P.nt + (k - 2));
            }
        };
        // receivers of level k (:551-555)
        auto record = [&](int k) {
            const float* p = sm + t.o_p[k & 1];
#pragma unroll 1
            for (int e = ct; e < nrec; e += RES_COMM) {
                const float v = p[recs[e].off];
                float* at = S.rec + (size_t)recs[e].ridx * P.nt;
                at[k - 2] = v;
                if (k == P.nt) at[P.nt - 1] = v;  // Rec_point(nt,:) = Rec_point(nt-1,:)  (solver_acoustic_SS.f90:588)
            }
        };
        __syncthreads();
        sources(2);
        // The thread's pairs, RES_WORDS at a time: where the words from pair b0 on
        // lie (e: edge_pair, 0 beyond the last one).
        const int in0 = in[0], in1 = in[1], in2 = in[2], in3 = in[3], rows = R * t.pitch;
        auto words = [&](EdgeWords& w, int b0, const unsigned* e) {
#pragma unroll
            for (int i = 0; i < RES_WORDS; ++i) {
                // a pair's own cell lies R rows or four columns inside the halo cell that the same pair reads
                const bool hi = e[i] >> 16 & 1, row = e[i] >> 17 & 1;
                const int off = row ? rows : 4;
                w.e[i] = e[i];
                w.cell[i] = (int)(e[i] & 0xffff) + (hi ? -off : off);
                w.at[i] = (row ? (hi ? in3 : in2) : (hi ? in1 : in0)) + 2 * (b0 + i * RES_COMM);
            }
        };
        constexpr int STRIDE = RES_WORDS * RES_COMM;
        __syncthreads();
        // those of the first passes stay in registers: shared loads take long while the others compute
        EdgeWords first, more;
        unsigned e[RES_WORDS], second[RES_WORDS];
        auto load = [&](int b0, unsigned* e) {
#pragma unroll
            for (int i = 0; i < RES_WORDS; ++i) e[i] = b0 + i * RES_COMM < npair ? pairs[b0 + i * RES_COMM] : 0;
        };
        load(ct, e);
        words(first, ct, e);
        load(ct + STRIDE, second);
        auto next_words = [&](int b0) {
            if (b0 >= 2 * STRIDE) {
                load(b0, e);
                words(more, b0, e);
            } else {
                words(more, b0, second);
            }
        };
        const int nwords = (npair + RES_COMM - 1) / RES_COMM;  // of a thread
        for (int k = 2; k <= P.steps; ++k) {
            float* nxt = sm + t.o_p[k & 1];
            uint2* out = P.out + (k & 1) * P.plane;
            uint2* own = out + t.out / 2 + 2 * ct;
            const unsigned tag = (unsigned)k;
            if (k > 2) record(k - 1);
            bool ok = true;
            if (k < P.steps) {
                sources(k + 1);
                edges_wait();
                if (nwords <= 1) send_words<1>(nxt, own, tag, first);
                else if (nwords == 2) send_words<2>(nxt, own, tag, first);
                else if (nwords == 3) send_words<3>(nxt, own, tag, first);
                else send_words<RES_WORDS>(nxt, own, tag, first);
#pragma unroll 1
                for (int b0 = ct + STRIDE; b0 < npair; b0 += STRIDE) {
                    next_words(b0);
                    send_words<RES_WORDS>(nxt, own + 2 * (b0 - ct), tag, more);
                }
                if (nwords <= 1) ok = receive_words<1>(nxt, out, tag, first, P.err);
                else if (nwords == 2) ok = receive_words<2>(nxt, out, tag, first, P.err);
                else if (nwords == 3) ok = receive_words<3>(nxt, out, tag, first, P.err);
                else ok = receive_words<RES_WORDS>(nxt, out, tag, first, P.err);
#pragma unroll 1
                for (int b0 = ct + STRIDE; b0 < npair && ok; b0 += STRIDE) {
                    next_words(b0);
                    ok = receive_words<RES_WORDS>(nxt, out, tag, more, P.err);
                }
            }
            if (step_done(!ok)) {
                if (ct == 0) *(volatile int*)P.err = 1;
                return;
            }
        }
        record(P.steps);
        return;
    }
    __syncthreads();
    __syncthreads();
    int l = 1, snap = MODE == 0 ? 0 : P.nt_store;
    for (int k = 2; k <= P.steps; ++k) {
        const float* cur = sm + t.o_p[(k - 1) & 1];
        float* nxt = sm + t.o_p[k & 1];
        const int par = k & 1;
        load_c2(work[0]);
        bool ev = false;
        if (++l == P.store_snap) {
            l = 0;
            ev = MODE == 1 || P.store;
            if (MODE == 0) ++snap;
            else --snap;
        }
        // the cells the neighbours read (phase 0), then the rest
#pragma unroll 1
        for (int ph = 0; ph < 2; ++ph) {
            const ResThread h = unpack(ph ? work[1] : work[0]);
            if (h.kind == 0) {
                if (ev) quads_snapshot<R, MODE>(P, S, h, cur, nxt, par, snap);
                else quads_interior<R, MODE>(P, h, cur, nxt, c4, par);
            } else if (h.kind == 1) {
                quads_bottom<R>(P, S, h, cur, nxt, k);
            } else if (h.kind == 2) {
                if (ev) strip_columns<R, MODE, true, false>(P, S, h, cur, nxt, k, snap);
                else strip_columns<R, MODE, false, false>(P, S, h, cur, nxt, k, -1);
            } else if (h.kind == 3) {
                strip_columns<R, MODE, false, true>(P, S, h, cur, nxt, k, snap);
            }
            if (ph) break;
            if (k < P.steps) edges_done();
            load_c2(work[1]);
        }
        if (step_done(false)) return;
    }
}

using ResKernel = void (*)(const ResParams);

ResKernel kernel_of(int acc, int mode) {
    if (acc == 3) return mode == 0 ? k_resident<3, 0> : k_resident<3, 1>;
    return mode == 0 ? k_resident<4, 0> : k_resident<4, 1>;
}

}  // namespace

cudaError_t configure_resident() {
    int dev = 0, most = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    for (int acc = 3; acc <= 4; ++acc)
        for (int mode = 0; mode < 2; ++mode) {
            ResKernel k = kernel_of(acc, mode);
            cudaFuncAttributes a;
            if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, k);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)a.sharedSizeBytes);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout,
                                         cudaSharedmemCarveoutMaxShared);
        }
    return e;
}

cudaError_t resident_blocks(int acc, size_t smem, int* blocks) {
    int a = 0, b = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, kernel_of(acc, 0), RES_BLOCK, smem);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kernel_of(acc, 1), RES_BLOCK, smem);
    *blocks = a < b ? a : b;
    return e;
}

cudaError_t launch_resident(int acc, int mode, const ResParams& p, int tiles, size_t smem, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)tiles);
    cfg.blockDim = dim3(RES_BLOCK);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeCooperative;  // every block resident, or the launch fails
    at.val.cooperative = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel_of(acc, mode), p);
}

}  // namespace fwi
