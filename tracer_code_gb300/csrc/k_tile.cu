// k_tile.cu -- FP32 smoother visits (iterate_stream, iterative_solver.f90:
// 860-963, with enforceBCs_stream after each sweep) on two-dimensional tiles
// with register patches: the smoother of the mixed solve.
//
// What bounds a sweep.  A level of 4K..260K points fits the chip's registers
// and shared memory, so a sweep is bound by instruction issue, shared-memory
// wavefronts and the latency of handing a tile's edge to its neighbours, not
// by HBM.  Two things cut those:
//
//   patches   a thread owns 2 columns x 2 or 4 rows and keeps their 13
//             operator coefficients, RHS, pseudo-time step and current values
//             in registers.  A sweep then takes 16 64-bit shared loads and 4
//             64-bit stores for 8 points (2 loads a point where one point a
//             thread takes 13), its multiply-add chains are independent;
//   halos     a tile carries a halo 2*S points deep and runs S sweeps
//             between exchanges: the points of the neighbouring tiles that
//             the later sweeps need are computed here too, from the same
//             coefficients and so with the same values, and the edge is
//             handed over once every S sweeps.
//
// A whole visit is one launch: of one thread-block cluster (a tile per CTA, up to
// 16 CTAs; levels of up to about 30K points), or of a cooperative grid (a tile
// per SM; larger levels).  Visits of 70 sweeps at 1024x256, with this kernel and
// with the kernels it took over from (one launch per sweep at level 1, six
// sweeps per launch at level 2, k_visit_cluster below): level 1 112 us against
// 197, level 2 65 against 82 (transfers to its neighbour levels included against
// not), level 3 42.6 against 50, level 4 24.5 against 30.
//
// Arithmetic per point is that of k_sweep32 / k_sweep_g32 (the folded taps in
// their order, c = 2/(cA + cB*temp) on the per-point Chebyshev level,
// v = fma(c*dt, r, psi)), so a level ends in the same state bit for bit as
// with one launch per sweep.
#include "tc_cluster.cuh"
#include "tc_device.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace {

constexpr int kMaxSweeps = 128;
constexpr int kMaxCluster = 16;
constexpr int kWaitLimit = 1 << 20;      // polls of a halo wait
constexpr int kTestWaitLimit = 1 << 14;  // polls of the timeout-path test's word
constexpr long long kDrain = 200000;     // cycles; edges land within about 1000
constexpr int PC = 2;                    // columns of a patch; its rows PR are a template parameter

// A tile's shared buffer starts HX columns left of its owned points and 2S rows
// above them: HX is 2S rounded up to a multiple of 4, so that edges move in
// 16-byte pieces.  Patches are laid out PL to a row (PW of them in use), PL a
// multiple of 16, and the row stride W is a compile-time multiple of 8: the
// patches of 16 consecutive threads lie in one row on different banks, and the
// stencil's offsets fold into the load instructions.
struct TileGeom {
    int S, HX;       // sweeps between exchanges; columns of the halo
    int TX, TY;      // owned points of a tile, multiples of 4
    int NX, NY;      // tiles across and down
    int W, R;        // shared buffer: row stride and rows
    int PW, PQ, PL;  // patches across and down the computed region; patches laid out per row
};

struct TileParams {
    Lay L;
    TileGeom G;
    int nsweeps, per_point, Vbc, g32;
    float c[kMaxSweeps];     // uniform Chebyshev/Richardson factor of sweep n
    float temp[kMaxSweeps];  // Chebyshev node of sweep n (per-point factor)
    FoldG32 F;               // weights of the viscosity fields (level 1)
    // transfers fused into the visit (nullptr: none), as k_visit_cluster's
    const float* ec;
    Lay Lc;
    float* rc;
    Lay Lr;
    float* zc;  // with the restriction: the coarser correction (layout Lr) set to zero
    const int* test_flag;
};

// ---- patches --------------------------------------------------------------------
// The two columns of a patch row travel together (64-bit shared loads and
// stores).  The packed FP32 instructions (fma.rn.f32x2) were tried for them and
// not kept: the taps one column off need register moves, and a sweep is bound by
// latency, not by multiply-add issue (256x64: 42.9 us a visit against 41.8).
typedef float2 f2;
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) { return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)); }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) { return make_float2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ f2 ld2(const float* p) { return *reinterpret_cast<const f2*>(p); }
__device__ __forceinline__ void st2(float* p, f2 v) { *reinterpret_cast<f2*>(p) = v; }
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

template <int PR>
struct Patch {
    f2 cf[PR][TC_NCOEF];  // negated coefficients (and the ghost taps' signs)
    f2 rh[PR], dt[PR];
    f2 own[PR];           // current values
};

// Taps that fall on a ghost (enforceBCs_stream): column -1 mirrors column 1 and
// a+1 mirrors a-1 (sign -1); row -1 mirrors row 1 and b+1 mirrors b-1 (sign
// zsgn).  Only a point's own value is mirrored into the ghost its taps reach, so
// a ghost's load is redirected to that value and the sign goes into the tap's
// coefficient (fma(-c, v, s) and fma(c, -v, s) round alike): no test and no
// select per sweep.  Where the ghost shares a load or a register with a wall
// (column a+1 when a is even, row b+1 when it lies inside the patch) patch_ghosts
// copies the value there.  Tile rows start at 1 modulo 4 and tile columns are
// even, so row 1 is a patch's first row and column 1 its second column.
struct PatchEdge {
    int l, r, t, b4, b5;  // offsets of the left and right pairs, of row -2, of the middle of row 4 and of row 5
    bool fix;             // patch_ghosts has work
    int jr, qb;           // the patch's column a-1 (or -1) and row b-1 (or -1)
};
template <int PR, int W>
__device__ __forceinline__ PatchEdge patch_edge(const Lay& L, int x, int y) {
    PatchEdge e;
    e.jr = (L.a - 1 - x >= 0 && L.a - 1 - x < PC) ? L.a - 1 - x : -1;
    e.qb = (L.b - 1 - y >= 0 && L.b - 1 - y < PR) ? L.b - 1 - y : -1;
    e.l = (x == 0) ? 0 : -2;
    e.r = (e.jr == 0) ? 0 : 2;
    e.t = (y == 1) ? 0 : -2 * W;
    e.b4 = (e.qb == PR - 2) ? (PR - 2) * W : PR * W;
    e.b5 = (e.qb == PR - 1) ? (PR - 1) * W : (PR + 1) * W;
    e.fix = e.jr == 1 || (e.qb >= 0 && e.qb < PR - 2);
    return e;
}

// coefficients and dt of the patch at (x, y): zero where a point is not an
// interior point of the level (its value then never changes)
template <int PR>
__device__ __forceinline__ void patch_coefs(Patch<PR>& P, const PatchEdge& E, const Lay& L, int x, int y,
                                            const float* __restrict__ coef, int g32, const FoldG32& F,
                                            const float* __restrict__ g, const float* __restrict__ dts, float zsgn) {
    const size_t pl = L.plane;
#pragma unroll
    for (int q = 0; q < PR; q++) {
        float cf[PC][TC_NCOEF], dt[PC];
#pragma unroll
        for (int j = 0; j < PC; j++) {
            const bool act = x + j >= 1 && x + j <= L.a - 1 && y + q >= 1 && y + q <= L.b - 1;
            const size_t xg = act ? IX(L, x + j, y + q) : 0;
            if (g32) {
                float G[5];
#pragma unroll
                for (int f = 0; f < 5; f++) G[f] = act ? __ldg(g + xg + f * pl) : 0.f;
                fold_from_fields(F, G, cf[j]);
#pragma unroll
                for (int d = 0; d < TC_NCOEF; d++) cf[j][d] = act ? cf[j][d] : 0.f;
            } else {
#pragma unroll
                for (int d = 0; d < TC_NCOEF; d++) cf[j][d] = act ? -__ldg(coef + xg + d * pl) : 0.f;
            }
            dt[j] = act ? __ldg(dts + xg) : 0.f;
            if (y == 1 && q == 0) cf[j][7] = zsgn * cf[j][7];
            if (E.qb == q) cf[j][8] = zsgn * cf[j][8];
        }
        if (x == 0) cf[1][3] = -cf[1][3];
        if (E.jr == 0) cf[0][4] = -cf[0][4];
        if (E.jr == 1) cf[1][4] = -cf[1][4];
#pragma unroll
        for (int d = 0; d < TC_NCOEF; d++) P.cf[q][d] = make_float2(cf[0][d], cf[1][d]);
        P.dt[q] = make_float2(dt[0], dt[1]);
    }
}
template <int PR>
__device__ __forceinline__ void patch_rhs(Patch<PR>& P, const Lay& L, int x, int y, const float* rhs) {
#pragma unroll
    for (int q = 0; q < PR; q++) {
        float r[PC];
#pragma unroll
        for (int j = 0; j < PC; j++) {
            const bool act = x + j >= 1 && x + j <= L.a - 1 && y + q >= 1 && y + q <= L.b - 1;
            r[j] = act ? ld_state(rhs + IX(L, x + j, y + q)) : 0.f;
        }
        P.rh[q] = make_float2(r[0], r[1]);
    }
}
template <int W, int PR>
__device__ __forceinline__ void patch_own(Patch<PR>& P, const float* p) {
#pragma unroll
    for (int q = 0; q < PR; q++) P.own[q] = ld2(p + q * W);
}
// (p: the patch's first point in the buffer its values were just put into)
template <int W, int PR>
__device__ __forceinline__ void patch_ghosts(Patch<PR>& P, const PatchEdge& E, float* p) {
    if (!E.fix) return;
    if (E.jr == 1) {
#pragma unroll
        for (int q = 0; q < PR; q++) p[q * W + 3] = P.own[q].y;
    }
#pragma unroll
    for (int q = 0; q + 2 < PR; q++)
        if (E.qb == q) P.own[q + 2] = P.own[q];
}

// r = rhs - A psi of the patch's points: the taps around it from shared
// memory (p: its first point), its own values from registers; the folded
// operator's tap order (0,0) (-1,0) (1,0) (-2,0) (2,0) (0,-1) (0,1) (0,-2)
// (0,2) (-1,-1) (1,-1) (-1,1) (1,1), the chains of the rows interleaved
template <int W, int PR>
__device__ __forceinline__ void patch_residual(const Patch<PR>& P, const PatchEdge& E, const float* p, f2 (&acc)[PR]) {
    const float *pl = p + E.l, *pr = p + E.r;
    // column pairs at offsets -2, 0, 2 (M) and -1, 1 (A, B) of rows -2..5
    f2 Lf[PR + 2], Rt[PR + 2], M[PR + 4], A[PR + 2], B[PR + 2];
    M[0] = ld2(p + E.t);
    M[1] = ld2(p - W);
    M[PR + 2] = ld2(p + E.b4);
    M[PR + 3] = ld2(p + E.b5);
#pragma unroll
    for (int q = 0; q < PR + 2; q++) {
        Lf[q] = ld2(pl + (q - 1) * W);
        Rt[q] = ld2(pr + (q - 1) * W);
        if (q >= 1 && q <= PR) M[q + 1] = P.own[q - 1];
    }
#pragma unroll
    for (int q = 0; q < PR + 2; q++) {
        A[q] = make_float2(Lf[q].y, M[q + 1].x);
        B[q] = make_float2(M[q + 1].y, Rt[q].x);
    }
#pragma unroll
    for (int q = 0; q < PR; q++) acc[q] = fma2(P.cf[q][0], M[q + 2], P.rh[q]);
#pragma unroll
    for (int q = 0; q < PR; q++) acc[q] = fma2(P.cf[q][1], A[q + 1], acc[q]);
#pragma unroll
    for (int q = 0; q < PR; q++) acc[q] = fma2(P.cf[q][2], B[q + 1], acc[q]);
#pragma unroll
    for (int q = 0; q < PR; q++) acc[q] = fma2(P.cf[q][3], Lf[q + 1], acc[q]);
#pragma unroll
    for (int q = 0; q < PR; q++) acc[q] = fma2(P.cf[q][4], Rt[q + 1], acc[q]);
#pragma unroll
    for (int q = 0; q < PR; q++) acc[q] = fma2(P.cf[q][5], M[q + 1], acc[q]);
#pragma unroll
    for (int q = 0; q < PR; q++) acc[q] = fma2(P.cf[q][6], M[q + 3], acc[q]);
#pragma unroll
    for (int q = 0; q < PR; q++) acc[q] = fma2(P.cf[q][7], M[q], acc[q]);
#pragma unroll
    for (int q = 0; q < PR; q++) acc[q] = fma2(P.cf[q][8], M[q + 4], acc[q]);
#pragma unroll
    for (int q = 0; q < PR; q++) acc[q] = fma2(P.cf[q][9], A[q], acc[q]);
#pragma unroll
    for (int q = 0; q < PR; q++) acc[q] = fma2(P.cf[q][10], B[q], acc[q]);
#pragma unroll
    for (int q = 0; q < PR; q++) acc[q] = fma2(P.cf[q][11], A[q + 2], acc[q]);
#pragma unroll
    for (int q = 0; q < PR; q++) acc[q] = fma2(P.cf[q][12], B[q + 2], acc[q]);
}

// one sweep of a patch: c2 the uniform factor in both halves, or (PP) the
// per-point Chebyshev factor 2 / (ca + cb * temp)
template <int W, bool PP, int PR>
__device__ __forceinline__ void patch_sweep(Patch<PR>& P, const PatchEdge& E, const f2 (&ca)[PR],
                                            const f2 (&cb)[PR], float c, float temp, const float* p, float* pn) {
    f2 acc[PR];
    patch_residual<W>(P, E, p, acc);
    // points that are not interior points keep their value (dt = 0): a wall
    // next to an interior point is stored again with it
#pragma unroll
    for (int q = 0; q < PR; q++) {
        const f2 cp = PP ? make_float2(2.0f / (ca[q].x + cb[q].x * temp), 2.0f / (ca[q].y + cb[q].y * temp))
                         : make_float2(c, c);
        P.own[q] = fma2(mul2(cp, P.dt[q]), acc[q], P.own[q]);
        st2(pn + q * W, P.own[q]);
    }
    patch_ghosts<W>(P, E, pn);
}

// ---- initial state ---------------------------------------------------------------
// bilinear prolongation of the coarse correction at fine point (i,k)
// (prolong, iterative_solver.f90:175-233), in k_prolong_add's order; the four
// corners are loaded whatever the parities, so that loads of several points
// are in flight together
__device__ __forceinline__ float prolong_at(const Lay& C, const float* ec, int i, int k) {
    const int i0 = i >> 1, i1 = (i + 1) >> 1, k0 = k >> 1, k1 = (k + 1) >> 1;
    const float e00 = ld_state(ec + IX(C, i0, k0)), e10 = ld_state(ec + IX(C, i1, k0));
    const float e11 = ld_state(ec + IX(C, i1, k1)), e01 = ld_state(ec + IX(C, i0, k1));
    const bool ie = (i & 1) == 0, ke = (k & 1) == 0;
    const float two = (e00 + (ie ? e01 : e10)) / 2.f;
    const float four = (e00 + e10 + e11 + e01) / 4.f;
    return (ie && ke) ? e00 : (ie || ke) ? two : four;
}
// the level's state at (ii,kk), ghosts and walls included, after the fused
// prolongation if there is one; 0 outside the ghost box
template <bool PRO>
__device__ __forceinline__ float start_value(const Lay& L, const Lay& C, const float* S, const float* ec, int ii,
                                             int kk, float zsgn) {
    const int a = L.a, b = L.b;
    if (ii < -SP || ii > a + SP || kk < -SP || kk > b + SP) return 0.f;
    const int mi = ii < 0 ? -ii : (ii > a ? 2 * a - ii : ii), mk = kk < 0 ? -kk : (kk > b ? 2 * b - kk : kk);
    const bool inner = PRO && mi >= 1 && mi <= a - 1 && mk >= 1 && mk <= b - 1;
    if (!inner) return ld_state(S + IX(L, ii, kk));
    const float si = (mi != ii) ? -1.f : 1.f, sk = (mk != kk) ? zsgn : 1.f;
    return (si * sk) * (ld_state(S + IX(L, mi, mk)) + prolong_at(C, ec, mi, mk));
}
// the tile's values (R rows of W from (gx, gy)) into NBUF buffers bsz apart;
// eight rows' loads of a warp are in flight before the first store
template <int W, int NBUF, bool PRO>
__device__ __forceinline__ void load_tile(float* buf, int bsz, int R, const Lay& L, const Lay& C, const float* S,
                                          const float* ec, int gx, int gy, float zsgn) {
    constexpr int U = 8;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, NW = blockDim.x >> 5;
    for (int c = lane; c < W; c += 32)
        for (int r0 = warp; r0 < R; r0 += U * NW) {
            float v[U];
#pragma unroll
            for (int u = 0; u < U; u++)
                v[u] = (r0 + u * NW < R) ? start_value<PRO>(L, C, S, ec, gx + c, gy + r0 + u * NW, zsgn) : 0.f;
#pragma unroll
            for (int u = 0; u < U; u++)
                if (r0 + u * NW < R) {
#pragma unroll
                    for (int q = 0; q < NBUF; q++) buf[q * bsz + (r0 + u * NW) * W + c] = v[u];
                }
        }
}

// ---- a whole visit in one launch ------------------------------------------------------
// The visit runs in periods of S sweeps, each followed by an exchange of the
// tiles' edges.  Two forms of the exchange:
//
// Cluster (GRID = false; a level of at most 16 tiles).  Period p reads its first
// sweep from buffer 2*(p&1) and alternates between that and 2*(p&1)+1; its last
// sweep writes the owned points into the first buffer of the other pair, from
// where, after a block barrier, the edges go to the neighbours' copies of the
// same buffer with st.async on their mbarriers.  A neighbour that is a period
// ahead therefore writes only buffers this CTA has left (it cannot be further
// ahead: it needs this CTA's edge of the period between).
//
// Grid (GRID = true; a tile per SM, a cooperative launch).  Edges go through
// the neighbours' inboxes in global memory, every value in one 64-bit word with
// the exchange's number: a word is taken when its number is right, so data and
// signal arrive together and no fence is needed.  An inbox has two sides used in
// turn; a side is written again only after its owner has sent the edge of the
// exchange between, i.e. after it has read the side.  Numbers go on from visit
// to visit: a level has one count per tile of its largest tiling, all of them
// equal between visits (the uniform and the per-point factor may take different
// tilings, so a visit also moves on the counts of tiles that it does not have).
//
// Waits are bounded: past the limit the CTA waits no more, finishes its loop
// and reports the timeout.  In a cluster it also arms its mbarriers no more (the
// phase it gave up on is still open) and, after the last cluster barrier, when
// every neighbour has sent its edges, stays for kDrain cycles while they land.
struct Exchange {
    unsigned long long* inbox;  // per tile 2 sides of W * R words (grid)
    unsigned* count;            // per tile of the level's largest tiling: exchanges so far (grid)
    int counts;                 // how many
};
__device__ __forceinline__ void st_words(unsigned long long* p, unsigned long long a, unsigned long long b) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void ld_words(const unsigned long long* p, unsigned long long& a, unsigned long long& b) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ unsigned long long word(float v, unsigned n) {
    return (unsigned long long)__float_as_uint(v) | ((unsigned long long)n << 32);
}

// (at most NT threads, one per laid-out patch, rounded up to a warp)
template <int W, int PR, int NT, bool PP, bool GRID>
__global__ void __launch_bounds__(NT, 1) k_tile_visit(const __grid_constant__ TileParams Q, float* Sg,
                                                      const float* __restrict__ coef, const float* __restrict__ g,
                                                      const float* rhs, const float* __restrict__ dts,
                                                      const float* __restrict__ cA, const float* __restrict__ cB,
                                                      float* res, int* timeout_flag, Exchange X) {
    const Lay& L = Q.L;
    const TileGeom& G = Q.G;
    const int a = L.a, b = L.b, S = G.S, HX = G.HX, nth = (int)blockDim.x;
    const int me = (int)blockIdx.x, tx = me % G.NX, ty = me / G.NX;  // one cluster: the CTA's rank is its index
    const int x0 = tx * G.TX, y0 = 1 + ty * G.TY;  // first owned column (column 0 is the wall) and row
    constexpr int NBUF = GRID ? 2 : 4;
    const int gx = x0 - HX, gy = y0 - 2 * S;  // buffer origin
    extern __shared__ __align__(16) unsigned char sm_raw[];
    unsigned long long* bar = reinterpret_cast<unsigned long long*>(sm_raw);  // 2 mbarriers (cluster)
    float* buf = reinterpret_cast<float*>(sm_raw + 32);
    const int bsz = W * G.R;
    uint3* push = reinterpret_cast<uint3*>(buf + NBUF * (size_t)bsz);
    const int tid = threadIdx.x;
    const float zsgn = (Q.Vbc == 1) ? 1.f : -1.f;
    const int pc = tid % G.PL, pr = tid / G.PL;
    const int x = x0 - 2 * (S - 1) + PC * pc, y = y0 - 2 * (S - 1) + PR * pr;
    const bool on = pc < G.PW && pr < G.PQ && x + PC - 1 >= 1 && x <= a - 1 && y + PR - 1 >= 1 && y <= b - 1;
    const int o = on ? (y - gy) * W + (x - gx) : 2 * W + 2;  // threads without a patch stay in the buffer
    // distance of the patch from the owned points: a sweep that is followed by
    // r more before the exchange is computed up to 2r points outside
    const int dist = max(max(max(x0 - (x + PC - 1), x - (x0 + G.TX - 1)), max(y0 - (y + PR - 1), y - (y0 + G.TY - 1))),
                         0);
    Patch<PR> P;
    f2 ca[PR], cb[PR];
    // coefficients, dt and Chebyshev denominators are fixed within a solve:
    // loaded before waiting for the previous kernel of the stream
    const PatchEdge E = patch_edge<PR, W>(L, x, y);
    patch_coefs(P, E, L, on ? x : -8, y, coef, Q.g32, Q.F, g, dts, zsgn);
    if (PP) {
#pragma unroll
        for (int q = 0; q < PR; q++) {
            float A[PC], B[PC];
#pragma unroll
            for (int j = 0; j < PC; j++) {
                const bool act = on && x + j >= 1 && x + j <= a - 1 && y + q >= 1 && y + q <= b - 1;
                A[j] = act ? __ldg(cA + IX(L, x + j, y + q)) : 1.f;
                B[j] = act ? __ldg(cB + IX(L, x + j, y + q)) : 0.f;
            }
            ca[q] = make_float2(A[0], A[1]);
            cb[q] = make_float2(B[0], B[1]);
        }
    }
    // the exchange list, in pieces of four columns: for each neighbour the owned
    // points within its halo (source, destination), and, rectangle for
    // rectangle, what comes back from it
    int expect = 0, np = 0;
    if (!GRID && tid == 0) {
        mbar_init(smem_addr(&bar[0]), 1);
        mbar_init(smem_addr(&bar[1]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int d = 0; d < 9; d++) {
        const int ox = d % 3 - 1, oy = d / 3 - 1;
        const int nx = tx + ox, ny = ty + oy;
        if (d == 4 || nx < 0 || nx >= G.NX || ny < 0 || ny >= G.NY) continue;
        const int sx = (ox > 0) ? G.TX : HX;  // first column and row in this CTA's buffer
        const int sy = (oy > 0) ? G.TY : 2 * S;
        const int wp = (ox == 0) ? G.TX / 4 : HX / 4, hh = (oy == 0) ? G.TY : 2 * S;
        const int rank = ny * G.NX + nx;
        uint32_t rb = 0, rbar = 0;
        if (!GRID) {
            rb = cluster_addr(smem_addr(buf), rank);
            rbar = cluster_addr(smem_addr(bar), rank);
        }
        for (int t = tid; t < wp * hh; t += nth) {
            const int cx = 4 * (t % wp), cy = t / wp;
            const int px = sx + cx, py = sy + cy;
            const int dst = (py - oy * G.TY) * W + px - ox * G.TX;
            const int rx = (ox < 0) ? 0 : (ox > 0 ? HX + G.TX : HX), ry = (oy < 0) ? 0 : (oy > 0 ? 2 * S + G.TY : 2 * S);
            push[np + t] = GRID ? make_uint3((unsigned)(py * W + px), (unsigned)(rank * 2 * bsz + dst),
                                             (unsigned)((ry + cy) * W + rx + cx))
                                : make_uint3((unsigned)(py * W + px), rb + 4u * (unsigned)dst, rbar);
        }
        np += wp * hh;
        expect += wp * hh * 16;
    }
    pdl_entry();
    const unsigned count0 = GRID ? __ldcg(X.count + me) : 0u;
    patch_rhs(P, L, on ? x : -8, y, rhs);
    if (Q.ec != nullptr) load_tile<W, NBUF, true>(buf, bsz, G.R, L, Q.Lc, Sg, Q.ec, gx, gy, zsgn);
    else load_tile<W, NBUF, false>(buf, bsz, G.R, L, L, Sg, nullptr, gx, gy, zsgn);
    if (GRID) __syncthreads();
    else cg::this_cluster().sync();  // buffers loaded and mbarriers initialised cluster-wide
    bool dead = false;
    if (Q.test_flag != nullptr) {
        int gave_up = 0;
        if (tid == 0) {
            int it = 0;
            while (*(volatile const int*)Q.test_flag == 0 && ++it <= kTestWaitLimit) {
            }
            gave_up = 1;
        }
        dead = __syncthreads_or(gave_up) != 0;
    }
    const bool need_res = res != nullptr || Q.rc != nullptr;
    float* mine = buf + o;
    const int reach = on ? (dist + 1) / 2 : 1 << 20;  // the patch is computed while that many sweeps or more follow
    int first = 0;  // the buffer the period starts from
    int p = 0;
    if (!dead) {
        for (int n0 = 0; n0 < Q.nsweeps; n0 += S, p++) {
            const int m = min(S, Q.nsweeps - n0);
            const bool exch = np > 0 && (n0 + S < Q.nsweeps || need_res);
            // the next kernel's launch and its loads of solve-constant data
            // overlap the last period (it waits for this grid's end before
            // touching anything else)
            if (n0 + S >= Q.nsweeps) pdl_done();
            const int alt = first ^ 1, next = GRID ? ((m & 1) ? alt : first) : 2 - (first & 2);
            float* from = mine + first * bsz;
            float* to = mine + alt * bsz;
            patch_own<W>(P, from);
            if (on) patch_ghosts<W>(P, E, from);
#pragma unroll 1
            for (int s = 0; s < m - 1; s++) {
                if (reach <= m - 1 - s)
                    patch_sweep<W, PP>(P, E, ca, cb, PP ? 0.f : Q.c[n0 + s], PP ? Q.temp[n0 + s] : 0.f, from, to);
                __syncthreads();
                float* t = from;
                from = to;
                to = t;
            }
            if (reach == 0)
                patch_sweep<W, PP>(P, E, ca, cb, PP ? 0.f : Q.c[n0 + m - 1], PP ? Q.temp[n0 + m - 1] : 0.f, from,
                                   mine + next * bsz);
            __syncthreads();
            first = next;
            if (!exch) continue;
            float* edge = buf + (size_t)next * bsz;
            if (GRID) {
                const unsigned n = count0 + (unsigned)p + 1u;
                const int side = (int)(n & 1u) * bsz;
                for (int t = tid; t < np; t += nth) {
                    const uint3 e = push[t];
                    const float4 v = ld4(edge + e.x);
                    unsigned long long* q = X.inbox + e.y + side;
                    st_words(q, word(v.x, n), word(v.y, n));
                    st_words(q + 2, word(v.z, n), word(v.w, n));
                }
                const unsigned long long* in = X.inbox + (size_t)me * 2 * bsz + side;
                for (int t = tid; t < np; t += nth) {
                    const unsigned at = push[t].z;
                    unsigned long long w0, w1, w2, w3;
                    int it = 0;
                    do {
                        ld_words(in + at, w0, w1);
                        ld_words(in + at + 2, w2, w3);
                        if (dead || ++it > kWaitLimit) {
                            dead = true;
                            break;
                        }
                    } while ((unsigned)(w0 >> 32) != n || (unsigned)(w1 >> 32) != n || (unsigned)(w2 >> 32) != n ||
                             (unsigned)(w3 >> 32) != n);
                    *reinterpret_cast<float4*>(edge + at) =
                        make_float4(__uint_as_float((unsigned)w0), __uint_as_float((unsigned)w1),
                                    __uint_as_float((unsigned)w2), __uint_as_float((unsigned)w3));
                }
                __syncthreads();
            } else {
                const int par = (p + 1) & 1;
                const uint32_t off = (uint32_t)(next * bsz) * 4u, boff = 8u * (uint32_t)par;
                if (tid == 0 && !dead) mbar_arrive_expect(smem_addr(&bar[par]), expect);
                for (int t = tid; t < np; t += nth) {
                    const uint3 e = push[t];
                    st_async4(e.y + off, ld4(edge + e.x), e.z + boff);
                }
                if (!dead) {
                    int it = 0;
                    while (!mbar_try_wait(smem_addr(&bar[par]), (p >> 1) & 1)) {
                        if (++it > kWaitLimit) { dead = true; break; }
                    }
                }
            }
        }
    }
    dead = __syncthreads_or(dead ? 1 : 0) != 0;
    if (GRID) {
        // every CTA counts the same exchanges, whether its waits ran out or not, and those
        // of the tiles beyond this visit's tiling
        for (int t = me + tid * (int)gridDim.x; t < X.counts; t += nth * (int)gridDim.x)
            X.count[t] = count0 + (unsigned)((Q.nsweeps + S - 1) / S);
    } else {
        cluster_arrive();  // this CTA's halos have landed: it needs no other CTA any more
    }
    if (dead) {
        if (tid == 0) atomicExch(timeout_flag, 1);
    } else {
        const bool owned = on && dist == 0;
        if (owned) {
#pragma unroll
            for (int q = 0; q < PR; q++)
#pragma unroll
                for (int j = 0; j < PC; j++)
                    if (x + j >= 1 && x + j <= a - 1 && y + q <= b - 1)
                        store_stream<float>(L, Sg, x + j, y + q, j ? P.own[q].y : P.own[q].x, Q.Vbc);
        }
        if (need_res) {
            float* rb = buf + (size_t)(first ^ 1) * bsz;
            if (on && dist <= 1) {
                f2 acc[PR];
                patch_own<W>(P, mine + first * bsz);
                patch_ghosts<W>(P, E, mine + first * bsz);
                patch_residual<W>(P, E, mine + first * bsz, acc);
#pragma unroll
                for (int q = 0; q < PR; q++)
#pragma unroll
                    for (int j = 0; j < PC; j++) {
                        const float r = j ? acc[q].y : acc[q].x;
                        if (Q.rc != nullptr) rb[o + q * W + j] = r;
                        else if (owned && x + j >= 1 && x + j <= a - 1 && y + q <= b - 1)
                            res[IX(L, x + j, y + q)] = r;
                    }
            }
            if (Q.rc != nullptr) {
                __syncthreads();
                // restrict (iterative_solver.f90:596-626; restrict9's terms and
                // order, the repeated corner included) for the coarse points
                // whose fine centre this CTA owns
                const int I0 = max(1, x0 / 2), I1 = min(Q.Lr.a - 1, (x0 + G.TX - 1) / 2);
                const int K0 = max(1, (y0 + 1) / 2), K1 = min(Q.Lr.b - 1, (y0 + G.TY - 1) / 2);
                const int ncol = I1 - I0 + 1, nrow = K1 - K0 + 1;
                for (int t = tid; ncol > 0 && t < nrow * ncol; t += nth) {
                    const int K = K0 + t / ncol, I = I0 + t % ncol;
                    const float* q = rb + (2 * K - gy) * W + (2 * I - gx);
                    const float corners = (q[-W - 1] + q[W - 1] + q[W + 1] + q[W - 1]) / 16.f;
                    const float sides = (q[-1] + q[-W] + q[1] + q[W]) / 8.f;
                    const float centre = q[0] / 4.f;
                    Q.rc[IX(Q.Lr, I, K)] = corners + sides + centre;
                }
                if (Q.zc != nullptr) {
                    // the coarser correction over this tile's footprint (its
                    // neighbours, which may still read it when they start, have
                    // started: they sent their edges), padding included
                    const int c0 = (tx == 0) ? 0 : x0 / 2 + SP, c1 = (tx == G.NX - 1) ? Q.Lr.ld : (x0 + G.TX) / 2 + SP;
                    const int r0 = (ty == 0) ? 0 : (y0 + 1) / 2 + SP,
                              r1 = (ty == G.NY - 1) ? Q.Lr.nk : (y0 + G.TY + 1) / 2 + SP;
                    const int nc = c1 - c0;
                    for (int t = tid; t < (r1 - r0) * nc; t += nth)
                        Q.zc[(size_t)(r0 + t / nc) * Q.Lr.ld + c0 + t % nc] = 0.f;
                }
            }
        }
    }
    if (!GRID) {
        cluster_wait();  // no CTA leaves while another may still write its shared memory
        if (dead)
            for (const long long t0 = clock64(); clock64() - t0 < kDrain;) {
            }
    }
}

// ---- host side ----------------------------------------------------------------------
// row strides that are compiled
constexpr int kStride[] = {40, 72, 104};

// geometry of NX x NY tiles with S sweeps per exchange; false if a tile is
// smaller than the halo or wider than the largest stride
bool geom(const Lay& L, int S, int PR, int NX, int NY, TileGeom* G) {
    const int cols = L.a, rows = L.b - 1;  // columns 0..a-1 (the wall rides along), rows 1..b-1
    G->S = S;
    G->HX = (2 * S + 3) / 4 * 4;
    G->TX = 4 * ((cols + 4 * NX - 1) / (4 * NX));
    G->TY = 4 * ((rows + 4 * NY - 1) / (4 * NY));
    G->NX = (cols + G->TX - 1) / G->TX;
    G->NY = (rows + G->TY - 1) / G->TY;
    if ((G->NX > 1 && G->TX < G->HX) || (G->NY > 1 && G->TY < 2 * S)) return false;
    G->PW = (G->TX + 4 * (S - 1)) / PC;
    G->PQ = (G->TY + 4 * (S - 1)) / PR;
    G->PL = (G->PW + 15) / 16 * 16;
    G->W = 0;
    for (int w : kStride)
        if (G->W == 0 && w >= G->TX + 2 * G->HX) G->W = w;
    G->R = G->TY + 4 * S;
    return G->W != 0;
}

struct VisitPlan {
    int PR, threads;
    TileGeom G;
    size_t smem;
};

// pushes of a tile with eight neighbours (at most)
int push_count(const TileGeom& G) {
    const int nx = G.NX > 2 ? 2 : G.NX - 1, ny = G.NY > 2 ? 2 : G.NY - 1;
    return ny * 2 * G.S * (G.TX / 4) + nx * (G.HX / 4) * G.TY + nx * ny * (G.HX / 4) * 2 * G.S;
}

int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Cycles of one sweep, a fit to measured visits (70 sweeps at 64x16..512x128):
// a latency per sweep, the warps of the busiest scheduler in turn, and an S-th
// of the exchange (about 0.45 us between the CTAs of a cluster, 1.5 us through
// global memory).
double sweep_cost(const TileGeom& G, int PR, int pushes, bool grid) {
    const int turns = ceil_div(ceil_div(G.PL * G.PQ, 32), 4);
    const double exchange = pushes > 0 ? (grid ? 3100.0 : 915.0) + pushes : 0.0;
    return (PR == 2 ? 60.0 + 130.0 * turns : 120.0 + 300.0 * turns) + exchange / G.S;
}

// The plan of a whole-visit launch: patch rows, tiles and sweeps per exchange of
// the least cost among those whose patches fit a CTA; false if the level needs
// more than `most` tiles.  Patches of 2 x 2 points have twice the warps of
// 2 x 4 to hide a sweep's latencies (128x32: 24.5 us a visit against 28.4, 64x16:
// 19.8 against 25.8, 256x64: 42.6 against 43.1), patches of 2 x 4 hold larger
// tiles (the register file); visits over the grid use 2 x 4.
bool visit_plan(const Lay& L, int most, bool grid, bool per_point, VisitPlan* best) {
    double cost = 1e30;
    for (int PR : {2, 4}) {
        if (PR == 2 && grid) continue;
        for (int S : {3, 5})
            for (int NX = 1; NX <= most; NX++)
                for (int NY = 1; NX * NY <= most; NY++) {
                    VisitPlan p;
                    p.PR = PR;
                    if (!geom(L, S, PR, NX, NY, &p.G) || p.G.NX != NX || p.G.NY != NY) continue;
                    p.threads = 32 * ceil_div(p.G.PL * p.G.PQ, 32);
                    if (p.threads > (PR == 2 ? 512 : per_point ? 256 : 384)) continue;
                    const int np = push_count(p.G);
                    p.smem = 32 + sizeof(float) * (grid ? 2 : 4) * (size_t)p.G.W * p.G.R + 16 + 12 * (size_t)np;
                    if (p.smem > 200 * 1024) continue;
                    // fewer CTAs among equals: the SMs they leave serve other cases
                    const double c = sweep_cost(p.G, PR, np, grid) * (1.0 + 1e-3 * NX * NY);
                    if (c < cost) {
                        cost = c;
                        *best = p;
                    }
                }
    }
    return cost < 1e30;
}

void fill_params(TileParams* Q, const Level& lv, const TileGeom& G, int nsweeps, const float* c, const float* temp,
                 int per_point, int Vbc) {
    Q->L = lv.L;
    Q->G = G;
    Q->nsweeps = nsweeps;
    Q->per_point = per_point;
    Q->Vbc = Vbc;
    for (int n = 0; n < nsweeps; n++) {
        Q->c[n] = c[n];
        Q->temp[n] = temp[n];
    }
    Q->g32 = lv.g32 != nullptr && lv.use_g32;
    Q->F = lv.gw;
    Q->ec = nullptr;
    Q->rc = nullptr;
    Q->zc = nullptr;
    Q->test_flag = nullptr;
}

struct VisitCall {
    const VisitPlan* p;
    const TileParams* Q;
    const Level* lv;
    float *S, *res;
    int* flag;
};

template <int W, int PR, int NT, bool PP, bool GRID>
int launch_visit(cudaStream_t s, const VisitCall& c) {
    auto k = k_tile_visit<W, PR, NT, PP, GRID>;
    static PerDevice set;
    if (set.get([k] {
            return (GRID || cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
                           cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) ==
                               cudaSuccess
                       ? 0
                       : -1;
        }) != 0)
        return 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(c.p->G.NX * c.p->G.NY), 1, 1);
    cfg.blockDim = dim3((unsigned)c.p->threads, 1, 1);
    cfg.dynamicSmemBytes = c.p->smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    if (GRID) {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.numAttrs = 1;
    } else {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = cfg.gridDim.x;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs = 2;
    }
    cfg.attrs = attr;
    const Level& lv = *c.lv;
    const Exchange X{lv.tile_inbox, lv.tile_count, lv.tile_counts};
    return cudaLaunchKernelEx(&cfg, k, *c.Q, c.S, (const float*)lv.coef32, (const float*)lv.g32,
                              (const float*)lv.rhs32, (const float*)lv.dts32, (const float*)lv.cA32,
                              (const float*)lv.cB32, c.res, c.flag, X) == cudaSuccess
               ? 0
               : 2;
}
template <int W, bool GRID>
int launch_visit_w(cudaStream_t s, const VisitCall& c) {
    if constexpr (!GRID) {
        if (c.p->PR == 2)
            return c.Q->per_point ? launch_visit<W, 2, 512, true, GRID>(s, c)
                                  : launch_visit<W, 2, 512, false, GRID>(s, c);
    }
    if (c.Q->per_point) return launch_visit<W, 4, 256, true, GRID>(s, c);
    return c.p->threads <= 256 ? launch_visit<W, 4, 256, false, GRID>(s, c) : launch_visit<W, 4, 384, false, GRID>(s, c);
}
template <bool GRID>
int launch_visit_any(cudaStream_t s, const VisitCall& c) {
    switch (c.p->G.W) {
        case 40: return launch_visit_w<40, GRID>(s, c);
        case 72: return launch_visit_w<72, GRID>(s, c);
        default: return launch_visit_w<104, GRID>(s, c);
    }
}

}  // namespace

// Can a visit of this level run as one cluster launch of k_tile_visit?
bool tile_visit_fits(const Lay& L, int nsweeps, int per_point) {
    VisitPlan p;
    return nsweeps <= kMaxSweeps && visit_plan(L, kMaxCluster, false, per_point != 0, &p);
}
// The inbox words and tiles of a visit over the grid (0 tiles: none)
int tile_grid_tiles(const Lay& L, int nsweeps, size_t* words) {
    int most = 0;
    *words = 0;
    for (int pp = 0; pp < 2; pp++) {
        VisitPlan p;
        if (nsweeps > kMaxSweeps || nsweeps <= 5 || !visit_plan(L, tc_sm_count(), true, pp != 0, &p)) continue;
        const size_t w = (size_t)p.G.NX * p.G.NY * 2 * p.G.W * p.G.R;
        if (w > *words) *words = w;
        if (p.G.NX * p.G.NY > most) most = p.G.NX * p.G.NY;
    }
    return most;
}

// A whole visit in one launch; 0 if it was launched, 1 if the level does not
// fit, 2 on a launch error.  res: the residual's plane (null: none).
int launch_tile_visit(cudaStream_t s, const Level& lv, bool grid, float* S, const float* c, const float* temp,
                      int nsweeps, int per_point, int Vbc, float* res, int* timeout_flag, const VisitXfer<float>* x,
                      const int* test_flag) {
    VisitPlan p;
    if (lv.no_cluster || nsweeps > kMaxSweeps || (grid && (nsweeps <= 5 || lv.tile_inbox == nullptr)) ||
        !visit_plan(lv.L, grid ? tc_sm_count() : kMaxCluster, grid, per_point != 0, &p))
        return 1;
    TileParams Q;
    fill_params(&Q, lv, p.G, nsweeps, c, temp, per_point, Vbc);
    if (x) {
        Q.ec = x->ec;
        Q.Lc = x->Lc;
        Q.rc = x->rc;
        Q.Lr = x->Lr;
        Q.zc = x->rc ? x->zc : nullptr;
    }
    Q.test_flag = test_flag;
    const VisitCall call{&p, &Q, &lv, S, res, timeout_flag};
    const int r = grid ? launch_visit_any<true>(s, call) : launch_visit_any<false>(s, call);
    if (r == 0) tc_note_launch();
    else cudaGetLastError();  // the caller's other kernels run instead: leave no error behind
    return r;
}
