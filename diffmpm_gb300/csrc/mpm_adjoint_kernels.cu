// Reverse passes of the explicit MPM step (USF or USL, per-step volume set-up).
//
// Notation of the forward USF step, particle p in cell c with corners k = 0..3
// (diffmpm/element.py, particle.py; the step order of diffmpm/scheme.py:22-67;
// USL, scheme.py:112-133, uses sig and V0 in F and updates sig, rho after G2P
// with r = flush(G^T vB), c = flush(Gc^T vB) at the start-of-step positions):
//   m    = V0 rho,           V0 = V_el / count(c)            (solver.py:81-85)
//   M_n  = sum N m,  P_n = flush(sum N m v),  vA = C(flush(P / M))
//   r    = flush(G^T vA) (xx, yy, xy),  c = flush(Gc^T vA),  dvol = dt (c0 + c1)
//   sig' = sig + D(E) r dt,  V = V0 (1 + dvol),  rho' = rho / (1 + dvol)
//   F_n  = sum -V (Gx sxx' + Gy sxy', Gy syy' + Gx sxy') + N m g
//   a    = F / M,  vB = flush(C(vA + a dt)),  aB = flush(C0(a))
//   v'   = velocity_update ? sum N vB : v + dt sum N aB,  x' = x + dt sum N vB
// C sets constrained velocity components, C0 zeroes constrained accelerations.
// flush(a) = 0 for |a| < 1e-12, so its derivative is 0 there and 1 elsewhere:
// a component that is exactly 0 after the flush passes no adjoint.  Cell ids,
// counts and masks are piecewise constant in the positions and pass none.
// The velocity a node with zero mass keeps from the previous step only
// reaches particles whose shape function at that node is exactly zero, so its
// dependence is dropped.
#include <cuda_runtime.h>
#include <cstdint>
#include "mpm_adjoint.h"
#include "mpm_device.cuh"

namespace mpm {

namespace {

constexpr int PART_THREADS = 256;
static_assert(PART_THREADS == ADJ_BLOCK, "the batched block map counts ADJ_BLOCK particles per chunk");

// Particles currently in cell (ci, cj) at the step start, in the order of the
// forward gathers: the cell's own sort-cell, and neighbouring sort-cells whose
// drift flag is set (positions tested).
template <class F>
__device__ __forceinline__ void visit_tape_cell(const AdjStep& A, int ci, int cj, const CellGeo& g,
                                                F&& f) {
    #pragma unroll 1
    for (int dj = -1; dj <= 1; ++dj) {
        const int sj = cj + dj;
        if (sj < 0 || sj >= A.ny) continue;
        #pragma unroll 1
        for (int di = -1; di <= 1; ++di) {
            const int si = ci + di;
            if (si < 0 || si >= A.nx) continue;
            const int s = sj * A.nx + si;
            const bool flagged = A.cflag[s] != 0;
            if (!(di == 0 && dj == 0) && !flagged) continue;
            const int b = A.cstart[s], e = A.cstart[s + 1];
            #pragma unroll 1
            for (int q = b; q < e; ++q) {
                if (flagged && !in_cell(g, A.x[q], A.y[q])) continue;
                f(q);
            }
        }
    }
}

__device__ __forceinline__ void particle_cell(const AdjStep& A, float x, float y, int& ci, int& cj) {
    ci = min(max(locate_axis(x, A.hx, A.nx), 0), A.nx - 1);
    cj = min(max(locate_axis(y, A.hy, A.ny), 0), A.ny - 1);
}

// Batched launches: the CTA copies its simulation's arguments into shared
// memory (one word per thread).
__device__ __forceinline__ void load_step_args(const AdjStep* __restrict__ src, AdjStep& dst) {
    static_assert(sizeof(AdjStep) % 4 == 0, "arguments copied in 4-byte words");
    const int* a = reinterpret_cast<const int*>(src);
    int* b = reinterpret_cast<int*>(&dst);
    for (int i = threadIdx.x; i < (int)(sizeof(AdjStep) / 4); i += blockDim.x) b[i] = a[i];
    __syncthreads();
}

// Adjoint seeds of G2P: (v-hat bar, a-hat bar) of a particle.
__device__ __forceinline__ void g2p_seeds(const AdjStep& A, float lx, float ly, float lvx, float lvy, float& gx,
                                          float& gy, float& hx, float& hy) {
    gx = fm(lx, A.dt);
    gy = fm(ly, A.dt);
    if (A.velocity_update) {
        gx = fa(gx, lvx);
        gy = fa(gy, lvy);
        hx = 0.0f;
        hy = 0.0f;
    } else {
        hx = fm(lvx, A.dt);
        hy = fm(lvy, A.dt);
    }
}

// ---------------------------------------------------------------------------
// Tiles of the two node passes: the forward kernels' tiles (a CTA of
// TILE_THREADS threads covers TILE_CX x TILE_CY cells and owns the nodes at
// the upper-right corners of all but its first column and row), with each
// thread summing the corner contributions of its cell's particles.  Fast
// path: the cell rows are staged with coalesced 16-byte copies (row_pass16),
// issued before the drift flags are known; slow path (a particle near the tile
// was outside its sort-cell at the step start): the tape's drift flags and
// visit_tape_cell.
// ---------------------------------------------------------------------------

// Slots of a staged row per pass of the reverse node passes: a row of 4
// particles in each of 32 cells, starting anywhere in a 16-byte piece, fits
// one pass.  The staged arrays (tape slots, adjoint and scratch arrays) start
// on 16-byte boundaries and hold a multiple of 4 slots.
constexpr int REV_ROW_P = 132;

// Reverse nodal update of node n from the G2P adjoint sums (vB-bar, aB-bar):
// vB = flush(C(vA + a dt)), aB = flush(C0(a)), a = F / M (element.py:305-329).
// USL adds the vB-bar of its stress update, gathered by pass G into vabx, vaby.
template <bool USL>
__device__ __forceinline__ void rev_node_update(const AdjStep& A, int n, float vbx, float vby,
                                                float abx, float aby) {
    if (USL) {
        vbx = fa(vbx, A.vabx[n]);
        vby = fa(vby, A.vaby[n]);
    }
    float fbx = 0.0f, fby = 0.0f, mb = 0.0f, wbx = 0.0f, wby = 0.0f;
    const float M = A.nm[n];
    if (M != 0.0f) {
        const uint16_t code = A.ncons[n];
        const bool cx = (code & 0xff) != 0, cy = (code >> 8) != 0;
        const float vBx = A.nvbx[n], vBy = A.nvby[n], aBx = A.nax[n], aBy = A.nay[n];
        wbx = (cx || vBx == 0.0f) ? 0.0f : vbx;
        wby = (cy || vBy == 0.0f) ? 0.0f : vby;
        const float ax = fa((cx || aBx == 0.0f) ? 0.0f : abx, fm(wbx, A.dt));
        const float ay = fa((cy || aBy == 0.0f) ? 0.0f : aby, fm(wby, A.dt));
        fbx = fdv(ax, M);
        fby = fdv(ay, M);
        mb = -fdv(fa(fm(ax, aBx), fm(ay, aBy)), M);
    }
    A.fbx[n] = fbx;
    A.fby[n] = fby;
    A.mb[n] = mb;
    A.vabx[n] = wbx;
    A.vaby[n] = wby;
}

// ---------------------------------------------------------------------------
// Pass 1: transposed G2P (v-hat bar = x-bar dt [+ v-bar], a-hat bar = v-bar dt
// gathered to the nodes with the shape functions), the reverse nodal update
// and the particle count of every cell (particle.py:208-247, element.py:305-329).
// ---------------------------------------------------------------------------
template <bool USL>
__device__ __forceinline__ void rev_nodal_update_tile(const AdjStep& A, const int4 T) {
    constexpr int NQ = 16;   // [v-hat bar x, y, a-hat bar x, y] x corner
    __shared__ float s_c[NQ][SC_STRIDE];
    __shared__ __align__(16) float s_row[TILE_CY][6][REV_ROW_P];
    __shared__ TileGeo G;
    const int tid = threadIdx.x, tx = tid % TILE_CX, ty = tid / TILE_CX;
    const int c0x = T.y * TILE_NX - 1, c0y = T.z * TILE_NY - 1;
    const int ci = c0x + tx, cj = c0y + ty;
    const TileLoads L = tile_loads(A, c0x, c0y, cj, tx);
    const bool node_ok = tx < TILE_NX && ty < TILE_NY && c0x + 1 + tx <= A.nx && c0y + 1 + ty <= A.ny;
    const int node = (c0y + 1 + ty) * (A.nx + 1) + c0x + 1 + tx;
    const bool own_cell = tx >= 1 && ty >= 1 && ci < A.nx && cj < A.ny;
    build_geo(A, c0x, c0y, G);
    const RowRange R(L, tx);
    const float* const src[6] = {A.x, A.y, A.lx, A.ly, A.lvx, A.lvy};
    float (*buf)[REV_ROW_P] = s_row[ty];
    row_issue16<6, REV_ROW_P>(buf, src, R.rb & ~3, R.re, tx);
    const bool slow = __syncthreads_or(L.drift()) != 0;
    const CellGeo g = geo_of(G, tx + 1, ty + 1);
    float acc[NQ];
    #pragma unroll
    for (int k = 0; k < NQ; ++k) acc[k] = 0.0f;
    int cnt = 0;
    auto add = [&](float x, float y, float lxv, float lyv, float lvx, float lvy) {
        float N[4];
        shape4(natural(x, g.cx, g.rx), natural(y, g.cy, g.ry), N);
        float gx = fm(lxv, A.dt), gy = fm(lyv, A.dt), hx = 0.0f, hy = 0.0f;
        if (A.velocity_update) {
            gx = fa(gx, lvx);
            gy = fa(gy, lvy);
        } else {
            hx = fm(lvx, A.dt);
            hy = fm(lvy, A.dt);
        }
        #pragma unroll
        for (int k = 0; k < 4; ++k) {
            acc[k] = fa(acc[k], fm(N[k], gx));
            acc[4 + k] = fa(acc[4 + k], fm(N[k], gy));
            acc[8 + k] = fa(acc[8 + k], fm(N[k], hx));
            acc[12 + k] = fa(acc[12 + k], fm(N[k], hy));
        }
        ++cnt;
    };
    if (!slow) {
        row_pass16<6, REV_ROW_P, true>(buf, src, R.rb, R.re, R.cb, R.ce, tx, [&](int, int j) {
            add(buf[0][j], buf[1][j], buf[2][j], buf[3][j], buf[4][j], buf[5][j]);
        });
    } else {
        cp_async_wait<0>();
        if (ci >= 0 && ci < A.nx && cj >= 0 && cj < A.ny)
            visit_tape_cell(A, ci, cj, g, [&](int q) {
                add(A.x[q], A.y[q], A.lx[q], A.ly[q], A.lvx[q], A.lvy[q]);
            });
    }
    #pragma unroll
    for (int k = 0; k < NQ; ++k) s_c[k][tid] = acc[k];
    if (own_cell) A.cnt[cj * A.nx + ci] = cnt;
    __syncthreads();
    if (node_ok)
        rev_node_update<USL>(A, node, node_sum(s_c + 0, tid), node_sum(s_c + 4, tid), node_sum(s_c + 8, tid),
                             node_sum(s_c + 12, tid));
}

template <bool USL>
__global__ void __launch_bounds__(TILE_THREADS, 2)
k_rev_nodal_update(const __grid_constant__ AdjStep A, const int4* __restrict__ tiles) {
    const int4 T = tiles[blockIdx.x];
    if (T.x < 0) return;   // past the listed tiles
    rev_nodal_update_tile<USL>(A, T);
}

template <bool USL>
__global__ void __launch_bounds__(TILE_THREADS, 2)
k_rev_nodal_update_batch(const AdjStep* __restrict__ table, const int4* __restrict__ tiles) {
    __shared__ AdjStep sA;
    const int4 T = tiles[blockIdx.x];
    if (T.x < 0) return;   // past the listed tiles
    load_step_args(table + T.x, sA);
    rev_nodal_update_tile<USL>(sA, T);
}

// ---------------------------------------------------------------------------
// Particle passes, in two forms with the same per-particle functions.
//   By particle: a thread locates its particle and gathers the node values of
//   its cell's corners through L2.  Every particle is in flight at once.
//   By tile: a CTA of TILE_THREADS threads takes the particles stored in the
//   tile's owned sort-cells (warp w: row w + 1), their fields staged a chunk
//   ahead by 16-byte copies, with the tile's node values and cell geometry in
//   shared memory: no locate, no division and no gather for a particle still
//   in its sort-cell (one of a drifted sort-cell is located and gathers).
// ---------------------------------------------------------------------------

// Particle fields a pass reads, by index.
enum RevField { RF_X, RF_Y, RF_RHO, RF_LX, RF_LY, RF_LVX, RF_LVY, RF_LRHO, RF_VX, RF_VY, RF_SXX, RF_SYY, RF_SZZ,
                RF_SXY, RF_LSXX, RF_LSYY, RF_LSZZ, RF_LSXY, RF_LE, RF_N };
__device__ __forceinline__ const float* rev_array(const AdjStep& A, int f) {
    switch (f) {
        case RF_X: return A.x;
        case RF_Y: return A.y;
        case RF_RHO: return A.rho;
        case RF_LX: return A.lx;
        case RF_LY: return A.ly;
        case RF_LVX: return A.lvx;
        case RF_LVY: return A.lvy;
        case RF_LRHO: return A.lrho;
        case RF_VX: return A.vx;
        case RF_VY: return A.vy;
        case RF_SXX: return A.sxx;
        case RF_SYY: return A.syy;
        case RF_SZZ: return A.szz;
        case RF_SXY: return A.sxy;
        case RF_LSXX: return A.lsxx;
        case RF_LSYY: return A.lsyy;
        case RF_LSZZ: return A.lszz;
        case RF_LSXY: return A.lsxy;
        default: return A.lE;
    }
}
// The fields of each pass and their places in its staged chunks.
template <int... F>
struct FieldList {
    static constexpr int N = sizeof...(F);
    static __device__ __forceinline__ constexpr int field(int i) {
        const int f[] = {F...};
        return f[i];
    }
    static __device__ __forceinline__ constexpr int at(int want) {
        const int f[] = {F...};
        for (int i = 0; i < N; ++i)
            if (f[i] == want) return i;
        return -1;
    }
};
using ForceFields = FieldList<RF_X, RF_Y, RF_RHO, RF_LX, RF_LY, RF_LVX, RF_LVY, RF_LRHO, RF_SXX, RF_SYY, RF_SZZ,
                              RF_SXY, RF_LSXX, RF_LSYY, RF_LSZZ, RF_LSXY, RF_LE>;
using MassFields = FieldList<RF_X, RF_Y, RF_RHO, RF_LX, RF_LY, RF_LVX, RF_LVY, RF_LRHO, RF_VX, RF_VY>;
using StressFields = FieldList<RF_X, RF_Y, RF_RHO, RF_LRHO, RF_LSXX, RF_LSYY, RF_LSZZ, RF_LSXY, RF_LE>;

// A particle's fields: from global memory, or from a staged chunk.
struct GlobalFields {
    const AdjStep& A;
    int q;
    template <int F>
    __device__ __forceinline__ float get() const { return rev_array(A, F)[q]; }
};
template <class LIST>
struct StagedFieldsOf {
    const float (*b)[32];
    int lane;
    template <int F>
    __device__ __forceinline__ float get() const {
        constexpr int i = LIST::at(F);
        static_assert(i >= 0, "the pass stages this field");
        return b[i][lane];
    }
};

// Node accessors: float4 (a, b) of corner k from arrays of 1 or 2 float4 a node.
struct TileNodes {
    const float4* n1;
    const float4* n2;
    __device__ __forceinline__ int at(int k) const { return k == 0 ? 0 : k == 1 ? 1 : k == 2 ? G_W + 1 : G_W; }
    __device__ __forceinline__ float4 a(int k) const { return n1[at(k)]; }
    __device__ __forceinline__ float4 b(int k) const { return n2[at(k)]; }
};
template <class LA, class LB>
struct GatheredNodes {
    int ids[4];
    const LA& la;
    const LB& lb;
    __device__ __forceinline__ float4 a(int k) const { return la(ids[k]); }
    __device__ __forceinline__ float4 b(int k) const { return lb(ids[k]); }
};

// la(n), lb(n): the values of node n (lb unused unless TWO); body(q, fields,
// x, y, geometry, volume, nodes) for particle q at (x, y), located.
template <bool REINIT, class LA, class LB, class In, class F>
__device__ __forceinline__ void rev_located(const AdjStep& A, int q, const In& in, float x, float y, LA& la, LB& lb,
                                            F& body) {
    int ci, cj;
    particle_cell(A, x, y, ci, cj);
    const int n = cj * (A.nx + 1) + ci;
    const int c = REINIT ? A.cnt[cj * A.nx + ci] : 0;
    body(q, in, x, y, cell_geo(ci, cj, A.hx, A.hy), c ? fdv(A.vol_el, (float)c) : 0.0f,
         GatheredNodes<LA, LB>{{n, n + 1, n + A.nx + 2, n + A.nx + 1}, la, lb});
}

// ... for every particle of the tile.
template <class LIST, int DEPTH, bool TWO, bool REINIT, class LA, class LB, class F>
__device__ __forceinline__ void rev_tile_particles(const AdjStep& A, const int4 T, LA& la, LB& lb, F& body) {
    constexpr int NF = LIST::N;
    __shared__ __align__(16) float s_stage[TILE_CY][DEPTH][NF][32];
    __shared__ float4 s_a[G_W * G_H];
    __shared__ float4 s_b[TWO ? G_W * G_H : 1];
    __shared__ int s_cs[TILE_CY][33];
    __shared__ unsigned char s_map[TILE_CY][G2P_MAP];
    __shared__ float s_V0[TILE_CY][32];   // V_el / count per sort-cell (per-step volume set-up)
    __shared__ TileGeo G;
    const int tid = threadIdx.x, lane = tid & 31, w = tid / 32;
    const int c0x = T.y * TILE_NX - 1, c0y = T.z * TILE_NY - 1;
    const int sj = c0y + 1 + w, si = c0x + 1 + lane;
    const bool row_ok = w < TILE_NY && sj < A.ny, cell_ok = row_ok && lane < TILE_NX && si < A.nx;
    const int cs = row_ok ? A.cstart[sj * A.nx + min(si, A.nx)] : 0;
    const uint8_t fl = cell_ok ? A.cflag[sj * A.nx + si] : 0;
    const int cnt = REINIT && cell_ok ? A.cnt[sj * A.nx + si] : 0;
    float4 na[2], nb[2];
    #pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int idx = tid + e * TILE_THREADS;
        const int I = c0x + idx % G_W, J = c0y + idx / G_W;
        if (idx < G_W * G_H && I >= 0 && I <= A.nx && J >= 0 && J <= A.ny) {
            const int n = J * (A.nx + 1) + I;
            na[e] = la(n);
            if (TWO) nb[e] = lb(n);
        }
    }
    const unsigned drifted = __ballot_sync(0xffffffffu, fl != 0);
    const int rb = __shfl_sync(0xffffffffu, cs, 0), re = __shfl_sync(0xffffffffu, cs, 31);
    const int next = __shfl_down_sync(0xffffffffu, cs, 1);
    const float* src[NF];
    #pragma unroll
    for (int f = 0; f < NF; ++f) src[f] = rev_array(A, LIST::field(f));
    RowStage16<NF, DEPTH> st(&s_stage[w][0][0][0], src, rb, re, lane);
    st.prime();
    build_geo(A, c0x, c0y, G);
    s_cs[w][lane] = cs;
    if (REINIT) s_V0[w][lane] = cnt ? fdv(A.vol_el, (float)cnt) : 0.0f;
    if (row_ok && lane < TILE_NX)
        for (int j = cs - rb; j < min(next - rb, G2P_MAP); ++j) s_map[w][j] = (unsigned char)lane;
    #pragma unroll
    for (int e = 0; e < 2; ++e)
        if (tid + e * TILE_THREADS < G_W * G_H) {
            s_a[tid + e * TILE_THREADS] = na[e];
            if (TWO) s_b[tid + e * TILE_THREADS] = nb[e];
        }
    __syncthreads();
    #pragma unroll 1
    for (int c = 0; c < st.nch; ++c) {
        const StagedFieldsOf<LIST> in{st.advance(c), lane};
        const int q = st.rb4 + 32 * c + lane;
        if (q < rb || q >= re) continue;
        const int l = q - rb < G2P_MAP ? s_map[w][q - rb] : cell_of(s_cs[w], 30, q);   // sort-cell c0x + 1 + l
        const float x = in.template get<RF_X>(), y = in.template get<RF_Y>();
        if (!((drifted >> l) & 1u)) {
            const int at = (w + 1) * G_W + 1 + l;
            body(q, in, x, y, geo_of(G, l + 2, w + 2), REINIT ? s_V0[w][l] : 0.0f,
                 TileNodes{s_a + at, TWO ? s_b + at : nullptr});
        } else {
            rev_located<REINIT>(A, q, in, x, y, la, lb, body);
        }
    }
    cp_async_wait<0>();
}

// Strain rates (xx, yy, xy) and centroid rates of a particle from the nodal
// velocities v(k) of its cell's corners, the left-to-right sums of
// strain_rate4 with its flushes; sx, sy: signed sums + - + - of the corner
// velocities (d Gx_k / d eta and d Gy_k / d xi carry these signs).
template <class V>
__device__ __forceinline__ void rates_at(const float Gx[4], const float Gy[4], const float Gcx[4],
                                         const float Gcy[4], V&& v, float& r0, float& r1, float& r3, float& c0,
                                         float& c1, float& sx, float& sy) {
    float r3a = 0.0f, r3b_ = 0.0f;
    #pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 vk = v(k);
        const float vx = vk.x, vy = vk.y;
        if (k == 0) {
            r0 = fm(Gx[0], vx);
            r1 = fm(Gy[0], vy);
            r3a = fm(Gx[0], vy);
            r3b_ = fm(Gy[0], vx);
            c0 = fm(Gcx[0], vx);
            c1 = fm(Gcy[0], vy);
            sx = vx;
            sy = vy;
        } else {
            r0 = fa(r0, fm(Gx[k], vx));
            r1 = fa(r1, fm(Gy[k], vy));
            r3a = fa(r3a, fm(Gx[k], vy));
            r3b_ = fa(r3b_, fm(Gy[k], vx));
            c0 = fa(c0, fm(Gcx[k], vx));
            c1 = fa(c1, fm(Gcy[k], vy));
            sx = (k & 1) ? fs(sx, vx) : fa(sx, vx);
            sy = (k & 1) ? fs(sy, vy) : fa(sy, vy);
        }
    }
    r0 = flush(r0);
    r1 = flush(r1);
    r3 = flush(fa(r3a, r3b_));
    c0 = flush(c0);
    c1 = flush(c1);
}

// Reverse of the stress update for the stress adjoint sb: the strain-rate
// adjoints (zero where the forward flushed the rate), dL/dE, the adjoint of
// the updated centroid volumetric strain (vscb) and whether the update is a
// total stress (the start-of-step stress then passes no adjoint).
//   LinearElastic, SimpleMaterial: sig' = sig + D(E) r dt;
//   Newtonian (the build's definition): sig' = K vsc' I + 2 mu dev(r) with
//   r_zz = 0, s_xy = mu r_xy (material.py has no Newtonian).
template <bool NEWT>   // NEWT: the run has Newtonian particles
__device__ __forceinline__ void stress_reverse(const MatDev& mat, float Ep, float dt, float r0, float r1,
                                               float r3, float sbxx, float sbyy, float sbzz, float sbxy,
                                               float& r0b, float& r1b, float& r3b, float& Eb,
                                               float& vscb, bool& total) {
    const float d0 = fm(r0, dt), d1 = fm(r1, dt), d3 = fm(r3, dt);
    float d0b = 0.0f, d1b = 0.0f, d3b = 0.0f;
    Eb = 0.0f;
    vscb = 0.0f;
    total = false;
    if (NEWT && mat.type == MAT_NEWTONIAN) {
        const float tr = fa(fa(sbxx, sbyy), sbzz);
        const float t3b = -fm(mat.twomu, tr);              // t3 = (r0 + r1) / 3
        vscb = fm(mat.K, tr);                              // kv = K vsc'
        const float r0n = fa(fm(mat.twomu, sbxx), fdv(t3b, 3.0f));
        const float r1n = fa(fm(mat.twomu, sbyy), fdv(t3b, 3.0f));
        r0b = r0 != 0.0f ? r0n : 0.0f;
        r1b = r1 != 0.0f ? r1n : 0.0f;
        r3b = r3 != 0.0f ? fm(mat.mu, sbxy) : 0.0f;
        total = true;
        return;
    }
    if (mat.type == MAT_LINEAR_ELASTIC) {
        float a1 = mat.a1, a2 = mat.a2, G = mat.G;
        if (Ep >= 0.0f) {
            a1 = fm(Ep, mat.c1);
            a2 = fm(Ep, mat.c2);
            G = fm(Ep, mat.c3);
        }
        d0b = fa(fa(fm(a1, sbxx), fm(a2, sbyy)), fm(a2, sbzz));
        d1b = fa(fa(fm(a2, sbxx), fm(a1, sbyy)), fm(a2, sbzz));
        d3b = fm(G, sbxy);
        Eb = fa(fa(fm(mat.c1, fa(fm(d0, sbxx), fm(d1, sbyy))),
                   fm(mat.c2, fa(fa(fm(d1, sbxx), fm(d0, sbyy)), fm(fa(d0, d1), sbzz)))),
                fm(mat.c3, fm(d3, sbxy)));
    } else if (mat.type == MAT_SIMPLE) {
        const float E = Ep >= 0.0f ? Ep : mat.E;
        d0b = fm(E, sbxx);
        d1b = fm(E, sbyy);
        d3b = fm(E, sbxy);
        Eb = fa(fa(fm(d0, sbxx), fm(d1, sbyy)), fm(d3, sbxy));
    }
    r0b = r0 != 0.0f ? fm(d0b, dt) : 0.0f;
    r1b = r1 != 0.0f ? fm(d1b, dt) : 0.0f;
    r3b = r3 != 0.0f ? fm(d3b, dt) : 0.0f;
}

// ---------------------------------------------------------------------------
// Particle velocity constraints (applied after the G2P velocity update, an
// extension): a constrained component of the end-of-step velocity is a
// constant, so its adjoint is cleared before the reverse passes.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void rev_pvc_at(const AdjStep& A, int q) {
    if (q >= A.np || !A.pvc) return;
    const uchar2 c = reinterpret_cast<const uchar2*>(A.pvc)[q];
    if (c.x) A.lvx[q] = 0.0f;
    if (c.y) A.lvy[q] = 0.0f;
}

__global__ void __launch_bounds__(PART_THREADS) k_rev_pvc(const __grid_constant__ AdjStep A) {
    rev_pvc_at(A, blockIdx.x * blockDim.x + threadIdx.x);
}

__global__ void __launch_bounds__(PART_THREADS)
k_rev_pvc_batch(const AdjStep* __restrict__ table, const int2* __restrict__ blocks) {
    __shared__ AdjStep sA;
    const int2 bm = blocks[blockIdx.x];
    load_step_args(table + bm.x, sA);
    #pragma unroll 1
    for (int k = 0; k < ADJ_ITER; ++k) rev_pvc_at(sA, (bm.y * ADJ_ITER + k) * PART_THREADS + threadIdx.x);
}

// ---------------------------------------------------------------------------
// USL pass U (before pass 1): reverse of the strain / density / stress update
// that USL runs after G2P from the updated nodal velocities vB, at the
// positions of the step start (scheme.py:127-133, particle.py:249-327).  The
// stress adjoint passes through unchanged; the strain-rate and centroid-rate
// adjoints go to pass G (their transposed gather) and to pass 2 (their
// position terms); the density adjoint becomes that of the step start.
// ---------------------------------------------------------------------------
template <bool REINIT, bool NEWT, class In, class Nodes>
__device__ __forceinline__ void rev_stress_usl_at(const AdjStep& A, int q, const In& in, float x, float y,
                                                  const CellGeo& g, const Nodes& nd) {
    float Gx[4], Gy[4], Gcx[4], Gcy[4];
    dshape4(natural(x, g.cx, g.rx), natural(y, g.cy, g.ry), g.rx, g.ry, Gx, Gy);
    dshape4(0.0f, 0.0f, g.rx, g.ry, Gcx, Gcy);
    float r0, r1, r3, c0, c1, sx, sy;
    rates_at(Gx, Gy, Gcx, Gcy, [&](int k) { const float4 v = nd.a(k); return make_float2(v.x, v.y); }, r0, r1, r3,
             c0, c1, sx, sy);
    const float dvol = fm(A.dt, fa(c0, c1));
    const float f = fa(1.0f, dvol);
    const float rho1 = fdv(in.template get<RF_RHO>(), f);
    const MatDev& mat = A.mats[A.mat[q]];
    const float Ep = A.E ? A.E[q] : -1.0f;
    float r0b, r1b, r3b, Eb, vscb;
    bool total;
    stress_reverse<NEWT>(mat, Ep, A.dt, r0, r1, r3, in.template get<RF_LSXX>(), in.template get<RF_LSYY>(),
                         in.template get<RF_LSZZ>(), in.template get<RF_LSXY>(), r0b,
                         r1b, r3b, Eb, vscb, total);
    if (total) {   // the start-of-step stress passes no adjoint (pass 2 adds the forces')
        A.lsxx[q] = 0.0f;
        A.lsyy[q] = 0.0f;
        A.lszz[q] = 0.0f;
        A.lsxy[q] = 0.0f;
    }
    const float lrho = in.template get<RF_LRHO>();
    float fb = -fdv(fm(lrho, rho1), f);
    if (NEWT) {   // vsc' = vsc + dvol (only Newtonian stress reads vsc; else its adjoint is 0)
        const float lvsc = fa(A.lvsc[q], vscb);
        A.lvsc[q] = lvsc;
        fb = fa(fb, lvsc);
    }
    if (!REINIT) {   // solve semantics: V' = V f carries the volume to the next step
        const float lv = A.lvol[q];
        fb = fa(fb, fm(lv, A.vol[q]));
        A.lvol[q] = fm(lv, f);
    }
    A.r0b[q] = r0b;
    A.r1b[q] = r1b;
    A.r3b[q] = r3b;
    A.c0b[q] = c0 != 0.0f ? fm(fb, A.dt) : 0.0f;
    A.c1b[q] = c1 != 0.0f ? fm(fb, A.dt) : 0.0f;
    A.lrho[q] = fdv(lrho, f);
    A.lE[q] = fa(in.template get<RF_LE>(), Eb);
}

// The pass of a particle, or (TILE) of a tile's particles.
template <bool REINIT, bool NEWT, bool TILE>
__device__ __forceinline__ void rev_stress_usl(const AdjStep& A, const int4 T, int q) {
    auto la = [&](int n) { return make_float4(A.nvbx[n], A.nvby[n], 0.0f, 0.0f); };
    auto body = [&](int p, const auto& in, float x, float y, const CellGeo& g, float, const auto& nd) {
        rev_stress_usl_at<REINIT, NEWT>(A, p, in, x, y, g, nd);
    };
    if constexpr (TILE) rev_tile_particles<StressFields, 2, false, false>(A, T, la, la, body);
    else if (q < A.np) rev_located<false>(A, q, GlobalFields{A, q}, A.x[q], A.y[q], la, la, body);
}

// ---------------------------------------------------------------------------
// Pass 2: reverse of the forces (element.py:236-268, 842-901) and, for USF,
// of the strain / volume / stress update before them (particle.py:249-327,
// material.py:113-131).  USL forces use the start-of-step stress and the
// reset volume V0; the strain-rate adjoints of its later stress update come
// from pass U and only add their position terms here.
// ---------------------------------------------------------------------------
// nd.a: (fbx, fby, vBx, vBy), nd.b: (aBx, aBy, vAx, vAy).
template <bool USL, bool TRAC, bool REINIT, bool NEWT, class In, class Nodes>
__device__ __forceinline__ void rev_forces_at(const AdjStep& A, int q, const In& in, float x, float y,
                                              const CellGeo& g, float V0, const Nodes& nd) {
    const float xi = natural(x, g.cx, g.rx), eta = natural(y, g.cy, g.ry);
    float N[4], Gx[4], Gy[4];
    shape4(xi, eta, N);
    dshape4(xi, eta, g.rx, g.ry, Gx, Gy);
    // V0: the volume at the step start (the per-step set-up V_el / count, or
    // under solve semantics the carried volume); m: the particle mass
    if (!REINIT) V0 = A.vol[q];
    const float rho0 = in.template get<RF_RHO>();
    const float m = REINIT ? fm(V0, rho0) : A.mass[q];

    // the stress and volume of the forces: USF recomputes the strain rates
    // from vA and the stress update; sAx, sAy: signed sums of the corner
    // velocities the strain rates used (vA for USF, vB for USL)
    float r0 = 0.0f, r1 = 0.0f, r3 = 0.0f, c0 = 0.0f, c1 = 0.0f, sAx = 0.0f, sAy = 0.0f;
    PState p{};
    p.sxx = in.template get<RF_SXX>();
    p.syy = in.template get<RF_SYY>();
    p.szz = in.template get<RF_SZZ>();
    p.sxy = in.template get<RF_SXY>();
    p.rho = rho0;
    // taped when a material uses it (Newtonian); in a batch with such members the
    // others have none
    p.vsc = NEWT && A.vsc ? A.vsc[q] : 0.0f;
    float f = 1.0f, V = V0;
    const MatDev& mat = A.mats[A.mat[q]];
    const float Ep = A.E ? A.E[q] : -1.0f;
    if (!USL) {
        float Gcx[4], Gcy[4];
        dshape4(0.0f, 0.0f, g.rx, g.ry, Gcx, Gcy);
        rates_at(Gx, Gy, Gcx, Gcy, [&](int k) { const float4 v = nd.b(k); return make_float2(v.z, v.w); }, r0, r1,
                 r3, c0, c1, sAx, sAy);
        const float dvol = fm(A.dt, fa(c0, c1));
        f = strain_stress_update(mat, Ep, A.dt, r0, r1, r3, dvol, p);
        V = fm(V0, f);
    }

    // particle tractions t_d = f(t) tau_d V / size0 (mesh.py:60-77,
    // particle.py:329-343, element.py:286-303): t_d and d t_d / dV
    float trx = 0.0f, try_ = 0.0f, tqx = 0.0f, tqy = 0.0f;
    if (TRAC && A.tr_fn) {
        const float tt = step_time(A.step, A.dt);
        const float size0 = REINIT ? sqrtf(V0) : A.psize[q];
        #pragma unroll
        for (int d = 0; d < 2; ++d) {
            const int code = A.tr_fn[2 * q + d];
            if (!code) continue;
            const float tv = fm(fn_value(A, code, tt), A.tr_tau[2 * q + d]);
            const float tr = fdv(fm(tv, V), size0), tq = fdv(tv, size0);
            if (d == 0) {
                trx = tr;
                tqx = tq;
            } else {
                try_ = tr;
                tqy = tq;
            }
        }
    }

    // G2P, external and internal forces: adjoints of the shape functions (as
    // x-bar, y-bar contributions), of m and V, of the stress the forces used,
    // and the signed sums of the gradient adjoints
    float gx, gy, hx, hy;
    float xb = in.template get<RF_LX>(), yb = in.template get<RF_LY>();
    g2p_seeds(A, xb, yb, in.template get<RF_LVX>(), in.template get<RF_LVY>(), gx, gy, hx, hy);
    float mb = 0.0f, Vb = 0.0f, fsxx = 0.0f, fsyy = 0.0f, fsxy = 0.0f, sgx = 0.0f, sgy = 0.0f;
    #pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 n1 = nd.a(k), n2 = nd.b(k);
        const float fbx = n1.x, fby = n1.y, vBx = n1.z, vBy = n1.w;
        const float fg = fa(fm(fbx, A.gx), fm(fby, A.gy));   // F-bar . g
        float Nb = fa(fa(fa(fm(gx, vBx), fm(gy, vBy)), fa(fm(hx, n2.x), fm(hy, n2.y))),
                      fm(m, fg));
        if (TRAC) {
            Nb = fa(Nb, fa(fm(fbx, trx), fm(fby, try_)));   // F-bar . traction
            if (!USL || !REINIT) Vb = fa(Vb, fm(N[k], fa(fm(fbx, tqx), fm(fby, tqy))));
        }
        if (USL) {
            sAx = k == 0 ? vBx : (k & 1) ? fs(sAx, vBx) : fa(sAx, vBx);
            sAy = k == 0 ? vBy : (k & 1) ? fs(sAy, vBy) : fa(sAy, vBy);
        }
        mb = fa(mb, fm(N[k], fg));
        const float fx = fa(fm(Gx[k], p.sxx), fm(Gy[k], p.sxy));
        const float fy = fa(fm(Gy[k], p.syy), fm(Gx[k], p.sxy));
        if (!USL || !REINIT) Vb = fs(Vb, fa(fm(fbx, fx), fm(fby, fy)));
        fsxx = fa(fsxx, fm(fbx, Gx[k]));
        fsyy = fa(fsyy, fm(fby, Gy[k]));
        fsxy = fa(fsxy, fa(fm(fbx, Gy[k]), fm(fby, Gx[k])));
        const float gxk = -fm(V, fa(fm(fbx, p.sxx), fm(fby, p.sxy)));
        const float gyk = -fm(V, fa(fm(fbx, p.sxy), fm(fby, p.syy)));
        sgx = (k & 1) ? fs(sgx, gxk) : fa(sgx, gxk);
        sgy = (k & 1) ? fs(sgy, gyk) : fa(sgy, gyk);
        xb = fa(xb, fm(Nb, Gx[k]));
        yb = fa(yb, fm(Nb, Gy[k]));
    }
    // stress adjoint: loss/next-step part (through pass U for USL) + force part
    float sbxx = fs(in.template get<RF_LSXX>(), fm(V, fsxx));
    float sbyy = fs(in.template get<RF_LSYY>(), fm(V, fsyy));
    float sbzz = in.template get<RF_LSZZ>();
    float sbxy = fs(in.template get<RF_LSXY>(), fm(V, fsxy));

    float r0b, r1b, r3b, rhob;
    if (USL) {
        r0b = A.r0b[q];
        r1b = A.r1b[q];
        r3b = A.r3b[q];
        const float lrho = in.template get<RF_LRHO>();
        rhob = REINIT ? fa(lrho, fm(V0, mb)) : lrho;
        if (!REINIT) A.lvol[q] = fa(A.lvol[q], Vb);   // the forces used the start volume
    } else {
        float Eb, vscb;
        bool total;
        stress_reverse<NEWT>(mat, Ep, A.dt, r0, r1, r3, sbxx, sbyy, sbzz, sbxy, r0b, r1b, r3b, Eb, vscb,
                             total);
        if (total) sbxx = sbyy = sbzz = sbxy = 0.0f;   // total stress: no adjoint to the start
        // reverse of V = V0 (1 + dvol), rho' = rho / (1 + dvol), m = V0 rho,
        // vsc' = vsc + dvol (solve semantics: m is constant and V also
        // carries to the next step)
        const float lrho = in.template get<RF_LRHO>();
        const float Vt = REINIT ? Vb : fa(Vb, A.lvol[q]);
        float fb = fs(fm(Vt, V0), fdv(fm(lrho, p.rho), f));
        if (NEWT) {   // only Newtonian stress reads vsc; otherwise its adjoint is 0
            const float lvsc = fa(A.lvsc[q], vscb);
            A.lvsc[q] = lvsc;
            fb = fa(fb, lvsc);
        }
        rhob = REINIT ? fa(fdv(lrho, f), fm(V0, mb)) : fdv(lrho, f);
        if (!REINIT) A.lvol[q] = fm(Vt, f);
        A.lE[q] = fa(in.template get<RF_LE>(), Eb);
        A.r0b[q] = r0b;
        A.r1b[q] = r1b;
        A.r3b[q] = r3b;
        A.c0b[q] = c0 != 0.0f ? fm(fb, A.dt) : 0.0f;
        A.c1b[q] = c1 != 0.0f ? fm(fb, A.dt) : 0.0f;
    }

    // strain-rate part of the gradient adjoints: Gx_k-bar += r0b v_x,k + r3b
    // v_y,k, Gy_k-bar += r1b v_y,k + r3b v_x,k; their signed sums move x, y
    sgx = fa(sgx, fa(fm(r0b, sAx), fm(r3b, sAy)));
    sgy = fa(sgy, fa(fm(r1b, sAy), fm(r3b, sAx)));
    const float rxy = fm(fm(0.25f, g.rx), g.ry);
    xb = fa(xb, fm(rxy, sgy));
    yb = fa(yb, fm(rxy, sgx));

    A.lx[q] = xb;
    A.ly[q] = yb;
    A.lsxx[q] = sbxx;
    A.lsyy[q] = sbyy;
    A.lszz[q] = sbzz;
    A.lsxy[q] = sbxy;
    A.lrho[q] = rhob;
}

template <bool USL, bool TRAC, bool REINIT, bool NEWT, bool TILE>
__device__ __forceinline__ void rev_forces(const AdjStep& A, const int4 T, int q) {
    auto la = [&](int n) { return make_float4(A.fbx[n], A.fby[n], A.nvbx[n], A.nvby[n]); };
    auto lb = [&](int n) {
        return USL ? make_float4(A.nax[n], A.nay[n], 0.0f, 0.0f)
                   : make_float4(A.nax[n], A.nay[n], A.nvax[n], A.nvay[n]);
    };
    auto body = [&](int p, const auto& in, float x, float y, const CellGeo& g, float V0, const auto& nd) {
        rev_forces_at<USL, TRAC, REINIT, NEWT>(A, p, in, x, y, g, V0, nd);
    };
    if constexpr (TILE) rev_tile_particles<ForceFields, 2, true, REINIT>(A, T, la, lb, body);
    else if (q < A.np) rev_located<REINIT>(A, q, GlobalFields{A, q}, A.x[q], A.y[q], la, lb, body);
}

// ---------------------------------------------------------------------------
// Pass 3: transposed strain-rate gather (vA-bar += sum over particles of
// G r-bar + Gc c-bar) and the reverse nodal velocity vA = C(flush(P / M)),
// P = flush(sum N m v) (element.py:191-202, 331-334; particle.py:281-313).
// The same tile kernel is USL's pass G (the gather alone, of the pass-U
// adjoints, into vabx, vaby); USL's pass 3 has no gather.
// ---------------------------------------------------------------------------
enum RevKinMode { RK_USF, RK_GATHER, RK_NODES };
__device__ __forceinline__ void rev_node_velocity(const AdjStep& A, int n, float vbx, float vby) {
    float qbx = 0.0f, qby = 0.0f, mbt = A.mb[n];
    const float M = A.nm[n];
    if (M != 0.0f) {
        const uint16_t code = A.ncons[n];
        const bool cx = (code & 0xff) != 0, cy = (code >> 8) != 0;
        const float vAx = A.nvax[n], vAy = A.nvay[n];
        const float ubx = (cx || vAx == 0.0f) ? 0.0f : vbx;
        const float uby = (cy || vAy == 0.0f) ? 0.0f : vby;
        qbx = fdv(ubx, M);
        qby = fdv(uby, M);
        mbt = fs(mbt, fdv(fa(fm(ubx, vAx), fm(uby, vAy)), M));
    }
    A.qbx[n] = qbx;
    A.qby[n] = qby;
    A.mbt[n] = mbt;
}

template <int MODE>
__device__ __forceinline__ void rev_nodal_kinematics_tile(const AdjStep& A, const int4 T) {
    constexpr int NQ = 8;    // [vA-bar x, y] x corner
    __shared__ float s_c[NQ][SC_STRIDE];
    __shared__ __align__(16) float s_row[TILE_CY][7][REV_ROW_P];
    __shared__ TileGeo G;
    const int tid = threadIdx.x, tx = tid % TILE_CX, ty = tid / TILE_CX;
    const int c0x = T.y * TILE_NX - 1, c0y = T.z * TILE_NY - 1;
    const int ci = c0x + tx, cj = c0y + ty;
    const TileLoads L = tile_loads(A, c0x, c0y, cj, tx);
    const bool node_ok = tx < TILE_NX && ty < TILE_NY && c0x + 1 + tx <= A.nx && c0y + 1 + ty <= A.ny;
    const int node = (c0y + 1 + ty) * (A.nx + 1) + c0x + 1 + tx;
    build_geo(A, c0x, c0y, G);
    const RowRange R(L, tx);
    const float* const src[7] = {A.x, A.y, A.r0b, A.r1b, A.r3b, A.c0b, A.c1b};
    float (*buf)[REV_ROW_P] = s_row[ty];
    row_issue16<7, REV_ROW_P>(buf, src, R.rb & ~3, R.re, tx);
    const bool slow = __syncthreads_or(L.drift()) != 0;
    const CellGeo g = geo_of(G, tx + 1, ty + 1);
    float Gcx[4], Gcy[4];
    dshape4(0.0f, 0.0f, g.rx, g.ry, Gcx, Gcy);
    float acc[NQ];
    #pragma unroll
    for (int k = 0; k < NQ; ++k) acc[k] = 0.0f;
    auto add = [&](float x, float y, float r0b, float r1b, float r3b, float c0b, float c1b) {
        float Gx[4], Gy[4];
        dshape4(natural(x, g.cx, g.rx), natural(y, g.cy, g.ry), g.rx, g.ry, Gx, Gy);
        #pragma unroll
        for (int k = 0; k < 4; ++k) {
            acc[k] = fa(acc[k], fa(fa(fm(Gx[k], r0b), fm(Gy[k], r3b)), fm(Gcx[k], c0b)));
            acc[4 + k] = fa(acc[4 + k], fa(fa(fm(Gy[k], r1b), fm(Gx[k], r3b)), fm(Gcy[k], c1b)));
        }
    };
    if (!slow) {
        row_pass16<7, REV_ROW_P, true>(buf, src, R.rb, R.re, R.cb, R.ce, tx, [&](int, int j) {
            add(buf[0][j], buf[1][j], buf[2][j], buf[3][j], buf[4][j], buf[5][j], buf[6][j]);
        });
    } else {
        cp_async_wait<0>();
        if (ci >= 0 && ci < A.nx && cj >= 0 && cj < A.ny)
            visit_tape_cell(A, ci, cj, g, [&](int q) {
                add(A.x[q], A.y[q], A.r0b[q], A.r1b[q], A.r3b[q], A.c0b[q], A.c1b[q]);
            });
    }
    #pragma unroll
    for (int k = 0; k < NQ; ++k) s_c[k][tid] = acc[k];
    __syncthreads();
    if (!node_ok) return;
    const float sx = node_sum(s_c + 0, tid), sy = node_sum(s_c + 4, tid);
    if (MODE == RK_GATHER) {
        A.vabx[node] = sx;
        A.vaby[node] = sy;
    } else {
        rev_node_velocity(A, node, fa(A.vabx[node], sx), fa(A.vaby[node], sy));
    }
}

// USL pass 3: the reverse nodal velocity of the tile's nodes from vA-bar alone.
__device__ __forceinline__ void rev_node_velocity_tile(const AdjStep& A, const int4 T) {
    const int tid = threadIdx.x, tx = tid % TILE_CX, ty = tid / TILE_CX;
    const int c0x = T.y * TILE_NX - 1, c0y = T.z * TILE_NY - 1;
    if (tx < TILE_NX && ty < TILE_NY && c0x + 1 + tx <= A.nx && c0y + 1 + ty <= A.ny) {
        const int node = (c0y + 1 + ty) * (A.nx + 1) + c0x + 1 + tx;
        rev_node_velocity(A, node, A.vabx[node], A.vaby[node]);
    }
}

template <int MODE>
__global__ void __launch_bounds__(TILE_THREADS, 2)
k_rev_nodal_kinematics(const __grid_constant__ AdjStep A, const int4* __restrict__ tiles) {
    const int4 T = tiles[blockIdx.x];
    if (T.x < 0) return;   // past the listed tiles
    if (MODE == RK_NODES) rev_node_velocity_tile(A, T);
    else rev_nodal_kinematics_tile<MODE>(A, T);
}

template <int MODE>
__global__ void __launch_bounds__(TILE_THREADS, 2)
k_rev_nodal_kinematics_batch(const AdjStep* __restrict__ table, const int4* __restrict__ tiles) {
    __shared__ AdjStep sA;
    const int4 T = tiles[blockIdx.x];
    if (T.x < 0) return;   // past the listed tiles
    load_step_args(table + T.x, sA);
    if (MODE == RK_NODES) rev_node_velocity_tile(sA, T);
    else rev_nodal_kinematics_tile<MODE>(sA, T);
}

// ---------------------------------------------------------------------------
// Pass 4: reverse of the mass and momentum P2G (element.py:122-189) and of
// m = V0 rho (particle.py:158-178).
// ---------------------------------------------------------------------------
// nd.a: (qbx, qby, mbt, -).
template <bool REINIT, class In, class Nodes>
__device__ __forceinline__ void rev_mass_momentum_at(const AdjStep& A, int q, const In& in, float x, float y,
                                                     const CellGeo& g, float V0, const Nodes& nd) {
    const float xi = natural(x, g.cx, g.rx), eta = natural(y, g.cy, g.ry);
    float N[4], Gx[4], Gy[4];
    shape4(xi, eta, N);
    dshape4(xi, eta, g.rx, g.ry, Gx, Gy);
    // (solve semantics: constant mass)
    const float m = REINIT ? fm(V0, in.template get<RF_RHO>()) : A.mass[q];
    const float vx = in.template get<RF_VX>(), vy = in.template get<RF_VY>();
    float mb = 0.0f, sqx = 0.0f, sqy = 0.0f, xb = in.template get<RF_LX>(), yb = in.template get<RF_LY>();
    #pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float4 n = nd.a(k);
        const float qx = n.x, qy = n.y;
        const float t = fa(fa(fm(qx, vx), fm(qy, vy)), n.z);
        mb = fa(mb, fm(N[k], t));
        sqx = fa(sqx, fm(N[k], qx));
        sqy = fa(sqy, fm(N[k], qy));
        const float nb = fm(m, t);
        xb = fa(xb, fm(nb, Gx[k]));
        yb = fa(yb, fm(nb, Gy[k]));
    }
    const float lvx = A.velocity_update ? 0.0f : in.template get<RF_LVX>();
    const float lvy = A.velocity_update ? 0.0f : in.template get<RF_LVY>();
    A.lvx[q] = fa(lvx, fm(m, sqx));
    A.lvy[q] = fa(lvy, fm(m, sqy));
    if (REINIT) A.lrho[q] = fa(in.template get<RF_LRHO>(), fm(V0, mb));
    A.lx[q] = xb;
    A.ly[q] = yb;
}

template <bool REINIT, bool TILE>
__device__ __forceinline__ void rev_mass_momentum(const AdjStep& A, const int4 T, int q) {
    auto la = [&](int n) { return make_float4(A.qbx[n], A.qby[n], A.mbt[n], 0.0f); };
    auto body = [&](int p, const auto& in, float x, float y, const CellGeo& g, float V0, const auto& nd) {
        rev_mass_momentum_at<REINIT>(A, p, in, x, y, g, V0, nd);
    };
    if constexpr (TILE) rev_tile_particles<MassFields, 3, false, REINIT>(A, T, la, la, body);
    else if (q < A.np) rev_located<REINIT>(A, q, GlobalFields{A, q}, A.x[q], A.y[q], la, la, body);
}

// The particle passes as kernels: pass U (USL), pass 2 or pass 4, by tile or by
// particle.
enum RevPass { RP_STRESS, RP_FORCES, RP_MASS };
template <int PASS, bool USL, bool TRAC, bool REINIT, bool NEWT, bool TILE>
__device__ __forceinline__ void rev_pass(const AdjStep& A, const int4 T, int q) {
    if constexpr (PASS == RP_STRESS) rev_stress_usl<REINIT, NEWT, TILE>(A, T, q);
    else if constexpr (PASS == RP_FORCES) rev_forces<USL, TRAC, REINIT, NEWT, TILE>(A, T, q);
    else rev_mass_momentum<REINIT, TILE>(A, T, q);
}

template <int PASS, bool USL, bool TRAC, bool REINIT, bool NEWT>
__global__ void __launch_bounds__(TILE_THREADS, 2)
k_rev_tiles(const __grid_constant__ AdjStep A, const int4* __restrict__ tiles) {
    const int4 T = tiles[blockIdx.x];
    if (T.x < 0) return;   // past the listed tiles
    rev_pass<PASS, USL, TRAC, REINIT, NEWT, true>(A, T, 0);
}

template <int PASS, bool USL, bool TRAC, bool REINIT, bool NEWT>
__global__ void __launch_bounds__(TILE_THREADS, 2)
k_rev_tiles_batch(const AdjStep* __restrict__ table, const int4* __restrict__ tiles) {
    __shared__ AdjStep sA;
    const int4 T = tiles[blockIdx.x];
    if (T.x < 0) return;   // past the listed tiles
    load_step_args(table + T.x, sA);
    rev_pass<PASS, USL, TRAC, REINIT, NEWT, true>(sA, T, 0);
}

template <int PASS, bool USL, bool TRAC, bool REINIT, bool NEWT>
__global__ void __launch_bounds__(PART_THREADS, 4)
k_rev_particles(const __grid_constant__ AdjStep A) {
    rev_pass<PASS, USL, TRAC, REINIT, NEWT, false>(A, int4{}, blockIdx.x * blockDim.x + threadIdx.x);
}

template <int PASS, bool USL, bool TRAC, bool REINIT, bool NEWT>
__global__ void __launch_bounds__(PART_THREADS, 4)
k_rev_particles_batch(const AdjStep* __restrict__ table, const int2* __restrict__ blocks) {
    __shared__ AdjStep sA;
    const int2 bm = blocks[blockIdx.x];
    load_step_args(table + bm.x, sA);
    #pragma unroll 1
    for (int k = 0; k < ADJ_ITER; ++k)
        rev_pass<PASS, USL, TRAC, REINIT, NEWT, false>(sA, int4{}, (bm.y * ADJ_ITER + k) * PART_THREADS + threadIdx.x);
}

// table[i] = bases[i] with the tape pointers moved to slot t.
__global__ void k_adj_table(const AdjStep* __restrict__ bases, int n, int t,
                            AdjStep* __restrict__ table) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    AdjStep a = bases[i];
    const size_t op = (size_t)t * a.sp, on = (size_t)t * a.sn, oc = (size_t)t * a.sc;
    a.x += op; a.y += op; a.vx += op; a.vy += op;
    a.sxx += op; a.syy += op; a.szz += op; a.sxy += op; a.rho += op;
    if (a.vol) a.vol += op;
    if (a.vsc) a.vsc += op;
    a.cflag += oc;
    a.nm += on; a.nvax += on; a.nvay += on; a.nvbx += on; a.nvby += on; a.nax += on; a.nay += on;
    a.step += t;
    table[i] = a;
}

inline int blocks_for(int n, int t) { return (n + t - 1) / t; }

}  // namespace

namespace {

// What a reverse step's launches work over: one simulation (A) or a batch
// (table), the node passes' tiles and the particle passes' tiles or blocks.
struct RevLaunch {
    const AdjStep& A;
    const AdjStep* table;
    const int4* tiles;
    int nt;
    const int2* blocks;
    int nb;
    bool by_tile;
    cudaStream_t s;
};

template <int PASS, bool USL, bool TRAC, bool REINIT, bool NEWT>
void rev_particles(const RevLaunch& r) {
    if (r.by_tile) {
        if (r.table) k_rev_tiles_batch<PASS, USL, TRAC, REINIT, NEWT><<<r.nt, TILE_THREADS, 0, r.s>>>(r.table, r.tiles);
        else k_rev_tiles<PASS, USL, TRAC, REINIT, NEWT><<<r.nt, TILE_THREADS, 0, r.s>>>(r.A, r.tiles);
    } else {
        if (r.table)
            k_rev_particles_batch<PASS, USL, TRAC, REINIT, NEWT><<<r.nb, PART_THREADS, 0, r.s>>>(r.table, r.blocks);
        else
            k_rev_particles<PASS, USL, TRAC, REINIT, NEWT><<<r.nb, PART_THREADS, 0, r.s>>>(r.A);
    }
}

using RevParticlesFn = void (*)(const RevLaunch&);
#define MPM_REV(u, t, r) rev_particles<RP_FORCES, u, t, r, false>, rev_particles<RP_FORCES, u, t, r, true>
constexpr RevParticlesFn kRevForces[16] = {
    MPM_REV(false, false, false), MPM_REV(false, false, true), MPM_REV(false, true, false),
    MPM_REV(false, true, true),   MPM_REV(true, false, false), MPM_REV(true, false, true),
    MPM_REV(true, true, false),   MPM_REV(true, true, true)};
#undef MPM_REV
constexpr RevParticlesFn kRevStress[4] = {
    rev_particles<RP_STRESS, true, false, false, false>, rev_particles<RP_STRESS, true, false, false, true>,
    rev_particles<RP_STRESS, true, false, true, false>, rev_particles<RP_STRESS, true, false, true, true>};

// The particle passes go by tile from this many listed tiles on: a wave of two
// CTAs on each of the 152 SMs.  Below it a tile's rows leave most of the chip
// idle and a thread per particle fills it; above it the gathers through L2
// bind.  A reverse USF step of one simulation by tile / by particle: 117 tiles
// 29.1 / 25.8 us, 216 tiles 38.9 / 34.8, 294 tiles 40.2 / 40.8, 442 tiles
// 62.9 / 67.4, 672 tiles 100 / 109; 40 simulations in a batch (1.94M
// particles), forces pass 72 / 91 us, mass pass 30 / 38.
constexpr int REV_BY_TILE = 304;

// The passes of one reverse step (but the particle constraints) over a tile list.
void rev_passes(const RevLaunch& r, bool usl, bool trac, bool reinit, bool newt) {
    auto nodes = [&](auto single, auto batch) {
        if (r.table) batch<<<r.nt, TILE_THREADS, 0, r.s>>>(r.table, r.tiles);
        else single<<<r.nt, TILE_THREADS, 0, r.s>>>(r.A, r.tiles);
    };
    const RevParticlesFn forces = kRevForces[usl * 8 + trac * 4 + reinit * 2 + newt];
    if (usl) {
        kRevStress[reinit * 2 + newt](r);
        nodes(k_rev_nodal_kinematics<RK_GATHER>, k_rev_nodal_kinematics_batch<RK_GATHER>);
        nodes(k_rev_nodal_update<true>, k_rev_nodal_update_batch<true>);
        forces(r);
        nodes(k_rev_nodal_kinematics<RK_NODES>, k_rev_nodal_kinematics_batch<RK_NODES>);
    } else {
        nodes(k_rev_nodal_update<false>, k_rev_nodal_update_batch<false>);
        forces(r);
        nodes(k_rev_nodal_kinematics<RK_USF>, k_rev_nodal_kinematics_batch<RK_USF>);
    }
    if (reinit) rev_particles<RP_MASS, false, false, true, false>(r);
    else rev_particles<RP_MASS, false, false, false, false>(r);
}

}  // namespace

cudaError_t launch_rev_step(const AdjStep& A, bool usl, bool trac, const int4* tiles, int ntiles,
                            cudaStream_t s) {
    const int nb = A.np > 0 ? blocks_for(A.np, PART_THREADS) : 0;
    if (A.pvc && nb > 0) k_rev_pvc<<<nb, PART_THREADS, 0, s>>>(A);
    if (ntiles > 0 && nb > 0)
        rev_passes(RevLaunch{A, nullptr, tiles, ntiles, nullptr, nb, ntiles >= REV_BY_TILE, s}, usl, trac,
                   A.reinit != 0, A.vsc != nullptr);
    return cudaGetLastError();
}

cudaError_t launch_adj_table(const AdjStep* bases, int n, int t, AdjStep* table, cudaStream_t s) {
    if (n > 0) k_adj_table<<<blocks_for(n, 128), 128, 0, s>>>(bases, n, t, table);
    return cudaGetLastError();
}

cudaError_t launch_rev_batch(const AdjStep* table, bool usl, bool trac, bool pvc, bool reinit, bool newt,
                             const int4* tiles, int ntiles, const int2* part_blocks, int n_part_blocks,
                             cudaStream_t s) {
    static const AdjStep unused{};   // the batched launches read the device table
    if (pvc && n_part_blocks > 0) k_rev_pvc_batch<<<n_part_blocks, PART_THREADS, 0, s>>>(table, part_blocks);
    if (ntiles > 0 && n_part_blocks > 0)
        rev_passes(RevLaunch{unused, table, tiles, ntiles, part_blocks, n_part_blocks, ntiles >= REV_BY_TILE, s},
                   usl, trac, reinit, newt);
    return cudaGetLastError();
}

}  // namespace mpm
