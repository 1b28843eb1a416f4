// One-dimensional explicit MPM on two-node line elements (Linear1D,
// diffmpm/element.py:343-600) -- the same phases as the 2-D step, for meshes
// of `nx` elements of length hx with nodes at float(i) * hx.
//
// Layout: particles are re-sorted by element at the start of every step (the
// 2-D sort machinery with a single row of cells), each element's particles in
// original-index order, and eid[q] holds the element of storage slot q for
// the step.  Node-centric kernels (one thread per node) merge the particles of
// the node's two elements by original index, so every nodal sum adds the
// particle contributions in the order of the reference's sequential scatter
// (a `lax.fori_loop` of `.at[].add`, element.py:138-152): the 1-D step gives
// the oracle's float32 results bit for bit.
//
// Build definitions where the reference's 1-D path does not run as written:
// the element volume is x_{e+1} - x_e (the reference's `ediff1d` broadcast
// only works for one element, element.py:543-546) and the strain rate is
// [dN/dx . v, 0, 0, 0, 0, 0] (the reference indexes a 1 x 1 matrix at [1, 1],
// particle.py:304-305).
#include <cuda_runtime.h>

#include "mpm_device.cuh"
#include "mpm_handle.h"
#include "mpm_kernels.h"

namespace mpm {
namespace {

constexpr int LINE_THREADS = 256;

struct LineElem {
    float x0, x1, c, r;   // nodes, centre, 2 / length
};

__device__ __forceinline__ LineElem line_elem(int e, float h) {
    LineElem g;
    g.x0 = node_coord(e, h);
    g.x1 = node_coord(e + 1, h);
    g.c = fm(fa(g.x0, g.x1), 0.5f);
    g.r = fdv(2.0f, fs(g.x1, g.x0));
    return g;
}

// Shape function of node k (0 left, 1 right) at natural coordinate xi
// (element.py:430-454): (1/2)(1 -/+ xi).
__device__ __forceinline__ float shape2(int k, float xi) {
    return k ? fm(0.5f, fa(1.0f, xi)) : fm(0.5f, fs(1.0f, xi));
}

// dN_k/dx = (-/+ 1/2) * 2 / length (element.py:456-515).
__device__ __forceinline__ float dshape2(int k, float r) { return fm(k ? 0.5f : -0.5f, r); }

// Volume at the per-step reset of solve_jit (particle.py:158-178): element
// length / particles in the element.
__device__ __forceinline__ float reset_volume(const SimDev& S, int e) {
    const LineElem g = line_elem(e, S.hx);
    return fdv(fs(g.x1, g.x0), (float)(S.cstart[e + 1] - S.cstart[e]));
}

// Visit the particles of elements i-1 (as their right node) and i (as their
// left node) in increasing original index; f(q, e, k).
template <class F>
__device__ __forceinline__ void for_node_particles(const SimDev& S, int i, F&& f) {
    int a = 0, ae = 0, b = 0, be = 0;
    if (i >= 1) { a = S.cstart[i - 1]; ae = S.cstart[i]; }
    if (i < S.nx) { b = S.cstart[i]; be = S.cstart[i + 1]; }
    #pragma unroll 1
    while (a < ae || b < be) {
        const bool left = a < ae && (b >= be || S.pid[a] < S.pid[b]);
        if (left) { f(a, i - 1, 1); ++a; }
        else { f(b, i, 0); ++b; }
    }
}

// Nodal constraint of direction 0 (constraint.py:29-44): slot + 1, or 0.
__device__ __forceinline__ int cons0(const SimDev& S, int i) { return S.ncons[i] & 0xff; }

template <bool REINIT>
__global__ void __launch_bounds__(LINE_THREADS)
k_line_nodal_kinematics(const __grid_constant__ SimDev S, int par) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > S.nx) return;
    const float* rho = S.rho[par];
    float m = 0.0f, p = 0.0f;
    for_node_particles(S, i, [&](int q, int e, int k) {
        const LineElem g = line_elem(e, S.hx);
        const float N = shape2(k, natural(S.x[q], g.c, g.r));
        const float mp = REINIT ? fm(reset_volume(S, e), rho[q]) : S.mass[q];
        m = fa(m, fm(mp, N));                       // element.py:138-152
        p = fa(p, fm(N, fm(mp, S.vx[q])));          // element.py:166-184
    });
    p = flush(p);                                    // element.py:185-189
    float v = m == 0.0f ? S.nvbx[i] : fdv(p, m);     // element.py:191-202
    v = flush(v);
    const int c = cons0(S, i);
    if (c) v = S.cons_vel[c - 1];                    // constraint.py:29-44
    S.nm[i] = m;
    S.nvax[i] = v;
    if (c) S.nax[i] = 0.0f;
}

// Strain rate, strain, volume and stress of each particle from the nodal
// velocities `nv` (particle.py:249-327), reading ping-pong slot `par` and
// writing `par ^ 1`.
template <bool REINIT>
__global__ void __launch_bounds__(LINE_THREADS)
k_line_stress(const __grid_constant__ SimDev S, const int* __restrict__ eid,
              const float* __restrict__ nv, int par) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= S.np) return;
    const int e = eid[q];
    const LineElem g = line_elem(e, S.hx);
    const float r = flush(fa(fm(dshape2(0, g.r), nv[e]), fm(dshape2(1, g.r), nv[e + 1])));
    const float dvol = fm(S.dt, r);     // the centroid rate equals r in 1-D
    const int o = par ^ 1;
    PState ps{S.sxx[par][q], S.syy[par][q], S.szz[par][q], S.sxy[par][q],
              S.exx[q], S.eyy[q], S.exy[q], S.rho[par][q], S.vsc[par][q]};
    const MatDev M = S.mats[S.mat[q]];
    const float Ep = S.E ? S.E[q] : -1.0f;
    const float f = strain_stress_update(M, Ep, S.dt, r, 0.0f, 0.0f, dvol, ps);
    S.sxx[o][q] = ps.sxx; S.syy[o][q] = ps.syy; S.szz[o][q] = ps.szz; S.sxy[o][q] = ps.sxy;
    S.exx[q] = ps.exx; S.eyy[q] = ps.eyy; S.exy[q] = ps.exy;
    S.rho[o][q] = ps.rho; S.vsc[o][q] = ps.vsc;
    const float V0 = REINIT ? reset_volume(S, e) : S.vol[par][q];
    S.vol[o][q] = fm(V0, f);            // particle.py:324-327
}

// External and internal nodal forces, then the nodal update
// (element.py:204-329).  `spar` is the slot holding the stress and volume the
// forces use (after the USF update, or before the USL one).
template <bool REINIT>
__global__ void __launch_bounds__(LINE_THREADS)
k_line_forces(const __grid_constant__ SimDev S, int par, int spar, int step) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > S.nx) return;
    const float* rho = S.rho[par];
    const float* sxx = S.sxx[spar];
    const float* vol = S.vol[spar];
    const bool usl_reset = REINIT && spar == par;   // USL under solve_jit: reset volume
    float fext = 0.0f, fint = 0.0f;
    for_node_particles(S, i, [&](int q, int e, int k) {
        const LineElem g = line_elem(e, S.hx);
        const float N = shape2(k, natural(S.x[q], g.c, g.r));
        const float mp = REINIT ? fm(reset_volume(S, e), rho[q]) : S.mass[q];
        fext = fa(fext, fm(N, fm(mp, S.gx)));                       // element.py:236-268
        const float V = usl_reset ? reset_volume(S, e) : vol[q];
        fint = fa(fint, fm(fm(-V, sxx[q]), dshape2(k, g.r)));       // element.py:548-600
    });
    if (S.cnf_ptr) {                                                 // element.py:270-284
        const float t = step_time(step, S.dt);
        #pragma unroll 1
        for (int j = S.cnf_ptr[i]; j < S.cnf_ptr[i + 1]; ++j)
            fext = fa(fext, fm(fn_value(S, S.cnf_fn[j], t), S.cnf_val[j]));
    }
    const float m = S.nm[i];
    float a = nan_to_num(fdv(fa(fa(fint, fext), 0.0f), m));          // element.py:305-329
    float v = fa(S.nvax[i], fm(a, S.dt));
    const int c = cons0(S, i);
    if (c) {
        v = S.cons_vel[c - 1];
        a = 0.0f;
    }
    S.nvbx[i] = flush(v);
    S.nax[i] = flush(a);
}

// G2P (particle.py:208-247) and the element check of the moved particle.
__global__ void __launch_bounds__(LINE_THREADS)
k_line_g2p(const __grid_constant__ SimDev S, const int* __restrict__ eid, Control* __restrict__ ctl) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= S.np) return;
    const int e = eid[q];
    const LineElem g = line_elem(e, S.hx);
    const float xi = natural(S.x[q], g.c, g.r);
    const float N0 = shape2(0, xi), N1 = shape2(1, xi);
    const float vh = fa(fm(N0, S.nvbx[e]), fm(N1, S.nvbx[e + 1]));
    const float ah = fa(fm(N0, S.nax[e]), fm(N1, S.nax[e + 1]));
    float v = S.velocity_update ? vh : fa(S.vx[q], fm(ah, S.dt));
    if (S.pvc && S.pvc[2 * q]) v = S.pvc_vel[S.pvc[2 * q] - 1];   // particle velocity constraint
    S.vx[q] = v;
    const float x = fa(S.x[q], fm(vh, S.dt));
    S.x[q] = x;
    const int ne = locate_axis(x, S.hx, S.nx);
    if (ne < 0 || ne >= S.nx) atomicOr(&ctl->status, ST_OUT_OF_MESH);
}

// ---------------------------------------------------------------------------
// Whole runs of steps in one CTA, for bars of at most LINE_FUSED_MAX particles
// and elements (every known use of the 1-D elements).  A step as separate
// kernels is ~26 dependent launches of one or two CTAs, so launches are all of
// its time (216 particles: 102 us a step).  Here a thread keeps its particles
// in registers for all steps, nodes and element lists live in shared memory,
// and a step is six barriers.  The lists are rebuilt only after a step in
// which a particle changed element.  Bound by the latency of the barriers and
// of the serial node sums: 216 particles 102 -> 4.5 us a step, one particle
// with its adjoint 163 -> 6 us a step.  Contributions are formed once per
// particle and stored in list order; a node adds them in the order of
// for_node_particles, so every sum has the same terms in the same order as
// the separate kernels: the same bits.
// ---------------------------------------------------------------------------
struct LineTape {   // of the whole run (LineTapeSlot by step), or P == nullptr
    float* P;       // [step][9][np]
    int* pid;       // [step][np]
    int* cs;        // [step][nx + 2]
    float* N;       // [step][4][nn]
};

struct LineShared {
    float *m, *va, *vb, *a, *V0, *c;   // nodes, reset volume per element, contributions [4][np] in list order
    int *start, *cnt, *pid;            // element lists: starts [nx + 2], scratch [nx + 1], original index per slot
    __device__ LineShared(char* raw, int np, int nx) {
        float* f = reinterpret_cast<float*>(raw);
        const int nn = nx + 1;
        m = f; va = m + nn; vb = va + nn; a = vb + nn; V0 = a + nn; c = V0 + nx;
        start = reinterpret_cast<int*>(c + 4 * (size_t)np);
        cnt = start + nx + 2;
        pid = cnt + nn;
    }
};
inline size_t line_shared_bytes(int np, int nx) {
    return 4 * ((size_t)4 * (nx + 1) + nx + 4 * (size_t)np + (nx + 2) + (nx + 1) + (size_t)np);
}

// Sum the two contribution rows of node i in for_node_particles' order.
__device__ __forceinline__ void line_node_sums(const LineShared& W, int np, int nx, int i, float& s0, float& s1) {
    int a = 0, ae = 0, b = 0, be = 0;
    if (i >= 1) { a = W.start[i - 1]; ae = W.start[i]; }
    if (i < nx) { b = W.start[i]; be = W.start[i + 1]; }
    const float *l0 = W.c, *r0 = W.c + np, *l1 = W.c + 2 * np, *r1 = W.c + 3 * np;
    s0 = s1 = 0.0f;
    #pragma unroll 1
    while (a < ae || b < be) {
        const bool left = a < ae && (b >= be || W.pid[a] < W.pid[b]);
        if (left) { s0 = fa(s0, r0[a]); s1 = fa(s1, r1[a]); ++a; }
        else { s0 = fa(s0, l0[b]); s1 = fa(s1, l1[b]); ++b; }
    }
}

// A particle's element lists entry: bucket (nx: outside the mesh), geometry, slot.
struct LineP {
    float x, v;
    PState s;
    float vol, mass, Ep, mp, N0, N1, gc, gr, x0, x1;
    int e, slot, pid, mat, code;
};

template <bool REINIT, bool USL, int PPT>
__global__ void __launch_bounds__(1024)
k_line_steps(const __grid_constant__ SimDev S, int par, int step0, int nsteps, Control* __restrict__ ctl,
             const LineTape tape) {
    extern __shared__ char s_raw[];
    __shared__ int s_warp[32];
    __shared__ int s_carry;
    const int np = S.np, nx = S.nx, nn = nx + 1, T = blockDim.x, tid = threadIdx.x;
    const LineShared W(s_raw, np, nx);
    LineP P[PPT];
    int status = 0;
    #pragma unroll
    for (int u = 0; u < PPT; ++u) {
        const int q = tid + u * T;
        if (q >= np) continue;
        LineP& p = P[u];
        p.x = S.x[q]; p.v = S.vx[q];
        p.s = PState{S.sxx[par][q], S.syy[par][q], S.szz[par][q], S.sxy[par][q],
                     S.exx[q], S.eyy[q], S.exy[q], S.rho[par][q], S.vsc[par][q]};
        p.vol = S.vol[par][q];
        p.mass = REINIT ? 0.0f : S.mass[q];
        p.Ep = S.E ? S.E[q] : -1.0f;
        p.pid = S.pid[q];
        p.mat = S.mat[q];
        p.code = S.pvc ? S.pvc[2 * q] : 0;
        p.e = locate_axis(p.x, S.hx, nx);
        if (p.e < 0 || p.e >= nx) { status |= ST_OUT_OF_MESH; p.e = nx; }
    }
    for (int i = tid; i < nn; i += T) { W.vb[i] = S.nvbx[i]; W.a[i] = 0.0f; }
    bool rebuild = true;
    #pragma unroll 1
    for (int t = 0; t < nsteps; ++t) {
        if (rebuild) {
            // counting sort by element, each element's entries by original index
            for (int i = tid; i <= nx; i += T) W.cnt[i] = 0;
            if (tid == 0) s_carry = 0;
            __syncthreads();
            #pragma unroll
            for (int u = 0; u < PPT; ++u)
                if (tid + u * T < np) P[u].slot = atomicAdd(&W.cnt[P[u].e], 1);
            __syncthreads();
            #pragma unroll 1
            for (int base = 0; base <= nx; base += T) {   // exclusive scan of the counts
                const int i = base + tid, lane = tid & 31;
                const int v = i <= nx ? W.cnt[i] : 0;
                int x = v;
                #pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                if (lane == 31) s_warp[tid >> 5] = x;
                __syncthreads();
                int before = s_carry;
                for (int w = 0; w < (tid >> 5); ++w) before += s_warp[w];
                if (i <= nx) W.start[i] = before + x - v;
                __syncthreads();
                if (tid == T - 1) s_carry = before + x;
            }
            if (tid == 0) W.start[nx + 1] = np;
            __syncthreads();
            #pragma unroll
            for (int u = 0; u < PPT; ++u)
                if (tid + u * T < np) W.pid[W.start[P[u].e] + P[u].slot] = P[u].pid;
            __syncthreads();
            #pragma unroll
            for (int u = 0; u < PPT; ++u)
                if (tid + u * T < np) {
                    LineP& p = P[u];
                    int rank = 0;
                    for (int j = W.start[p.e]; j < W.start[p.e + 1]; ++j) rank += W.pid[j] < p.pid;
                    p.slot = W.start[p.e] + rank;
                    const LineElem g = line_elem(p.e, S.hx);
                    p.gc = g.c; p.gr = g.r; p.x0 = g.x0; p.x1 = g.x1;
                }
            for (int e = tid; e < nx; e += T) {
                const LineElem g = line_elem(e, S.hx);
                W.V0[e] = fdv(fs(g.x1, g.x0), (float)(W.start[e + 1] - W.start[e]));
            }
            __syncthreads();
            #pragma unroll
            for (int u = 0; u < PPT; ++u)
                if (tid + u * T < np) W.pid[P[u].slot] = P[u].pid;
            __syncthreads();
        }
        if (tape.P) {
            float* o = tape.P + (size_t)t * 9 * np;
            #pragma unroll
            for (int u = 0; u < PPT; ++u)
                if (tid + u * T < np) {
                    const LineP& p = P[u];
                    const float v[9] = {p.x, p.v, p.s.sxx, p.s.syy, p.s.szz, p.s.sxy, p.s.rho, p.vol, p.s.vsc};
                    #pragma unroll
                    for (int k = 0; k < 9; ++k) o[(size_t)k * np + p.slot] = v[k];
                    tape.pid[(size_t)t * np + p.slot] = p.pid;
                }
            for (int i = tid; i < nx + 2; i += T) tape.cs[(size_t)t * (nx + 2) + i] = W.start[i];
        }
        // mass and momentum of the nodes
        #pragma unroll
        for (int u = 0; u < PPT; ++u)
            if (tid + u * T < np) {
                LineP& p = P[u];
                const float xi = natural(p.x, p.gc, p.gr);
                p.N0 = shape2(0, xi);
                p.N1 = shape2(1, xi);
                p.mp = REINIT ? fm(p.e < nx ? W.V0[p.e] : 0.0f, p.s.rho) : p.mass;
                const float mv = fm(p.mp, p.v);
                W.c[p.slot] = fm(p.mp, p.N0);
                W.c[np + p.slot] = fm(p.mp, p.N1);
                W.c[2 * np + p.slot] = fm(p.N0, mv);
                W.c[3 * np + p.slot] = fm(p.N1, mv);
            }
        __syncthreads();
        for (int i = tid; i < nn; i += T) {
            float m, mom;
            line_node_sums(W, np, nx, i, m, mom);
            mom = flush(mom);
            float v = m == 0.0f ? W.vb[i] : fdv(mom, m);
            v = flush(v);
            const int c = cons0(S, i);
            if (c) v = S.cons_vel[c - 1];
            W.m[i] = m;
            W.va[i] = v;
        }
        __syncthreads();
        // (USF) stress update; internal and external force contributions
        auto stress = [&](LineP& p, const float* nv) {
            const int e = min(p.e, nx - 1);
            const float r = flush(fa(fm(dshape2(0, p.gr), nv[e]), fm(dshape2(1, p.gr), nv[e + 1])));
            const float dvol = fm(S.dt, r);
            const float f = strain_stress_update(S.mats[p.mat], p.Ep, S.dt, r, 0.0f, 0.0f, dvol, p.s);
            p.vol = fm(REINIT ? W.V0[e] : p.vol, f);
        };
        #pragma unroll
        for (int u = 0; u < PPT; ++u)
            if (tid + u * T < np) {
                LineP& p = P[u];
                const float Vs = REINIT ? W.V0[min(p.e, nx - 1)] : p.vol;
                if (!USL) stress(p, W.va);
                const float mg = fm(p.mp, S.gx), vs = fm(-(USL ? Vs : p.vol), p.s.sxx);
                W.c[p.slot] = fm(p.N0, mg);
                W.c[np + p.slot] = fm(p.N1, mg);
                W.c[2 * np + p.slot] = fm(vs, dshape2(0, p.gr));
                W.c[3 * np + p.slot] = fm(vs, dshape2(1, p.gr));
            }
        __syncthreads();
        for (int i = tid; i < nn; i += T) {
            float fext, fint;
            line_node_sums(W, np, nx, i, fext, fint);
            if (S.cnf_ptr) {
                const float time = step_time(step0 + t, S.dt);
                #pragma unroll 1
                for (int j = S.cnf_ptr[i]; j < S.cnf_ptr[i + 1]; ++j)
                    fext = fa(fext, fm(fn_value(S, S.cnf_fn[j], time), S.cnf_val[j]));
            }
            float a = nan_to_num(fdv(fa(fa(fint, fext), 0.0f), W.m[i]));
            float v = fa(W.va[i], fm(a, S.dt));
            const int c = cons0(S, i);
            if (c) {
                v = S.cons_vel[c - 1];
                a = 0.0f;
            }
            W.vb[i] = flush(v);
            W.a[i] = flush(a);
        }
        __syncthreads();
        if (tape.P) {
            float* o = tape.N + (size_t)t * 4 * nn;
            for (int i = tid; i < nn; i += T) {
                o[i] = W.m[i];
                o[nn + i] = W.va[i];
                o[2 * nn + i] = W.vb[i];
                o[3 * nn + i] = W.a[i];
            }
        }
        bool moved = false;
        #pragma unroll
        for (int u = 0; u < PPT; ++u)
            if (tid + u * T < np) {
                LineP& p = P[u];
                const int e = min(p.e, nx - 1);
                const float vh = fa(fm(p.N0, W.vb[e]), fm(p.N1, W.vb[e + 1]));
                const float ah = fa(fm(p.N0, W.a[e]), fm(p.N1, W.a[e + 1]));
                float v = S.velocity_update ? vh : fa(p.v, fm(ah, S.dt));
                if (p.code) v = S.pvc_vel[p.code - 1];
                p.v = v;
                p.x = fa(p.x, fm(vh, S.dt));
                if (USL) stress(p, W.vb);
                if (!(p.e < nx && p.x >= p.x0 && p.x < p.x1)) {
                    int ne = locate_axis(p.x, S.hx, nx);
                    if (ne < 0 || ne >= nx) { status |= ST_OUT_OF_MESH; ne = nx; }
                    moved = moved || ne != p.e;
                    p.e = ne;
                }
            }
        rebuild = __syncthreads_or(moved) != 0;
    }
    const int o = (par + nsteps) & 1;
    #pragma unroll
    for (int u = 0; u < PPT; ++u) {
        const int q = tid + u * T;
        if (q >= np) continue;
        const LineP& p = P[u];
        S.x[q] = p.x; S.vx[q] = p.v;
        S.sxx[o][q] = p.s.sxx; S.syy[o][q] = p.s.syy; S.szz[o][q] = p.s.szz; S.sxy[o][q] = p.s.sxy;
        S.exx[q] = p.s.exx; S.eyy[q] = p.s.eyy; S.exy[q] = p.s.exy;
        S.rho[o][q] = p.s.rho; S.vsc[o][q] = p.s.vsc; S.vol[o][q] = p.vol;
    }
    for (int i = tid; i < nn; i += T) {
        S.nm[i] = W.m[i];
        S.nvax[i] = W.va[i];
        S.nvbx[i] = W.vb[i];
        S.nax[i] = W.a[i];
    }
    // the element starts of the last step, as a sort before every step leaves them
    // (a momentum read counts by them; the particles stay in their storage slots,
    // which the next use sorts)
    for (int i = tid; i < nx + 2; i += T) S.cstart[i] = W.start[i];
    if (status) atomicOr(&ctl->status, status);
}

template <bool REINIT, bool USL>
cudaError_t launch_line_steps(const SimDev& S, int par, int step0, int n, Control* ctl, const LineTape& tape,
                              cudaStream_t s) {
    const size_t bytes = line_shared_bytes(S.np, S.nx);
    // a thread per particle and node up to 1024 threads, two particles a thread above
    const int want = S.np > S.nx ? S.np : S.nx + 1;
    const int T = want >= 1024 ? 1024 : (want + 31) / 32 * 32;
    auto go = [&](auto kernel) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return e;
        kernel<<<1, T, bytes, s>>>(S, par, step0, n, ctl, tape);
        return cudaGetLastError();
    };
    return S.np <= T ? go(k_line_steps<REINIT, USL, 1>) : go(k_line_steps<REINIT, USL, 2>);
}

// Element of each storage slot: the bucket it was sorted into.  Particles outside
// the mesh (the last bucket; the call ends with an error) get the last element, so
// that the kernels until then stay within their arrays.
__global__ void k_line_eid(const int* __restrict__ cstart, int nx, int* __restrict__ eid) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e > nx) return;
    #pragma unroll 1
    for (int q = cstart[e]; q < cstart[e + 1]; ++q) eid[q] = min(e, nx - 1);
}

// Each element's particles in increasing original index (insertion sort of a
// bucket by pid; buckets hold a few particles).
__global__ void k_line_segsort(int nbucket, const int* __restrict__ start, int* __restrict__ perm,
                               const int* __restrict__ pid) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nbucket) return;
    const int b = start[c], e = start[c + 1];
    #pragma unroll 1
    for (int i = b + 1; i < e; ++i) {
        const int v = perm[i];
        const int pv = pid[v];
        int j = i - 1;
        #pragma unroll 1
        while (j >= b && pid[perm[j]] > pv) {
            perm[j + 1] = perm[j];
            --j;
        }
        perm[j + 1] = v;
    }
}

// V = element length / count, m = V rho, size = V (solve semantics set-up,
// particle.py:158-178).
__global__ void k_line_setup_volume(const __grid_constant__ SimDev S, const int* __restrict__ eid, int par) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= S.np) return;
    const float V = reset_volume(S, eid[q]);
    S.vol[par][q] = V;
    S.mass[q] = fm(V, S.rho[par][q]);
    S.psize[q] = V;
}

inline int blocks(int n) { return (n + LINE_THREADS - 1) / LINE_THREADS; }

}  // namespace

cudaError_t launch_line_segsort(int nbucket, const int* start, int* perm, const int* pid, cudaStream_t s) {
    if (nbucket > 0) k_line_segsort<<<blocks(nbucket), LINE_THREADS, 0, s>>>(nbucket, start, perm, pid);
    return cudaGetLastError();
}

cudaError_t launch_line_eid(const int* cstart, int nx, int* eid, cudaStream_t s) {
    if (nx > 0) k_line_eid<<<blocks(nx + 1), LINE_THREADS, 0, s>>>(cstart, nx, eid);
    return cudaGetLastError();
}

namespace host {

int line_setup_volume(MpmHandle* h, cudaStream_t s) {
    if (h->np > 0)
        k_line_setup_volume<<<blocks((int)h->np), LINE_THREADS, 0, s>>>(h->hs, h->line_eid, parity(h));
    CK(h, cudaGetLastError());
    return MPM_OK;
}

// One step: re-sort by element, nodal kinematics, (USF) stress update, forces
// and nodal update, G2P, (USL) stress update.
static int line_step(MpmHandle* h, cudaStream_t s, const LineTapeSlot* tape) {
    TRY(resort(h, s));
    const SimDev& S = h->hs;
    const int par = parity(h), nb = blocks(h->nx + 1), pb = blocks((int)h->np);
    const int step = (int)h->step;
    const size_t fb = sizeof(float) * (size_t)h->np, nbytes = sizeof(float) * (size_t)h->nn;
    if (tape) {
        const float* src[9] = {S.x, S.vx, S.sxx[par], S.syy[par], S.szz[par], S.sxy[par], S.rho[par],
                               S.vol[par], S.vsc[par]};
        for (int k = 0; k < 9; ++k) CK(h, cudaMemcpyAsync(tape->p[k], src[k], fb, cudaMemcpyDeviceToDevice, s));
        CK(h, cudaMemcpyAsync(tape->pid, S.pid, sizeof(int) * (size_t)h->np, cudaMemcpyDeviceToDevice, s));
        CK(h, cudaMemcpyAsync(tape->cs, S.cstart, sizeof(int) * (size_t)(h->nx + 2), cudaMemcpyDeviceToDevice, s));
    }
    if (h->reinit) k_line_nodal_kinematics<true><<<nb, LINE_THREADS, 0, s>>>(S, par);
    else k_line_nodal_kinematics<false><<<nb, LINE_THREADS, 0, s>>>(S, par);
    if (!h->usl) {
        if (h->reinit) k_line_stress<true><<<pb, LINE_THREADS, 0, s>>>(S, h->line_eid, h->nvax, par);
        else k_line_stress<false><<<pb, LINE_THREADS, 0, s>>>(S, h->line_eid, h->nvax, par);
    }
    const int spar = h->usl ? par : par ^ 1;
    if (h->reinit) k_line_forces<true><<<nb, LINE_THREADS, 0, s>>>(S, par, spar, step);
    else k_line_forces<false><<<nb, LINE_THREADS, 0, s>>>(S, par, spar, step);
    k_line_g2p<<<pb, LINE_THREADS, 0, s>>>(S, h->line_eid, h->ctl);
    if (h->usl) {
        if (h->reinit) k_line_stress<true><<<pb, LINE_THREADS, 0, s>>>(S, h->line_eid, h->nvbx, par);
        else k_line_stress<false><<<pb, LINE_THREADS, 0, s>>>(S, h->line_eid, h->nvbx, par);
    }
    CK(h, cudaGetLastError());
    if (tape) {
        const float* src[4] = {h->nm, h->nvax, h->nvbx, h->nax};
        for (int k = 0; k < 4; ++k) CK(h, cudaMemcpyAsync(tape->n[k], src[k], nbytes, cudaMemcpyDeviceToDevice, s));
    }
    h->step++;
    h->needs_resort = true;
    return MPM_OK;
}

// n steps in one launch (bars of at most LINE_FUSED_MAX particles and elements).
static int line_steps_fused(MpmHandle* h, int n, cudaStream_t s, const LineTapeSlot* tape) {
    const int par = parity(h);
    const LineTape tp = tape ? LineTape{tape->p[0], tape->pid, tape->cs, tape->n[0]} : LineTape{};
    const int step = (int)h->step;
    cudaError_t e;
    if (h->reinit)
        e = h->usl ? launch_line_steps<true, true>(h->hs, par, step, n, h->ctl, tp, s)
                   : launch_line_steps<true, false>(h->hs, par, step, n, h->ctl, tp, s);
    else
        e = h->usl ? launch_line_steps<false, true>(h->hs, par, step, n, h->ctl, tp, s)
                   : launch_line_steps<false, false>(h->hs, par, step, n, h->ctl, tp, s);
    CK(h, e);
    h->step += n;
    h->resorts += n;
    h->needs_resort = true;
    return MPM_OK;
}

int line_steps(MpmHandle* h, int n, cudaStream_t s, const LineTapeSlot* tape) {
    if (n > 0 && line_fused(h)) return line_steps_fused(h, n, s, tape);
    LineTapeSlot slot;
    if (tape) slot = *tape;
    for (int t = 0; t < n; ++t) {
        TRY(line_step(h, s, tape ? &slot : nullptr));
        if (!tape) continue;
        for (float*& p : slot.p) p += 9 * (size_t)h->np;
        slot.pid += h->np;
        slot.cs += h->nx + 2;
        for (float*& p : slot.n) p += 4 * (size_t)h->nn;
    }
    return MPM_OK;
}

}  // namespace host
}  // namespace mpm
