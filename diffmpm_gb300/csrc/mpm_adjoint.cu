// Differentiation of the explicit step: a recorded forward run (mpm_record) and
// the hand-written discrete adjoint (mpm_adjoint).
//
// The tape holds, for a run of consecutive steps, each step's start state and
// nodal results.  Taped steps write it as they go: a step's kernels read the
// particles from its slot and write them to the next one, and write the nodal
// results to its slot, so a tape costs no copies but the first slot of a block
// and the nodes of its last (as copies around every step it was a third of the
// forward time).  The last step of a block writes the handle's own arrays,
// where re-sorts, snapshots and reads find the state.
//
// mpm_record tapes the whole run when that fits a bounded share of the device
// memory and a bounded multiple of what the checkpoints asked for would take;
// mpm_adjoint then only runs the reverse passes of mpm_adjoint.h from
// the last step to the first.  A longer run is cut into segments of K steps,
// with a full copy of the state at the start of every segment (and at the
// end) and the steps before which the particles were re-sorted: record tapes
// the last segment, and mpm_adjoint restores each earlier one's checkpoint,
// re-runs its steps with the tape (re-sorting at the recorded steps, so the
// storage order of every step matches the recorded run, and checking that it
// ends bit for bit in the next checkpoint) and reverses it.
// The adjoint arrays follow the storage order of the step being reversed;
// where a re-sort separates two steps they are permuted through the original
// particle order, and after a segment they are left in the order of its
// checkpoint, which is the order the previous segment ends in.
// Memory: per taped step 9 floats per particle, 7 per node and 1 byte per cell
// (one more float per particle for the volume under solve semantics and one
// for the volumetric strain of a run with Newtonian particles), the material
// ids, moduli and cell starts of each sort, and one checkpoint per segment when
// there are several.
//
// mpm_batch_record / mpm_batch_adjoint do the same for every simulation of a
// batch in lockstep: each step and reverse pass is one launch for all
// simulations (the tile records carry the tape, and the reverse passes work
// over a table of per-simulation arguments).
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <map>
#include <vector>

#include "mpm_adjoint.h"
#include "mpm_batch.h"
#include "mpm_handle.h"

using namespace mpm;
using namespace mpm::host;


namespace mpm {

namespace {

constexpr int NLAM = 12;   // adjoint arrays: x y vx vy sxx syy szz sxy rho E vol vsc
constexpr int NTP = 9;     // tape per particle: x y vx vy sxx syy szz sxy rho
constexpr int NTN = 7;     // tape per node: m vAx vAy vBx vBy aBx aBy
constexpr int NPS = 5;     // per-particle scratch: r0b r1b r3b c0b c1b
constexpr int NNS = 8;     // per-node scratch: fbx fby mb vabx vaby qbx qby mbt

struct Epoch {               // arrays of one sort epoch inside a segment
    int* pid = nullptr;
    uint8_t* mat = nullptr;
    float* E = nullptr;
    int* cstart = nullptr;
    int8_t* tr_fn = nullptr;   // particle tractions (2 per particle), when present
    float* tr_tau = nullptr;
    uint8_t* pvc = nullptr;    // velocity constraint codes (2 per particle), when present
    float* mass = nullptr;     // solve semantics: the constant mass and size
    float* psize = nullptr;
};

}  // namespace

using GraphKey = std::array<int64_t, 4>;
// Executable graphs by what varies between them; a null entry has run once
// without a graph (the second time captures it: a run that happens once does
// not pay for capturing).
using GraphMap = std::map<GraphKey, cudaGraphExec_t>;

// The graphs of one configuration of the step launches: taped runs of steps
// (first slot, length, parity) and reverse runs (first and last slot, sort
// epoch, tiles), with the copy tables of the handle's buffers.
struct AdjGraphs {
    StepKey key;
    GraphMap fwd, rev;
    SegBuf tp[2], tn;          // slot copies of the start state (by parity) and of the nodal results
};

struct AdjointState {
    int interval = 0;          // the checkpoint interval asked for
    int K = 0, nseg = 0;       // the segments kept: K steps each, nseg of them
    int64_t step0 = 0, nsteps = 0;
    uint64_t gen = 0;
    bool valid = false, recording = false;
    std::vector<int64_t> resort_steps;
    std::vector<Checkpoint> ck;   // ck[s]: start of segment s; ck[nseg]: end state (several segments)
    int tape_seg = -1;         // the segment whose steps the tape holds, or -1
    uint64_t taped_with = 0;   // what taped it: BatchAdjoint::tape_id, or 0 for the handle alone
    // sized for np_alloc particles and tape_slots steps
    int64_t np_alloc = -1;
    int tape_slots = 0;
    float* tp[NTP] = {};
    float* tvol = nullptr;     // volume at each step start (solve semantics only)
    float* tvsc = nullptr;     // centroid volumetric strain at each step start (Newtonian only)
    uint8_t* tflag = nullptr;
    float* tn[NTN] = {};
    std::vector<Epoch> epochs;
    std::vector<int> epoch_of;
    int nep = 0;               // epochs captured in the current segment
    int64_t seg_first = 0;     // first step of the taped segment
    // the tiles with particles in any sort of the taped segment (the reverse
    // node passes' list), valid while every run had its empty tiles apart;
    // else (all_tiles) they visit every tile
    int* tile_union = nullptr;
    int4 *rtiles = nullptr, *rempty = nullptr;
    int nrtiles = -1;          // grid over rtiles; -1: not formed since the segment was taped
    bool all_tiles = false;
    float* lam[NLAM] = {};
    float* lam_tmp = nullptr;
    float* pscr[NPS] = {};
    float* nscr[NNS] = {};
    int* cnt = nullptr;
    int* mismatch = nullptr;   // device counter of the re-run check
    int* h_mismatch = nullptr; // pinned
    // for the most recently used configurations first; dropped whenever a
    // buffer here is (re)allocated
    std::vector<AdjGraphs> graphs;
};

// Scratch of a batched record and adjoint (owned by the batch).
struct BatchAdjoint {
    AdjStep* d_bases = nullptr;
    AdjStep* d_table = nullptr;
    std::vector<AdjStep> bases;
    int2* part_blocks = nullptr;
    int n_part_blocks = 0;
    TapeDev* d_tapes = nullptr;
    SegBuf misc;
    int* mismatch = nullptr;
    int* h_mismatch = nullptr;
    // the tiles with particles in any sort of the segment that the batch taped
    // (the one of its members whose taped_with is tape_id, unique per taping)
    uint64_t tape_id = 0;
    int* tile_union = nullptr;
    int4 *rtiles = nullptr, *rempty = nullptr;
    int nrtiles = -1;          // grid over rtiles; -1: not formed yet, -2: the set lacks a replay's sorts
    // graphs of the reverse steps (first and last slot, tiles, particle
    // blocks), valid for the buffers in `gsig`
    GraphMap g_rev;
    std::vector<uintptr_t> gsig;
};

namespace {

void free_graphs(GraphMap& m) {
    for (auto& kv : m)
        if (kv.second) cudaGraphExecDestroy(kv.second);
    m.clear();
}

void free_adj_graphs(AdjGraphs& g) {
    free_graphs(g.fwd);
    free_graphs(g.rev);
    for (SegBuf& b : g.tp) segbuf_free(b);
    segbuf_free(g.tn);
}

void drop_adj_graphs(AdjointState* a) {
    for (AdjGraphs& g : a->graphs) free_adj_graphs(g);
    a->graphs.clear();
}

void free_tape(MpmHandle* h, AdjointState* a) {
    drop_adj_graphs(a);
    for (float*& p : a->tp) { dfree(h, p); p = nullptr; }
    for (float*& p : a->tn) { dfree(h, p); p = nullptr; }
    dfree(h, a->tvol);
    a->tvol = nullptr;
    dfree(h, a->tvsc);
    a->tvsc = nullptr;
    dfree(h, a->tflag);
    a->tflag = nullptr;
    a->tape_slots = 0;
    a->tape_seg = -1;
}

void free_epochs(MpmHandle* h, AdjointState* a) {
    drop_adj_graphs(a);
    for (Epoch& e : a->epochs) {
        dfree(h, e.pid);
        dfree(h, e.mat);
        dfree(h, e.E);
        dfree(h, e.cstart);
        dfree(h, e.tr_fn);
        dfree(h, e.tr_tau);
        dfree(h, e.pvc);
        dfree(h, e.mass);
        dfree(h, e.psize);
    }
    a->epochs.clear();
}

void free_buffers(MpmHandle* h, AdjointState* a) {
    free_tape(h, a);
    for (auto& c : a->ck) checkpoint_free(h, c);
    a->ck.clear();
    dfree(h, a->tile_union);
    dfree(h, a->rtiles);
    dfree(h, a->rempty);
    a->tile_union = nullptr;
    a->rtiles = a->rempty = nullptr;
    free_epochs(h, a);
    for (float*& p : a->lam) { dfree(h, p); p = nullptr; }
    for (float*& p : a->pscr) { dfree(h, p); p = nullptr; }
    for (float*& p : a->nscr) { dfree(h, p); p = nullptr; }
    dfree(h, a->lam_tmp);
    dfree(h, a->cnt);
    dfree(h, a->mismatch);
    if (a->h_mismatch) cudaFreeHost(a->h_mismatch);
    a->mismatch = nullptr;
    a->h_mismatch = nullptr;
    a->lam_tmp = nullptr;
    a->cnt = nullptr;
    a->np_alloc = -1;
    a->valid = false;
}

// Drop everything sized for another particle count.
void fit(MpmHandle* h, AdjointState* a) {
    if (a->np_alloc != h->np) {
        free_buffers(h, a);
        a->np_alloc = h->np;
    }
}

int save_checkpoint(MpmHandle* h, AdjointState* a, size_t idx, std::vector<CopySeg>& v) {
    if (a->ck.size() <= idx) a->ck.resize(idx + 1);
    TRY(checkpoint_alloc(h, a->ck[idx]));
    checkpoint_segments(h, a->ck[idx], true, v);
    return MPM_OK;
}

int restore_checkpoint(MpmHandle* h, Checkpoint& c, cudaStream_t s) {
    std::vector<CopySeg> v;
    checkpoint_segments(h, c, false, v);
    TRY(run_segments(h, h->segbuf, v, s));
    TRY(clear_status(h, s));
    return sync(h, s);
}

// Particle slots between consecutive tape slots (np rounded up to 4).
size_t tape_stride(const MpmHandle* h) { return ((size_t)h->np + 3) & ~(size_t)3; }

bool newtonian(const MpmHandle* h) {
    for (const MatDev& m : h->mats)
        if (m.type == MAT_NEWTONIAN) return true;
    return false;
}

// A tape of `slots` steps.  Particle arrays and tape slots hold a multiple of
// 4 slots, so that every slot starts on a 16-byte boundary for the row staging
// of the step kernels and the reverse node passes (which may read up to 3
// slots past a row's end).
int ensure_tape(MpmHandle* h, AdjointState* a, int slots) {
    const size_t np = tape_stride(h), nn = (size_t)h->nn;
    if (a->tape_slots >= slots && (h->reinit || a->tvol) && (!newtonian(h) || a->tvsc)) return MPM_OK;
    free_tape(h, a);
    auto alloc = [&]() -> int {
        for (float*& p : a->tp) TRY(dalloc(h, &p, np * slots));
        if (!h->reinit) TRY(dalloc(h, &a->tvol, np * slots));
        if (newtonian(h)) TRY(dalloc(h, &a->tvsc, np * slots));
        for (float*& p : a->tn) TRY(dalloc(h, &p, nn * slots));
        return dalloc(h, &a->tflag, (size_t)h->ncell * slots);
    };
    const int r = alloc();
    if (r != MPM_OK) {
        cudaGetLastError();
        free_tape(h, a);
        return r;
    }
    a->tape_slots = slots;
    return MPM_OK;
}

int ensure_adjoint_buffers(MpmHandle* h, AdjointState* a) {
    const size_t np = tape_stride(h), nn = (size_t)h->nn;
    if (!a->lam[0]) {
        drop_adj_graphs(a);
        for (float*& p : a->lam) TRY(dalloc(h, &p, np));
        for (float*& p : a->pscr) TRY(dalloc(h, &p, np));
        for (float*& p : a->nscr) TRY(dalloc(h, &p, nn));
        TRY(dalloc(h, &a->lam_tmp, np * NLAM));
        TRY(dalloc(h, &a->cnt, (size_t)h->ncell));
        TRY(dalloc(h, &a->mismatch, 1));
        CK(h, cudaMallocHost(&a->h_mismatch, sizeof(int)));
    }
    return MPM_OK;
}

// Bytes of a taped step, with a sort epoch of its own.
size_t tape_step_bytes(const MpmHandle* h) {
    const size_t np = tape_stride(h);
    return np * (4 * (NTP + 2) + 9 + (h->has_trac ? 10 : 0) + (h->has_pvc ? 2 : 0) + (h->reinit ? 0 : 8)) +
           (size_t)h->nn * 4 * NTN + (size_t)h->ncell * 5;
}

// Bytes of a checkpoint (Checkpoint).
size_t checkpoint_bytes(MpmHandle* h) {
    const size_t nf = movable_f32(h, h->ps[h->pcur], false).size();
    return (size_t)h->np * (4 * nf + 1 + (h->has_trac ? 10 : 0) + (h->has_pvc ? 2 : 0)) + (size_t)h->ncell * 5 +
           (size_t)h->nn * 8;
}

// What a recording of one handle, or of all members of a batch, holds or would.
struct TapeNeed {
    size_t step = 0, checkpoint = 0, have = 0;   // bytes of a taped step, of a checkpoint; of the tape held
    int64_t limit = -1;                          // mpm_set_tape_limit, of a batch the least; negative: none
    void add(MpmHandle* h) {
        step += tape_step_bytes(h);
        checkpoint += checkpoint_bytes(h);
        have += tape_step_bytes(h) * (size_t)h->adj->tape_slots;
        if (h->tape_limit >= 0 && (limit < 0 || h->tape_limit < limit)) limit = h->tape_limit;
    }
};

// Whether a run of nsteps steps is taped whole rather than in segments of the
// K steps that the caller asked for: within the caller's bound, or without one
// within TAPE_OVER times what checkpoints every K steps and a segment's tape
// take (K is how a caller trades memory for re-runs), and at most a tenth of
// the device's memory and a quarter of what is free.
bool tape_whole(const TapeNeed& m, int nsteps, int K) {
    const size_t need = m.step * (size_t)nsteps, nseg = ((size_t)nsteps + K - 1) / (size_t)K;
    const size_t asked = m.checkpoint * (nseg + 1) + m.step * (size_t)std::min(K, nsteps);
    if (need > (m.limit >= 0 ? (size_t)m.limit : TAPE_OVER * asked)) return false;
    if (need <= m.have) return true;
    size_t free_b = 0, total = 0;
    if (cudaMemGetInfo(&free_b, &total) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return need <= total / 10 && need - m.have <= free_b / 4;
}

// Before a recording of `slots` taped steps: give back a longer tape (and the
// sort epochs) that is over the caller's bound or TAPE_OVER times as long, and
// the checkpoints when it keeps none.
void shrink(MpmHandle* h, AdjointState* a, const TapeNeed& m, int slots, bool checkpoints) {
    const bool over = m.limit >= 0 && m.have > (size_t)m.limit;
    if (a->tape_slots > slots && (over || (size_t)a->tape_slots > TAPE_OVER * (size_t)slots)) {
        free_tape(h, a);
        free_epochs(h, a);
    }
    if (!checkpoints) {
        for (auto& c : a->ck) checkpoint_free(h, c);
        a->ck.clear();
    }
}

void add_seg(std::vector<CopySeg>& v, const void* src, void* dst, size_t bytes, size_t step) {
    CopySeg c;
    c.src = src;
    c.dst = dst;
    c.bytes = bytes;
    c.dst_step = step;
    v.push_back(c);
}

// Segments copying the current sort epoch's order-dependent arrays into epoch slot e.
int epoch_segments(MpmHandle* h, AdjointState* a, size_t e, std::vector<CopySeg>& v) {
    const size_t np = (size_t)h->np;
    if (a->epochs.size() <= e) {
        drop_adj_graphs(a);
        Epoch ep;
        TRY(dalloc(h, &ep.pid, np));
        TRY(dalloc(h, &ep.mat, np));
        TRY(dalloc(h, &ep.cstart, (size_t)h->ncell + 2));
        a->epochs.push_back(ep);
    }
    Epoch& ep = a->epochs[e];
    if (h->has_E && !ep.E) {
        drop_adj_graphs(a);
        TRY(dalloc(h, &ep.E, np));
    }
    if (h->has_trac && !ep.tr_fn) {
        drop_adj_graphs(a);
        TRY(dalloc(h, &ep.tr_fn, 2 * np));
        TRY(dalloc(h, &ep.tr_tau, 2 * np));
    }
    if (h->has_pvc && !ep.pvc) {
        drop_adj_graphs(a);
        TRY(dalloc(h, &ep.pvc, 2 * np));
    }
    if (!h->reinit && !ep.mass) {
        drop_adj_graphs(a);
        TRY(dalloc(h, &ep.mass, np));
        TRY(dalloc(h, &ep.psize, np));
    }
    const PSet& p = h->ps[h->pcur];
    add_seg(v, p.pid, ep.pid, sizeof(int) * np, 0);
    add_seg(v, p.mat, ep.mat, np, 0);
    if (h->has_E) add_seg(v, p.E, ep.E, sizeof(float) * np, 0);
    if (h->has_trac) {
        add_seg(v, p.tr_fn, ep.tr_fn, 2 * np, 0);
        add_seg(v, p.tr_tau, ep.tr_tau, sizeof(float) * 2 * np, 0);
    }
    if (h->has_pvc) add_seg(v, p.pvc, ep.pvc, 2 * np, 0);
    if (!h->reinit) {
        add_seg(v, p.mass, ep.mass, sizeof(float) * np, 0);
        add_seg(v, p.psize, ep.psize, sizeof(float) * np, 0);
    }
    add_seg(v, h->cstart[h->cs_cur], ep.cstart, sizeof(int) * ((size_t)h->ncell + 2), 0);
    return MPM_OK;
}

int capture_epoch(MpmHandle* h, AdjointState* a, cudaStream_t s) {
    std::vector<CopySeg> v;
    TRY(epoch_segments(h, a, (size_t)a->nep, v));
    a->nep++;
    return run_segments(h, h->segbuf, v, s);
}

// Tape copies of a step that starts with ping-pong parity `par`: the particle
// state and drift flags (before the step) into slot 0 + t * stride.
void tape_particle_segments(MpmHandle* h, AdjointState* a, int par, std::vector<CopySeg>& v) {
    const PSet& p = h->ps[h->pcur];
    const size_t np = (size_t)h->np, stride = tape_stride(h);
    const float* src[NTP] = {p.x, p.y, p.vx, p.vy, p.sxx[par], p.syy[par], p.szz[par],
                             p.sxy[par], p.rho[par]};
    for (int k = 0; k < NTP; ++k) add_seg(v, src[k], a->tp[k], sizeof(float) * np, sizeof(float) * stride);
    if (!h->reinit) add_seg(v, p.vol[par], a->tvol, sizeof(float) * np, sizeof(float) * stride);
    if (a->tvsc) add_seg(v, p.vsc[par], a->tvsc, sizeof(float) * np, sizeof(float) * stride);
    add_seg(v, h->cflag, a->tflag, (size_t)h->ncell, (size_t)h->ncell);
}

// ... and the nodal results (after the step).
void tape_node_segments(MpmHandle* h, AdjointState* a, std::vector<CopySeg>& v) {
    const size_t nn = (size_t)h->nn;
    const float* src[NTN] = {h->nm, h->nvax, h->nvay, h->nvbx, h->nvby, h->nax, h->nay};
    for (int k = 0; k < NTN; ++k) add_seg(v, src[k], a->tn[k], sizeof(float) * nn, sizeof(float) * nn);
}

// Pairs (re-run state, recorded state of the next checkpoint) for the bitwise check.
void check_segments(MpmHandle* h, AdjointState* a, int seg, std::vector<CopySeg>& v) {
    const Checkpoint& next = a->ck[seg + 1];
    std::vector<float**> f = movable_f32(h, h->ps[h->pcur], false);
    for (size_t i = 0; i < f.size(); ++i) add_seg(v, *f[i], next.f[i], sizeof(float) * h->np, 0);
}

bool resorts_at(const AdjointState* a, int64_t step) {
    return std::binary_search(a->resort_steps.begin(), a->resort_steps.end(), step);
}

// The graphs of the handle's current step configuration (the first of
// a->graphs), with the tape copy tables of its buffers.
int prepare_adj_graphs(MpmHandle* h, AdjointState* a, cudaStream_t s) {
    constexpr size_t KEEP = 4;
    const StepKey key = step_key(h);
    size_t at = 0;
    while (at < a->graphs.size() && !(a->graphs[at].key == key)) ++at;
    if (at < a->graphs.size()) {
        std::rotate(a->graphs.begin(), a->graphs.begin() + at, a->graphs.begin() + at + 1);
        return MPM_OK;
    }
    if (a->graphs.size() == KEEP) {
        TRY(sync(h, s));       // none of its graphs is running
        free_adj_graphs(a->graphs.back());
        a->graphs.pop_back();
    }
    a->graphs.insert(a->graphs.begin(), AdjGraphs{key, {}, {}, {}, {}});
    AdjGraphs& g = a->graphs[0];
    for (int par = 0; par < 2; ++par) {
        std::vector<CopySeg> v;
        tape_particle_segments(h, a, par, v);
        TRY(upload_segments(h, g.tp[par], v, s));
    }
    std::vector<CopySeg> vn;
    tape_node_segments(h, a, vn);
    return upload_segments(h, g.tn, vn, s);
}

// Launch what `body` issues: directly the first time, as a graph captured on
// the handle's capture stream and kept at map[key] after that (at most
// GRAPHS_KEPT of them).
constexpr size_t GRAPHS_KEPT = 64;
template <class F>
int run_cached_graph(MpmHandle* h, GraphMap& map, const GraphKey& key, cudaStream_t s, F&& body) {
    auto it = map.find(key);
    if (it == map.end()) {
        if (map.size() >= GRAPHS_KEPT) {
            TRY(sync(h, s));   // none of them is running
            free_graphs(map);
        }
        map.emplace(key, nullptr);
        return body(s);
    }
    if (!it->second) {
        cudaGraph_t g = nullptr;
        CK(h, cudaStreamBeginCapture(h->cap, cudaStreamCaptureModeThreadLocal));
        const int r = body(h->cap);
        const cudaError_t e = cudaStreamEndCapture(h->cap, &g);
        if (r != MPM_OK || e != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            if (r != MPM_OK) return r;
            CK(h, e);
        }
        cudaGraphExec_t ex = nullptr;
        const cudaError_t ei = cudaGraphInstantiate(&ex, g, 0);
        cudaGraphDestroy(g);
        CK(h, ei);
        it->second = ex;
    }
    CK(h, cudaGraphLaunch(it->second, s));
    return MPM_OK;
}

// The handle's descriptor for step k of a taped run of len steps from slot
// `slot` (ping-pong parity par at the run's start).
SimDev slot_desc(MpmHandle* h, AdjointState* a, int slot, int k, int len, int par) {
    SimDev S = h->hs;
    const size_t sp = tape_stride(h), nn = (size_t)h->nn, nc = (size_t)h->ncell, i = (size_t)(slot + k);
    const int p = (par + k) & 1;
    const bool last = k == len - 1;
    float** in[4] = {&S.x, &S.y, &S.vx, &S.vy};
    float** to[4] = {&S.xo, &S.yo, &S.vxo, &S.vyo};
    for (int f = 0; f < 4; ++f) {
        *in[f] = a->tp[f] + i * sp;
        if (!last) *to[f] = a->tp[f] + (i + 1) * sp;
    }
    float** pair[TAPE_P - 4] = {S.sxx, S.syy, S.szz, S.sxy, S.rho, S.vol, S.vsc};
    float* tape[TAPE_P - 4] = {a->tp[4], a->tp[5], a->tp[6], a->tp[7], a->tp[8], h->reinit ? nullptr : a->tvol,
                               a->tvsc};
    for (int f = 0; f < TAPE_P - 4; ++f) {
        if (!tape[f]) continue;
        pair[f][p] = tape[f] + i * sp;
        if (!last) pair[f][p ^ 1] = tape[f] + (i + 1) * sp;
    }
    float** node[NTN] = {&S.nm, &S.nvax, &S.nvay, &S.nvbx, &S.nvby, &S.nax, &S.nay};
    if (!last)
        for (int f = 0; f < NTN; ++f) *node[f] = a->tn[f] + i * nn;
    if (k > 0) {
        S.nvpx = a->tn[3] + (i - 1) * nn;
        S.nvpy = a->tn[4] + (i - 1) * nn;
    }
    S.cflag = a->tflag + i * nc;
    if (!last) S.cflago = a->tflag + (i + 1) * nc;
    return S;
}

// The taped segment starts: its first epoch and its tile set are the current
// sort's.  Taped by a batch (`batched`), which captures the epochs of all members
// together and keeps one tile set for them, the member has no tile set of its
// own: its own adjoint then visits every tile.
int tape_begin(MpmHandle* h, AdjointState* a, int len, cudaStream_t s, bool batched = false) {
    if (!a->tile_union) {
        TRY(dalloc(h, &a->tile_union, (size_t)h->ntiles));
        TRY(dalloc(h, &a->rtiles, (size_t)h->ntiles));
        TRY(dalloc(h, &a->rempty, (size_t)h->ntiles));
    }
    if (!batched) CK(h, cudaMemsetAsync(a->tile_union, 0, sizeof(int) * (size_t)h->ntiles, s));
    // (a step writes the flags of its listed tiles' cells; those of an empty tile,
    // which a listed one beside it reads, are clear in every slot)
    CK(h, cudaMemsetAsync(a->tflag, 0, (size_t)h->ncell * (size_t)len, s));
    a->nrtiles = -1;
    a->all_tiles = batched;
    a->tape_seg = -1;
    a->taped_with = 0;
    a->seg_first = h->step;
    a->epoch_of.assign(len, 0);
    a->nep = 0;
    return batched ? MPM_OK : capture_epoch(h, a, s);
}

// Advance len steps within one sort, tape slots slot .. slot + len - 1.
int run_taped(MpmHandle* h, AdjointState* a, int slot, int len, cudaStream_t s) {
    TRY(classify_tiles(h, s));
    if (h->step_tiles == h->d_active) CK(h, launch_or_flags(a->tile_union, h->d_tile_flags, h->ntiles, s));
    else a->all_tiles = true;
    TRY(prepare_adj_graphs(h, a, s));
    AdjGraphs& g = a->graphs[0];
    const int par = parity(h);
    auto body = [&](cudaStream_t c) -> int {
        CK(h, launch_copy_segments(g.tp[par].blk, g.tp[par].nblocks, slot, c));
        for (int k = 0; k < len; ++k) {
            const SimDev S = slot_desc(h, a, slot, k, len, par);
            for (int p = 0; p < 3; ++p) TRY(launch_phase(h, S, p, k, c));
        }
        CK(h, launch_advance_step(h->ctl, len, c));
        CK(h, launch_copy_segments(g.tn.blk, g.tn.nblocks, slot + len - 1, c));
        return MPM_OK;
    };
    if (len < GRAPH_STEPS) TRY(body(s));
    else TRY(run_cached_graph(h, g.fwd, GraphKey{slot, len, par, 0}, s, body));
    for (int k = 0; k < len; ++k) a->epoch_of[slot + k] = a->nep - 1;
    h->step += len;
    return MPM_OK;
}

// replay_block with the tape: the block's B steps from slot `slot`.
int replay_taped(MpmHandle* h, AdjointState* a, int64_t step0, int slot, int B, int& st, cudaStream_t s) {
    h->rollbacks++;
    TRY(restore_snapshot(h, step0, s));
    st = 0;
    for (int i = 0; i < B; ++i) {
        if (st & ST_DRIFTED) {
            TRY(resort(h, s));
            TRY(capture_epoch(h, a, s));
        }
        TRY(run_taped(h, a, slot + i, 1, s));
        TRY(take_ctl(h, s));
        TRY(check_status(h, st));
        if (st & ST_DRIFT_VIOLATION)
            return fail(h, MPM_ERR_CFL, "a particle crossed more than one cell in one step (step %lld)",
                        (long long)h->step - 1);
    }
    return MPM_OK;
}

// Steps of the block at step `done` of a recorded run: blocks end at multiples
// of the checkpoint interval however the run is kept, so that its re-sorts,
// and with them the last bits of its sums, do not depend on that.
int block_length(const AdjointState* a, int done, int n, int block_steps) {
    return std::min({n - done, block_steps, a->interval - done % a->interval});
}

// mpm_step of the n steps of the segment being taped, the same blocks.
int taped_steps(MpmHandle* h, AdjointState* a, int n, cudaStream_t s) {
    h->gen++;
    TRY(tape_begin(h, a, n, s));
    for (int slot = 0; slot < n;) {
        const int B = block_length(a, slot, n, h->block_steps);
        if (h->needs_resort) {
            TRY(resort(h, s));
            TRY(capture_epoch(h, a, s));
        }
        const int64_t step0 = h->step;
        TRY(take_snapshot(h, s));
        TRY(run_taped(h, a, slot, B, s));
        TRY(take_ctl(h, s));
        int st = h->h_ctl->status;
        if (st & ST_DRIFT_VIOLATION) TRY(replay_taped(h, a, step0, slot, B, st, s));
        else TRY(check_status(h, st));
        h->needs_resort = (st & ST_DRIFTED) != 0;
        slot += B;
    }
    return MPM_OK;
}

// Re-run segment `seg` of one simulation from its checkpoint, filling tape
// slots 0..len-1, and check that it ends in the next checkpoint's state.
int recompute_segment(MpmHandle* h, AdjointState* a, int seg, int len, cudaStream_t s) {
    TRY(restore_checkpoint(h, a->ck[seg], s));
    const int64_t first = a->ck[seg].step;
    TRY(tape_begin(h, a, len, s));
    for (int t = 0; t < len;) {
        if (resorts_at(a, first + t)) {
            TRY(resort(h, s));
            TRY(capture_epoch(h, a, s));
        }
        int t1 = t + 1;
        while (t1 < len && !resorts_at(a, first + t1)) ++t1;
        TRY(run_taped(h, a, t, t1 - t, s));
        t = t1;
    }
    TRY(read_ctl(h, s));
    int st = 0;
    TRY(check_status(h, st));
    // the re-run must end bit for bit in the recorded state of the next checkpoint
    std::vector<CopySeg> vc;
    check_segments(h, a, seg, vc);
    SegBuf cb;
    int r = upload_segments(h, cb, vc, s);
    if (r == MPM_OK) {
        cudaError_t e = cudaMemsetAsync(a->mismatch, 0, sizeof(int), s);
        if (e == cudaSuccess) e = launch_compare_segments(cb.blk, cb.nblocks, a->mismatch, s);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(a->h_mismatch, a->mismatch, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e != cudaSuccess) r = fail(h, MPM_ERR_CUDA, "re-run check: %s", cudaGetErrorString(e));
        if (r == MPM_OK) r = sync(h, s);
    }
    segbuf_free(cb);
    TRY(r);
    if ((st & ST_DRIFT_VIOLATION) || *a->h_mismatch != 0 || h->step != a->ck[seg + 1].step)
        return fail(h, MPM_ERR_STATE,
                    "re-run of steps %lld..%lld did not reproduce the recorded run (%d words differ)",
                    (long long)first, (long long)(first + len - 1), *a->h_mismatch);
    a->tape_seg = seg;
    return clear_status(h, s);
}

// Adjoint arrays first .. first + ncomp - 1, stored in the order `pid`,
// against the original-order array `aos`.
FieldMap lam_map(MpmHandle* h, AdjointState* a, int first, int ncomp, const int* pid, const float* aos) {
    FieldMap F{};
    for (int k = 0; k < ncomp; ++k) {
        F.comp[k] = a->lam[first + k];
        F.slot[k] = -1;
    }
    F.ncomp = ncomp;
    F.np = (int)h->np;
    F.pid = pid;
    F.aos = const_cast<float*>(aos);
    return F;
}

// Move the adjoint arrays from the storage order `from` to the storage order `to`.
int permute(MpmHandle* h, AdjointState* a, const int* from, const int* to, cudaStream_t s) {
    if (from == to) return MPM_OK;
    CK(h, launch_field(lam_map(h, a, 0, NLAM, from, a->lam_tmp), false, s));
    CK(h, launch_field(lam_map(h, a, 0, NLAM, to, a->lam_tmp), true, s));
    return MPM_OK;
}

// Reverse-pass arguments with the tape at slot 0 and the epoch of slot t.
AdjStep base_args(MpmHandle* h, AdjointState* a, int epoch) {
    const Epoch& ep = a->epochs[epoch];
    AdjStep A{};
    A.nx = h->nx;
    A.ny = h->ny;
    A.np = (int)h->np;
    A.hx = h->hx;
    A.hy = h->hy;
    A.dt = h->dt;
    A.vol_el = h->vol_el;
    A.gx = h->gx;
    A.gy = h->gy;
    A.velocity_update = h->velocity_update;
    A.ncons = h->d_ncons;
    A.mats = h->d_mats;
    A.cstart = ep.cstart;
    A.mat = ep.mat;
    A.E = h->has_E ? ep.E : nullptr;
    A.tr_fn = h->has_trac ? ep.tr_fn : nullptr;
    A.tr_tau = h->has_trac ? ep.tr_tau : nullptr;
    A.pvc = h->has_pvc ? ep.pvc : nullptr;
    A.reinit = h->reinit ? 1 : 0;
    A.vol = h->reinit ? nullptr : a->tvol;
    A.mass = h->reinit ? nullptr : ep.mass;
    A.psize = h->reinit ? nullptr : ep.psize;
    A.vsc = a->tvsc;
    A.fn_off = h->d_fn_off;
    A.fn_x = h->d_fn_x;
    A.fn_y = h->d_fn_y;
    A.step = (int)a->seg_first;
    const float** tp[NTP] = {&A.x, &A.y, &A.vx, &A.vy, &A.sxx, &A.syy, &A.szz, &A.sxy, &A.rho};
    for (int k = 0; k < NTP; ++k) *tp[k] = a->tp[k];
    A.cflag = a->tflag;
    const float** tn[NTN] = {&A.nm, &A.nvax, &A.nvay, &A.nvbx, &A.nvby, &A.nax, &A.nay};
    for (int k = 0; k < NTN; ++k) *tn[k] = a->tn[k];
    float** lam[NLAM] = {&A.lx, &A.ly, &A.lvx, &A.lvy, &A.lsxx, &A.lsyy, &A.lszz, &A.lsxy,
                         &A.lrho, &A.lE, &A.lvol, &A.lvsc};
    for (int k = 0; k < NLAM; ++k) *lam[k] = a->lam[k];
    float** ps[NPS] = {&A.r0b, &A.r1b, &A.r3b, &A.c0b, &A.c1b};
    for (int k = 0; k < NPS; ++k) *ps[k] = a->pscr[k];
    float** ns[NNS] = {&A.fbx, &A.fby, &A.mb, &A.vabx, &A.vaby, &A.qbx, &A.qby, &A.mbt};
    for (int k = 0; k < NNS; ++k) *ns[k] = a->nscr[k];
    A.cnt = a->cnt;
    A.sp = (long long)tape_stride(h);
    A.sn = h->nn;
    A.sc = h->ncell;
    return A;
}

// The tiles the reverse node passes visit: those with particles in some sort
// of the taped segment (an empty tile's node adjoints and cell counts are
// read by no particle), or every tile.
int reverse_tiles(MpmHandle* h, AdjointState* a, const int4*& tiles, int& ntiles, cudaStream_t s) {
    if (a->all_tiles) {
        tiles = h->dtiles;
        ntiles = h->ntiles;
        return MPM_OK;
    }
    if (a->nrtiles < 0) {
        CK(h, launch_compact_tiles(a->tile_union, h->dtiles, h->ntiles, a->rtiles, a->rempty, h->d_tile_counts, s));
        CK(h, cudaMemcpyAsync(h->h_tile_counts, h->d_tile_counts, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
        TRY(sync(h, s));
        a->nrtiles = tile_grid(h->h_tile_counts[0], h->ntiles);
    }
    tiles = a->rtiles;
    ntiles = a->nrtiles;
    return MPM_OK;
}

int reverse_step(MpmHandle* h, AdjointState* a, int t, const int4* tiles, int ntiles, cudaStream_t s) {
    AdjStep A = base_args(h, a, a->epoch_of[t]);
    const size_t op = (size_t)t * A.sp, on = (size_t)t * A.sn, oc = (size_t)t * A.sc;
    A.x += op; A.y += op; A.vx += op; A.vy += op;
    A.sxx += op; A.syy += op; A.szz += op; A.sxy += op; A.rho += op;
    if (A.vol) A.vol += op;
    if (A.vsc) A.vsc += op;
    A.cflag += oc;
    A.nm += on; A.nvax += on; A.nvay += on; A.nvbx += on; A.nvby += on; A.nax += on; A.nay += on;
    A.step += t;
    CK(h, launch_rev_step(A, h->usl, h->has_trac, tiles, ntiles, s));
    return MPM_OK;
}

// The reverse steps t1 .. t0, of one sort epoch (tractions need the step
// number, which a graph would hold by value).
int reverse_run(MpmHandle* h, AdjointState* a, int t0, int t1, cudaStream_t s) {
    const int4* tiles;
    int ntiles;
    TRY(reverse_tiles(h, a, tiles, ntiles, s));
    auto body = [&](cudaStream_t c) -> int {
        for (int t = t1; t >= t0; --t) TRY(reverse_step(h, a, t, tiles, ntiles, c));
        return MPM_OK;
    };
    if (h->has_trac || t1 - t0 + 1 < GRAPH_STEPS) return body(s);
    TRY(prepare_adj_graphs(h, a, s));
    const int64_t grid = (int64_t)ntiles * 2 + (tiles == a->rtiles);
    return run_cached_graph(h, a->graphs[0].rev, GraphKey{t0, t1, a->epoch_of[t0], grid}, s, body);
}

// Zero the adjoint arrays; particle (n, 2) seeds in original order -> lam[0..3]
// in the storage order `pid`.
int seed(MpmHandle* h, AdjointState* a, const float* dl_dloc, const float* dl_dvel,
         const int* pid, int on_device, cudaStream_t s) {
    CK(h, launch_field(lam_map(h, a, 0, NLAM, pid, nullptr), true, s));
    const float* src[2] = {dl_dloc, dl_dvel};
    for (int k = 0; k < 2; ++k) {
        if (!src[k]) continue;
        const void* d = nullptr;
        TRY(to_device(h, src[k], sizeof(float) * 2 * h->np, on_device, s, &d));
        CK(h, launch_field(lam_map(h, a, 2 * k, 2, pid, static_cast<const float*>(d)), true, s));
        TRY(sync(h, s));
    }
    return MPM_OK;
}

// Adjoint arrays lam[first..] in storage order `pid` -> particle (n, ncomp)
// array in original order.
int emit(MpmHandle* h, AdjointState* a, float* dst, int first, int ncomp, const int* pid,
         int on_device, cudaStream_t s) {
    if (!dst) return MPM_OK;
    const size_t bytes = sizeof(float) * ncomp * h->np;
    float* d = dst;
    if (!on_device) {
        TRY(ensure_stage(h, bytes));
        d = static_cast<float*>(h->stage);
    }
    CK(h, launch_field(lam_map(h, a, first, ncomp, pid, d), false, s));
    if (!on_device) CK(h, cudaMemcpyAsync(dst, d, bytes, cudaMemcpyDeviceToHost, s));
    return sync(h, s);
}

int emit_all(MpmHandle* h, AdjointState* a, float* dl_dE, float* dl_dloc0, float* dl_dvel0,
             int on_device, cudaStream_t s) {
    const int* pid = a->epochs[0].pid;   // the order of the first checkpoint
    TRY(emit(h, a, dl_dE, 9, 1, pid, on_device, s));
    TRY(emit(h, a, dl_dloc0, 0, 2, pid, on_device, s));
    return emit(h, a, dl_dvel0, 2, 2, pid, on_device, s);
}

int check_supported(MpmHandle* h) {
    if (h->ndim != 2) return fail(h, MPM_ERR_UNSUPPORTED, "the adjoint implements Quadrilateral4Node meshes");
    return MPM_OK;
}

// Record the run in segments of K steps.
void record_segments(AdjointState* a, int K) {
    a->K = K;
    a->nseg = (int)((a->nsteps + K - 1) / K);
}

// Start a recording on h: checks, state and bookkeeping.
int record_begin(MpmHandle* h, int nsteps, int K) {
    if (!h->initialized) return fail(h, MPM_ERR_STATE, "initialize first");
    if (nsteps < 1 || K < 1) return fail(h, MPM_ERR_INVALID, "nsteps and checkpoint_steps must be >= 1");
    if (h->np <= 0) return fail(h, MPM_ERR_STATE, "no particles");
    TRY(check_supported(h));
    if (!h->adj) h->adj = new AdjointState();
    AdjointState* a = h->adj;
    fit(h, a);
    a->valid = false;
    a->tape_seg = -1;
    a->resort_steps.clear();
    a->step0 = h->step;
    a->nsteps = nsteps;
    a->interval = K;
    record_segments(a, K);
    a->recording = true;
    return MPM_OK;
}

void record_end(MpmHandle* h, bool ok) {
    AdjointState* a = h->adj;
    a->recording = false;
    if (!ok) return;
    std::sort(a->resort_steps.begin(), a->resort_steps.end());
    a->resort_steps.erase(std::unique(a->resort_steps.begin(), a->resort_steps.end()),
                          a->resort_steps.end());
    a->gen = h->gen;
    a->valid = true;
}

int check_recorded(MpmHandle* h) {
    AdjointState* a = h->adj;
    if (!a || !a->valid || a->np_alloc != h->np) return fail(h, MPM_ERR_STATE, "call mpm_record first");
    if (a->gen != h->gen) return fail(h, MPM_ERR_STATE, "the simulation changed since mpm_record");
    return MPM_OK;
}

}  // namespace

void adjoint_note_resort(MpmHandle* h) {
    if (h->adj && h->adj->recording) h->adj->resort_steps.push_back(h->step);
}

void adjoint_free(MpmHandle* h) {
    if (!h->adj) return;
    free_buffers(h, h->adj);
    delete h->adj;
    h->adj = nullptr;
}

// The buffers the batched reverse graphs hold; the cached graphs are dropped
// when any of them changed.
void check_batch_adj_graphs(MpmBatch* b, BatchAdjoint* x) {
    const std::vector<uintptr_t> sig = {(uintptr_t)x->d_bases, (uintptr_t)x->d_table, (uintptr_t)x->part_blocks,
                                        (uintptr_t)x->n_part_blocks, (uintptr_t)x->rtiles,
                                        (uintptr_t)b->sims.size()};
    if (sig != x->gsig) {
        free_graphs(x->g_rev);
        x->gsig = sig;
    }
}

void batch_adjoint_free(MpmBatch* b) {
    BatchAdjoint* x = b->badj;
    if (!x) return;
    free_graphs(x->g_rev);
    cudaFree(x->d_tapes);
    cudaFree(x->tile_union);
    cudaFree(x->rtiles);
    cudaFree(x->rempty);
    cudaFree(x->d_bases);
    cudaFree(x->d_table);
    cudaFree(x->part_blocks);
    cudaFree(x->mismatch);
    if (x->h_mismatch) cudaFreeHost(x->h_mismatch);
    segbuf_free(x->misc);
    delete x;
    b->badj = nullptr;
}

}  // namespace mpm

using namespace mpm::batch;

namespace {

int ensure_batch_tape(MpmBatch* b) {
    if (!b->badj) b->badj = new BatchAdjoint();
    BatchAdjoint* x = b->badj;
    const size_t nt = (size_t)b->ntiles;
    if (!x->tile_union) BCK(b, cudaMalloc(&x->tile_union, sizeof(int) * nt));
    if (!x->rtiles) BCK(b, cudaMalloc(&x->rtiles, sizeof(int4) * nt));
    if (!x->rempty) BCK(b, cudaMalloc(&x->rempty, sizeof(int4) * nt));
    if (!x->d_tapes) BCK(b, cudaMalloc(&x->d_tapes, sizeof(TapeDev) * b->sims.size()));
    return MPM_OK;
}

// Capture the current sort of the listed members as their next epoch.
int capture_epochs(MpmBatch* b, BatchAdjoint* x, const std::vector<int>& members, cudaStream_t s) {
    std::vector<CopySeg> v;
    for (int i : members) {
        AdjointState* a = b->sims[i]->adj;
        BTRY(b, i, epoch_segments(b->sims[i], a, (size_t)a->nep, v));
        a->nep++;
    }
    BTRY(b, 0, run_segments(b->sims[0], x->misc, v, s));
    return MPM_OK;
}

// tape_begin for every member.
int batch_tape_begin(MpmBatch* b, BatchAdjoint* x, int len, cudaStream_t s) {
    static std::atomic<uint64_t> tapings{0};   // (a member may belong to several batches)
    std::vector<int> every;
    BCK(b, cudaMemsetAsync(x->tile_union, 0, sizeof(int) * (size_t)b->ntiles, s));
    x->nrtiles = -1;
    x->tape_id = ++tapings;
    for (int i = 0; i < (int)b->sims.size(); ++i) {
        BTRY(b, i, tape_begin(b->sims[i], b->sims[i]->adj, len, s, true));
        b->sims[i]->adj->taped_with = x->tape_id;
        every.push_back(i);
    }
    return capture_epochs(b, x, every, s);
}

// run_taped for every member (slots slot .. slot + len - 1 of each).
int batch_run_taped(MpmBatch* b, BatchAdjoint* x, int slot, int len, cudaStream_t s) {
    const int n = (int)b->sims.size();
    std::vector<TapeDev> tapes(n);
    std::vector<CopySeg> v;
    for (int i = 0; i < n; ++i) {
        MpmHandle* h = b->sims[i];
        AdjointState* a = h->adj;
        TapeDev& T = tapes[i];
        for (int k = 0; k < NTP; ++k) T.p[k] = a->tp[k];
        T.p[NTP] = h->reinit ? nullptr : a->tvol;
        T.p[NTP + 1] = a->tvsc;
        for (int k = 0; k < NTN; ++k) T.n[k] = a->tn[k];
        T.cflag = a->tflag;
        T.sp = (long long)tape_stride(h);
        T.sn = h->nn;
        T.sc = h->ncell;
        T.step0 = (int)a->seg_first;
        T.first = (int)h->step;
        T.last = (int)h->step + len - 1;
        T.pad = 0;
        tape_particle_segments(h, a, parity(h), v);
    }
    BCK(b, cudaMemcpyAsync(x->d_tapes, tapes.data(), sizeof(TapeDev) * n, cudaMemcpyHostToDevice, s));
    BTRY(b, 0, upload_segments(b->sims[0], x->misc, v, s));
    BCK(b, launch_copy_segments(x->misc.blk, x->misc.nblocks, slot, s));
    int r = prepare_tiles(b, s, x->d_tapes);
    if (r != MPM_OK) return r;
    BCK(b, launch_or_flags(x->tile_union, b->d_tflags, b->ntiles, s));
    r = run_batch_steps(b, len, s);
    if (r != MPM_OK) return r;
    v.clear();
    for (MpmHandle* h : b->sims) tape_node_segments(h, h->adj, v);
    BTRY(b, 0, upload_segments(b->sims[0], x->misc, v, s));
    BCK(b, launch_copy_segments(x->misc.blk, x->misc.nblocks, slot + len - 1, s));
    for (MpmHandle* h : b->sims) {
        for (int k = 0; k < len; ++k) h->adj->epoch_of[slot + k] = h->adj->nep - 1;
        h->step += len;
    }
    return MPM_OK;
}

// batch_steps of the n steps of the segment being taped, the same blocks.
int batch_taped_steps(MpmBatch* b, BatchAdjoint* x, int n, cudaStream_t s) {
    int r = batch_tape_begin(b, x, n, s);
    for (int slot = 0; slot < n && r == MPM_OK;) {
        const int B = block_length(b->sims[0]->adj, slot, n, b->block_steps);
        std::vector<int> resorted;
        r = block_resorts(b, resorted, s);
        if (r == MPM_OK && !resorted.empty()) r = capture_epochs(b, x, resorted, s);
        if (r == MPM_OK) r = snapshot_all(b, s);
        if (r != MPM_OK) break;
        std::vector<int64_t> step0;
        for (MpmHandle* h : b->sims) step0.push_back(h->step);
        r = batch_run_taped(b, x, slot, B, s);
        if (r == MPM_OK) r = read_statuses(b, s);
        for (int i = 0; i < (int)b->sims.size() && r == MPM_OK; ++i) {
            MpmHandle* h = b->sims[i];
            h->gen++;
            int st = b->h_status[i].status;
            if (st & ST_DRIFT_VIOLATION) {
                BTRY(b, i, replay_taped(h, h->adj, step0[i], slot, B, st, s));
                x->nrtiles = -2;   // the replay's sorts are not in the batch's tile set
            } else if (st & ST_OUT_OF_MESH) {
                return bfail(b, MPM_ERR_OUT_OF_MESH, "simulation %d: a particle left the mesh", i);
            }
            h->needs_resort = (st & ST_DRIFTED) != 0;
        }
        slot += B;
    }
    return r;
}

// The tiles of the batched reverse node passes (reverse_tiles): every tile when a
// member's segment was not taped with the batch's present tile set (members may
// be recorded one by one).
int batch_reverse_tiles(MpmBatch* b, BatchAdjoint* x, const int4*& tiles, int& ntiles, cudaStream_t s) {
    bool apart = x->nrtiles == -2;
    for (const MpmHandle* h : b->sims) apart = apart || !x->tape_id || h->adj->taped_with != x->tape_id;
    if (apart) {
        tiles = b->d_tiles;
        ntiles = b->ntiles;
        return MPM_OK;
    }
    if (x->nrtiles < 0) {
        BCK(b, launch_compact_tiles(x->tile_union, b->d_tiles, b->ntiles, x->rtiles, x->rempty, b->d_tcounts, s));
        BCK(b, cudaMemcpyAsync(b->h_tcounts, b->d_tcounts, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
        BCK(b, cudaStreamSynchronize(s));
        x->nrtiles = tile_grid(b->h_tcounts[0], b->ntiles);
    }
    tiles = x->rtiles;
    ntiles = x->nrtiles;
    return MPM_OK;
}

// Batched re-run of segment `seg` of every simulation (tape slots 0..len-1),
// with the bitwise check against the next checkpoints.
int batch_recompute(MpmBatch* b, BatchAdjoint* x, int seg, int len, cudaStream_t s) {
    const int n = (int)b->sims.size();
    std::vector<CopySeg> v;
    for (int i = 0; i < n; ++i) checkpoint_segments(b->sims[i], b->sims[i]->adj->ck[seg], false, v);
    BTRY(b, 0, run_segments(b->sims[0], x->misc, v, s));
    int r = read_statuses(b, s);   // (clears the restored status words)
    if (r == MPM_OK) r = batch_tape_begin(b, x, len, s);
    if (r != MPM_OK) return r;
    std::vector<int64_t> first(n);
    for (int i = 0; i < n; ++i) first[i] = b->sims[i]->step;
    for (int t = 0; t < len;) {
        std::vector<int> due;
        for (int i = 0; i < n; ++i)
            if (resorts_at(b->sims[i]->adj, first[i] + t)) due.push_back(i);
        if (!due.empty()) {
            r = resort_many(b, due, s);
            if (r == MPM_OK) r = capture_epochs(b, x, due, s);
            if (r != MPM_OK) return r;
        }
        int t1 = t + 1;
        auto any_due = [&](int u) {
            for (int i = 0; i < n; ++i)
                if (resorts_at(b->sims[i]->adj, first[i] + u)) return true;
            return false;
        };
        while (t1 < len && !any_due(t1)) ++t1;
        r = batch_run_taped(b, x, t, t1 - t, s);
        if (r != MPM_OK) return r;
        t = t1;
    }
    r = read_statuses(b, s);
    if (r != MPM_OK) return r;
    v.clear();
    for (int i = 0; i < n; ++i) {
        const int st = b->h_status[i].status;
        if (st & (ST_DRIFT_VIOLATION | ST_OUT_OF_MESH))
            return bfail(b, MPM_ERR_STATE, "simulation %d: re-run of segment %d left the recorded run",
                         i, seg);
        if (b->sims[i]->step != b->sims[i]->adj->ck[seg + 1].step)
            return bfail(b, MPM_ERR_STATE, "simulation %d: step count of the re-run differs", i);
        check_segments(b->sims[i], b->sims[i]->adj, seg, v);
    }
    BTRY(b, 0, upload_segments(b->sims[0], x->misc, v, s));
    BCK(b, cudaMemsetAsync(x->mismatch, 0, sizeof(int), s));
    BCK(b, launch_compare_segments(x->misc.blk, x->misc.nblocks,
                                   x->mismatch, s));
    BCK(b, cudaMemcpyAsync(x->h_mismatch, x->mismatch, sizeof(int), cudaMemcpyDeviceToHost, s));
    BCK(b, cudaStreamSynchronize(s));
    if (*x->h_mismatch != 0)
        return bfail(b, MPM_ERR_STATE, "re-run of segment %d did not reproduce the recorded run "
                     "(%d words differ)", seg, *x->h_mismatch);
    for (MpmHandle* h : b->sims) h->adj->tape_seg = seg;
    return MPM_OK;
}

// seed() for every member, one launch per seed array.  A host seed is staged in
// its member's own staging buffer; the second seed's copy follows the first
// one's transfer on the stream.
int batch_seed(MpmBatch* b, const float* const* dl_dloc, const float* const* dl_dvel, int len, int on_device,
               cudaStream_t s) {
    const int n = (int)b->sims.size();
    std::vector<FieldMap> maps;
    auto order = [&](MpmHandle* h) { return h->adj->epochs[h->adj->epoch_of[len - 1]].pid; };
    for (MpmHandle* h : b->sims) maps.push_back(lam_map(h, h->adj, 0, NLAM, order(h), nullptr));
    int r = fields_many(b, maps, true, s);
    const float* const* src[2] = {dl_dloc, dl_dvel};
    for (int k = 0; k < 2 && r == MPM_OK; ++k) {
        if (!src[k]) continue;
        maps.clear();
        for (int i = 0; i < n; ++i) {
            MpmHandle* h = b->sims[i];
            if (!src[k][i]) continue;
            const void* d = nullptr;
            BTRY(b, i, to_device(h, src[k][i], sizeof(float) * 2 * h->np, on_device, s, &d));
            maps.push_back(lam_map(h, h->adj, 2 * k, 2, order(h), static_cast<const float*>(d)));
        }
        r = fields_many(b, maps, true, s);
    }
    return r;
}

// emit() for every member with a destination, one launch; the caller
// synchronises the stream before it returns.
int batch_emit(MpmBatch* b, float* const* dst, int first, int ncomp, int on_device, cudaStream_t s) {
    const int n = (int)b->sims.size();
    std::vector<FieldMap> maps;
    for (int i = 0; i < n; ++i) {
        MpmHandle* h = b->sims[i];
        if (!dst[i]) continue;
        float* d = dst[i];
        if (!on_device) {
            BTRY(b, i, ensure_stage(h, sizeof(float) * ncomp * h->np));
            d = static_cast<float*>(h->stage);
        }
        maps.push_back(lam_map(h, h->adj, first, ncomp, h->adj->epochs[0].pid, d));
    }
    const int r = fields_many(b, maps, false, s);
    if (r != MPM_OK || on_device) return r;
    for (int i = 0; i < n; ++i) {
        MpmHandle* h = b->sims[i];
        if (dst[i])
            BCK(b, cudaMemcpyAsync(dst[i], h->stage, sizeof(float) * ncomp * h->np, cudaMemcpyDeviceToHost, s));
    }
    return MPM_OK;
}

int ensure_batch_adjoint(MpmBatch* b, cudaStream_t s) {
    if (!b->badj) b->badj = new BatchAdjoint();
    BatchAdjoint* x = b->badj;
    const int n = (int)b->sims.size();
    if (!x->d_bases) {
        BCK(b, cudaMalloc(&x->d_bases, sizeof(AdjStep) * n));
        BCK(b, cudaMalloc(&x->d_table, sizeof(AdjStep) * n));
        BCK(b, cudaMalloc(&x->mismatch, sizeof(int)));
        BCK(b, cudaMallocHost(&x->h_mismatch, sizeof(int)));
    }
    // block maps (particle counts may have changed since the last call)
    std::vector<int2> pb;
    for (int i = 0; i < n; ++i) {
        const MpmHandle* h = b->sims[i];
        for (int c = 0; c * ADJ_BLOCK * ADJ_ITER < h->np; ++c) pb.push_back(make_int2(i, c));
    }
    cudaFree(x->part_blocks);
    x->part_blocks = nullptr;
    BCK(b, cudaMalloc(&x->part_blocks, sizeof(int2) * pb.size()));
    BCK(b, cudaMemcpyAsync(x->part_blocks, pb.data(), sizeof(int2) * pb.size(), cudaMemcpyHostToDevice, s));
    BCK(b, cudaStreamSynchronize(s));
    x->n_part_blocks = (int)pb.size();
    return MPM_OK;
}

}  // namespace

extern "C" {

int mpm_record(MpmHandle* h, int nsteps, int checkpoint_steps, void* stream) {
    if (!h) return MPM_ERR_INVALID;
    if (h->ndim == 1) return line_record(h, nsteps, S(stream));   // full tape, no checkpoints
    TRY(record_begin(h, nsteps, checkpoint_steps));
    cudaStream_t s = S(stream);
    AdjointState* a = h->adj;
    TapeNeed need;
    need.add(h);
    if (tape_whole(need, nsteps, checkpoint_steps)) record_segments(a, nsteps);
    shrink(h, a, need, std::min(a->K, nsteps), a->nseg > 1);
    bool taped = ensure_tape(h, a, std::min(a->K, nsteps)) == MPM_OK;
    if (!taped && a->K > checkpoint_steps) {
        record_segments(a, checkpoint_steps);
        taped = ensure_tape(h, a, std::min(a->K, nsteps)) == MPM_OK;
    }
    // (without memory for a tape the run keeps checkpoints only)
    const bool checkpoints = !taped || a->nseg > 1;
    int r = MPM_OK;
    for (int seg = 0; seg <= a->nseg && r == MPM_OK; ++seg) {
        if (checkpoints) {
            std::vector<CopySeg> v;
            r = save_checkpoint(h, a, seg, v);
            if (r == MPM_OK) r = run_segments(h, h->segbuf, v, s);
        }
        if (r != MPM_OK || seg == a->nseg) break;
        const int len = std::min(a->K, nsteps - seg * a->K);
        if (taped && seg == a->nseg - 1) r = taped_steps(h, a, len, s);
        else r = mpm_step(h, len, stream);
    }
    if (r == MPM_OK) r = sync(h, s);
    if (r == MPM_OK && taped) a->tape_seg = a->nseg - 1;
    record_end(h, r == MPM_OK);
    return r;
}

int mpm_adjoint(MpmHandle* h, const float* dl_dloc, const float* dl_dvel, float* dl_dE,
                float* dl_dloc0, float* dl_dvel0, int on_device, void* stream) {
    if (!h) return MPM_ERR_INVALID;
    if (h->ndim == 1)
        return line_adjoint(h, dl_dloc, dl_dvel, dl_dE, dl_dloc0, dl_dvel0, on_device, S(stream));
    TRY(check_recorded(h));
    if (!dl_dloc) return fail(h, MPM_ERR_INVALID, "dl_dloc is null");
    AdjointState* a = h->adj;
    cudaStream_t s = S(stream);
    TRY(ensure_adjoint_buffers(h, a));
    TRY(ensure_tape(h, a, (int)std::min<int64_t>(a->K, a->nsteps)));
    int r = MPM_OK;
    bool moved = false;
    for (int seg = a->nseg - 1; seg >= 0 && r == MPM_OK; --seg) {
        const int len = (int)std::min<int64_t>(a->K, a->nsteps - (int64_t)seg * a->K);
        if (a->tape_seg != seg) {
            moved = true;
            r = recompute_segment(h, a, seg, len, s);
        }
        // the seeds go to the order of the last step, the recorded end state's
        if (r == MPM_OK && seg == a->nseg - 1)
            r = seed(h, a, dl_dloc, dl_dvel, a->epochs[a->epoch_of[len - 1]].pid, on_device, s);
        for (int t1 = len - 1; t1 >= 0 && r == MPM_OK;) {
            const int e = a->epoch_of[t1];
            if (t1 < len - 1) r = permute(h, a, a->epochs[a->epoch_of[t1 + 1]].pid, a->epochs[e].pid, s);
            int t0 = t1;
            while (t0 > 0 && a->epoch_of[t0 - 1] == e) --t0;
            if (r == MPM_OK) r = reverse_run(h, a, t0, t1, s);
            t1 = t0 - 1;
        }
        if (r == MPM_OK && a->epoch_of[0] != 0)
            r = permute(h, a, a->epochs[a->epoch_of[0]].pid, a->epochs[0].pid, s);
    }
    if (r == MPM_OK) r = emit_all(h, a, dl_dE, dl_dloc0, dl_dvel0, on_device, s);
    // leave the handle at the recorded end state (where the re-runs moved it)
    const int r2 = moved ? restore_checkpoint(h, a->ck[a->nseg], s) : sync(h, s);
    TRY(r);
    return r2;
}

int mpm_batch_record(MpmBatch* b, int nsteps, int checkpoint_steps, void* stream) {
    if (!b) return MPM_ERR_INVALID;
    int r = check_ready(b);
    if (r != MPM_OK) return r;
    const int n = (int)b->sims.size();
    for (int i = 0; i < n; ++i) BTRY(b, i, record_begin(b->sims[i], nsteps, checkpoint_steps));
    cudaStream_t s = S(stream);
    TapeNeed need;   // of the whole batch
    for (MpmHandle* h : b->sims) need.add(h);
    auto ensure_tapes = [&](int K) {
        for (MpmHandle* h : b->sims) {
            record_segments(h->adj, K);
            if (ensure_tape(h, h->adj, std::min(K, nsteps)) != MPM_OK) return false;
        }
        return true;
    };
    const bool whole = tape_whole(need, nsteps, checkpoint_steps);
    const int slots = whole ? nsteps : std::min(checkpoint_steps, nsteps);
    for (MpmHandle* h : b->sims) shrink(h, h->adj, need, slots, slots < nsteps);
    bool taped = ensure_batch_tape(b) == MPM_OK && ensure_tapes(whole ? nsteps : checkpoint_steps);
    if (!taped && whole) {
        for (MpmHandle* h : b->sims) free_tape(h, h->adj);
        taped = ensure_batch_tape(b) == MPM_OK && ensure_tapes(checkpoint_steps);
    }
    // (without memory for the tapes the run keeps checkpoints only)
    for (MpmHandle* h : b->sims)
        if (!taped) record_segments(h->adj, checkpoint_steps);
    const int K = b->sims[0]->adj->K, nseg = b->sims[0]->adj->nseg;
    const bool checkpoints = !taped || nseg > 1;
    for (int seg = 0; seg <= nseg && r == MPM_OK; ++seg) {
        if (checkpoints) {
            std::vector<CopySeg> v;
            for (int i = 0; i < n && r == MPM_OK; ++i) {
                r = save_checkpoint(b->sims[i], b->sims[i]->adj, seg, v);
                if (r != MPM_OK) r = from_sim(b, i, r);
            }
            if (r == MPM_OK && run_segments(b->sims[0], b->segbuf, v, s) != MPM_OK)
                r = from_sim(b, 0, MPM_ERR_CUDA);
        }
        if (r != MPM_OK || seg == nseg) break;
        const int len = std::min(K, nsteps - seg * K);
        r = taped && seg == nseg - 1 ? batch_taped_steps(b, b->badj, len, s) : batch_steps(b, len, s);
    }
    if (r == MPM_OK && cudaStreamSynchronize(s) != cudaSuccess) r = bfail(b, MPM_ERR_CUDA, "synchronise");
    for (MpmHandle* h : b->sims) {
        if (r == MPM_OK && taped) h->adj->tape_seg = nseg - 1;
        record_end(h, r == MPM_OK);
    }
    return r;
}

int mpm_batch_adjoint(MpmBatch* b, const float* const* dl_dloc, const float* const* dl_dvel,
                      float* const* dl_dE, float* const* dl_dloc0, float* const* dl_dvel0,
                      int on_device, void* stream) {
    if (!b) return MPM_ERR_INVALID;
    if (!dl_dloc) return bfail(b, MPM_ERR_INVALID, "dl_dloc is null");
    const int n = (int)b->sims.size();
    for (int i = 0; i < n; ++i) {
        MpmHandle* h = b->sims[i];
        BTRY(b, i, check_recorded(h));
        if (h->adj->nsteps != b->sims[0]->adj->nsteps || h->adj->K != b->sims[0]->adj->K)
            return bfail(b, MPM_ERR_STATE, "simulation %d was recorded apart from the batch", i);
        if (!dl_dloc[i]) return bfail(b, MPM_ERR_INVALID, "dl_dloc[%d] is null", i);
    }
    cudaStream_t s = S(stream);
    const int K = b->sims[0]->adj->K, nseg = b->sims[0]->adj->nseg;
    const int64_t nsteps = b->sims[0]->adj->nsteps;
    int r = ensure_batch_adjoint(b, s);
    if (r != MPM_OK) return r;
    BatchAdjoint* x = b->badj;
    r = ensure_batch_tape(b);
    if (r != MPM_OK) return r;
    for (int i = 0; i < n; ++i) {
        MpmHandle* h = b->sims[i];
        BTRY(b, i, ensure_adjoint_buffers(h, h->adj));
        BTRY(b, i, ensure_tape(h, h->adj, (int)std::min<int64_t>(K, nsteps)));
    }
    bool any_pvc = false, any_newt = false, moved = false;
    for (MpmHandle* h : b->sims) {
        any_pvc = any_pvc || h->has_pvc;
        any_newt = any_newt || h->adj->tvsc != nullptr;
    }
    std::vector<int> cur(n, -1);   // epoch whose order the member's adjoint arrays are in
    for (int seg = nseg - 1; seg >= 0 && r == MPM_OK; --seg) {
        const int len = (int)std::min<int64_t>(K, nsteps - (int64_t)seg * K);
        bool have = true;
        for (MpmHandle* h : b->sims) have = have && h->adj->tape_seg == seg;
        if (!have) {
            moved = true;
            r = batch_recompute(b, x, seg, len, s);
            if (r != MPM_OK) break;
        }
        for (int i = 0; i < n; ++i) cur[i] = b->sims[i]->adj->epoch_of[len - 1];
        if (seg == nseg - 1) {
            r = batch_seed(b, dl_dloc, dl_dvel, len, on_device, s);
            if (r != MPM_OK) break;
        }
        const int4* rtiles = nullptr;
        int nrtiles = 0;
        r = batch_reverse_tiles(b, x, rtiles, nrtiles, s);
        if (r != MPM_OK) break;
        x->bases.assign(n, AdjStep{});
        for (int t1 = len - 1; t1 >= 0 && r == MPM_OK;) {
            // the steps down to t0 keep every member's sort
            for (int i = 0; i < n && r == MPM_OK; ++i) {
                MpmHandle* h = b->sims[i];
                AdjointState* a = h->adj;
                const int e = a->epoch_of[t1];
                if (e != cur[i]) r = permute(h, a, a->epochs[cur[i]].pid, a->epochs[e].pid, s);
                if (r != MPM_OK) {
                    r = from_sim(b, i, r);
                    break;
                }
                cur[i] = e;
                x->bases[i] = base_args(h, a, e);
            }
            if (r != MPM_OK) break;
            BCK(b, cudaMemcpyAsync(x->d_bases, x->bases.data(), sizeof(AdjStep) * n, cudaMemcpyHostToDevice, s));
            int t0 = t1;
            auto same = [&](int t) {
                for (int i = 0; i < n; ++i)
                    if (b->sims[i]->adj->epoch_of[t] != cur[i]) return false;
                return true;
            };
            while (t0 > 0 && same(t0 - 1)) --t0;
            auto body = [&](cudaStream_t c) -> int {
                for (int t = t1; t >= t0; --t) {
                    CK(b->sims[0], launch_adj_table(x->d_bases, n, t, x->d_table, c));
                    CK(b->sims[0], launch_rev_batch(x->d_table, b->cfg.usl, b->cfg.traction, any_pvc,
                                                    b->cfg.reinit, any_newt, rtiles, nrtiles, x->part_blocks,
                                                    x->n_part_blocks, c));
                }
                return MPM_OK;
            };
            if (t1 - t0 + 1 < GRAPH_STEPS) {
                r = body(s);
            } else {
                check_batch_adj_graphs(b, x);
                const int64_t grid = (int64_t)nrtiles * 2 + (rtiles == x->rtiles);
                const int64_t opts = (int64_t)x->n_part_blocks * 4 + any_pvc * 2 + any_newt;
                r = run_cached_graph(b->sims[0], x->g_rev, GraphKey{t0, t1, grid, opts}, s, body);
            }
            if (r != MPM_OK) r = from_sim(b, 0, r);
            t1 = t0 - 1;
            // (the host copy of the arguments must outlive the upload)
            if (r == MPM_OK && cudaStreamSynchronize(s) != cudaSuccess) r = bfail(b, MPM_ERR_CUDA, "synchronise");
        }
        for (int i = 0; i < n && r == MPM_OK; ++i) {
            MpmHandle* h = b->sims[i];
            AdjointState* a = h->adj;
            if (a->epoch_of[0] != 0) {
                const int e = permute(h, a, a->epochs[a->epoch_of[0]].pid, a->epochs[0].pid, s);
                if (e != MPM_OK) r = from_sim(b, i, e);
            }
        }
    }
    if (r == MPM_OK && dl_dE) r = batch_emit(b, dl_dE, 9, 1, on_device, s);
    if (r == MPM_OK && dl_dloc0) r = batch_emit(b, dl_dloc0, 0, 2, on_device, s);
    if (r == MPM_OK && dl_dvel0) r = batch_emit(b, dl_dvel0, 2, 2, on_device, s);
    // leave every simulation at the recorded end state, where the re-runs moved
    // it (the wait also completes the gradients' copies)
    int r2 = MPM_OK;
    if (moved) {
        std::vector<CopySeg> v;
        for (MpmHandle* h : b->sims) checkpoint_segments(h, h->adj->ck[nseg], false, v);
        r2 = run_segments(b->sims[0], x->misc, v, s);
        if (r2 == MPM_OK) r2 = read_statuses(b, s);
        else r2 = from_sim(b, 0, r2);
    }
    if (cudaStreamSynchronize(s) != cudaSuccess && r2 == MPM_OK) r2 = bfail(b, MPM_ERR_CUDA, "synchronise");
    return r != MPM_OK ? r : r2;
}

}  // extern "C"
