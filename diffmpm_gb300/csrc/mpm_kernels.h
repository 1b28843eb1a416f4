// Host-side launchers of the MPM kernels (implemented in mpm_kernels.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <cmath>
#include <string>
#include "mpm_types.h"

namespace mpm {

// Element volume of an hx x hy Quadrilateral4Node element by the reference's
// formula in float32 (diffmpm/element.py:903-909), on the host.
inline float element_volume(float hx, float hy) {
    const float a = hy, c = hy, b = hx, d = hx;
    const float p = std::sqrt(a * a + b * b), q = p;
    const float t = ((a * a + c * c) - b * b) - d * d;
    const float x = (((4.0f * p) * p) * q) * q - t * t;
    return 0.25f * std::sqrt(x);
}

struct StepConfig {
    bool usl;          // scheme: USL (else USF)
    bool reinit;       // solve_jit semantics: volume/mass reset each step
    bool traction;     // particle tractions present
    // resident CTAs per SM the nodal kinematics and USF G2P kernels are
    // built for: 3 (40 registers a thread) or 2 (up to 64).  (G2P, 2.1M particles:
    // 20.2 us with 3, 21.2 with 2; a batch of 64, 2.27M: 29.0 and 31.4.)
    int nk_ctas = 3;
    int g2p_ctas = 3;
    // forces kernel fast path: particle per lane with row slots (0), lane
    // per cell (1), particle per lane on a staged row (2); the same bits
    // every way
    int forces_lpc = 0;
    bool operator==(const StepConfig& o) const {
        return usl == o.usl && reinit == o.reinit && traction == o.traction && nk_ctas == o.nk_ctas &&
               g2p_ctas == o.g2p_ctas && forces_lpc == o.forces_lpc;
    }
};

// One explicit step = three launches over the (active) tile list.  The descriptor is
// passed by value (a __grid_constant__ kernel parameter), so a captured graph
// holds the descriptor current at capture time.
cudaError_t launch_nodal_kinematics(const StepConfig& c, const SimDev& S, const int4* tiles,
                                    int ntiles, Control* ctl, int k, cudaStream_t s);
cudaError_t launch_forces(const StepConfig& c, const SimDev& S, const int4* tiles, int ntiles,
                          Control* ctl, int k, cudaStream_t s);
cudaError_t launch_particle_kinematics(const StepConfig& c, const SimDev& S, const int4* tiles,
                                       int ntiles, Control* ctl, int k, cudaStream_t s);
// n whole steps over at most one tile per SM in one cooperative launch, with
// the default forces path; advances the step counter.  `arrived`: one word of
// scratch.  ST_STALLED in the status means that a wait of `polls` reads ran out
// (BARRIER_POLLS reads take seconds, a step of such a run microseconds).  One
// such launch is shorter than the launches of its steps for any n (a call of one
// step, of seven: 160 particles 40 -> 32 us, 138 -> 65; 136k particles 74 -> 69,
// 212 -> 160), but not than the launches of a replayed step, whose status the
// host waits for anyway (a thrown block of 200 of them: 26.0 ms with, 21 without).
constexpr unsigned BARRIER_POLLS = 1u << 22;
cudaError_t launch_steps_resident(const StepConfig& c, const SimDev& S, const int4* tiles, int ntiles, Control* ctl,
                                  unsigned* arrived, int n, unsigned polls, cudaStream_t s);
// Split the tile list into active tiles (cells or their ring store a
// particle; the step kernels' grid) and empty ones (node updates only,
// k_empty_nodes), in tile order, both padded to ntiles entries with
// (-1, 0, 0, 0), and write their counts to counts[0..1]; flags is ntiles
// ints of scratch.  Valid until the sort changes.
cudaError_t launch_classify_tiles(const SimDev& S, const int4* tiles, int ntiles, int* flags, int4* active,
                                  int4* empty, int* counts, cudaStream_t s);
// The same split from flags alone, and flags[t] |= more[t] (the tiles that hold
// particles in any of several sorts).
cudaError_t launch_compact_tiles(const int* flags, const int4* tiles, int ntiles, int4* active, int4* empty,
                                 int* counts, cudaStream_t s);
cudaError_t launch_or_flags(int* flags, const int* more, int n, cudaStream_t s);
// A single simulation launches its empty tiles apart only when it has at
// least this many (mpm_set_empty_split changes it per handle).
constexpr int EMPTY_SPLIT_MIN = 128;
// Grid of a launch over `count` tiles of such a list: the count rounded up to
// a multiple of TILE_GRID_QUANTUM (at most the list's length), so that the
// captured graphs, keyed by their grids, serve the small changes of the
// counts that re-sorts bring; the CTAs past the count read a (-1, ...) entry
// and return.
constexpr int TILE_GRID_QUANTUM = 64;
inline int tile_grid(int count, int ntiles) {
    if (count <= 0) return 0;
    const int q = (count + TILE_GRID_QUANTUM - 1) / TILE_GRID_QUANTUM * TILE_GRID_QUANTUM;
    return q < ntiles ? q : ntiles;
}
// The step's node updates of the empty tiles (before the nodal kinematics).
// Without concentrated nodal forces a massless node's update is idempotent
// (velocity kept or constrained and flushed, mass and acceleration 0) and no
// other tile writes it, so step k of a launched sequence repeats what its
// first step left: only that one launches the kernel (4096^2 mixed: 97 us of
// a 745 us step; 1024^2: 5.8 of 92 us).
inline bool empty_nodes_due(int k, bool nodal_forces) { return k == 0 || nodal_forces; }
cudaError_t launch_empty_nodes(const SimDev& S, const int4* empty, int ntiles, Control* ctl, int k,
                               cudaStream_t s);
// The same for a batch: tiles of every simulation (sims[tile.x]); the empty
// tiles' records (launch_gather_tiles of the empty list).
cudaError_t launch_classify_tiles_batch(const SimDev* const* sims, const int4* tiles, int ntiles, int* flags,
                                        int4* active, int4* empty, int* counts, cudaStream_t s);
cudaError_t launch_empty_nodes_batch(const TileDesc* td, int ntiles, int k, cudaStream_t s);
// Steps of a captured step graph (a block of steps launches it repeatedly and
// the remainder without a graph): a graph of a whole block of 100 steps cost
// 1.2 ms to capture and instantiate, one of 20 a fifth, and 20 steps on the GPU
// last longer than the host needs for the next launch.
constexpr int GRAPH_STEPS = 20;
// The kernels above work on step (ctl->step + k); these advance the counter
// once a sequence of steps has been launched.
cudaError_t launch_advance_step(Control* ctl, int by, cudaStream_t s);
cudaError_t launch_advance_steps(Control* const* ctls, int n, int by, cudaStream_t s);

// The same three phases for a batch of simulations in one launch each: tile
// t works on simulation tiles[t].x, whose descriptor is sims[tiles[t].x] and
// whose step counter and status are in ctls[tiles[t].x].
// out[t] = {tiles[t], ctls[tiles[t].x], *sims[tiles[t].x], row starts,
// occupancy, tapes[tiles[t].x] if any} for t < ntiles (only out[t].T for a
// tile (-1, ...)).
cudaError_t launch_gather_tiles(const SimDev* const* sims, Control* const* ctls, const TapeDev* tapes,
                                const int4* tiles, int ntiles, TileDesc* out, cudaStream_t s);
cudaError_t launch_nodal_kinematics_batch(const StepConfig& c, const TileDesc* td, int ntiles,
                                          int k, cudaStream_t s);
cudaError_t launch_forces_batch(const StepConfig& c, const TileDesc* td, int ntiles, int k,
                                cudaStream_t s);
cudaError_t launch_particle_kinematics_batch(const StepConfig& c, const TileDesc* td, int ntiles,
                                             int k, cudaStream_t s);

// Re-sort of a simulation's particles by current cell, stable in storage
// order (mpm_sort.cu): the arguments of one simulation, current arrays to the
// other buffer set.
struct SortScratch {
    int* count;        // ncell + 1 (last bucket: particles outside the mesh)
    int* key;          // np
    int* rank;         // np
    int* perm;         // np
    int* block_sums;   // ceil((ncell + 2) / 1024) + 1
};
constexpr int SORT_FIELDS = 18;   // 4-byte arrays that move with a particle
struct SortJob {
    int np, nx, ny, nf;
    float hx, hy;
    const float *x, *y;
    int *count, *key, *rank, *perm, *start;
    uint8_t* cflag;
    Control* ctl;
    const uint32_t* src[SORT_FIELDS];
    uint32_t* dst[SORT_FIELDS];
    const uint8_t* mat_src;
    uint8_t* mat_dst;
    const uint16_t* pvc_src;    // byte pairs; null when absent
    uint16_t* pvc_dst;
    const uint16_t* trfn_src;   // byte pairs; null when absent
    uint16_t* trfn_dst;
    const float2* trtau_src;
    float2* trtau_dst;
};
// count, start and perm (each bucket in storage order with `buckets`), and the
// drift flags cleared; the arrays' move is apart.  With `buckets` the counts
// are zero before and after.
cudaError_t launch_sort_order(const SortJob& J, int* block_sums, bool buckets, cudaStream_t s);
cudaError_t launch_sort_move(const SortJob& J, cudaStream_t s);
// Meshes of at most SORT_MANY_CELLS cells take one launch for the scan, and
// several simulations (device table) are sorted together.
constexpr int SORT_MANY_CELLS = 1 << 18;
cudaError_t launch_sort_many(const SortJob* jobs, int n, int most_np, int most_cells, cudaStream_t s);
// *puts[i].dst = puts[i].S
struct DescPut {
    SimDev* dst;
    SimDev S;
};
cudaError_t launch_put_descs(const DescPut* puts, int n, cudaStream_t s);

// Solve-semantics volume set-up after a sort (V = V_el / count, m = V rho, size = sqrt V).
cudaError_t launch_setup_volume(const SimDev* sim, int np, int parity, cudaStream_t s);

// dst[i] = src[perm[i]] for pairs of bytes and of floats.
cudaError_t launch_gather_pairs(const uint16_t* src, uint16_t* dst, const int* perm, int n, cudaStream_t s);
cudaError_t launch_gather_pairs(const float2* src, float2* dst, const int* perm, int n, cudaStream_t s);

// Transfer of a field between original order (aos: ncomp values per particle,
// null reads as zeros) and storage order (an array per component; a component
// without one lives in slot[c] of the original-order `passive` array, or is
// zero); pid: storage -> original (null: the same order).
constexpr int PASSIVE_N = 5;
struct FieldMap {
    float* comp[12];
    signed char slot[12];
    int ncomp, np;
    const int* pid;
    float* passive;
    float* aos;
};
cudaError_t launch_field(const FieldMap& F, bool in, cudaStream_t s);
cudaError_t launch_field_many(const FieldMap* maps, int n, int most_np, bool in, cudaStream_t s);
cudaError_t launch_gather_in_u8(uint8_t* dst, const int* pid, int np, const int32_t* in,
                                cudaStream_t s);
cudaError_t launch_scatter_out_u8(const uint8_t* src, const int* pid, int np, int32_t* out,
                                  cudaStream_t s);

// Derived per-particle outputs in original order: element id, volume, mass
// (solve_jit semantics: the volume set-up at the current positions), momentum.
// 1-D (mpm_line.cu): buckets ordered by original index; element per storage slot
cudaError_t launch_line_segsort(int nbucket, const int* start, int* perm, const int* pid, cudaStream_t s);
cudaError_t launch_line_eid(const int* cstart, int nx, int* eid, cudaStream_t s);
cudaError_t launch_derived_out(const SimDev* sim, int ndim, int np, int parity, bool reinit, int what,
                               const int* pid, void* out, cudaStream_t s);

// Interleave / de-interleave nodal vectors.
cudaError_t launch_interleave2(const float* a, const float* b, int n, float* out, cudaStream_t s);
cudaError_t launch_deinterleave2(const float* in, int n, float* a, float* b, cudaStream_t s);
cudaError_t launch_node_momentum(const float* m, const float* vx, const float* vy, int n,
                                 float* out, cudaStream_t s);

// Copy of many device-memory segments in one launch (snapshots and checkpoints
// of whole batches, the adjoint's tape).  Segment i is cut into chunks of
// COPY_CHUNK bytes, chunks first[i] .. first[i+1]-1, first[nseg] being their
// number.  The chunk table (source, destination and length of every chunk)
// is formed on the device once per upload (launch_chunk_table), so a CTA of
// the copy kernel starts its chunk after one dependent load.  The
// destination of a launch with slot t is dst + t * dst_step.
struct CopySeg {
    const void* src;
    void* dst;
    unsigned long long bytes;
    unsigned long long dst_step;
};
struct CopyChunk {
    const char* src;
    char* dst;
    unsigned long long dst_step;
    unsigned long long bytes;
};
constexpr unsigned COPY_CHUNK = 16384;
cudaError_t launch_chunk_table(const CopySeg* segs, const unsigned* first, int nseg, unsigned nchunks,
                               CopyChunk* chunks, cudaStream_t s);
cudaError_t launch_copy_segments(const CopyChunk* chunks, unsigned nchunks, int t, cudaStream_t s);
// *mismatch += number of differing 16-byte words or tail bytes between src and dst.
cudaError_t launch_compare_segments(const CopyChunk* chunks, unsigned nchunks, int* mismatch,
                                    cudaStream_t s);

// *ctls[i] = 0 for i < n.
cudaError_t launch_zero_controls(Control* const* ctls, int n, cudaStream_t s);
// The step counter advances, *host = *ctl (pinned host memory), and the drift
// bit of ctl->status is cleared (the bits of errors stay).
cudaError_t launch_take_control(Control* ctl, Control* host, int advance, cudaStream_t s);
// out[i] = *ctls[i], then ctls[i]->status = 0, for i < n.
cudaError_t launch_gather_status(Control* const* ctls, int n, Control* out, cudaStream_t s);

// Set the calling thread's message returned by mpm_last_error(NULL).
void set_thread_error(const std::string& msg);

}  // namespace mpm
