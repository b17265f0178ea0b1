// Kernel launchers of the simulation step (implemented in sph_kernels.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "sph_types.h"

namespace sph {

// Device pointers of one system's arenas, passed by value to every launcher.
struct DevArrays {
    const SceneDev* scenes;
    int* steps_left;          // per scene: -1 unlimited, 0 inactive, >0 remaining
    const Work* ptiles;       // particle tiles
    const int* n_ptiles;
    const Work* ctiles;       // scan chunks (start = chunk index within the scene)
    const int* n_ctiles;
    const Work* ttiles;       // terrain tiles
    const int* n_ttiles;
    const int* scene_list;    // active scene ids (diagnostics)
    // particles
    float4* pos;   // x y z id(bits)      current state
    float4* vel;   // vx vy vz sediment(bits)
    float4* spos;  // sorted copies
    float4* svel;
    float4* dyn;   // density, P/rho^2, m/rho, P
    uint32_t* key;
    uint32_t* slot;
    uint32_t* perm;
    int32_t* nbid;
    int32_t* snbid;
    float* rec;    // kRecFloats per particle (record mode)
    // keys
    uint32_t* counts;
    uint32_t* offsets;
    uint32_t* chunk_sum;
    const uint32_t* tab;
    // terrain
    const float* tbase;
    long long* tdelta;
    float* theight;
    // in-range neighbour lists written by the density pass and read by the
    // force pass (variant bit 3), in traversal order.  Each work tile of T
    // particles starting at sorted index t owns kNbCap * T entries from
    // t * kNbCap on, in groups of four: entry q of the tile's lane l at
    // ((q / 4) * T + l) * 4 + q % 4, so a lane writes 16 bytes at a time, next
    // to its neighbour lanes' (passes that take a group of lanes per particle
    // keep each particle's entries together instead).  ncnt[p] = in-range
    // count (may exceed kNbCap: that particle's force pass then walks the cells).
    uint32_t* nlist;
    int32_t* ncnt;
    // packed neighbour records, two float4 per sorted particle:
    // (x, y, z, P/rho^2) and (vx, vy, vz, m/rho)
    float4* fdat;
    // status word: bit 0 = ordered-mode neighbour overflow, bit 1 =
    // inconsistent sort counts, bit 2 = a bounded wait of the TMA force
    // pipeline ran out
    unsigned* status;
    // work counters of the dynamically scheduled neighbour kernels
    // ([0] density, [1] force), cleared by the reorder kernel every step;
    // null where no kernel is scheduled that way
    unsigned* ctr;
    int tile;      // lanes per work tile (the list stride)
    bool early;    // set by the launchers: the kernel overlaps the one before it and waits for it
};

// Slots per particle of the in-range neighbour lists.
constexpr int kNbCap = 192;

// The one-block sort of small scenes: most particles, and most shared memory
// (counts for 45,056 keys beside the order: the scan's odd share of a thread
// rounds the next key range, 49,152, up to 2 KB more).
constexpr int kSmallSort = 4096;
constexpr int kSmallSortBytes = 215040;

struct LaunchShape {
    int tile;        // threads per particle tile
    int grid_p;      // persistent grid of particle kernels
    int grid_c;      // persistent grid of the scan
    int grid_t;      // persistent grid of the terrain kernel
    int variant;     // sph_system_config.variant bits (bit 3 only with lists allocated)
    bool pack;       // the density pass writes packed records, the force pass gathers them
    size_t sort_smem;  // shared memory of the one-block sort; 0: a scene is too large for it
    int grid_sort;     // its blocks: one per scene, whose first tiles lead the work list
    bool early;      // few particles: each kernel's launch overlaps the kernel before it
    bool captured;   // the launches go into a graph
    int nsm;         // SMs of the device
    bool density_group, force_group, ordered_group;  // few particles: a group of lanes per particle (group_rules)
    bool record;     // some scene keeps its force records (SPH_FLAG_RECORD)
    int grid_dyn;    // grid of the dynamically scheduled neighbour kernels
    const void* fmap;  // host copy of the CUtensorMap over the packed records (null: none)
};

// Once per process and device: opt the list-traversal kernels into >48 KB of
// dynamic shared memory.
void configure_kernels();
// Shared memory of the one-block sort for scenes of at most max_n particles and
// max_keys keys; 0: too large for it.
size_t sort_small_smem(int64_t max_n, int64_t max_keys);
// Its block ranks a cell's particles against one another by itself, so a scene
// of more than two particles a thread whose average cell holds more than 16
// (cells of 4h and more) is not for it.  4,096 particles, 64 steps, us, one block
// and the whole chip: cells of 8h 6,821 vs 4,713, of 4h 3,113 vs 2,638 (three
// systems in turn 1,313 vs 1,388); 2,000 particles, cells of 4h 2,103 vs 2,247.
constexpr bool sort_crowded(int64_t n, int64_t keys) { return n > 2048 && n > 16 * keys; }
void launch_sort_small(const DevArrays& a, const LaunchShape& s, cudaStream_t st);
void launch_keys(const DevArrays& a, const LaunchShape& s, cudaStream_t st);
void launch_scan(const DevArrays& a, const LaunchShape& s, cudaStream_t st);
void launch_scatter(const DevArrays& a, const LaunchShape& s, cudaStream_t st);
void launch_reorder(const DevArrays& a, const LaunchShape& s, cudaStream_t st);
// Variants with the same value launch the same neighbour kernels.
int neighbour_kernels(const LaunchShape& s);
// Sets early and the three group members from the others.
void group_rules(LaunchShape& s);
void launch_density(const DevArrays& a, const LaunchShape& s, cudaStream_t st);
void launch_density_ordered(const DevArrays& a, const LaunchShape& s, cudaStream_t st);
void launch_force(const DevArrays& a, const LaunchShape& s, cudaStream_t st);
void launch_force_ordered(const DevArrays& a, const LaunchShape& s, cudaStream_t st);
void launch_terrain(const DevArrays& a, const LaunchShape& s, cudaStream_t st);
void launch_tick(const DevArrays& a, const LaunchShape& s, int nscenes, cudaStream_t st);

// Inspection and on-demand kernels.
void launch_neighbour_counts(const DevArrays& a, const LaunchShape& s, int32_t* out_by_id, cudaStream_t st);
// [rows visited, candidates tested, in-range pairs] of one scene's sorted state.
void launch_traversal_stats(const DevArrays& a, int scene, unsigned long long* out, cudaStream_t st);
// Scatter a scene's state into id order: any output may be null.
void launch_gather_by_id(const float4* pos, const float4* vel, const float4* dyn, int p_off, int n, float* pos3,
                         float* vel3, float* dens, int32_t* sed, int priority, cudaStream_t st);
// Per-scene FP64 partial sums: kDiagBlocks blocks per listed scene.
constexpr int kDiagBlocks = 32;
constexpr int kDiagDoubles = 8;  // mass-weighted momentum xyz, kinetic, potential, (pad)
void launch_diag(const DevArrays& a, int nlist, double* partial, long long* isums, int* nan_count,
                 cudaStream_t st);

}  // namespace sph
