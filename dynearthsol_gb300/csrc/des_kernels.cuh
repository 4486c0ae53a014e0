// des_kernels.cuh -- host-side launchers of the explicit-step kernels.
#pragma once

#include <algorithm>

#include <cuda_runtime.h>

#include "des_common.cuh"

namespace des {

// Threads per block of a kernel with one thread per element or node.  An SM
// issues two FP64 operations per clock however many of its warps wait, so a
// small mesh wants its warps spread over all 152 SMs, and a mesh of a few
// waves a fine last wave: blocks of 64 up to 152 SMs x 2048 threads.  Beyond,
// many waves follow one another, and blocks of 128 keep the neighbours'
// gathers of a block together.  Measured against blocks of 256 everywhere
// (ms per pass): 8,000 triangles x 200 steps 11.6 -> 9.1, 648 tets x 100 FP64
// steps 13.5 -> 9.9, 14,400 yielding tets x 100 mixed steps 12.3 -> 10.0,
// 118,326 tets x 10 loops of the per-function entry points 5.24 -> 4.67,
// 998,400 tets x 20 FP64 steps 39.5 -> 39.0 (128 and 64 alike), 998,400 tets
// x 50 mixed steps 28.3 -> 27.6 (128).  Blocks of 32 for all of them are slower
// than 64 at every size (launch and scheduling of blocks); for the few kernels
// of DES_LAUNCH_W they are not.
inline bool one_wave(long long n) { return n <= 152LL * 2048; }

constexpr int BLOCK_MOST = 128;   // of DES_LAUNCH
inline int block_threads(long long n) { return one_wave(n) ? 64 : BLOCK_MOST; }

inline int grid_blocks(long long n)
{
    const long long t = block_threads(n), b = (n + t - 1) / t;
    return (int)(b < 1 ? 1 : b);
}

// kernel<<<...>>> over n elements or nodes on stream s
#define DES_LAUNCH(KERNEL, n, s, ...) \
    KERNEL<<<des::grid_blocks(n), des::block_threads(n), 0, (s)>>>(__VA_ARGS__)

// DES_LAUNCH for the 3D FP64 geometry and reverse element kernels, which a
// small mesh's warps share an SM's FP64 pipe for: up to one wave a warp to a
// block, so that no SM has more of them than it must.  Measured (blocks of 64
// / 32 threads), windows of 20 steps and their reverse: 14,400 tets 4.03 / 3.94
// ms, 49,152 6.85 / 6.69, 105,600 11.90 / 11.89, 193,536 18.3 / 18.2, 301,056
// 23.1 / 23.1; 50 FP64 steps of 49,152 tets 6.66 / 6.53, of 105,600 12.14 /
// 12.17: nothing to choose from a third of a wave on.  The other kernels, and
// 2D, take the same time or 0.3% more.
#define DES_LAUNCH_W(KERNEL, n, s, ...)                                                  \
    do {                                                                                 \
        const long long nw_ = (n);                                                       \
        if (des::one_wave(nw_))                                                          \
            KERNEL<<<(unsigned)((nw_ + 31) / 32), 32, 0, (s)>>>(__VA_ARGS__);            \
        else                                                                             \
            DES_LAUNCH(KERNEL, nw_, s, __VA_ARGS__);                                     \
    } while (0)

// DES_LAUNCH for kernels of a few instructions a value (copies, layout
// conversions, the per-function motion, boundary condition and temperature
// updates): starting a block costs them as much as its work.  Blocks of 64 or
// 128 / 256, us a call: coordinates of 998,400 tets 6.3 / 4.3 in a mixed
// context, velocity BCs 5.8 / 4.3; an upload of 1,200 triangles 152 / 139.
#define DES_LAUNCH_LIGHT(KERNEL, n, s, ...) \
    KERNEL<<<(unsigned)std::max(1LL, ((long long)(n) + 255) / 256), 256, 0, (s)>>>(__VA_ARGS__)

// flags of the element geometry pass
enum GeoFlags : int {
    GEO_COPY_OLD = 1,    // volume_old <- volume        (dynearthsol.cxx:226)
    GEO_VOLUME = 2,      // compute_volume              (geometry.cxx:86-108)
    GEO_SHAPE = 4,       // compute_shape_fn            (geometry.cxx:368-455)
    GEO_ROTATE = 8,      // rotate_stress               (fields.cxx:411-483)
    GEO_DT = 16,         // compute_dt element terms    (geometry.cxx:254-292)
    GEO_DT_IF_STEP = 32, // ... only when steps % 10 == 0 (dynearthsol.cxx:349-361)
    GEO_MASS_TERMS = 64, // the element's mass and tmass terms -> me, tme (for launch_mass_sum)
    GEO_DT_FINAL = 128   // with GEO_DT, in one launch over the whole mesh: form dt too (launch_dt_finalize)
};

// Each launcher returns the number of kernels it launched.
int launch_strain_rate(const KP &p, cudaStream_t s);
int launch_update_temperature(const KP &p, cudaStream_t s);       // tdot -> p.tdot, T (FP64 contexts)
int launch_temperature_update(const KP &p, cudaStream_t s);       // T from p.tdot
int launch_dvoldt(const KP &p, cudaStream_t s);                   // -> ntmp
// the FP64 step's element-centric form of strain rate + heat gather + dvoldt
// (+ clock advance) and of the node sums + temperature update: the same bits
// (needs p.qv and, with heat, p.hc64)
int launch_elem_pass(const KP &p, cudaStream_t s, bool heat);
// mass_sums (a chained step): first the compute_mass sums of the look-ahead
// geometry pass's element terms, and the clock advance
int launch_node_pass(const KP &p, cudaStream_t s, bool heat, bool mass_sums = false);
int launch_edvoldt(const KP &p, cudaStream_t s);
int launch_update_stress(const KP &p, cudaStream_t s, bool fused);
// dp_nd -> ntmp; stored: the dp vol products of the fused mixed stress pass (KP::pv)
int launch_nmd_gather(const KP &p, cudaStream_t s, bool stored = false);
// fused: it also forms the elements' force terms from the corrected stress,
// which launch_force sums, and the stress-BC facets' forces
int launch_nmd_correct(const KP &p, cudaStream_t s, bool fused);
// the force terms and the facet forces alone, from the current stress
int launch_force_terms(const KP &p, cudaStream_t s);
int launch_force(const KP &p, cudaStream_t s, bool fused_motion);
int launch_velocity(const KP &p, cudaStream_t s, bool contract = false);
int launch_vbcs(const KP &p, cudaStream_t s);
int launch_coordinate(const KP &p, cudaStream_t s, bool contract = false);
int launch_swap_volume(const KP &p, cudaStream_t s);   // volume_old <- volume
int launch_geometry(const KP &p, cudaStream_t s, int flags);
// the chained step's geometry pass, which also does the next step's element
// pass (k_elem_pass's or k_elem_pass_mixed3's work)
int launch_geometry_ahead(const KP &p, cudaStream_t s, int flags);
// compute_mass from the element terms of a GEO_MASS_TERMS geometry pass (same sums, same order)
int launch_mass_sum(const KP &p, cudaStream_t s);
// compute_dt's element terms alone (for launch_dt_finalize)
int launch_dt_terms(const KP &p, cudaStream_t s);
int launch_dt_finalize(const KP &p, cudaStream_t s, bool only_on_step);
int launch_quality(const KP &p, cudaStream_t s, unsigned long long *red);
// red[2], red[3]: bad_mesh_quality's first tiny element and first drifted bottom node
int launch_quality_scans(const KP &p, cudaStream_t s, double smallest_vol, double bottom, double dist,
                         int check_bottom, unsigned long long *red);
// out[4][ne]: density, mesh quality, viscosity, material of an output frame
int launch_output_elem(const KP &p, double *out, cudaStream_t s);
// material constants: visc_coef[nmat], then 4 values per plastic table entry
int launch_material_table(const KP &p, cudaStream_t s, double *out);
// the per-element blended material properties (KP::eprop) from the marker
// counts; run whenever the counts change
int launch_elem_props(const KP &p, cudaStream_t s, double *out);

// the support-list entry of each (element, slot), slot-major, from the lists' n entries
void launch_sup_pos(const int *ent, int *pos, int ne, long long n, cudaStream_t s);
// a mixed 3D context's shape functions (p.shpdw non-null; else no launch):
// the double-word pairs -> FP64 p.shp, for a download
int launch_shp_join(const KP &p, cudaStream_t s);

// layout conversion between the reference's AoS rows and device SoA
int launch_aos_to_soa(const double *aos, double *soa, int n, int ncomp, cudaStream_t s);
int launch_soa_to_aos(const double *soa, double *aos, int n, int ncomp, cudaStream_t s);

// The same conversion for the rows [lo, hi) of several fields in one launch
// (one slab of the pipelined host step).
constexpr int ROWS_MAX = 12;
struct RowField {
    double *stage;   // AoS rows [n][nc]; rows lo..hi-1 are read (up) or written
    double *dev;     // SoA [nc][n]
    long long first; // index of the field's first value in the launch
    int n, nc, lo, hi;
    const float2 *dw; // download: read the double-word pairs here instead of dev, or null
};
struct RowTable {
    RowField f[ROWS_MAX];
    long long total;
    int count;
};
int launch_rows(const RowTable &t, bool up, cudaStream_t s);

}  // namespace des
