// Host-side declarations of the kernel launchers (one translation unit per stage).
#pragma once
#include <vector>
#include "gbt_common.cuh"

namespace gbt {

// launch geometry of one level of a batch: grid.y enumerates solves, grid.x covers the largest
// solve's box (blocks past a smaller solve's end return at once)
struct LaunchCtx {
    Batch batch;
    cudaStream_t stream;
    int maxIM = 0, maxJM = 0, maxKM = 0;     // maxima over the solves of this level
    long long pool_n = 0;                     // elements of one field pool of this level
    // optional stage profiler: called before (begin = 1) and after (begin = 0) a group of
    // launches with the group's name, the number of kernel launches in it and the grid level
    void (*hook)(void *user, const char *stage, int begin, int launches, int level) = nullptr;
    void *hook_user = nullptr;
    int level = 0;                            // grid level of these launches (1 = fine)
    // a second stream for what may run beside the launches of the first, and the events between the two (null: none)
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    const void *face_tma = nullptr;           // tables of the TMA-staged face stage (mixed form), or null
    const void *face_tma_host = nullptr;      // their header, on the host
    void mark(const char *stage, int begin, int launches = 1) const { if (hook) hook(hook_user, stage, begin, launches, level); }
    dim3 grid_n(long long n, int bs) const { return dim3((unsigned)((n + bs - 1) / bs), batch.nsolve); }
    dim3 grid_cells(int bs) const { return grid_n((long long)(maxIM - 1) * (maxJM - 1) * (maxKM - 1), bs); }
    dim3 grid_faces(int f, int bs) const
    {
        return grid_n((long long)(maxIM - 1 + (f == 0)) * (maxJM - 1 + (f == 1)) * (maxKM - 1 + (f == 2)), bs);
    }
    dim3 grid_plane(int bs) const { return grid_n((long long)(maxIM - 1) * (maxJM - 1), bs); }
};

// boundary patches in device form; every record names its solve
struct DevInOut { int solve, face, is, ie, js, je, ks, ke; };
struct DevWall { int solve, face, rotate, is, ie, js, je, ks, ke; };
// mixing plane: k+ face of slot s1 (rows is..ie, pitch range js1..je1) against the k- face of slot s2
struct DevMix { int s1, s2, is, ie, js1, je1, js2, je2; };
constexpr int kMixVals = 14;                    // per row: both sides' averaged d, u, v, w, p, c; the SA value
struct BcTables {
    const DevInOut *inlet = nullptr; int n_inlet = 0, max_inlet = 0;     // max cells of a patch
    const DevInOut *outlet = nullptr; int n_outlet = 0;
    const DevWall *wall = nullptr; int n_wall = 0, max_wall = 0;
    // walls grouped by their position in each solve's list (the reference applies them in order)
    int n_wall_slot = 0;
    int wall_slot_off[65] = {0};                  // first record of slot q; slot q has off[q+1]-off[q]
    int wall_slot_lines[64] = {0};                // most wall-normal lines of a patch in slot q
    // periodic exchange as a gather list: dst <- rotate(src, sign * delta_th of the solve)
    const long long *per_dst = nullptr, *per_src = nullptr;
    const int *per_meta = nullptr;                // solve * 4 + (sign + 1)
    const double *per_trig = nullptr;             // per solve: cos, sin of +delta_th, then of -delta_th
    long long n_per = 0;
    int max_outlet_im = 0, max_outlet_jm = 0;
    double *outlet_cu = nullptr;                  // per outlet patch: mass-weighted swirl of each radial row
    double2 *outlet_trig = nullptr;               // per outlet patch and face: sine and cosine of its polar angle
    long long outlet_trig_stride = 0;
    bool apart = false;                           // no ghost cell belongs to two of inlet, outlet, wall and periodic fills
    bool mix_apart = false;                       // nor one of a mixing plane to any of them
    double *integ_part = nullptr;                 // per solve and section: kIntegralBlocks partial sums of 3
    unsigned *integ_count = nullptr;              // per solve: blocks of a launch that are done
    // Baldwin-Lomax wall distances (fine level): record w holds, for point n0 = 1..N-1 of each of
    // its wall-normal lines t, the distance of cell n0 from the line's wall-face centre at
    // wall_dist[wall_dist_off[w] + (n0 - 1) * lines(w) + t], in the working precision
    void *wall_dist = nullptr;
    const long long *wall_dist_off = nullptr;
    const DevInOut *inlet_first = nullptr, *outlet_first = nullptr;   // per solve: Inlet[1], Outlet[1]
    // mixing planes (applied after every other boundary) and their per-row averages
    const DevMix *mix = nullptr;
    int n_mix = 0, max_mix_rows = 0, max_mix_j = 0;
    double *mix_avg = nullptr;
    // Spalart-Allmaras: ghost cells of the variable filled by interfaces and periodic pairs
    const long long *sa_dst = nullptr, *sa_src = nullptr;
    long long n_sa_gather = 0;
};

// where the integrals put an iteration's row of the history (12 values per case): row iter - *base
// With both (per slot, zero between iterations) the norm and the integrals may finish in either order, and the
// later one writes the row; without, the integrals, which then come after the norm.
struct HistorySink { double *out; const int *base; int rows, ncase; unsigned *both; };

// out-of-range cells of every slot (update.cuh): their list, its length, blocks of a launch that are done
struct LimitLists { int *list, cap, *count; unsigned *done; };

constexpr int kIntegralBlocks = 32;             // blocks per inlet/outlet section in the integrals

// The LU-SGS sweeps' tiles (wavefront.cu). A tile is a group of grid columns that a block marches
// along k, skewed by the columns' places in it; the tiles of a slot hold T steps each, tile (PI, PJ)
// from step0 + (PI * nPJ + PJ) * T on.
struct WaveSolve { int nI, nJ, nK, nPI, nPJ, T; long long step0; };
struct WaveCtl { unsigned epoch, ticket[2]; };     // sweeps started; tiles handed out, per direction
struct WaveBytes { int geo, flow, dq, pkt, area, var_flow, var_dq, var_pkt; };      // of a step
struct WaveTables {
    const WaveSolve *solve = nullptr;              // per slot
    const int2 *item = nullptr;                    // {slot, PI * nPJ + PJ}: every tile, after the two it reads from
    int n_item = 0, narrow = 0;
    int max_tiles = 0, max_T = 0;                  // largest of a slot: tiles, steps of a tile
    long long max_steps = 0;                       // and steps of all its tiles
    WaveCtl *ctl = nullptr;
    char *geo = nullptr, *flow = nullptr, *dq = nullptr;   // blocks of the steps, in step order
    void *area = nullptr;                          // mean area per cell and direction
    uint4 *pkt = nullptr;                          // terms that cross from tile to tile
};
// columns of a tile in i and j; bytes of a step's blocks (fp64: working type; narrow: the form for small grids, in FP64 half as wide in j;
// sa: with the Spalart-Allmaras variable)
void wave_patch(int fp64, int narrow, int &pa, int &pb);
void wave_bytes(int fp64, int narrow, int sa, WaveBytes &w);

void launch_geometry(const LaunchCtx &ctx, const Geo &G, double *totalvol);
// the periodic rotation's cosines and sines per solve (BcTables::per_trig), once at create
void launch_periodic_trig(const LaunchCtx &ctx, double *trig);
// the sines and cosines of the outlets' faces (BcTables::outlet_trig), once per level after the geometry
void launch_outlet_trig(const LaunchCtx &ctx, const Geo &G, const BcTables &bc);

template <typename T>
void launch_boundary(const LaunchCtx &ctx, const Phys &P, const Geo &G, Flow<T> F, const BcTables &bc);

// residual stages; level = 1 for the fine mesh (turbulence model only there)
// the mixed form's face stage with tiles staged in shared memory by TMA (csrc/face_tma.cu)
bool face_tma_eligible(const std::vector<Lvl> &lv);
void *build_face_tma(const std::vector<Lvl> &lv, const GeoW<float> &G, const Flow<float> &W, size_t *bytes,
                     unsigned char host_header[64]);
void launch_face_tma(const LaunchCtx &ctx, const Phys &P, const PhysW<float> &PC, const GeoW<float> &GW, Flow<float> W,
                     const DevWall *walls);

template <typename T>
void launch_resflux(const LaunchCtx &ctx, const Phys &P, const PhysW<T> &PC, const Geo &G, const GeoW<T> &GW, Flow<T> F,
                    const BcTables &bc, int level, T *scratch_dtmin);

// both sweeps, then Q_old = Q, Q += dQ, the primitive variables and the limiter (with the Spalart-Allmaras variable present, F.ev, its update too; VV:
// the tables of the variable's sweep)
template <typename T>
void launch_lusgs_sweeps(const LaunchCtx &ctx, const Phys &P, const PhysW<T> &PC, const Geo &G, Flow<T> F, const WaveTables &V,
                         const WaveTables &VV, int level, const LimitLists &q);

// Baldwin-Lomax wall distances of every wall line point (fine level, once; see BcTables)
template <typename T>
void launch_wall_distances(const LaunchCtx &ctx, const Geo &G, const BcTables &bc);

// FP32 copies of the geometry the working-precision kernels read (mixed form; once per level)
void launch_cell_norms(const LaunchCtx &ctx, const GeoW<double> &G);
void launch_geometry_working(const LaunchCtx &ctx, const Geo &G, const GeoW<float> &GW);

// the sweeps' geometry in step order (once per level, after the geometry kernels)
template <typename T>
void launch_wave_geometry(const LaunchCtx &ctx, const Geo &G, const WaveTables &V);

template <typename T>
void launch_res_norm(const LaunchCtx &ctx, const Geo &G, Flow<T> F, const double *totalvol, double *partials,
                     int nblk, unsigned *count, const HistorySink &hist);

// residual norm with scratch in a static device array; copies the norms to host_out if given
template <typename T>
void launch_res_norm_static(const LaunchCtx &ctx, const Geo &G, Flow<T> F, const double *totalvol, int ncase, double *host_out);

template <typename T>
void launch_integrals(const LaunchCtx &ctx, const Phys &P, const Geo &G, Flow<T> F, const BcTables &bc, const HistorySink &hist);

template <typename T>
void launch_primitive(const LaunchCtx &ctx, const Phys &P, Flow<T> F);

template <typename T>
void launch_limiter(const LaunchCtx &ctx, const Phys &P, Flow<T> F, int level, const LimitLists &q);

// multigrid transfer between fine (f) and coarse (c) levels
template <typename T>
void launch_restrict(const LaunchCtx &cf, const LaunchCtx &cc, const Geo &Gf, const Geo &Gc, Flow<T> Ff, Flow<T> Fc);
// restriction or prolongation with the receiving level's primitive variables and limiter
template <typename T>
void launch_restrict_primitive(const LaunchCtx &cf, const LaunchCtx &cc, const Phys &P, const Geo &Gf, const Geo &Gc, Flow<T> Ff,
                               Flow<T> Fc, int level, const LimitLists &q);
template <typename T>
void launch_interpolate_primitive(const LaunchCtx &cf, const LaunchCtx &cc, const Phys &P, Flow<T> Ff, Flow<T> Fc, int init_from_coarse,
                                  int level, const LimitLists &q);
template <typename T>
void launch_forcing(const LaunchCtx &cc, Flow<T> Fc);
template <typename T>
void launch_delta(const LaunchCtx &cc, Flow<T> Fc);
template <typename T>
void launch_forcing_keep(const LaunchCtx &cc, Flow<T> Fc);
template <typename T>
void launch_add_forcing(const LaunchCtx &cc, Flow<T> Fc);
template <typename T>
void launch_corner(const LaunchCtx &cc, Flow<T> Fc);
template <typename T>
void launch_delta_corner(const LaunchCtx &cc, Flow<T> Fc);
template <typename T>
void launch_interpolate(const LaunchCtx &cf, const LaunchCtx &cc, Flow<T> Ff, Flow<T> Fc, int init_from_coarse);

// per-solve scalar stages
void launch_cfl_ramp(const LaunchCtx &ctx, int iter);

// Spalart-Allmaras (sa.cu)
void launch_sa_wall_distance(const LaunchCtx &ctx, const Geo &G, const long long *face_p, const int *face_f, long long n,
                             double *scratch_xyz, const long long *case_off, double *dwall);
void launch_sa_init(const LaunchCtx &ctx, double *ev, double ev_ratio);
template <typename T>
void launch_sa_boundary(const LaunchCtx &ctx, const Phys &P, Flow<T> W, const BcTables &bc);
template <typename T>
void launch_sa_model(const LaunchCtx &ctx, const PhysW<T> &P, const GeoW<T> &GW, Flow<T> W);
template <typename T>
void launch_sa_update(const LaunchCtx &ctx, const Phys &P, Flow<T> W, int *bad_list, int bad_cap, int *bad_count);
template <typename T>
void launch_sa_limit(const LaunchCtx &ctx, Flow<T> W, int *bad_list, int bad_cap, int *bad_count);

}  // namespace gbt
