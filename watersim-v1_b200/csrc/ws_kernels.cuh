// ws_kernels.cuh — kernel parameter blocks and launcher declarations.
#pragma once
#include "ws_internal.cuh"

struct AdvectParams {
  double dt, dtLast, pic, maxSpeed, gravity, oceanR, coreR, atmosphereH;
  double rainTe, rainLiftAge;
  double windS[3];
  int ceilReflect;
  // what every particle's FP32 arithmetic uses of the above and the grid
  float picF, flipF, maxSpeedF, halfDt, lo[3], hi[3], domIn2, damp, drag, rockDrag;
};

struct HeatParams {
  int hasSun;
  double sun[3];
  double sunActivity, Tamb, shadeCool, heatK, coreR;
};

struct PhaseParams {
  double cloudT, cloudP, rainT, snowT, meltT, rainLiftAge, cloudBase, dt;
  int spinOn;
  uint32_t tick;
};

// ---- ws_grid.cu
void launch_static_types(const Dims& d, const TerrainDev& t, double coreR, uint8_t* st, uint8_t* nearRock, cudaStream_t s);
void launch_gravity_geometry(const Dims& d, double oceanR, float* g, cudaStream_t s);
// bricks: clear the accumulator of the last substep's work list only
void launch_clear_raster(const Dims& d, const GridDev& g, DevStatus* st, const BrickSet& B, bool bricks, cudaStream_t s);
void launch_brick_activity(const BrickSet& B, cudaStream_t s);
// the face passes over the active-brick list, or (all) over every brick of the grid
void launch_faces_normalize_bc(const Dims& d, const GridDev& g, const BrickSet& B, bool all, cudaStream_t s);
void launch_faces_forces(const Dims& d, const GridDev& g, const BrickSet& B, bool all, double coef, int viscOn, double dt,
                         double gs, cudaStream_t s);
void launch_project(const Dims& d, const GridDev& g, const BrickSet& B, bool all, int doClamp, double maxSpeed,
                    DevStatus* st, cudaStream_t s);
void launch_extrapolate(const Dims& d, const GridDev& g, const BrickSet& B, bool all, cudaStream_t s);
// cs: count every particle P2G will scatter in its cell (null: mark only)
void launch_mark_fluid(const Dims& d, const GridDev& g, const PartsDev& P, const TerrainDev& t,
                       double oceanR, double coreR, const CellSort* cs, DevStatus* st, cudaStream_t s);
void launch_p2g(const Dims& d, const GridDev& g, const PartsDev& P, DevStatus* st, cudaStream_t s);
// the fluid marking and P2G in index order in one pass (a substep without balls)
void launch_mark_p2g(const Dims& d, const GridDev& g, const PartsDev& P, const TerrainDev& t, double oceanR, double coreR,
                     DevStatus* st, cudaStream_t s);
size_t cell_sort_scratch_bytes(long long nKeys);
int launch_p2g_sorted(const Dims& d, const GridDev& g, const PartsDev& P, const CellSort& cs, const BrickSet& B,
                      bool binned, void* scratch, size_t scratchBytes, DevStatus* st, cudaStream_t s);
// over the brick list, or every brick of the grid (allBricks)
void launch_pressure_setup(const Dims& d, const GridDev& g, uint8_t* diag8, double omega, DevStatus* st,
                           const BrickSet& B, bool allBricks, cudaStream_t s);
void launch_sor_color(const Dims& d, const GridDev& g, int color, double om1, cudaStream_t s);
int residual_blocks(const Dims& d);
void launch_residual(const Dims& d, const GridDev& g, const uint8_t* diag8, double2* partials,
                     DevStatus* st, double* hostMirror, cudaStream_t s);
void launch_clamp_umax(const Dims& d, const GridDev& g, double maxSpeed, DevStatus* st, cudaStream_t s);
void launch_vorticity(const Dims& d, const GridDev& g, double eps, double dt, cudaStream_t s);
void launch_extract_weight(const Dims& d, const float2* acc, float* out, long long off, long long n, cudaStream_t s);

// ---- ws_particles.cu
void launch_g2p_advect(const Dims& d, const GridDev& g, const PartsDev& P, const TerrainDev& t,
                       const AdvectParams& ap, DevStatus* st, cudaStream_t s);
// copies between device memory and mapped host memory, in one launch
struct HostCopies { const void* from[16]; void* to[16]; unsigned bytes[16]; int n; };
void launch_host_copies(const HostCopies& c, cudaStream_t s);
void launch_compact(const uint8_t* fl, int nP, int mode, int* blockCounts, int* out, int* total, cudaStream_t s);
void launch_vapor_advect(const Dims& d, const GridDev& g, const PartsDev& P, const TerrainDev& t, const AdvectParams& ap,
                         const int* vIdx, const int* nV, uint32_t* rng, DevStatus* st, cudaStream_t s);
void launch_impulse_sphere(const PartsDev& P, double cx, double cy, double cz, double R, double fx, double fy, double fz, cudaStream_t s);
void launch_stir_at(const PartsDev& P, double cx, double cy, double cz, double vx, double vy, double vz, double R, double dt, cudaStream_t s);
void launch_stir_gaussian(const PartsDev& P, double pcx, double pcy, double pcz, double tx, double ty, double tz,
                          double sigma, double peak, cudaStream_t s);

// ---- ws_frame.cu
void launch_heat(const Dims& d, const GridDev& g, const PartsDev& P, const TerrainDev& t, const HeatParams& hp,
                 double dt, int* cnt, double* sumT, double* change, cudaStream_t s);
// Evaporation (exact _evS stream): prepare (flags, compaction, thresholds) once,
// then passes over the candidates from t0 until no irregular kick is reported.
struct EvapScratch {
  long long* thr; uint32_t* b; int* ejP; uint32_t* ejS;
  double* wsum; int* L; int* Ew; unsigned short* table;
};
size_t evaporation_scratch_bytes(int capacity);   // <= contacts_scratch_bytes: the two share one buffer
EvapScratch evap_carve(void* base, int capacity);
void launch_evap_prepare(const Dims& d, const GridDev& g, const PartsDev& P, double freezeT, double rate, double dt,
                         uint8_t* cand, int* blockCounts, int* list, int* nC, const EvapScratch& es, cudaStream_t s);
void launch_evap_pass(int nP, const int* list, const int* nC, const EvapScratch& es, int t0, int eoff,
                      const uint32_t* sStart, DevStatus* st, cudaStream_t s);
void launch_evap_apply(const Dims& d, const GridDev& g, const PartsDev& P, double freezeT, const EvapScratch& es,
                       int nEj, cudaStream_t s);
uint32_t evap_kick_end(uint32_t s);
void launch_phase(const Dims& d, const GridDev& g, const PartsDev& P, const PhaseParams& pp, int* cnt, cudaStream_t s);
void launch_push_surface(const Dims& d, const GridDev& g, const PartsDev& P, const TerrainDev& t,
                         double oceanR, double coreR, double atmosphereH, cudaStream_t s);
void launch_splat(const Dims& d, const GridDev& g, const PartsDev& P, double spacing, cudaStream_t s);
void launch_currents(const Dims& d, const PartsDev& P, const CurrField& F, double simTime, double strength,
                     double oceanR, double coreR, double dt, cudaStream_t s);
// marching tets in scratch (mt_scratch_bytes(d.nCells) bytes): the cells that
// straddle iso, then (at the same iso) the signed volume and the vertex count
// into out[0..1] (device or mapped host memory) and, with pos, the vertices, unless *err holds a fault; a mesh of
// more than maxVerts (0 or more) vertices: the count alone. Both return the kernels launched.
size_t mt_scratch_bytes(long long nCells);
int launch_mt_list(const Dims& d, const float* dens, double iso, void* scratch, cudaStream_t s);
int launch_mt_emit(const Dims& d, const float* dens, double iso, long long maxVerts, float* pos, float* nrm, double* out,
                   const int* err, void* scratch, cudaStream_t s);
// render-side particle prep: classify, bucket-sort far to near, emit the
// draw list (ws_render.cu); counts land in the first five scratch words
// balls (ws_balls.cu): moving-solid raster (after the static raster),
// particle push-out, and the per-substep histogram + integration
void launch_ball_raster(const Dims& d, uint8_t* type, float* sv, bool clearSv, const double* balls, int nb,
                        const GridDev& g, cudaStream_t s);
void launch_ball_push(const PartsDev& P, const double* balls, int nb, cudaStream_t s);
void launch_ball_update(const Dims& d, const float* vel, const TerrainDev& t, const PartsDev& P, double* balls, int nb,
                        int* hist, float* surfY, const BallEnv& env, double dt, cudaStream_t s);
// Metaballs.build's corner field on an (m+1)^3 lattice of spacing mdx
// (FP64 accumulation, float result; field untouched when *err holds a fault); 1 or 2 launches
void launch_metaball_field(const PartsDev& P, int m, double mdx, double R2, int rad, double* acc, float* field,
                           const int* err, cudaStream_t s);
size_t render_scratch_bytes(long long capacity);
void launch_render_particles(const RenderCfg& c, const PartsDev& P, void* scratch, RenderOut o, cudaStream_t s);
// ticket: zero before the first call (and after each); out: three doubles, device or mapped host memory
void launch_particle_reduce(const PartsDev& P, int mode, double mp, double* partials, unsigned* ticket, double* out, cudaStream_t s);

// ---- ws_queries.cu
void launch_wave_impulse(const Dims& d, const PartsDev& P, const double dir[3], uint32_t s0, double dvx, cudaStream_t s);
void launch_dry_land(const Dims& d, const TerrainDev& t, const uint8_t* type, double oceanR, int* dry, cudaStream_t s);
void launch_sample_vel(const Dims& d, const float* vel, const double* xyz, long long n, double* out, cudaStream_t s);
void launch_terrain_radius(const TerrainDev& t, double coreR, const double* xyz, long long n, double* out,
                           cudaStream_t s);
void launch_ocean_point(const Dims& d, const TerrainDev& t, double coreR, double oceanR, double need, uint32_t s0,
                        double* out, cudaStream_t s);

// ---- ws_sor_tb.cu (regions in shared memory on every SM) and ws_sor.cu (colour lists)
cudaError_t sor_init(void** statePtr, const Dims& d, int device);
void sor_free(void* statePtr);
// the whole solve of the last pressure setup's system; iterations, residual
// and path land in device memory
cudaError_t launch_sor_solve(void* statePtr, const Dims& d, const GridDev& g, const uint8_t* diag8, double omega,
                             int iters, int check, double tol, DevStatus* st, bool report, cudaStream_t s);
cudaError_t launch_sor_solve_lists(void* statePtr, const Dims& d, const GridDev& g, const uint8_t* diag8, double omega,
                                   int iters, int check, double tol, DevStatus* st, bool report, cudaStream_t s);
int sor_solve_launches(void* state);
int sor_list_solve_launches(void* state);

// ---- ws_contacts.cu
void launch_vapor_collisions(const Dims& d, const PartsDev& P, double spacing, double oceanR, int spinOn,
                             int hasSun, const double* sunRel, void* scratch, size_t scratchBytes,
                             DevStatus* st, cudaStream_t s);
void launch_ice_contacts(const PartsDev& P, double spacing, void* scratch, size_t scratchBytes, cudaStream_t s);
size_t contacts_scratch_bytes(int capacity, int rows);   // rows: ny * nz of the grid
