// Time loops on chip (stencil_resident.cu): a shot's whole wavefield stays in
// the shared and tensor memory of a group of CTAs for all steps of a launch.
// This header is what the engine needs to plan and launch them.
#pragma once

#include "fused.cuh"

namespace daw {

constexpr int kResCols = 27;       // most grid columns per CTA (column masks read 4 ahead)
constexpr int kResRowBlocks = 15;  // most 128-row blocks per CTA
constexpr int kResWarps = 16;      // most warps per CTA (128 registers a thread)
constexpr int kResShots = 16;      // most shots (CTA groups) per launch
constexpr int kResPolls = 1 << 22; // rounds after which a wait gives up (seconds)

// A rectangle of the extended grid whose pressure every step is kept for the
// Hicks gathers after the loop: rows [r0, r1), columns [c0, c1), step-major
// [step][row][col] with `ld` columns and `step` elements per step.
struct ResidentRect {
  float* buf;
  size_t step;
  int ld, r0, r1, c0, c1;
  int quad0;  // first quad of rows in the shared-memory staging (ResidentLaunch::quads)
};

// Injection tables of one station map for CTAs of C columns: CTA b's points
// are C columns x (rows of its header), `m` entries per point in station
// order (padded with zero coefficients).
struct ResidentInj {
  const int4* head;             // per CTA: first row (of 4), rows, first station, stations
  const float* cd;              // coefficient * dt   [cta][pts][m]
  const unsigned short* sta;    // station - first station of the CTA
  const float* kap;             // kappa of the point [cta][pts]
  int pts, m, nsta;             // capacities: points and stations per CTA, entries per point
};

struct ResidentShot {
  float *px, *pz, *vx, *vz;     // state at the start (load) and the end (save) of the launch
  void* hist;
  unsigned* amax;
  const float* amp;             // step-major amplitudes [step][nsta]
  int nsta;
  ResidentInj inj;              // pts = 0: no injection
  ResidentRect rect[2];         // buf = nullptr: unused
  float* wf;                    // optional (n1,n2,nt) pressure output, wf_acc: accumulated
  int wf_acc;
  int nt, first, last;          // record length; steps of this launch
};

struct ResidentLaunch {
  int C, G, RB, groups;         // columns per CTA, CTAs per shot, 128-row blocks, shots
  bool ps;                      // p in shared memory
  int CG, CW;                   // column groups and columns of a group (resident_launch)
  ulonglong2* halo;             // [phase][parity][cta][3][RB * 32][2]
  unsigned long long* slots;    // 72 words a CTA: stage A's maxima and their results
  int poll_limit;               // kResPolls but in tests
  unsigned tag0;                // step tags of this launch: tag0 + step
  int load, save;               // state from / to global memory (else zero / dropped)
  int slo;                      // pressure source margin (1: final esource)
  int n1h, hist_step0;
  int inj_pts, inj_m, inj_sta;  // shared-memory capacities of the injection tables
  int quads;                    // quads of rows staged for the rectangles, 0: written directly
  unsigned* err;
  unsigned long long nz;        // (-0, -0), set by resident_launch
  ResidentShot shot[kResShots];
};

// Dynamic shared memory of a CTA.
size_t resident_smem(int C, int RB, bool ps, int inj_pts, int inj_m, int inj_sta, int quads);
// Warps of a CTA: column groups and columns per group.
void resident_groups(int C, int RB, bool ps, int* cg, int* cw);
// CTAs per SM of (mode, fp16, density) with that much shared memory; 0 when it does not fit.
int resident_occupancy(int mode, bool fp16, bool rho, bool ps, int C, int RB, size_t smem);
cudaError_t resident_launch(const Grid& g, const ModelDev& m, const ResidentLaunch& L, int mode,
                            bool fp16, cudaStream_t st);
// Fills the injection tables of a station map for the CTAs' headers.
void resident_tables(const Grid& g, const ModelDev& m, const InjMapDev& map, int C, int G,
                     const int4* head, int pts, int mm, float* cd, unsigned short* sta, float* kap,
                     cudaStream_t st);
// Hicks sums of a station set for steps 0 .. nsteps-1 of a rectangle buffer,
// the support clipped to rows [lo1, hi1) and columns [lo2, hi2), and to the points that
// are updated (`off` rows and columns at the far edges are not), which the others'
// zeros add nothing to:
// out[row(step) + nt * station], row = row0 + step, or row0 - step when reverse.
void resident_gather(const Grid& g, const ResidentRect& r, const StationsDev& st, int off, int lo1,
                     int hi1, int lo2, int hi2, int nsteps, float* out, int nt, int row0, int reverse,
                     cudaStream_t s);

}  // namespace daw
