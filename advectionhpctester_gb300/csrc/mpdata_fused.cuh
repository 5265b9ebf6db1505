// Host interface of the fused single-precision MPDATA step (mpdata_fused.cu,
// mpdata_narrow.cu).
#pragma once
#include <cuda.h>

#include <vector>

#include "mpdata_stages.cuh"

namespace mpdata {

// Fields of the fused step's arena, each px*(mp+4)*lp floats (a halo of four
// columns and two rows on every side, none for the narrow kernels; rows a
// multiple of 4 elements so that every row starts on a 16-byte boundary, as TMA
// requires): the step's input field, the two ping-pong fields of the passes,
// pseudo and limited velocities, and two ping-pong pairs of running extrema.
enum FusedField { FZ_XIN = 0, FZ_X0, FZ_X1, FZ_V1, FZ_V2, FZ_V3, FZ_W1, FZ_W2, FZ_W3, FZ_MX0, FZ_MN0, FZ_MX1,
                  FZ_MN1, FZ_NF };

// The kernels a problem runs on: the gauge form on a grid that is periodic on
// every axis (wraps only) by 64x12 tiles or by narrow ones, the gauge form with
// open or wall axes, the standard form on any grid; FZ_NONE: the stage kernels
// (in a batch the tile kernels).
enum FusedClass { FZ_NONE = -1, FZ_PERIODIC = 0, FZ_NARROW, FZ_WALL, FZ_STD };

// Arguments of the fused kernels for one problem: caller arrays, the arena,
// the z-march chunk, and the arena fields of the current pass.
struct FusedArgs {
  Geo g;
  Arr<float> psi, u1, u2, u3, h, rhr;
  int stdf;                // the standard form
  const float *bcx, *bcy;  // Dirichlet halo values of psi on open x and y walls
  float* arena;
  int px;
  long fs;
  int ntx, nty;                       // tiles along x and y
  unsigned char* flags;               // per plane and tile: h and rhr all exactly 1 (written by the first kernel)
  int kchunk;
  int fin, fout;                      // pass input / output field
  int fmx_in, fmn_in, fmx_out, fmn_out;
  int* err;
};

struct FusedPlan {
  Geo g;
  FusedClass cls;
  Arr<float> psi, u1, u2, u3, h, rhr;  // caller arrays
  const float *bcx, *bcy;
  float* arena;
  int kchunk;   // planes per block of the z-march
  int* err;     // device error word (bit 1: a staging wait timed out)
  const CUtensorMap* tmap;  // one 4-D map over the arena (x, y, z, field)
  unsigned char* flags = nullptr;  // the unit flags, where they do not follow the FZ_NF fields
};

// Whether the fused kernels on 64x12 tiles can take a step: FP32, nonoscillatory,
// iord >= 2, not the density step.
bool fused_eligible(const Geo& g, int precision, int gauge, int nonos, int iord, int rho);
// The kernels of n problems that are stepped together (cls[p]).  FP32 steps with
// the limiter and iord >= 2, outside the density step, run on the fused kernels
// where these are the faster ones.
void fused_classes(const Geo* g, const int* gauge, int n, int precision, int nonos, int iord, FusedClass* cls);
// Arena geometry of a class: row pitch, elements per field, tiles, and the total
// elements of the FZ_NF fields and the flags.
struct FusedArena {
  int px, ntx, nty;
  long fs;
  size_t elems;
};
FusedArena fused_arena(const Geo& g, FusedClass c);
// An arena field's interior as an array view.
Arr<float> fused_view(float* arena, int field, const Geo& g, FusedClass c);
// Encodes the arena's tensor map (one field's box in a plane).  0 on success.
int fused_make_tmap(CUtensorMap* map, float* arena, const Geo& g, FusedClass c, int fields = FZ_NF);
// Planes per block of the z-march for each of the n problems that are stepped
// together (MPDATA_FUSED_KCHUNK overrides).
void fused_kchunk(const Geo* g, const FusedClass* c, int n, int* kchunk);
// One step; on return *mx_field / *mn_field name the arena fields that hold
// the running extrema of the step (-1 when iord = 2 keeps none).
int run_step_fused(const FusedPlan& F, int iord, Prof* prof, cudaStream_t s, int* mx_field, int* mn_field);

// The forward record of an iord-2 gauge step, left in the arena F names: the
// fields up to FZ_V3 (FZ_NREC of them, and the flags), of which FZ_X0 holds the
// upwind field and FZ_V1..3 the pseudo-velocities.  update: the step's output is
// written to F.psi as by run_step_fused; without it only the record is made.
constexpr int FZ_NREC = FZ_V3 + 1;
int run_record_fused(const FusedPlan& F, bool update, cudaStream_t s);

// Batches.  Each problem of the fused table gets work items (a tile and a z
// chunk) packed as problem | tile x << 16 | tile y << 32 | chunk << 48; one
// launch per fused kernel and work list (the periodic gauge problems; the walled
// and standard-form ones; the narrow ones, whose first kernel has its own tiles)
// then covers every problem.
FusedArgs fused_args(const FusedPlan& F);
enum FusedList { FZ_L_PERIODIC = 0, FZ_L_MIXED, FZ_L_NARROW_UP, FZ_L_NARROW, FZ_NLIST };
inline unsigned long long pack_item(int p, int x, int y, int z) {
  return (unsigned long long)p | ((unsigned long long)x << 16) | ((unsigned long long)y << 32) |
         ((unsigned long long)z << 48);
}
// Appends problem p's items to its lists (items[FZ_NLIST]).
void fused_items(const Geo& g, FusedClass c, int kchunk, int p, std::vector<unsigned long long>* items);
int fused_init();
// A device work list.
struct FusedItems {
  const unsigned long long* items;
  int n;
};
// One step of every problem of the table (device arrays: args, tensor maps;
// items[FZ_NLIST]: the lists, empty ones with n = 0).
int run_batch_fused(const FusedArgs* probs, const CUtensorMap* maps, const FusedItems* items, int iord, Prof* prof,
                    cudaStream_t s);

// The narrow kernels' part of the above.
FusedArena narrow_arena(const Geo& g);
int narrow_make_tmap(CUtensorMap* map, float* arena, const Geo& g);
void narrow_kchunk(const Geo* g, int n, int* kchunk);
void narrow_items(const Geo& g, int kchunk, int p, std::vector<unsigned long long>& up,
                  std::vector<unsigned long long>& rest);
int narrow_init();
int narrow_step(const FusedPlan& F, int iord, Prof* prof, cudaStream_t s, int* mx_field, int* mn_field);
int narrow_batch(const FusedArgs* probs, const CUtensorMap* maps, const FusedItems& up, const FusedItems& rest,
                 int iord, Prof* prof, cudaStream_t s);

}  // namespace mpdata
