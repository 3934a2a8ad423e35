/*
 * Internal interfaces shared by the CUDA translation units of the gravity
 * library (not part of the public C-ABI in include/).
 */
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "cuda_typedef.h"
#include "changa_gb300.h"

namespace chg {

enum Form : int { kF32 = 0, kF64 = 1, kMix = 2 };

/* Arguments of one interaction-list launch. */
struct ListArgs {
  const void* src;      // kF32: CudaMultipoleMoments* or CompactPartData*
                        // kF64: double* (12 or 5 per row); kMix: packed float4
  long long n_src;
  const void* tgt;      // kF32: CompactPartData*; kF64: double*; kMix: packed float4
  long long n_tgt;
  void* vars;           // kF32: VariablePartData*; kF64/kMix: double* (5 per row)
  const int2* list;     // ILCell {index, offsetID}
  long long n_entries;  // entries in list (markers are clamped to it)
  const int* markers;   // n_buckets + 1
  const int* starts;
  const int* sizes;
  int n_buckets;
  float fperiod_f;
  double fperiod_d;
  unsigned int* queue;  // work counter, zero at launch
  /* the launch before this one in the stream is a list kernel of the same
   * evaluation (same vars, its inputs ready before that one began): this one
   * may start as that one drains */
  bool after_list = false;
};

/* Packed FP32-mixed layouts (built by pack kernels from FP64 inputs):
 *   cell   : 4 float4 per node  {hi.xyz, M} {lo.xyz, soft} {xx,xy,xz,yy}
 *            {yz, zz, tr, 0}
 *   particle: 2 float4 per particle {hi.xyz, mass} {lo.xyz, soft}
 * hi = (float)x, lo = (float)(x - hi), both exact in FP64. */
constexpr int kCellPackF4 = 4;
constexpr int kPartPackF4 = 2;
/* hexadecapole cell: {hi.xyz, M} {lo.xyz, soft} then the radius and the 21
 * scaled reduced moments (xx xy xz yy yz, xxx xyy xxy yyy xxz yyz xyz,
 * xxxx xyyy xxxy yyyy xxxz yyyz xxyy xxyz xyyz) and two zeros */
constexpr int kCellHexPackF4 = 8;

/* launchers (grav_lists.cu) */
cudaError_t launch_list(int form, bool cell, const ListArgs& a, cudaStream_t s);
int list_variant_count();
int set_list_variant(int kernel, int variant);
int get_list_variant(int kernel);
int set_hex_variant(int v);
int get_hex_variant();
/* poll limit of the TMA variants' mbarrier waits (negative: the default) */
void set_tma_wait_polls(int polls);
/* TMA-variant launches since load */
unsigned long long tma_launches();
/* Synchronises the current device, then returns (in bits) and clears the
 * library's device status word (bit 0: a TMA wait ran out). */
cudaError_t read_device_status(unsigned* bits);
cudaError_t launch_pack_cells(const double* moments, long long n, float4* out, cudaStream_t s);
cudaError_t launch_pack_parts(const double* parts, long long n, float4* out, cudaStream_t s);
/* Both and kQueueInts zero words at queue, in one launch.  Cells: of 12 doubles,
 * or of 27 for the hexadecapole form, packed as list_kernel_hex (variant 0)
 * or as list_kernel_hex2 reads them. */
constexpr int kQueueInts = 192;
enum PackCells { kPackQuad = 0, kPackHex = 1, kPackHexPaired = 2 };
cudaError_t launch_pack_step(PackCells kind, const double* moments, long long n_moments, float4* cells,
                             const double* parts, long long n_parts, float4* packed,
                             unsigned int* queue, cudaStream_t s);
cudaError_t launch_zero_vars_f32(VariablePartData* v, long long n, cudaStream_t s);
/* hexadecapole build: cell lists over 27-double (kF64) or packed (kMix)
 * moments; the pack; cells as point-mass particles {M, soft, cm} */
/* variant: get_hex_variant() as the cells were packed by launch_pack_step */
cudaError_t launch_list_hex(int form, const ListArgs& a, int variant, cudaStream_t s);
cudaError_t launch_cells_as_parts(const double* moments, int stride, long long n, double* out,
                                  cudaStream_t s);

/* Ewald (ewald.cu) */
struct EwaldArgsF32;  // defined in ewald.cu
cudaError_t launch_ewald_f32(const CompactPartData* parts, VariablePartData* vars,
                             const int* markers, int largephase, int first, int last,
                             const EwaldReadOnlyData& ro, const EwtData* ewt,
                             cudaStream_t s);
/* hex: the hexadecapole build's expansion (p.momc required) */
cudaError_t launch_ewald_fp(int form, const double* parts, long long n_parts, const int* idx,
                            long long n_idx, const ChangaEwaldParams& p, double* vars,
                            cudaStream_t s, bool hex = false, bool after_list = false);

/* adjoint of the Ewald term (quadrupole root expansion, FP64): adds the
 * vector-Jacobian product of lam . a_ewald to grad (n x 4 {dL/dx, dL/dm});
 * acc: 10 doubles of device scratch */
cudaError_t launch_ewald_vjp(const double* parts, long long n_parts, const ChangaEwaldParams& p,
                             const double* lam, double* grad, double* acc, cudaStream_t s);

/* runtime helpers (hostcuda.cu) */
int sm_count();
void count_launch(unsigned n = 1);
/* Keeps memory freed with cudaFreeAsync cached in this device's default
 * pool (a process-local pool attribute, set once per device). */
void prepare_pool();
int record_error(int code, const char* what, const char* file, int line);

/* Kernel ids for the optional per-kernel event timing
 * (changa_gb300_set_timing / changa_gb300_kernel_time). */
enum KernelId : int {
  kKidListF32Cell = 0, kKidListF32Part, kKidListF64Cell, kKidListF64Part, kKidListMixCell,
  kKidListMixPart, kKidEwaldF32, kKidEwaldF64, kKidEwaldMix, kKidPack, kKidVjpCell, kKidVjpPart,
  kKidMoments, kKidCount
};
inline int list_kernel_id(int form, bool cell) { return 2 * form + (cell ? 0 : 1); }

/* Records CUDA events around one launch on stream s when timing is on. */
struct TimingScope {
  TimingScope(int kid, cudaStream_t s);
  ~TimingScope();
  int kid;
  cudaStream_t s;
  void* start;
};

#ifdef __CUDACC__
/* Launches of one evaluation that only meet in the sums they add to vars
 * overlap: the first lets its successor start once every one of its own
 * blocks has (open_to_next), the successor's blocks take the places that it
 * frees as it drains, and wait for its end (wait_for_last) before they touch
 * vars.  Without the attribute of launch_after both are no-operations.  A
 * kernel launched so has wait_for_last in every path that adds to vars and at
 * its end, so that it never ends before the one it overlaps, whose end the
 * launches after it rely on.  us a
 * step, one after another / so: 32768 Plummer particles 125 / 107, 6000 of
 * them 52 / 40, 1200 37 / 25; 12000 periodic with Ewald 87 / 51; 2^20 with
 * Ewald 2490 / 2350. */
__device__ __forceinline__ void open_to_next() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_for_last() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

/* The share of an SM's L1 kept as shared memory, in percent, asked for by every
 * kernel that overlaps another: an SM that must change its split first drains,
 * which cost more than the overlap gave (1200 periodic particles 82 us a step
 * with the runtime's choice per kernel, 35 with one split; 75 without
 * overlap).  60 holds each kernel's resident blocks, but the FP64 Ewald
 * kernel's, so the FP64 form asks for all of it. */
constexpr int kCarveoutFp32 = 60, kCarveoutFp64 = 100;
template <typename K>
inline void set_carveout(K kernel, int percent) {
  cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, percent);
}

template <typename... P, typename... A>
cudaError_t launch_after(void (*kernel)(P...), int grid, int threads, cudaStream_t s, bool overlap,
                         A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
#endif

}  // namespace chg

#define CHG_CUDA(call)                                                            \
  do {                                                                            \
    cudaError_t e_ = (call);                                                      \
    if (e_ != cudaSuccess) return ::chg::record_error((int)e_, #call, __FILE__, __LINE__); \
  } while (0)
