// Host-side launch interface between the plan builder (glqb_api.cu) and the translation units that
// instantiate the large kernel families (glqb_gemm_inst.cu: tensor-core GEMMs and tile decodes;
// glqb_fused.cu: single-launch decode).  Splitting them keeps every unit's compile time in check.
#pragma once
#include "glqb_internal.h"
#include "glqb_comm.cuh"
#include <cstdlib>

namespace glqb {

struct GemmItem;

// Launch with programmatic stream serialization: the kernel may start while the one before it on the stream is still running
// and orders itself behind it (pdl_wait).  What comes before the wait (scheduling, barriers, tensor memory, table fills, the
// decode of weights) overlaps the other kernel's tail.  GLQB_PDL=0 launches in the ordinary way.
// Whole calls back to back, ordinary / chained: one token of 14336 x 4096 (E8: the 224 KiB table is copied during the input
// transform) 52.2 / 47.3 us, 333 tokens of 2048 x 11008 44.2 / 40.9, 2048 tokens of 11008 x 2048 155 / 151, 700 tokens of
// 5376 x 21504 309 / 304.  Not chained: e8_tiles_kernel, whose gathers need the L1 that the input transform's shared memory
// would still hold (2048 tokens of 14336 x 4096 346 / 368 us), the streaming trellis kernel, which has nothing to do early, and the
// launches of experts but their trellis matmuls (MOE_CHAIN_MAX).  A kernel whose successor would take the room it needs, or find
// room on a few SMs only, does not trigger (glq_gemm_kernel).
inline bool pdl_enabled() {
  static const bool on = [] { const char* e = getenv("GLQB_PDL"); return !e || atoi(e) != 0; }();
  return on;
}
template <class... P, class... A>
inline cudaError_t launch_chained(bool chain, void (*kernel)(P...), int grid, int threads, size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = chain && pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// One launch of a streaming decode kernel: a set of layers that share format / bit widths /
// token-column blocks, contiguous in the device table.
struct Segment {
  int format, k1, k2, ns, nb;
  int tn;                    // 0: streaming decode kernel; else tensor-core GEMM with that token tile (glq_gemm_kernel: 128
                             // or 256, trellis_gemm_kernel: a multiple of 16 up to 192)
  int two_phase = 0;         // GEMM with many tokens: weight tiles decoded once beforehand (E8, large trellis layers)
  // single-launch form (input transform + decode + output transform in one kernel): all layers read one input
  bool fused = false;
  int total_units = 0, scratch_elems = 0;
  size_t fused_smem = 0;
  int first, count;          // range in the device table
  long long total_groups;
  int per_warp;
  int grid;
  int item_first, item_count;   // GEMM work items (range in the plan's item array)
  // E8 only: most of the codebook resident in shared memory (one CTA per SM)
  bool lut_table = false;    // trellis: table form of the streaming kernel (large batch-1 launches)
  bool smem_table = false;
  const uint32_t* big_table = nullptr;
  const uint32_t* small_table = nullptr;
  int small_entries = 0;
  int res_entries = 0;       // single-launch E8 form: table entries kept in shared memory (0: all gathers go to L1 / L2)
};

// does trellis_gemm_kernel run the segment's GEMM?  (Else glq_gemm_kernel: decoded tiles, E8, two stages with 256-token
// tiles.)  The activation layout follows from it.
inline bool trellis_form(const Segment& s) { return s.tn && s.tn < 256 && s.format == GLQB_FMT_TRELLIS_3INST && !s.two_phase; }

constexpr int GEMM_STAGES = 4;

// ---- glqb_gemm_inst.cu
bool gemm_available(const Segment& s);                       // is there a kernel for the segment's format / rates?
cudaError_t gemm_prepare(const Segment& s);                  // raises the kernel's dynamic shared-memory limit
cudaError_t tiles_smem_prepare(int ns);                      // same for the resident-table tile decode
// the segment's launches: (two-phase: tile decode, then) the GEMM over `items`, for at most `tokens` tokens per layer
void gemm_launch(const Segment& s, const DevLinear* layers, const GemmItem* items, uint8_t* ws, int* status,
                 int sm_count, int tokens, cudaStream_t stream);

// ---- glqb_fused.cu
bool fused_available(const Segment& s);                      // is there a single-launch kernel for the segment's format / rates?
cudaError_t fused_prepare(const Segment& s, size_t smem_limit, size_t smem, int* resident_ctas_out);
// `layers`: HOST copy of the segment's table entries (they are passed to the kernel by value)
// `comm`: null, or the communicator whose ranks' outputs are summed inside the kernel (layers with DevLinear::reduce)
void fused_launch(const Segment& s, const DevLinear* layers, const uint8_t* x_base, uint8_t* y_base, uint8_t* ws,
                  int* tickets, const CommDev* comm, cudaStream_t stream);

// ---- glqb_comm.cu
const CommDev* comm_dev(const GlqbComm* c);                  // null until the communicator is connected

}  // namespace glqb
