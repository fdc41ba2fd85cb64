// Helpers of the core library's runtime: options, and what brings a step's arrays to the device.
#include "common.cuh"

// Sets one of the ATOM_OPT_* options (common.cuh) in the core library.
ATOM_EXPORT int atom_set_option(int key, int value) { return atom::set_option(key, value); }

namespace atom {

constexpr int STEP_TABLES = 8;
struct StepTables {
  int count;
  int first[STEP_TABLES], width[STEP_TABLES], at[STEP_TABLES], pitch[STEP_TABLES];   // first: of the host's numbers
};

// dst[0..small) and the tables' live parts of a captured step, read from pinned host memory where they lie.  A captured step
// reads block tables whose rows are as long as the longest request the engine takes; a step brings only the rows of the live
// requests, as far as their longest context reaches.  It has no pdl_trigger(): what is launched behind it may read the arrays before
// it waits (common.cuh).  Bound by a round trip over PCIe, then by its rate: a thread brings one
// number, so that all reads are under way together.  In place of two copies, one of the small arrays and one of rows for a table
// (208, 4,608, 67,328 and 1,050,624 numbers, with a small kernel behind: 13.8, 12.2, 50.7 and 121 us) 3.9, 4.3, 9.2 and 87 us.
__global__ void __launch_bounds__(256) step_arrays_kernel(int* __restrict__ dst, const int* __restrict__ src, int small, int total,
                                                          const __grid_constant__ StepTables t) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= total) return;
  const int x = __ldcv(src + i);
  int64_t to = i;
  if (i >= small) {
    int k = 0;
    while (k + 1 < t.count && i >= t.first[k + 1]) ++k;
    const int e = i - t.first[k], row = e / t.width[k];
    to = t.at[k] + (int64_t)row * t.pitch[k] + (e - row * t.width[k]);
  }
  dst[to] = x;
}

}  // namespace atom

// The tables that one launch takes.
ATOM_EXPORT int atom_step_arrays_tables(void) { return atom::STEP_TABLES; }

// src: pinned host memory, `small` numbers for dst's start and then, for every table k < tables, rows x widths[k] numbers for the
// rows that begin at dst + ats[k] and lie pitches[k] apart.  dst_elems: the numbers that dst holds.
ATOM_EXPORT int atom_step_arrays(int* dst, int64_t dst_elems, const int* src, int small, int tables, int rows, const int* widths,
                                 const int* ats, const int* pitches, cudaStream_t stream) {
  if (dst == nullptr || src == nullptr || small < 0 || small > dst_elems || small > (1 << 30) || tables < 0 || tables > atom::STEP_TABLES || rows < 0)
    return ATOM_ERR_ARG;
  atom::StepTables t{};
  t.count = rows > 0 ? tables : 0;
  constexpr int64_t kMost = 1 << 30;
  int64_t total = small;
  for (int k = 0; k < t.count; ++k) {
    if (widths[k] <= 0 || pitches[k] < widths[k] || ats[k] < 0 || ats[k] + (int64_t)(rows - 1) * pitches[k] + widths[k] > dst_elems)
      return ATOM_ERR_ARG;
    t.first[k] = (int)total;
    t.width[k] = widths[k];
    t.at[k] = ats[k];
    t.pitch[k] = pitches[k];
    total += (int64_t)rows * widths[k];
    if (total > kMost) return ATOM_ERR_ARG;
  }
  if (total == 0) return ATOM_OK;
  atom::step_arrays_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(dst, src, small, (int)total, t);
  return atom::check_launch();
}
