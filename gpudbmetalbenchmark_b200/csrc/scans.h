// Launchers of the Q6/Q1 scan kernels (scans.cu), shared with the batch path (batch.cu).
#pragma once
#include "engine.h"

namespace gpudb {

constexpr size_t kQ6ResultBytes = 16;              // int64 revenue, uint64 rows matched
constexpr size_t kQ1ResultBytes = 6 * 6 * 16;      // 6 groups x {count, qty, base, disc_price, charge, discount} u128

// Enqueue one scan of device-resident columns on the call's stream, adding into `out`
// (device; kQ6ResultBytes / kQ1ResultBytes, zeroed before the first chunk). Q1 reports a
// value outside its exact-arithmetic domain in `status` (the call's status word if null).
// Q6 with `hstatus` (the status word of the call's mapped host slot, Call::begin_direct)
// overwrites `out` in that slot instead: one launch over the whole table.
int launch_q6(Call& call, const gpudb_lineitem& c, const gpudb_q6_params& p, void* out, uint32_t* hstatus = nullptr);
int launch_q1(Call& call, const gpudb_lineitem& c, const gpudb_q1_params& p, void* out, uint32_t* status = nullptr);
// One scan for n1 (1 or 2) Q1 requests that also evaluates up to 4 Q6 requests on the rows it reads
// (one read of the table for all of them), for columns that q1_shared_ok accepts; each request
// adds into its own words and, Q1, reports into its own status word.
int launch_q1_riders(Call& call, const gpudb_lineitem& c, int n1, const gpudb_q1_params* q1, void* const* q1out,
                     uint32_t* const* q1status, int n6, const gpudb_q6_params* q6, void* const* q6out);

// Whether launch_q1_riders would share one read of these columns between requests.
bool q1_shared_ok(const gpudb_ctx* ctx, const gpudb_lineitem& c);

// Loads the kernels a scan batch may use. The runtime loads a kernel at its first use (50 to 90 us
// each), which would hold up a served stream whenever a batch first has a new mix of requests; a
// server loads them all when it opens (1.3 ms, once per process).
int load_batch_kernels(gpudb_ctx* ctx);
int load_scan_kernels(gpudb_ctx* ctx);

// Host result from the kQ1ResultBytes device words of one Q1 scan.
void q1_result_from(const uint8_t* words, gpudb_q1_result* out);

}  // namespace gpudb
