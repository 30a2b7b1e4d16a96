// Device-side preparation of an uploaded CSR: 64-bit offsets narrowed to the
// 32-bit form the kernels read, and the row invariants the sampler relies on
// (ascending, unique, in range) checked without a host pass over the edges.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace silvan {

cudaError_t narrow_offsets(const uint64_t *in, uint32_t *out, uint32_t count, uint64_t limit,
                           uint32_t *bad, cudaStream_t s);
// rows[v] = (off[v], off[v + 1]) for v < n: a row's bounds in one 8-byte load
// (one memory transaction where two 4-byte loads take two).
cudaError_t make_rows(const uint32_t *off, uint2 *rows, uint32_t n, cudaStream_t s);
// *bad (device) becomes nonzero when a row is not ascending and unique, when
// an id is >= n, or when the offsets decrease.  The sums of the rows' entries
// (fwd: sums[0..1]) and of the reversed entries (bwd: sums[2..3]) are added to
// sums (device, 4 words, zeroed by the caller): the forward rows' first pair
// equals the reverse rows' second pair exactly when the two directions hold
// the same edges.
cudaError_t validate_rows(const uint32_t *off, const uint32_t *adj, uint32_t n, uint32_t *bad,
                          bool fwd, bool bwd, unsigned long long *sums, cudaStream_t s);

}  // namespace silvan
