// m2_internal.hpp -- what one part of libm2gpu reads from a context that the
// C ABI does not expose: its digit layout, creation options, stream and
// device-side state.  Every call is stream-ordered on the context's stream.
#pragma once
#include "../../include/m2gpu.h"
#include "m2_host.hpp"

#include <cuda_runtime_api.h>

namespace m2k { struct LargePlan; }

namespace m2i {

// Device-to-host copy behind the stream's work, with that work waited for first
// where the destination is pageable: the driver then waits for it inside the
// copy, under a lock that every other thread's allocation, event creation and
// stream creation needs (a thread beside a batch of 3 s had its first call back
// after 2.6 s, with the wait here 0.2 ms).
inline cudaError_t read_back(void* dst, const void* src, size_t bytes, cudaStream_t s) {
    cudaPointerAttributes at{};
    cudaError_t e = cudaPointerGetAttributes(&at, dst);
    if (e != cudaSuccess) cudaGetLastError();
    if (e != cudaSuccess || at.type == cudaMemoryTypeUnregistered) e = cudaStreamSynchronize(s);
    return e == cudaSuccess ? cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s) : e;
}

// plan of the three-pass path for exponent layout L (false: no plan fits);
// carry_pairs is the -B hint (columns per CTA), 0 for the default
bool plan_large(const m2::Layout& L, int span, uint32_t carry_pairs, m2k::LargePlan& P);

// digit widths and bit positions of the context's residue
const m2::Layout& layout(const m2_ctx* c);
// the options of m2_create (device, hints, path, fields), with the stream
// cleared: a second context built from them has the same transform
m2_opts creation_opts(const m2_ctx* c);
cudaStream_t stream(const m2_ctx* c);

// the state's n canonical digits, written into the context's canonical
// buffer (device memory, valid until the context's next call)
int canonical(m2_ctx* c, const unsigned long long** out);
// the state's n signed digit words (device memory) for a caller that writes
// a new state there and reads it back through canonical(); pending segment
// carries are cleared
int raw_state(m2_ctx* c, long long** digits);
// the context's canonical buffer (device memory, n words), allocated if needed
int canon_buffer(m2_ctx* c, unsigned long long** buf);
// where launches may have been called off (m2_board.hpp): waits for the context's
// work and runs their squarings.  A read on the device, like canonical(), comes
// after it.  The state's code
int settle(m2_ctx* c);
// m2_iterate by launches that are not called off; after it the state is read by
// canonical() or replaced by load_canon()
int iterate_unowed(m2_ctx* c, uint32_t k);
// the runs of these contexts are ordered by events: neither keeps the other off
// the device
void share_turns(m2_ctx* a, m2_ctx* b);
// state <- the canonical digits in the canonical buffer (balanced on the
// device), with the iteration counter set
int load_canon(m2_ctx* c, uint32_t iteration);

}  // namespace m2i
