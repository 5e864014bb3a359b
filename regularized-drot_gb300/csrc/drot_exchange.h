// drot_exchange.h -- rules of the exchange between the CTAs of a resident solve
// (drot_resident.cuh) that both the kernel and the host checks use.
#pragma once

#ifdef __CUDACC__
#define DROT_XHD __host__ __device__ __forceinline__
#else
#define DROT_XHD inline
#endif

namespace drot {

// The slot (of two) that the residual of iteration `it` is published in: the
// tested iterations take them in turn.  every: all iterations are tested, not
// only the even ones.
//   A slot is written again two tests later, and every CTA must have read it by
// then.  With two copies of X a CTA reads the residual of iteration t during t
// + 1, in a warp that nothing orders before its mass word of t + 1.
//   Tests on even iterations: CTA A publishes t + 4 into t's slot after it has
// seen every mass word of t + 2, which CTA B adds after its own round t + 1, the
// read included.  (A slot of the iteration's parity is written again at t + 2,
// which A enters on the mass words of t + 1: B may still be reading.)
//   Tests on every iteration: A publishes t + 2 after it has read t + 1 in the
// same warp, which B publishes after it has read t.
//   With one copy of X the read of t ends iteration t, and the next test comes
// after the mass words of an iteration in between.
DROT_XHD int residual_slot(int it, bool every) { return (every ? it : it >> 1) & 1; }

}  // namespace drot
