// Who may trust a "full" barrier's parity: the rule that the MMA issuers of the tensor-core Linear follow on their shared ring of
// slots. Host code as well, so that it can be checked against a model of the barriers without a GPU.
#pragma once

#ifdef __CUDACC__
#define TTB_RING_FN __host__ __device__ __forceinline__
#else
#define TTB_RING_FN inline
#endif

namespace ttb {
namespace ring {

// A ring of `stages` slots is filled block after block; block g goes to slot g % stages and is that slot's use number g / stages.
// Of a tile's blocks, issuer i of two takes those at offsets i, i + 2, ...
//
// A wait on a barrier names only the parity of the use it waits for, so that an issuer that waits for use n of a slot must know
// that use n - 1 has landed: were it still on its way, the barrier would show the parity of use n - 2, which is that of use n, and
// the issuer would multiply what the slot holds by then. Where use n - 1 was the issuer's own, it has waited for it before. Where it
// was the other's, nothing orders the two: loads may land in any order. That is so
//   - on every block when the number of slots is odd: the block `stages` earlier is at an offset of the other parity;
//   - on the first `stages` blocks of a tile when tiles have an odd number of blocks: the offsets of the tile before count on from
//     another parity. (With an even number of slots and of blocks, a slot belongs to one issuer throughout.)
// There the issuer first waits for the slot's "empty" barrier, as the producer does before it fills the slot: use n - 1 has then
// been read, hence had landed. That is no new dependency, the load that the issuer is about to wait for made the same wait.
//
// That wait is unambiguous in turn: it could only be mistaken for use n - 3, and use n - 2 has been read. An issuer is at most
// three blocks past its last one (an odd tile's end); the producer issued that one, block h >= g - 3, only once block
// h - stages had been read, and with it all before. With three slots or more that covers block g - 2 * stages, use n - 2.
constexpr int kMinStages = 3;

TTB_RING_FN constexpr bool wait_for_empty_first(int stages, int issuers, int tile_blocks, int offset) {
  return issuers == 2 && (stages % 2 != 0 || (tile_blocks % 2 != 0 && offset < stages));
}

}  // namespace ring
}  // namespace ttb
