// Page-locked host blocks shared by everything in the process that receives pixels from the GPU: the payloads of one
// download sit in blocks of about 8 MB, and a block lives as long as anybody still looks at one of them (reference counted).
//
// Why: a fresh pageable buffer per payload costs a page fault per 4 KB (2 GB/s on the virtual machines this runs on) and a
// staged copy by the driver; handing out views of the block the copy engine wrote costs neither.
//
// Blocks are private mappings that are page-locked afterwards (cudaHostRegister), not cudaHostAlloc memory: that is a shared
// mapping, so a forked child (a data loader's worker) that inherited a payload would see the parent's pool write the next
// one over it.  Page-locked private memory is copied when a process forks (0.3 s and 800 MB for 800 MB of blocks), so only
// blocks that somebody references go to the child (madvise).  They are quicker to make as well (48 of 768 KB: 2.1 ms, 50 ms with cudaHostAlloc; the copies run at the
// same 56 GB/s).
//
// Bounds: blocks nobody references are kept for reuse up to a limit (DATAGO_B200_HOST_BLOCKS_MB, default 1024) and freed
// beyond it, all of them when the last device context of the process goes away.  Requests that have an alternative (`optional`)
// are refused when they would bring what is referenced above the same amount, so a caller that hoards payloads does not lock
// all of its memory.  While there are feeders, whose batches have no alternative, blocks are kept for reuse up to the most that
// was referenced at one time: a batch of 512 photos is 1.6 GB, and locking that anew each time took longer than the decoding
// (8192 photos through a feeder: 589 images/s, 13 000 to 14 600 with blocks that stay).
#pragma once
#include <cstddef>

namespace dg {

int host_block_acquire(size_t nbytes, bool optional, void** out);  // dg_status; one reference
void host_block_retain(void* base);
void host_block_release(void* base);
bool host_blocks_scarce();  // whether more than the limit is referenced
bool host_blocks_room(size_t nbytes);  // whether optional requests for that much would be granted
void host_blocks_feeder(int change);  // +1 / -1 feeder
// +1 / -1 context on `device`.  Blocks are page-locked on a device that has one: the calling thread's current device may be
// another rank's, and locking there would create a context on it.
void host_blocks_context(int device, int change);

}  // namespace dg
