// Page-locked blocks for results that leave the library as arrays over its own memory.
//
// A result of megabytes that goes through the handle's staging buffer into ordinary memory is copied once
// more and, where that memory is fresh, pays a page fault per 4 KB: 56 MB of ids took 11 ms that way, the
// transfer from the device 1.1.  A caller that lets go of one result before it asks for the next but one
// (a loop over documents) needs two blocks, which the device fills directly.  A caller that keeps every
// result gets ordinary memory once the blocks are out.
#pragma once
#include <cstddef>

namespace gtok {

// A block of at least `bytes`, or nullptr when the pool's bounds (blocks and bytes, free ones and those
// handed out together) leave no room: then ordinary memory is to be used.  Any thread.
void* result_block_get(size_t bytes);
// Gives a block back; it is kept for a later call or returned to the system.  Any thread.
void result_block_put(void* block);
// +1 for each engine that is made, -1 when it goes: with the last one the free blocks go back to the system,
// and those still in use as they are given back.
void result_blocks_user(int change);

}  // namespace gtok
