// The batched solver for batches of up to 32 load cases.
#define WN_BATCH 32
#include "block_batch.cuh"
