// The batched solver for batches of up to 8 load cases.
#define WN_BATCH 8
#include "block_batch.cuh"
