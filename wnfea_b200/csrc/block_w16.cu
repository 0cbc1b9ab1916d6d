// The batched solver for batches of up to 16 load cases.
#define WN_BATCH 16
#include "block_batch.cuh"
