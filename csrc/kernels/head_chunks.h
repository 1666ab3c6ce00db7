// Prompts of the recurrences of head_recurrence.h by chunks of sixteen tokens (head_chunks.cu).
#pragma once
#include <cuda_runtime.h>
#include "head_recurrence.h"

namespace nkb {
bool head_chunks_ok(const NkbHeadRec& a);              // sizes, types and alignment fit
bool head_chunks_pay(const NkbHeadRec& a);             // sequences are long enough
int head_chunks(const NkbHeadRec& a, cudaStream_t s);
}  // namespace nkb
