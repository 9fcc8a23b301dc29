// attention_tc.cu: attention of many query rows on the tensor cores (f32 operands split into half-precision pairs)
#pragma once
#include "cached_attention.cuh"

// what decides the launch of a CACHED_ATTENTION step: its sizes, the keys all its rows together and one row can see at most
struct ZgAtcShape { uint32_t T, H, G, maps, dk, dv, reach, keys; };
bool zg_attention_tc_usable(const ZgAtcShape& s);
size_t zg_attention_tc_scratch_elems(const ZgAtcShape& s, int n_sm);
// args: CaArgs with 16-byte aligned rows.  *splits > 1: the key shares lie in *part, to be merged by the caller.
bool zg_attention_tc_launch(const ZgAtcShape& s, const void* args, float* scratch, int n_sm, cudaStream_t st, uint32_t* splits, float** part);
