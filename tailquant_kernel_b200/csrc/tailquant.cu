// libtailquant.so is one translation unit: the kernel files share the device-side status
// word and the PTX wrappers, and none of them needs relocatable device code.
#include "tq_api.cu"
#include "tq_prologue_fast.cu"
#include "tq_prologue.cu"
#include "tq_gemm.cu"
#include "tq_gemm_stream.cu"
#include "tq_split_gemm.cu"
#include "tq_gemm_pair.cu"
#include "tq_tail.cu"
#include "tq_misc.cu"
#include "tq_decode.cu"
#include "tq_decode_linear.cu"
#include "tq_linear.cu"
