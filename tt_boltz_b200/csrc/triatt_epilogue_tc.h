// Triangle-attention epilogue on tcgen05 (triatt_epilogue_tc.cu).
#pragma once
#include "common.cuh"

namespace b200pf {
namespace tae {

// z [rows][128] fp32 += (o * g) w_o^T, or (z null) upd [rows][128] bf16 = it; pointers 16-byte aligned, rows below 2^31 - 128
int launch(float* z, __nv_bfloat16* upd, const __nv_bfloat16* o, const __nv_bfloat16* g, const __nv_bfloat16* w_o, int rows, int sms, cudaStream_t st);

}  // namespace tae
}  // namespace b200pf
