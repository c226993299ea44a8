// The fp32 product's status word (linear_f32.cu), as the libraries' status calls see it.
#pragma once

namespace atma {
int linear_f32_status_fetch_and_clear(int* out);
}  // namespace atma
