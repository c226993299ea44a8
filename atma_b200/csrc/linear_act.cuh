// The status word of the MLPs' first product (linear_act.cu), as the libraries' status calls see it.
#pragma once

namespace atma {
int linear_act_status_fetch_and_clear(int* out);
}  // namespace atma
