/* game_gpu_numerics' operations of the FP64 path (numerics_f64.cu) */
#pragma once

namespace game {

constexpr int NUMERICS_F64 = 11, NUMERICS_OPS = 22; /* the first of them, one past the last */
__host__ __device__ inline bool numerics_two_inputs(int op) { return (op >= 9 && op <= 15) || op == 21; }
void launch_numerics_f64(int op, const double *in, double *out, long long n);

}  // namespace game
