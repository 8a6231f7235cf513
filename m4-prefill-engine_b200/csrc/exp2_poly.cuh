// Polynomials for 2^f, |f| <= 1/2, of the attention kernel's exponentials (host-compilable).
//   degree 5   minimax with the constant term held at 1 (linear programme over 4001 points on the relative error, 9.2e-8 before its
//              coefficients are rounded to fp32); evaluated with fp32 multiply-adds 1.6e-7.  (The Taylor series of that degree: 3e-6.)
//   degree 6   minimax with the constant term held at 1 (Remez exchange on the relative error, 3.9e-9 before its coefficients are
//              rounded to fp32); evaluated with fp32 multiply-adds 7.9e-8, two thirds of a unit in the last place (exp2f is documented
//              with two).
#pragma once
#ifndef __CUDACC__
#define __host__
#define __device__
#endif

namespace exp2poly {

template <int DEG> __host__ __device__ constexpr float coef(int i) {
    static_assert(DEG == 5 || DEG == 6, "degrees in use");
    if (DEG == 5) {
        const float c[6] = {1.0f, 6.9314697745e-1f, 2.4022242137e-1f, 5.5507341232e-2f, 9.6715109281e-3f, 1.3264601772e-3f};
        return c[i];
    }
    const float c[7] = {1.0f, 6.931472254e-1f, 2.4022651084e-1f, 5.5502973142e-2f, 9.6180307825e-3f, 1.3410000966e-3f, 1.5469731969e-4f};
    return c[i];
}

}  // namespace exp2poly
