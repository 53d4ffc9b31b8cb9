// 2^r on [-0.5, 0.5]: the polynomial of degree 5 of least relative error (Remez exchange in 64 bits, coefficients rounded to
// fp32).  By Horner's rule in fp32 its relative error is 2.1e-7, within the 2^-22 of the exponential unit beside which
// attention_tc05.cu evaluates it.  Plain constants, for device code and (for the tests) host code.
#pragma once

namespace ptv3 {

constexpr float EXP2_C0 = 1.0000001192092896f, EXP2_C1 = 0.6931469440460205f, EXP2_C2 = 0.24022120237350464f,
                EXP2_C3 = 0.05550713092088699f, EXP2_C4 = 0.009675540961325169f, EXP2_C5 = 0.0013276472454890609f;

}  // namespace ptv3
