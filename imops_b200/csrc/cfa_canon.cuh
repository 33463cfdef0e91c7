// cfa_canon.cuh -- the CFA patterns whose colours kernels compile in, and how a
// CFA is recognised as a shift of one of them.
#pragma once

#include "common.cuh"

namespace imops {
namespace canon {

// Canonical patterns, colour codes as parse_cfa assigns them (R 0, G 1, B 2),
// two bits a cell, packed at compile time.
__host__ __device__ constexpr int colour_code(char ch) { return ch == 'R' ? 0 : ch == 'G' ? 1 : 2; }
__host__ __device__ constexpr unsigned long long pack2(const char* p, int from, int n) {
    unsigned long long v = 0ull;
    for (int i = 0; i < n; i++) v |= (unsigned long long)colour_code(p[from + i]) << (2 * i);
    return v;
}
struct BayerCanon {  // RGGB
    static constexpr int PW = 2, PH = 2;
    static constexpr unsigned long long LO = pack2("RGGB", 0, 4), HI = 0ull;
    __host__ __device__ static constexpr int at(int r, int c) {
        return (int)((r * PW + c < 18 ? LO >> (2 * (r * PW + c)) : HI >> (2 * (r * PW + c - 18))) & 3ull);
    }
};
struct XTransCanon {  // the X-Trans sensors' 6x6 period
    static constexpr int PW = 6, PH = 6;
    static constexpr unsigned long long LO = pack2("GGRGGBGGBGGRBRGRBG", 0, 18);
    static constexpr unsigned long long HI = pack2("GGBGGRGGRGGBRBGBRG", 0, 18);
    __host__ __device__ static constexpr int at(int r, int c) {
        return (int)((r * PW + c < 18 ? LO >> (2 * (r * PW + c)) : HI >> (2 * (r * PW + c - 18))) & 3ull);
    }
};

// (ox, oy) with colour(y, x) == P::at((y - oy) mod PH, (x - ox) mod PW) for
// every site of c's period, or false when c is no shift of P.
template <class P>
bool canonical_offset(const CfaDev& c, int* ox, int* oy) {
    if (c.pw != P::PW || c.ph != P::PH) return false;
    for (int dy = 0; dy < P::PH; dy++)
        for (int dx = 0; dx < P::PW; dx++) {
            bool ok = true;
            for (int r = 0; r < P::PH && ok; r++)
                for (int q = 0; q < P::PW && ok; q++)
                    ok = c.col[r * P::PW + q] == P::at((r - dy + P::PH) % P::PH, (q - dx + P::PW) % P::PW);
            if (ok) {
                *ox = dx;
                *oy = dy;
                return true;
            }
        }
    return false;
}

}  // namespace canon
}  // namespace imops
