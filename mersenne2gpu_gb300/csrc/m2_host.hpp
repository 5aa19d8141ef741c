// m2_host.hpp -- host-side tables and state conversion for the GB300 engine.
//
// Exponent -> transform size, digit widths and IBDWT shift weights follow the
// reference definitions (mersenne2_gpu.cpp:286-293, 3921-3944) because they
// define the residue's digit layout, which must be identical for the state to
// be a drop-in.  The transform itself (generator, twiddle tables, step plan)
// is this engine's own; its tables are built on the device (m2_tables.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <string>
#include <vector>

namespace m2 {

using u64 = uint64_t;
using u32 = uint32_t;
using i64 = int64_t;

constexpr u64 P61 = (u64(1) << 61) - 1;
constexpr u32 P31 = (u32(1) << 31) - 1;

// The IBDWT shift lr x modulo m = 61 or 31 (lr < m): the factor x, up to n, is
// reduced first, so that the product fits 32 bits at every n.
constexpr u32 weight_shift(u32 lr, u32 x, u32 m) { return lr * (x % m) % m; }

// Dual-field element as stored in the twiddle tables: GF(P61^2) pair + GF(P31^2) pair.
struct alignas(8) Dual {
    u64 a, b;   // GF(P61^2): a + b i
    u32 c, d;   // GF(P31^2): c + d i
};
static_assert(sizeof(Dual) == 24, "Dual must be 24 bytes");

// Smallest ln >= 3 with ln + 2((p >> ln) + 1) < bound: 92 for the two fields
// (mersenne2_gpu.cpp:286-293), 61 for GF(P61^2) alone
// (gf61_ntt_prp_opencl_inplace_nobitrev_fused.cpp:124-132).
int transform_log2(u64 p, int bound = 92);

struct Layout {
    u32 p = 0;
    int ln = 0;            // log2 n
    u64 n = 0, h = 0;      // real digits, complex elements
    u32 q = 0;             // narrow digit width p >> ln
    // the first min(n, head) digits of these (make_layout):
    std::vector<uint8_t> width;   // n digit widths, q or q+1
    std::vector<u64> bitpos;      // n+1 bit positions ceil(p j / n)
};
Layout make_layout(u32 p, int bound = 92, u64 head = ~u64(0));

// Roots of unity of this engine: g61 of order 2^62 in GF(P61^2) and g31 of
// order 2^32 in GF(P31^2), chosen so that the order-4 root is +i.
Dual root_of_unity(u64 order);       // primitive root of the given power-of-two order

// Bound-driven number of digits through which an incoming segment carry is
// propagated before its remainder is added to the next digit (see the .cpp).
int carry_span(const Layout& L);

// ---- state conversion (exact, host side) ----
// Any n unsigned digit words -> canonical digits of the residue they denote.
std::vector<u64> canonical_from_unsigned(const Layout& L, const u64* d);
// Canonical (or any non-negative) digits -> balanced digits of the same residue.
std::vector<i64> balanced_digits(const Layout& L, const std::vector<u64>& canon);
// Small integer -> canonical digits.
std::vector<u64> digits_of_small(const Layout& L, u64 x);
}  // namespace m2
