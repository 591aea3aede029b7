// Host build of the packed df64 operations (df64.cuh's df2): each lane of each
// operation against the scalar df64 operation on the same values.
#include <cstdint>
#include <cstring>

#include "df64.cuh"

using namespace ddd;

static bool same(df64 a, df64 b) { return !std::memcmp(&a.hi, &b.hi, 4) && !std::memcmp(&a.lo, &b.lo, 4); }

// v: 4 doubles per case (two operands for each lane); bad[op] counts lanes that
// differ: + - * / recip sqrt log atan, then + - * with a float second operand.
extern "C" void df2_compare(const double* v, int64_t n, int64_t* bad) {
  for (int64_t i = 0; i < n; ++i) {
    const df64 a = df_from_double(v[4 * i]), b = df_from_double(v[4 * i + 1]);
    const df64 c = df_from_double(v[4 * i + 2]), d = df_from_double(v[4 * i + 3]);
    const df64 pa = a.hi < 0.0f ? -a : a, pc = c.hi < 0.0f ? -c : c;
    const df2 P = df2_make(a, c), Q = df2_make(b, d), PP = df2_make(pa, pc);
    auto check = [&](int op, df2 r, df64 x, df64 y) { bad[op] += !same(df2_x(r), x) + !same(df2_y(r), y); };
    check(0, P + Q, a + b, c + d);
    check(1, P - Q, a - b, c - d);
    check(2, P * Q, a * b, c * d);
    check(3, P / Q, a / b, c / d);
    check(4, df_recip(P), df_recip(a), df_recip(c));
    check(5, df_sqrt(PP), df_sqrt(pa), df_sqrt(pc));
    check(6, df_log(PP), df_log(pa), df_log(pc));
    check(7, df_atan(P), df_atan(a), df_atan(c));
    check(8, P + Q.hi, a + b.hi, c + d.hi);
    check(9, P - Q.hi, a - b.hi, c - d.hi);
    check(10, P * Q.hi, a * b.hi, c * d.hi);
  }
}
