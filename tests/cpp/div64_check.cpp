// FP64 division on the integer units (csrc/div64.cuh), host form: quotients
// of the doubles read from stdin (pairs a, b) to stdout.
#include <cstdio>

#include "div64.cuh"

int main() {
  double v[2];
  while (fread(v, sizeof(double), 2, stdin) == 2) {
    const double q = tridi::div64(v[0], tridi::invert64(v[1]));
    double qa, qc, qd;
    tridi::div64x3(v[0], -v[0], 2.0, v[1], qa, qc, qd);
    const double out[4] = {q, qa, qc, qd};
    fwrite(out, sizeof(double), 4, stdout);
  }
  return 0;
}
