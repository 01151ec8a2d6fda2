// Host-only probe of the rule for keeping every state of a forward pass
// (nb::adj_tape_fits in nb_internal.cuh); no device code runs.  Used by
// tests/test_adjoint_memory.py.
//   adj_tape_probe n steps ref limit
#include <cstdio>
#include <cstdlib>

#include "nb_internal.cuh"

int main(int argc, char **argv)
{
    if (argc != 5) return 2;
    printf("%d\n", (int)nb::adj_tape_fits(strtoull(argv[1], nullptr, 10), atoi(argv[2]), atoi(argv[3]) != 0,
                                          strtoull(argv[4], nullptr, 10)));
    return 0;
}
