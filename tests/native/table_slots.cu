// Host check of the sizes of global hash tables: prints the slots for the key
// counts given on the command line.
#include <cstdio>
#include <cstdlib>
#include "common.cuh"

int main(int argc, char** argv) {
    for (int i = 1; i < argc; i++) printf("%lld\n", (long long)pggc::global_table_slots(atoll(argv[i])));
    return 0;
}
