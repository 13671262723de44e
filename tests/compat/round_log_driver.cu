// Prints round_follows(k, before, k_max, size, alive) for each line of five numbers.
#include <cstdio>

#include "kt_device.cuh"

int main() {
    unsigned k, before, k_max, size, alive;
    while (scanf("%u %u %u %u %u", &k, &before, &k_max, &size, &alive) == 5)
        printf("%d\n", kt::round_follows(k, before, k_max, size, alive));
    return 0;
}
