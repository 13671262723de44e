// Prints what kt_list_rule.h decides: lines "most m", "small m cap", "repeat need cap",
// "buffer total limit", "walks m with total local least".
#include <cstdio>
#include <cstring>

#include "kt_list_rule.h"

int main() {
    char op[16];
    unsigned long long a, b = 0;
    while (scanf("%15s %llu", op, &a) == 2) {
        if (!strcmp(op, "most")) {
            printf("%llu\n", (unsigned long long)kt::most_entries(a));
            continue;
        }
        if (scanf("%llu", &b) != 1) return 1;
        unsigned long long c = 0;
        if (!strcmp(op, "walks")) {
            unsigned long long local = 0;
            unsigned least = 0;
            if (scanf("%llu %llu %u", &c, &local, &least) != 3) return 1;
            printf("%d\n", kt::walks_rows(a, b, c, local, least));
            continue;
        }
        if (!strcmp(op, "buffer")) {
            printf("%llu\n", (unsigned long long)kt::buffer_entries(a, b));
            continue;
        }
        printf("%d\n", !strcmp(op, "small") ? kt::small_lists(a, b) : kt::repeat_lists(a, b));
    }
    return 0;
}
