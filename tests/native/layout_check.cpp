// Reads "model nii njj situations levels" per line and prints 1 where the batch takes the interleaved layout.
#include <cstdio>

#include "batch_rules.h"

int main() {
    int m, ni, nj, n, v;
    while (std::scanf("%d %d %d %d %d", &m, &ni, &nj, &n, &v) == 5) std::printf("%d\n", gral::interleaved_pays(n, ni, nj, v, m));
    return 0;
}
