// Byte offsets of matrix columns (bie_fix64.cuh) against 128-bit arithmetic:
// prints 1 where all agree.
#include "bie_fix64.cuh"

#include <cstdio>

int main() {
    bool ok = true;
    const long long rows[] = {1, 129, (1LL << 28) - 1, 1LL << 28, (1LL << 28) + 1, 3LL << 29, 0x7fffffffLL};
    const int nodes[] = {0, 1, 2, 17, 40961, 0x7fffffff};
    for (long long m : rows)
        for (int n : nodes) {
            const unsigned __int128 want = (unsigned __int128)16 * (unsigned)n * (unsigned long long)m;
            if (want >> 63) continue;   // (no such buffer)
            ok = ok && bie::fix64::column_bytes(n, m) == (unsigned long long)want;
        }
    std::printf("%d\n", ok ? 1 : 0);
    return 0;
}
