// Asks recipe_dev_b200/csrc/rq_ring_rule.cuh: lines "type sm_count rows cols tokens" in, "stages block_values block_bytes" out. Built and run by tests/test_ring_rule.py.
#include <cstdio>

#include "rq_ring_rule.cuh"

int main() {
    int type, sms, tokens;
    long long rows, cols;
    while (std::scanf("%d %d %lld %lld %d", &type, &sms, &rows, &cols, &tokens) == 5)
        std::printf("%d %d %d\n", rqring::stages(type, sms, rows, cols, tokens), rqring::block_values(type), rqring::block_bytes(type));
    return 0;
}
