// Test build of host-callable rules of the entropy stage (falcons_b200/csrc), for tests/test_entropy_rules.py.
// Test infrastructure; the product never loads it.
#include "../../falcons_b200/csrc/entropy_rules.cuh"

extern "C" {
int rules_range_within(unsigned long long first, unsigned long long count, unsigned long long n) {
    return fb2::range_within(first, count, n);
}

unsigned long long rules_chain_part_count(unsigned long long n, unsigned long long part) {
    return fb2::chain_part_count(n, part);
}
}
