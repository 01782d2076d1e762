// Test build of host-callable parts of the entropy stage (falcons_b200/csrc), for tests/test_entropy_rules.py and
// tests/test_fse_tables_gpu.py.  Test infrastructure; the product never loads it.
#include "../../falcons_b200/csrc/entropy_rules.cuh"
#include "../../falcons_b200/csrc/fse.cuh"

extern "C" {
unsigned long long rules_chain_part_count(unsigned long long n, unsigned long long part) {
    return fb2::chain_part_count(n, part);
}

// An FSE block of n >= 3 symbols with a table of 2^log cells; `low` marks one-cell symbols as low-probability
// (-1, on the table's top cells).  Returns its size, 0 when the counts fill no such table.
long long rules_fse_block(const uint8_t *src, unsigned long long n, unsigned log, int low, uint8_t *dst,
                          unsigned long long cap) {
    using namespace fb2::fse;
    static BlockScratch w;
    unsigned top = 0;
    for (int s = 0; s < 256; s++) w.count[s] = 0;
    for (unsigned long long i = 0; i < n; i++) {
        w.count[src[i]]++;
        if (src[i] > top) top = src[i];
    }
    if (normalize_count(w.norm, log, w.count, n, top) != log) return 0;
    for (unsigned s = 0; low && s <= top; s++)
        if (w.norm[s] == 1) w.norm[s] = -1;
    const size_t hdr = write_ncount(dst, w.norm, top, log);
    if (!hdr || !build_ctable(w.state_table, w.sym_tt, w.sym, w.norm, top, log)) return 0;
    BitWriter bw;
    bw.init(dst + hdr, cap - hdr);
    uint32_t st[2];
    for (unsigned k = 0; k < 2; k++) {
        const SymTT t = w.sym_tt[src[(n - 1) % 2 == k ? n - 1 : n - 2]];
        const uint32_t nb = (t.deltaNbBits + (1u << 15)) >> 16, v = (nb << 16) - t.deltaNbBits;
        st[k] = w.state_table[(int32_t)(v >> nb) + t.deltaFindState];
    }
    for (unsigned long long i = n - 2; i-- > 0;) {
        uint32_t &x = st[i & 1];
        const SymTT t = w.sym_tt[src[i]];
        const uint32_t nb = (x + t.deltaNbBits) >> 16;
        bw.add(x, nb);
        x = w.state_table[(int32_t)(x >> nb) + t.deltaFindState];
        bw.flush();
    }
    bw.add(st[1], log);
    bw.add(st[0], log);
    bw.flush();
    const size_t body = bw.close();
    return bw.overflow ? 0 : (long long)(hdr + body);
}
}
