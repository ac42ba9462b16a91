// Host-only harness for the chunked decoder's symbol tables (build_sym,
// mmrecode_gb300/csrc/huffman_lut.h): looks every 16-bit window up as the kernels do.
#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "huffman_lut.h"

// key: 16 counts then the symbols (a DHT table body). sym and skip: 65536 entries each,
// of the windows p << 16; meta: entries, first_long, last, whether the table may be read
// without clamping the window, and the largest entry any window then indexes. `before` entries precede the
// table, as in a batch of several.
extern "C" void mmr_test_sym(const uint8_t *key, size_t key_len, int ac, size_t before, uint16_t *sym, uint32_t *skip,
                             uint32_t *meta) {
    std::vector<uint16_t> s(before, 0xabcd);
    const mmr::LutMeta m = mmr::build_sym(key, key_len, ac != 0, &s);
    std::vector<uint32_t> k(m.off + m.len);
    for (uint32_t x = 0; x < m.len; x++) k[m.off + x] = mmr::skip_entry_of(s.data() + m.off, m.first_long, x);
    for (uint32_t p = 0; p < 65536; p++) {
        const uint32_t at = m.off + mmr::lut_entry_index(std::min(p << 16, m.last), m.first_long);
        sym[p] = at < s.size() ? s[at] : 0xffff;
        skip[p] = at < k.size() ? k[at] : 0xffffffffu;
    }
    meta[0] = m.len;
    meta[1] = m.first_long;
    meta[2] = m.last;
    meta[3] = mmr::lut_fits_shared(m);
    meta[4] = 0;
    for (uint32_t p = 0; p < 65536; p++) meta[4] = std::max(meta[4], mmr::lut_entry_index(p << 16 | 0xffffu, m.first_long));
}
