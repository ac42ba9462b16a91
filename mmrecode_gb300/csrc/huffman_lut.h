// Host construction of a baseline Huffman table's lookup records (HuffLut, plan.h)
// from its DHT counts and symbols (crates/codecs/mjpeg/src/entropy.rs:18-70 builds
// the same canonical code). Shared by the engine and the table tests.
#pragma once

#include <string.h>

#include <vector>

#include "plan.h"

namespace mmr {

// key: 16 counts then the symbols; sym_off: the table's first symbol in the batch's
// symbol pool.
inline void build_canon(const uint8_t *key, uint32_t sym_off, HuffCanon *c) {
    memset(c, 0, sizeof(*c));
    for (int l = 0; l < 18; l++) c->maxcode[l] = -1;
    uint32_t code = 0, k = 0;
    for (int l = 1; l <= 16; l++, code <<= 1) {
        const uint32_t n = key[l - 1];
        if (n) {
            c->valptr[l] = (int32_t)k - (int32_t)code;
            c->maxcode[l] = (int32_t)(code + n - 1);
        }
        for (uint32_t i = 0; i < n; i++, code++, k++) {
            if (l > 9) continue;
            const uint32_t first = code << (9 - l), cnt = 1u << (9 - l);
            for (uint32_t j = 0; j < cnt; j++)  // the first code of each 9-bit pattern wins
                if (!c->fast[first + j]) c->fast[first + j] = (uint16_t)((l << 8) | key[16 + k]);
        }
    }
    c->sym_off = sym_off;
}

// ac: an AC table (run/size symbols, EOB, ZRL) or a DC one.
inline void build_lut(const uint8_t *key, size_t key_len, uint32_t sym_off, bool ac, HuffLut *lut) {
    memset(lut, 0, sizeof(*lut));
    for (int l = 0; l < 18; l++) lut->maxcode[l] = -1;
    const uint8_t *counts = key;
    const uint8_t *symbols = key + 16;
    constexpr uint32_t FB = kHuffFastBits;
    uint32_t code = 0, k = 0;
    for (int l = 1; l <= 16; l++) {
        uint32_t n = counts[l - 1];
        if (n) {
            lut->valptr[l] = (int32_t)k - (int32_t)code;
            lut->maxcode[l] = (int32_t)(code + n - 1);
        }
        for (uint32_t i = 0; i < n; i++) {
            const uint8_t sym = symbols[k];
            if (l <= 9) {
                uint32_t first = code << (9 - l), cnt = 1u << (9 - l);
                for (uint32_t j = 0; j < cnt; j++)  // the first code of each 9-bit pattern wins
                    if (!lut->fast[first + j]) lut->fast[first + j] = (uint16_t)((l << 8) | sym);
            }
            if ((uint32_t)l <= FB) {
                uint32_t size = 0, adv = 1, eob = 0;
                bool ok;
                if (ac) {
                    size = sym & 15;
                    adv = (sym >> 4) + 1;
                    if (sym == 0x00) eob = kFastEob, adv = 0, ok = true;
                    else if (sym == 0xf0) adv = 16, ok = true;
                    else ok = size >= 1 && size <= 10;
                } else {
                    size = sym;
                    ok = size <= 11;
                }
                if (ok && l + size > FB) {  // the code alone: the magnitude follows it
                    const uint32_t e = (size << 16) | kFastCode | (adv << 5) | (uint32_t)l;
                    const uint32_t base = code << (FB - l);
                    for (uint32_t j = 0; j < (1u << (FB - l)); j++)
                        if (!lut->fastv[base + j]) lut->fastv[base + j] = e;
                }
                if (ok && l + size <= FB) {
                    const uint32_t rest = FB - l - size;  // bits after the magnitude
                    for (uint32_t m = 0; m < (1u << size); m++) {
                        int32_t v = 0;
                        if (size) {
                            v = (int32_t)m;
                            if (v < (1 << (size - 1))) v += 1 - (1 << size);  // receive_extend
                        }
                        const uint32_t e = ((uint32_t)v << 16) | eob | (adv << 5) | (l + size);
                        const uint32_t base = (code << (FB - l)) | (m << rest);
                        for (uint32_t j = 0; j < (1u << rest); j++)
                            if (!lut->fastv[base + j]) lut->fastv[base + j] = e;
                    }
                }
            }
            code++;
            k++;
        }
        code <<= 1;
    }
    // pairs: an AC symbol whose bits leave room for the whole next one
    for (uint32_t x = 0; x < (1u << FB); x++) {
        const uint32_t e1 = lut->fastv[x];
        lut->fastp[x] = e1;
        if (!ac || !e1 || (e1 & (kFastCode | kFastEob))) continue;
        const uint32_t l1 = e1 & 31, adv1 = (e1 >> 5) & 127;
        const int32_t v1 = (int32_t)e1 >> 16;
        if (l1 + 2 > FB || v1 < -64 || v1 > 63) continue;
        const uint32_t e2 = lut->fastv[(x << l1) & ((1u << FB) - 1)];
        if (!e2 || (e2 & kFastCode)) continue;
        const uint32_t l2 = e2 & 31;  // the entry depends only on its first l2 bits
        if (l2 > FB - l1) continue;
        const int32_t v2 = (int32_t)e2 >> 16;
        const uint32_t adv2 = (e2 & kFastEob) ? 0 : (e2 >> 5) & 127;
        if (v2 < -32 || v2 > 31) continue;
        lut->fastp[x] = ((uint32_t)v2 << 26) | (((uint32_t)v1 & 127) << 19) | (adv2 << 14) | kFastPair | (adv1 << 5) |
                        (l1 + l2);
    }
    lut->sym_off = sym_off;
    lut->nsym = (uint32_t)(key_len - 16);
}

// The chunked decoder's lookups of the same table (plan.h), appended to *sym. The table
// is not oversubscribed.
inline LutMeta build_sym(const uint8_t *key, size_t key_len, bool ac, std::vector<uint16_t> *sym) {
    constexpr uint32_t FB = kHuffFastBits;
    const uint8_t *symbols = key + 16;
    LutMeta m;
    m.off = (uint32_t)sym->size();
    m.first_long = m.last = 0xffffffffu;
    uint64_t end = 0;  // of the used code space, left-aligned
    {
        uint64_t code = 0;
        for (uint32_t l = 1; l <= 16; l++, code <<= 1) {
            if (l == FB + 1) m.first_long = (uint32_t)(code << (32 - l) > 0xffffffffull ? 0xffffffffu : code << (32 - l));
            code += key[l - 1];
            if (key[l - 1]) end = code << (32 - l);
        }
    }
    if (end <= m.first_long) m.first_long = 0xffffffffu;  // no long codes
    if (m.first_long != 0xffffffffu && (0x100000000ull - m.first_long) >> 16 > kSharedLong && end <= 0xffffffffull)
        m.last = (uint32_t)end;
    m.len = (lut_entry_index(m.last, m.first_long) + 1 + 7) & ~7u;
    sym->resize(m.off + m.len, 0);
    uint16_t *e = sym->data() + m.off;
    uint32_t code = 0, k = 0;
    for (uint32_t l = 1; l <= 16; l++, code <<= 1) {
        for (uint32_t i = 0; i < key[l - 1] && k < key_len - 16; i++, code++, k++) {
            const uint32_t s = symbols[k], size = ac ? s & 15 : s, run = s >> 4;
            uint32_t adv = ac ? run + 1 : 1;
            if (size > (ac ? 10u : 11u)) continue;
            if (ac && size == 0) {
                if (run != 0 && run != 15) continue;
                if (run == 0) adv = kSymEob;
            }
            const uint16_t entry = (uint16_t)(l | size << 5 | adv << 9);
            if (l <= FB) {
                const uint32_t first = code << (FB - l);
                for (uint32_t j = first; j < first + (1u << (FB - l)) && j < m.len; j++) e[j] = entry;
            } else {  // (its patterns may straddle an 11-bit prefix: one entry further there)
                for (uint32_t j = 0; j < 1u << (16 - l); j++) {
                    const uint32_t at = lut_entry_index((code << (32 - l)) + (j << 16), m.first_long);
                    if (at < m.len) e[at] = entry;
                }
            }
        }
    }
    return m;
}

}  // namespace mmr
