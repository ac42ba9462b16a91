"""The chunked decoder's symbol tables (build_sym, mmrecode_gb300/csrc/huffman_lut.h):
the entry the kernels find for every 16-bit window, against a canonical decode of the
same bits (tests/test_huffman_lut.py), for Annex K's tables, seeded random codes and
codes at the limits (none longer than 11 bits, all of one length, one short code and
255 long ones, a complete code, long codes over several 11-bit prefixes)."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import oracle
from test_huffman_lut import codes_of, dht_tables, first_code, random_key

ROOT = Path(__file__).resolve().parents[1]
FB, EOB = 11, 96


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    so = tmp_path_factory.mktemp("sym") / "sym_harness.so"
    subprocess.run([gxx, "-O1", "-shared", "-fPIC", "-std=c++17", f"-I{ROOT / 'mmrecode_gb300' / 'csrc'}",
                    "-o", str(so), str(ROOT / "tests" / "cuda" / "sym_harness.cpp")], check=True)
    lib = ctypes.CDLL(str(so))
    lib.mmr_test_sym.argtypes = [ctypes.c_char_p, ctypes.c_size_t, ctypes.c_int, ctypes.c_size_t] + [ctypes.c_void_p] * 3
    return lib


def symbol(codes, bits, nbits, ac, max_len):
    """(code bits, size, advance) of the symbol at the top of bits, None where there is
    none of at most max_len bits or the reference rejects it."""
    found = first_code(codes, bits, nbits, max_len)
    if found is None:
        return None
    length, s = found
    if not ac:
        return (length, s, 1) if s <= 11 else None
    if s & 15 == 0:
        return (length, 0, EOB if s == 0 else 16) if s in (0x00, 0xF0) else None
    return (length, s & 15, (s >> 4) + 1) if s & 15 <= 10 else None


def check(lib, key, ac, before=0):
    sym, skip, meta = np.zeros(65536, np.uint16), np.zeros(65536, np.uint32), np.zeros(5, np.uint32)
    lib.mmr_test_sym(key, len(key), int(ac), before, sym.ctypes.data, skip.ctypes.data, meta.ctypes.data)
    codes, pairs = codes_of(key), 0
    long_patterns = sum(n << (16 - i) for i, n in enumerate(key[:16], 1) if i > FB)
    assert meta[0] <= (1 << FB) + max(512, long_patterns + 1) + 7
    assert not meta[3] or meta[4] < meta[0] <= 2560  # unclamped windows stay inside a shared table
    for p in range(65536):
        one = symbol(codes, p, 16, ac, 16)
        assert int(sym[p]) == (one[0] | one[1] << 5 | one[2] << 9 if one else 0), (hex(p), one, hex(int(sym[p])))
        if not ac:
            continue
        want = 0
        if one:
            bits, adv = one[0] + one[1], one[2]
            two = None
            if one[0] <= FB and adv != EOB and bits < FB:  # a second code whole within the first 11 bits
                rest = FB - bits
                two = symbol(codes, (p >> 5) & ((1 << rest) - 1), rest, ac, rest)
            pairs += two is not None
            want = adv << 24 | bits << 16 | (adv + (two[2] if two else 0)) << 8 | (bits + (two[0] + two[1] if two else 0))
        assert int(skip[p]) == want, (hex(p), one, hex(int(skip[p])), hex(want))
    return meta, pairs


def test_tables_of_the_encoders_streams(lib):
    rng = np.random.default_rng(12)
    planes = [(32, 32, rng.integers(0, 256, (32, 32), dtype=np.uint8).tobytes())] * 3
    seen, all_pairs = set(), 0
    for annex_k in (True, False):
        for key, ac in dht_tables(oracle.jpeg_encode(4, 32, 32, planes, 75, annex_k=annex_k)):
            if (key, ac) not in seen:
                seen.add((key, ac))
                meta, pairs = check(lib, key, ac, before=8 * len(seen))
                assert meta[3]  # read from shared memory
                all_pairs += pairs
    assert len(seen) >= 4 and all_pairs > 0  # (the reference encoder's own AC codes are all long: no pairs)


@pytest.mark.parametrize("seed", range(4))
def test_random_canonical_codes(lib, seed):
    rng = np.random.default_rng(200 + seed)
    check(lib, random_key(rng, 16, False), False)
    check(lib, random_key(rng, int(rng.integers(20, 160)), True), True)


AC = [0x00, 0xF0] + [(r << 4) | s for r in range(16) for s in range(1, 11)] + [0x0B, 0x10, 0xFF]


@pytest.mark.parametrize("counts", [
    {1: 1},                                  # one code, half the space unused
    {2: 1, 16: 150},                         # one short code, the rest of 16 bits: an incomplete code
    {1: 1, 2: 1, 3: 1, 4: 1, 5: 1, 6: 1, 7: 1, 8: 1, 9: 1, 10: 1, 11: 2},  # complete, none longer than 11 bits
    {1: 1, 2: 1, 3: 1, 4: 1, 5: 1, 6: 1, 7: 1, 8: 1, 9: 1, 10: 1, 11: 1, 12: 1, 13: 1, 14: 1, 15: 1, 16: 2},  # complete
    {12: 160},                               # only long codes, over 80 prefixes
    {16: 160},                               # a few patterns of the whole space
    {11: 3, 12: 5, 13: 7, 14: 9, 15: 11, 16: 13},
    {8: 160},
    {3: 7, 16: 100},                         # long codes up to the end of their prefix
])
def test_codes_at_the_limits(lib, counts):
    n = sum(counts.values())
    key = bytes(counts.get(i, 0) for i in range(1, 17)) + bytes(AC[:n])
    check(lib, key, True, before=16)
