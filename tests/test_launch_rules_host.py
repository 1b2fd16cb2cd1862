"""The launchers' rules on the CPU (csrc/launch_rules.h compiled by itself)."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "cumm-rocm_b200" / "csrc"


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text('#include "launch_rules.h"\n'
                                 'extern "C" int wgrad(int chunks, int groups, int ctas) '
                                 '{ return scb::wgrad_row_splits(chunks, groups, ctas); }\n'
                                 'extern "C" int wide(long long rows, int columns, int sms) '
                                 '{ return scb::simt_wide_columns(rows, columns, sms); }\n'
                                 'extern "C" long long simt_rows(long long rows, int tiles, int sms) '
                                 '{ return scb::simt_wgrad_rows(rows, tiles, sms, 64, 1024); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", str(CSRC), str(d / "rules.cpp"), "-o",
                    str(d / "rules.so")], check=True)
    lib = ctypes.CDLL(str(d / "rules.so"))
    lib.wide.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int]
    lib.simt_rows.argtypes, lib.simt_rows.restype = lib.wide.argtypes, ctypes.c_longlong
    return lib


@pytest.mark.parametrize("ctas", [148, 296, 132, 7])
def test_wgrad_chain_never_longer_than_with_filled_ctas(rules, ctas):
    """A split's chunks are one chain of additions: its length bounds dW's
    error, so rounding the splits must not lengthen it; and the splits leave no
    wave of fewer CTAs than the rounded-up ones would."""
    for groups in list(range(1, 60)) + [108, 147, 148, 149, 200, 296, 297, 700]:
        for chunks in (1, 2, 3, 7, 30, 79, 157, 313, 625, 938, 3125, 40625):
            s = rules.wgrad(chunks, groups, ctas)
            assert 1 <= s <= chunks
            filled = min(-(-ctas // groups), chunks)
            chain = -(-chunks // s)
            assert chain <= -(-chunks // filled), (groups, chunks)
            assert -(-chunks // chain) == s  # no empty split
            waves = lambda n: -(-n * groups // ctas)
            full = -(-chunks // -(-chunks // filled))
            assert waves(s) <= max(waves(full), 2), (groups, chunks)
            assert waves(s) * chain <= waves(full) * -(-chunks // filled), (groups, chunks)


@pytest.mark.parametrize("sms", [148, 132, 20])
def test_simt_rules_follow_the_sm_count(rules, sms):
    """64 columns from two 64-row blocks per SM; about six row ranges' blocks
    per SM between the least and the most rows of a block."""
    assert rules.wide(128 * sms, 33, sms) and not rules.wide(128 * sms - 1, 33, sms)
    assert not rules.wide(128 * sms, 32, sms)
    for tiles in (1, 27, 108):
        for rows in (1, 1000, 20000, 300000, 70000000):
            r = rules.simt_rows(rows, tiles, sms)
            assert r % 64 == 0 and 256 <= r <= 1024
            blocks = -(-rows // r) * tiles
            assert r == 256 or blocks >= 3 * sms
            assert r == 1024 or blocks <= 6 * sms + tiles
