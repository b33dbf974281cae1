"""The rule by which the NVFP4 GEMM takes pairs of SMs (muser_b200/csrc/nvfp4_pairs_rule.h), held on the CPU against times that both
forms took on a B200 (148 SMs, 74 pairs), weights from HBM, launches back to back."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
PLAIN, GROUP, FUSED = range(3)
# (form, weight-row tiles, slabs, tokens, us single, us pairs)
MEASURED = [
    (PLAIN, 4, 4, 1, 4.46, 4.76), (PLAIN, 40, 4, 16, 4.78, 5.81), (PLAIN, 74, 4, 64, 5.95, 7.19), (PLAIN, 74, 4, 128, 6.50, 7.69),
    (PLAIN, 28, 4, 128, 6.38, 5.70), (PLAIN, 8, 4, 256, 6.31, 5.53), (PLAIN, 74, 11, 1, 9.93, 11.36), (PLAIN, 40, 11, 16, 8.22, 8.90),
    (PLAIN, 44, 10, 64, 8.70, 9.73), (PLAIN, 44, 12, 80, 9.89, 10.92), (PLAIN, 28, 11, 128, 9.22, 8.18), (PLAIN, 74, 11, 128, 11.48, 10.19),
    (PLAIN, 40, 20, 16, 11.59, 12.97), (PLAIN, 28, 20, 64, 11.72, 11.07), (PLAIN, 74, 20, 128, 15.88, 13.57), (PLAIN, 74, 47, 16, 24.21, 29.11),
    (PLAIN, 40, 9, 128, 9.35, 8.48), (PLAIN, 20, 20, 2048, 32.3, 27.7), (PLAIN, 20, 108, 2048, 138, 120),
    (FUSED, 4, 4, 1, 7.11, 7.53), (FUSED, 74, 4, 16, 7.44, 9.91), (FUSED, 74, 4, 256, 9.18, 9.98), (FUSED, 16, 20, 16, 13.11, 12.68),
    (FUSED, 40, 20, 16, 14.12, 18.00), (FUSED, 74, 20, 1, 16.48, 19.16), (FUSED, 74, 20, 48, 16.72, 18.61), (FUSED, 74, 20, 128, 16.85, 16.01),
    (FUSED, 74, 12, 300, 17.31, 18.42), (FUSED, 216, 20, 384, 55, 60), (FUSED, 216, 20, 2048, 237, 220),
    (PLAIN, 40, 4, 128, 6.64, 6.29), (PLAIN, 56, 32, 32, 18.37, 16.90), (PLAIN, 54, 32, 48, 18.4, 17.0), (FUSED, 56, 108, 16, 54.59, 49.18),
    (FUSED, 20, 108, 16, 43.7, 38.1), (FUSED, 56, 108, 48, 51.0, 46.3),
    (GROUP, 72, 32, 128, 20.5, 18.7), (GROUP, 52, 20, 128, 13.2, 12.8), (GROUP, 37, 4, 100, 5.51, 5.96), (GROUP, 8, 11, 384, 8.58, 7.72), (GROUP, 37, 12, 384, 9.93, 10.58), (GROUP, 28, 13, 96, 8.78, 8.34),
    (GROUP, 74, 5, 384, 9.41, 10.30), (GROUP, 28, 20, 2048, 37.7, 32.4),
]


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    out = tmp_path_factory.mktemp("rule")
    (out / "rule.cpp").write_text('''#include "muser_b200/csrc/nvfp4_pairs_rule.h"
extern "C" int pays(uint32_t sms, uint32_t room, uint32_t n_tiles, uint32_t tokens, uint32_t slabs, int form) {
    return muser::pairs_pay(sms, room, n_tiles, tokens, slabs, (muser::PairForm)form);
}''')
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{ROOT}", str(out / "rule.cpp"), "-o", str(out / "rule.so")], check=True)
    return C.CDLL(str(out / "rule.so")).pays


@pytest.mark.parametrize("form,tiles,slabs,tokens,single,pairs", MEASURED)
def test_the_faster_form_is_taken(rule, form, tiles, slabs, tokens, single, pairs):
    assert rule(148, 74, tiles, tokens, slabs, form) == (pairs < single)


def test_a_device_without_pairs_takes_none(rule):
    assert not any(rule(148, 0, tiles, tokens, 20, form) for tiles in (1, 40, 200) for tokens in (1, 128, 4096) for form in range(3))
