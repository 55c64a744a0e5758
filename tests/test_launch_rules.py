"""The rules that choose a launch by sizes (csrc/launch_rules.hpp, host code):
compiled on their own and asked at their edges."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CHECKS = {
    # two CTAs of 113 KB fit an SM (228 KB, 1 KB reserved for each); more planes than SMs
    "rhs_plane_threads(196, 148, 2 * 48 * 48 * 16, 233472, 1024)": 256,
    "rhs_plane_threads(148, 148, 2 * 48 * 48 * 16, 233472, 1024)": 512,
    "rhs_plane_threads(169, 148, 115712, 233472, 1024)": 256,
    "rhs_plane_threads(169, 148, 115713, 233472, 1024)": 512,
    "rhs_plane_threads(169, 148, 2 * 65 * 56 * 16, 233472, 1024)": 512,
    "staged_stage_us(false, false, true, 0)": 9,
    "staged_stage_us(false, true, false, 1e5)": 17,
    "staged_stage_us(true, false, true, 0)": 20,
    "staged_stage_us(true, true, true, 0)": 26,
    "staged_stage_us(true, false, false, 0)": 24,
    "(double)ws_ipa_bytes(12, false)": 12 << 20,
    "(double)ws_ipa_bytes(16, false)": 12 << 20,
    "(double)ws_ipa_bytes(15, true)": 12 << 20,
    "(double)ws_ipa_bytes(16, true)": 14 << 20,
    "(double)ws_ipa_bytes(17, true)": 12 << 20,
    "obs_by_thread(1)": 1,
    "obs_by_thread(4)": 1,
    "obs_by_thread(5)": 0,
}


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("rules")
    src = d / "rules.cpp"
    src.write_text('#include <cstdio>\n#include "launch_rules.hpp"\nusing namespace edus;\nint main() {\n'
                   + "".join(f'    std::printf("%.17g\\n", (double)({c}));\n' for c in CHECKS) + "}\n")
    subprocess.run([gxx, "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "edus_2.0_b200", "csrc"), str(src),
                    "-o", str(d / "rules")], check=True)
    out = subprocess.run([str(d / "rules")], check=True, capture_output=True, text=True).stdout.split()
    return dict(zip(CHECKS, map(float, out)))


@pytest.mark.parametrize("call", CHECKS)
def test_rule(rules, call):
    assert rules[call] == CHECKS[call]
