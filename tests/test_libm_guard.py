"""The strict table's fingerprint covers everything that was checked when the
table was made: with any of those forms or bounds changed in the headers, the
fingerprint, and with it the refusal of an older table, has to follow."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG_DIR

CSRC = os.path.join(PKG_DIR, "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include <cmath>
#include "exact_libm.h"
#include "libm_file.h"
int main()
{
  const mcg_libm_tab t = MCG_LIBM_TAB_INIT;
  printf("%016llx\n", (unsigned long long)mcg_libm_fingerprint(&t));
}
"""

CHANGES = {  # file, text, replacement
    "none": None,
    "short form, mid": ("exact_libm.h", "MCG_FMA(-u, 1.0f / 720.0f, 1.0f / 120.0f)",
                        "MCG_FMA(-u, 1.0f / 640.0f, 1.0f / 120.0f)"),
    "short form, thin": ("exact_libm.h", "MCG_FMA(-u, 1.0f / 6.0f, 0.5f)", "MCG_FMA(-u, 1.0f / 5.0f, 0.5f)"),
    "residue, mid": ("exact_libm.h", "d = MCG_FMA(-0.5f, e, d);", ""),
    "bound, mid": ("libm_file.h", "1.0 / 2048.0", "1.0 / 4096.0"),
    "bound, thin": ("libm_file.h", "(c + 16.0)", "(c + 1.0)"),
    "range, mid": ("exact_libm.h", "MCG_OM_MID_MAX 0x1p-4f", "MCG_OM_MID_MAX 0x1p-3f"),
}


def _fingerprint(folder, change):
    os.makedirs(folder)
    for f in ("exact_libm.h", "libm_file.h", "libm_tables.inc"):
        shutil.copy(os.path.join(CSRC, f), folder)
    if change:
        path = os.path.join(folder, change[0])
        text = open(path).read()
        assert text.count(change[1]) == 1
        open(path, "w").write(text.replace(change[1], change[2]))
    src = os.path.join(folder, "fp.cpp")
    open(src, "w").write(PROGRAM)
    exe = os.path.join(folder, "fp")
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-I" + str(folder), src, "-o", exe],
                   check=True, capture_output=True, text=True)
    return subprocess.run([exe], check=True, capture_output=True, text=True).stdout.strip()


@pytest.mark.parametrize("what", [k for k in CHANGES if k != "none"])
def test_fingerprint_follows(tmp_path, what):
    assert _fingerprint(str(tmp_path / "a"), CHANGES[what]) != _fingerprint(str(tmp_path / "b"), None)
