"""Every ctypes struct of zorch_gb300/_lib.py has the size and the field offsets
that a C compiler gives the struct of that name in include/zc.h."""

from __future__ import annotations

import ctypes
import re
import shutil
import subprocess
from pathlib import Path

import pytest

from zorch_gb300 import _lib

ROOT = Path(__file__).resolve().parent.parent
STRUCTS = {"zc_leaves": _lib.Leaves, "zc_lde_job": _lib.LdeJob, "zc_merkle_job": _lib.MerkleJob,
           "zc_fold_rounds_desc": _lib.FoldRoundsDesc, "zc_open_job": _lib.OpenJob}


def test_every_struct_is_compared():
    mirrors = {c for c in vars(_lib).values()
               if isinstance(c, type) and issubclass(c, ctypes.Structure)}
    assert mirrors == set(STRUCTS.values())
    header = re.sub(r"/\*.*?\*/", "", (ROOT / "include" / "zc.h").read_text(), flags=re.S)
    assert set(re.findall(r"\}\s*(zc_\w+)\s*;", header)) - {"zc_status", "zc_field"} == set(STRUCTS)


def test_layouts(tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        pytest.skip("no C compiler")
    lines = ["#include <stdio.h>", "#include <stddef.h>", '#include "zc.h"', "int main(void) {"]
    for c, py in STRUCTS.items():
        lines.append(f'  printf("{c} size %zu 0\\n", sizeof({c}));')
        for name, _ in py._fields_:
            lines.append(f'  printf("{c} {name} %zu %zu\\n", offsetof({c}, {name}), '
                         f"sizeof((({c}*)0)->{name}));")
    src = tmp_path / "layout.c"
    src.write_text("\n".join(lines + ["  return 0;", "}"]) + "\n")
    exe = tmp_path / "layout"
    subprocess.run([cc, "-std=c11", "-I", str(ROOT / "include"), str(src), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    got = {(c, f): (int(o), int(s)) for c, f, o, s in (line.split() for line in out.splitlines())}
    for c, py in STRUCTS.items():
        assert got[c, "size"][0] == ctypes.sizeof(py), c
        for name, _ in py._fields_:
            field = getattr(py, name)
            assert got[c, name] == (field.offset, field.size), (c, name)
