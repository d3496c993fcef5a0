"""Rows that the decode attention copies from the caches (ops/csrc/tile_rows.h): every valid one but the one being written."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "create_llm_by_cupy_b200" / "ops" / "csrc"

PROGRAM = r"""
#include <cassert>
#include <initializer_list>
#include "tile_rows.h"

int main() {
  for (int tile : {1, 8, 32})
    for (int len = 1; len <= 100; ++len)
      for (int pos = -1; pos <= 101; ++pos) {
        int copied[200] = {};
        for (int key0 = 0; key0 < len; key0 += tile) {
          const b200::TileRows r = b200::tile_rows(key0, tile, len, pos);
          assert(r.first >= 0 && r.rest >= 0 && r.first + (r.rest > 0 ? 1 + r.rest : 0) <= tile);
          for (int i = 0; i < r.first; ++i) ++copied[key0 + i];
          for (int i = 0; i < r.rest; ++i) ++copied[key0 + r.first + 1 + i];
        }
        for (int k = 0; k < 200; ++k) assert(copied[k] == (k < len && k != pos));
      }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_every_valid_row_but_the_new_one(tmp_path):
    src, exe = tmp_path / "rows.cpp", tmp_path / "rows"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-UNDEBUG", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)


def test_every_copy_goes_by_them():
    text = re.sub(r"//[^\n]*", "", (CSRC / "decode.cu").read_text())
    kernel = text[text.index("decode_attn_kernel("):].split("\n}\n", 1)[0]
    fetch = kernel[kernel.index("auto fetch"):]
    fetch = fetch[:fetch.index("\n  };")]
    assert "tile_rows(t * DA_TILE, DA_TILE, len, APPEND ? p.pos : -1)" in fetch
    assert kernel.count("bulk_load(") == fetch.count("bulk_load(") == 2
    for call in re.findall(r"bulk_load\(.*?\);", fetch, re.S):
        assert re.search(r"rows\.(first|rest)\) \* D \* 2, bar\)", call), call
