"""The check of a claimed task record, on the CPU: what would index out of a
table, the board or the path is refused, everything else is taken."""
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG

PROGRAM = r"""
#include <stdio.h>
#include <string.h>
#include "sp_defs.h"
int main() {
  int w, plen;
  unsigned char b[28];
  while (scanf("%d %d", &w, &plen) == 2) {
    for (int i = 0; i < 28; ++i) {
      unsigned v;
      if (scanf("%u", &v) != 1) return 1;
      b[i] = (unsigned char)v;
    }
    uint32_t word[7];
    memcpy(word, b, 28);
    putchar(sp::record_ok(w, word, plen) ? '1' : '0');
  }
  return 0;
}
"""


@pytest.mark.parametrize("width", [4, 5])
def test_records(tmp_path, width):
    src, exe = tmp_path / "records.cpp", tmp_path / "records"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(PKG, "csrc"), str(src), "-o", str(exe)], check=True)
    n = width * width
    rng = np.random.default_rng(width)
    rows, want = [], []

    def add(board, blank, plen):
        cells = np.zeros(28, np.int64)
        cells[:n] = board
        cells[25], cells[26], cells[27] = blank, rng.integers(0, 256), rng.integers(0, 16)
        rows.append("%d %d %s" % (width, plen, " ".join(map(str, cells))))
        want.append(all(t < n for t in board) and blank < n and plen <= 160)

    for _ in range(200):  # boards of the search; the blank's own byte may hold any tile
        board = rng.permutation(n)
        blank = int(np.argmin(board))
        board[blank] = rng.integers(0, n)
        add(board, blank, int(rng.integers(0, 161)))
        assert want[-1]
    for cell in range(n):  # one bad byte anywhere
        for tile in (n - 1, n, n + 1, 31, 32, 127, 128, 200, 255):
            board = rng.permutation(n)
            board[cell] = tile
            add(board, 0, 0)
    for blank in (n - 1, n, 127, 128, 255):
        add(rng.permutation(n), blank, 0)
    for plen in (0, 1, 159, 160, 161, 255):
        add(rng.permutation(n), 0, plen)
    out = subprocess.run([str(exe)], input="\n".join(rows), capture_output=True, text=True, check=True).stdout
    assert [c == "1" for c in out] == want
