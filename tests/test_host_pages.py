"""Outputs that a call maps before its result is known keep their contents
(host_pages.hpp, compiled here)."""
import os
import shutil
import subprocess

import pytest

from helpers import ROOT

SOURCE = r"""
#include <cstdlib>
#include <vector>
#include "host_pages.hpp"
int main()
{
	for (size_t n : {(size_t)0, (size_t)1, (size_t)4095, (size_t)4096, (size_t)4097, (size_t)100000})
		for (size_t off : {0, 1, 63}) {
			std::vector<char> v(n + off + 64);
			for (size_t i = 0; i < v.size(); i++) v[i] = (char)(i * 131 + 7);
			const std::vector<char> was = v;
			bm4dof::touch_pages(v.data() + off, n);
			if (v != was) return 1;
		}
	// pages that do not exist yet read as zeros afterwards
	const size_t n = 64 << 20;
	char *p = static_cast<char *>(std::calloc(n, 1));
	bm4dof::touch_pages(p, n);
	for (size_t i = 0; i < n; i++)
		if (p[i]) return 2;
	std::free(p);
	return 0;
}
"""


def test_touched_pages_keep_their_contents(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "t.cpp").write_text(SOURCE)
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "bm4d-of_gb300", "csrc"), str(tmp_path / "t.cpp"),
                    "-o", str(tmp_path / "t")], check=True)
    assert subprocess.run([str(tmp_path / "t")]).returncode == 0
