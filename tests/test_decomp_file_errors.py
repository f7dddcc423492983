"""The .decompCPU writer opens its file once the whole text is on the host: a
copy from the device that fails leaves a file that was there as it was."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include <cstdio>
#include <cstring>
#include "dc_textout.hpp"

// argv: path, bytes of text, whether the copy fails after half of them
int main(int, char** argv) {
    const uint64_t n = strtoull(argv[2], nullptr, 10);
    const bool fails = atoi(argv[3]) != 0;
    const int rc = dc::write_fetched(argv[1], "7\n", 2, n, [&](char* to) {
        memset(to, 'x', fails ? n / 2 : n);
        return fails ? dc::set_error(DC_ERR_CUDA, "copy failed") : DC_OK;
    });
    std::printf("%d %s\n", rc, dc_last_error());
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_failed_copy_leaves_the_file(dc, tmp_path):
    src, exe, out = tmp_path / "t.cpp", tmp_path / "t", tmp_path / "out"
    src.write_text("#include <cstdlib>\n" + DRIVER)
    libdir = os.path.dirname(dc.LIB_PATH)
    subprocess.run(["g++", "-std=c++17", str(src), "-I", os.path.join(libdir, "csrc"), "-L", libdir, "-ldcore_b200",
                    f"-Wl,-rpath,{libdir}", "-o", str(exe)], check=True)

    def write(path, n, fails):
        r = subprocess.run([str(exe), str(path), str(n), str(int(fails))], capture_output=True, text=True, check=True)
        return r.stdout.strip()

    n = 5 << 20
    out.write_bytes(b"as before")
    assert write(out, n, True) == "-2 copy failed"
    assert out.read_bytes() == b"as before"
    assert write(tmp_path / "new", n, True) == "-2 copy failed"
    assert not (tmp_path / "new").exists()
    assert write(out, n, False).startswith("0")
    assert out.read_bytes() == b"7\n" + b"x" * n
    assert write(out, 0, False).startswith("0")
    assert out.read_bytes() == b"7\n"
    assert write(tmp_path / "no" / "such", n, False).startswith("-4 cannot write")
