"""n and p may each be up to 2^31 - 1.  Tile counts and element places near that
end, on the host: no such V is made on the GPU."""
from __future__ import annotations

import re
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "rust-nmf_b200" / "csrc"
END = 2**31 - 1


def _source(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def test_tile_count(tmp_path):
    """tile_count() as the kernels have it, compiled for the host."""
    text = _source("kernels.cuh")
    at = text.index("__host__ __device__ inline int tile_count(")
    body = text[at:text.index("\n}\n", at) + 3]
    lens = [0, 1, 31, 32, 33, 2**31 - 33, 2**31 - 32, 2**31 - 31, END]
    lines = "".join(f'std::printf("%d %d\\n", tile_count({n}, 32), tile_count({n}, 16));' for n in lens)
    src = tmp_path / "t.cpp"
    src.write_text("#include <cstdio>\n#define __host__\n#define __device__\n" + body +
                   "int main() {" + lines + "}\n")
    exe = tmp_path / "t"
    subprocess.run(["g++", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover", "-o", str(exe),
                    str(src)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert [list(map(int, x.split())) for x in out.splitlines()] == [
        [-(-n // 32), -(-n // 16)] for n in lens]


def test_tiles_are_counted_by_it():
    for name in ("kernels.cuh", "stream.cuh"):
        counts = re.findall(r"const int tiles = ([^;]*);", _source(name))
        assert counts and all(c.startswith("tile_count(") for c in counts), (name, counts)


def test_f32_copy_places():
    """The copy's column is past 32 bits in a block that reaches past p."""
    text = _source("kernels.cuh")
    at = text.index("convert_f64_f32(")
    body = text[at:text.index("\n}\n", at)]
    assert re.search(r"const int64_t j = \(\(int64_t\)blockIdx\.x", body)


def test_csc_tiles_end_within_range():
    """The copy by tiles counts columns in whole tiles."""
    text = _source("sparse.cu")
    cols = int(re.search(r"kCscCols = (\d+);", text).group(1))
    rule = re.search(r"const bool tiles = ([^;]*);", text).group(1)
    assert "p <= INT32_MAX - kCscCols" in rule
    assert -(-(END - cols) // cols) * cols <= END
