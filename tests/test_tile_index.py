"""Offsets within a group of tiles, compiled for the host from the header that the warp kernel uses."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mask_b200", "csrc")


def test_ids_of_the_last_tiles_of_a_long_group(tmp_path):
    """2^28 tiles are 2^31 ids: their offsets do not fit int32, whatever type the tile's number has where it is used."""
    source, program = tmp_path / "offsets.cpp", tmp_path / "offsets"
    source.write_text("""#include <cinttypes>
#include <cstdio>
#include "tile_index.h"
int main() {
    const uint32_t tiles[] = {0, 1, (1u << 28) - 1, 1u << 28, (1u << 28) + 5, (1u << 31) - 1, (1u << 31) + 40};
    for (uint32_t t : tiles) printf("%" PRIu32 " %" PRId64 "\\n", t, mask::ids_before_tile(t));
}
""")
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, "-o", str(program), str(source)], check=True)
    lines = subprocess.run([str(program)], check=True, capture_output=True, text=True).stdout.split("\n")[:-1]
    assert len(lines) == 7
    for line in lines:
        tile, offset = map(int, line.split())
        assert offset == 8 * tile
