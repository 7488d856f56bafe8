"""The step's upload (csrc/fp_upload.h) never reaches past what the step reserves for it.

The layout's arithmetic is plain C++ without a device: it is compiled here and asked, for every
room and count of simulations around the sizes where the parameters' end is and is not on the
scenes' 256-byte boundary, where the last scene ends and how many bytes are reserved.
"""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "threejs-fire-pro_b200" / "csrc"
PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "fp_upload.h"
int main() {
  for (int room : {1, 2, 3, 31, 256, 511, 512, 513, 517, 600, 1023, 1025, 4099})
    for (int count = 1; count <= room; count = count < 8 || count + 8 >= room ? count + 1 : count + 7)
      for (size_t scene : {(size_t)0, (size_t)256, (size_t)4096, (size_t)1 << 20}) {
        const size_t scenes = fp_upload_scenes(room, count);
        if (scenes % 256 || scenes < fp_upload_params(room) + count * sizeof(SimParams) ||
            scenes + scene > fp_upload_bytes(room, scene)) {
          std::printf("room %d count %d: scenes at %zu end at %zu, reserved %zu\n", room, count, scenes,
                      scenes + scene, fp_upload_bytes(room, scene));
          return 1;
        }
      }
  return 0;
}
"""


def test_upload_ends_within_its_reservation(tmp_path):
    source, program = tmp_path / "layout.cpp", tmp_path / "layout"
    source.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-I", "/usr/local/cuda/include", str(source), "-o",
                    str(program)], check=True)
    r = subprocess.run([str(program)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
