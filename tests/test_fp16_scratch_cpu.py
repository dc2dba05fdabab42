"""The FP16 launcher reads the registered scratch once per call: what its plan was made for is what the kernel gets."""
import subprocess
from pathlib import Path

from llmmm_b200 import build

HERE = Path(__file__).resolve().parent


def test_scratch_changed_by_another_thread_during_the_call(tmp_path):
    src, obj = build.CSRC / "fp16_mm.cu", build.OBJ / "fp16_mm.o"
    headers = [*build.CSRC.glob("*.h"), *build.CSRC.glob("*.cuh"), build.PKG.parent / "include" / "llmmm_c.h"]
    if not build._newer(obj, [src, *headers]):
        obj = tmp_path / "fp16_mm.o"
        subprocess.run([build.NVCC, *build.FLAGS, "-c", str(src), "-o", str(obj)], check=True, capture_output=True)
    exe = tmp_path / "fp16_scratch_lookup"
    cuda_include = Path(build.NVCC).resolve().parent.parent / "include"
    r = subprocess.run(["g++", "-O1", "-std=c++17", f"-I{cuda_include}", "-o", str(exe), str(HERE / "cpp" / "fp16_scratch_lookup.cc"), str(obj)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
