"""The host side of the batches, without a GPU: csrc/vf_batch.cu linked with a CUDA
runtime of host functions (host/batch_host.cu), which runs one scenario a time."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "volumefluxes.jl_gb300" / "csrc"


def compile_driver(out: Path, *flags: str) -> Path:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = Path(nvcc).resolve().parent.parent / "include"
    cc = [nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O1", "-g", f"-I{CSRC}", "-w",
          *(f for flag in flags for f in ("-Xcompiler", flag)), "-c"]
    objs = [out / "batch.o", out / "driver.o", out / "cudart.o"]
    jobs = [subprocess.Popen([*cc, str(CSRC / "vf_batch.cu"), "-o", str(objs[0])]),
            subprocess.Popen([*cc, str(HERE / "host" / "batch_host.cu"), "-o", str(objs[1])]),
            subprocess.Popen(["g++", "-std=c++17", "-O1", "-g", *flags, f"-I{cuda}", "-c", str(HERE / "host" / "fake_cudart.cpp"),
                              "-o", str(objs[2])])]
    assert [j.wait() for j in jobs] == [0, 0, 0]
    exe = out / "driver"
    subprocess.run(["g++", *flags, *map(str, objs), "-o", str(exe), "-pthread"], check=True)
    return exe


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    return compile_driver(tmp_path_factory.mktemp("batch"))


@pytest.mark.parametrize("scenario", ["error", "stall", "capture"])
def test_batch_host(driver, scenario):
    r = subprocess.run([str(driver), scenario], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_feeder_and_launches_share_no_table(tmp_path):
    driver = compile_driver(tmp_path, "-fsanitize=thread")
    r = subprocess.run([str(driver), "slots"], capture_output=True, text=True, timeout=300)
    if "unexpected memory mapping" in r.stderr:
        pytest.skip("the thread sanitizer does not start under this kernel's address layout")
    assert r.returncode == 0 and "data race" not in r.stderr, r.stdout + r.stderr[-6000:]
