"""Failed CUDA calls while a data set's plans are made (tests/cpp/test_plan_failures.cu: a fake runtime, no GPU)."""
import glob
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
WRAP = ["cudaMalloc", "cudaFree", "cudaMemcpy", "cudaMemcpyAsync", "cudaStreamSynchronize", "cudaGetLastError",
        "cudaLaunchKernel", "__cudaLaunchKernel", "cudaFuncSetAttribute", "cudaOccupancyMaxActiveClusters",
        "cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags", "cudaGetDriverEntryPointByVersion"]


def test_every_failing_call(tmp_path):
    from fiuncho_gb300 import build
    build.build()
    exe = str(tmp_path / "failures")
    subprocess.run([build.nvcc()] + build.NVFLAGS + [os.path.join(ROOT, "tests", "cpp", "test_plan_failures.cu")] +
                   sorted(glob.glob(os.path.join(build.OBJ, "*.o"))) + ["-Xlinker=--wrap=" + f for f in WRAP] +
                   ["-lcudart_static", "-lrt", "-ldl", "-lpthread", "-o", exe], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
