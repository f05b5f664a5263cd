"""Builds tests/kernels/_build/<name> (test infrastructure: kernel-level checks of the
tensor-core contractions)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(os.path.dirname(HERE))
CSRC = os.path.join(ROOT, "cc4s_b200", "csrc")


def build(name="split_check"):
    OUT = os.path.join(HERE, "_build", name)
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    parts = ("ops_cuda.cu",) if name == "stage_check" else ("split_gemm.cu", "gemm_f64.cu")
    srcs = [os.path.join(HERE, name + ".cu")] + [os.path.join(CSRC, p) for p in parts]
    deps = srcs + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    if os.path.exists(OUT) and os.path.getmtime(OUT) > max(os.path.getmtime(d) for d in deps):
        return OUT
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-lineinfo", "-o", OUT] + srcs + ["-lcuda"], check=True)
    return OUT


if __name__ == "__main__":
    print(build())
