"""Small pieces of the launch path's host code, compiled by themselves and run without a GPU."""
import subprocess
from pathlib import Path

from orinmllm_b200 import build as b

CPP = Path(__file__).resolve().parent / "cpp"


def test_a_refused_launch_leaves_no_error_behind(tmp_path):
    exe = tmp_path / "launch_error"
    subprocess.run([b._nvcc(), *b.NVCC_FLAGS, "-o", exe, CPP / "test_launch_error.cu", "-Xlinker",
                    "--wrap=cudaLaunchKernelExC", "-Xlinker", "--wrap=cudaGetLastError"], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout


def test_a_device_value_is_worked_out_once(tmp_path):
    exe = tmp_path / "per_device"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", b.CSRC, "-o", exe, CPP / "test_per_device.cpp"], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout


def test_narrow_cluster_forms_share_an_sm(tmp_path):
    exe = tmp_path / "cluster_forms"
    subprocess.run([b._nvcc(), *b.NVCC_FLAGS, "-o", exe, CPP / "test_cluster_forms.cu", "-lcuda"], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout


def test_prefill_work_lists(tmp_path):
    exe = tmp_path / "prefill_plan"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", b.CSRC, "-o", exe, CPP / "test_prefill_plan.cpp"], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout


def test_form_of_the_rope_kernel(tmp_path):
    exe = tmp_path / "rope_form"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", b.CSRC, "-o", exe, CPP / "test_rope_form.cpp"], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
