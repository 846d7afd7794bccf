"""Host-side parts of the library, compiled by themselves and run on the CPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "tioga_b200", "csrc")


def _run(tmp_path, source, *command):
    exe = str(tmp_path / "check")
    subprocess.run([*command, "-std=c++17", "-I", CSRC, "-o", exe, os.path.join(ROOT, "tests", "host", source)],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr


def test_buffers_go_back_after_the_work_that_reads_them(tmp_path):
    """A buffer that is let go is handed out again only after everything
    queued on the instance's streams, and not while one of them is being
    captured."""
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    _run(tmp_path, "devmem_check.cc", "g++", "-I", os.path.join(cuda, "include"))


def test_kernels_work_on_arrays_of_their_own_device_only(tmp_path):
    """A caller's array that a kernel may not reach (another GPU's, host or
    misaligned memory) is left to copies."""
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    _run(tmp_path, "reach_check.cc", "g++", "-I", os.path.join(cuda, "include"))


def test_donor_slots_refuse_indices_outside_their_arrays(tmp_path):
    """Both kernels that fill the donor slots take their places from here."""
    _run(tmp_path, "donor_slots_check.cu", os.environ.get("NVCC", "nvcc"))


def test_one_page_locked_allocation_per_instance(tmp_path):
    """Each such allocation takes milliseconds: the small buffers and the data
    update's slots share one, and outgrow it safely."""
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    _run(tmp_path, "pinned_check.cc", "g++", "-I", os.path.join(cuda, "include"))
