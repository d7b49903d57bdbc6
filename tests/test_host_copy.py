"""The copies of fields and state to the host (csrc/host_copy.cpp) against stand-ins for the CUDA calls, without a GPU: the
bytes of every size and number of threads; a kernel whose steps are still queued does not hold up the read-out of another;
pinned memory, streams or copies that fail."""
import os
import subprocess

from lbm_b200 import abi

TESTS = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(TESTS)


def test_host_copy(tmp_path):
    program = str(tmp_path/'host_copy')
    cuda = os.environ.get('CUDA_HOME', '/usr/local/cuda')
    source = os.path.join(os.path.dirname(abi.__file__), 'csrc')
    subprocess.run(['g++', '-std=c++17', '-O1', '-pthread', '-I' + os.path.join(ROOT, 'include'), '-I' + source,
                    '-I' + os.path.join(cuda, 'include'), os.path.join(TESTS, 'host_copy_fakes.cpp'),
                    os.path.join(source, 'host_copy.cpp'), '-o', program], check=True)
    run = subprocess.run([program], timeout=120, capture_output=True, text=True)
    assert run.returncode == 0, run.stdout + run.stderr
