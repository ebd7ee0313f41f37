"""Launch facts that differ by device (grid sizes, the opt-in to large shared
memory): one entry per device, safe from several threads."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, 'vision_b200', 'csrc')
CUDA_INCLUDE = os.path.join(os.environ.get('CUDA_HOME', '/usr/local/cuda'), 'include')


def test_two_devices_and_several_threads(tmp_path):
    # Against a runtime of two devices that the program itself stands in for.
    if not os.path.exists(os.path.join(CUDA_INCLUDE, 'cuda_runtime.h')):
        pytest.skip('no CUDA headers')
    exe = str(tmp_path / 'resident_devices')
    subprocess.run(['g++', '-std=c++17', '-O1', '-pthread', '-I', CSRC, '-I', CUDA_INCLUDE,
                    os.path.join(ROOT, 'tests', 'cpp', 'resident_devices.cpp'), '-o', exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == 'ok', r.stdout


def test_no_process_wide_launch_facts():
    # A plain static in a launch function holds one device's value for all of
    # them, and is written by every thread.
    found = []
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(('.cu', '.cuh', '.h')):
            for k, line in enumerate(open(os.path.join(CSRC, name)), 1):
                if re.match(r'\s+static (bool|int|unsigned|uint32_t|size_t) \w+', line) and '(' not in line:
                    found.append('%s:%d: %s' % (name, k, line.strip()))
    assert not found
