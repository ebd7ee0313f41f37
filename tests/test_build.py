"""The build's content digests."""
import importlib.util
import os
import shutil

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _module(path):
    spec = importlib.util.spec_from_file_location('build_copy', path)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_digests_do_not_depend_on_the_folder(tmp_path):
    shutil.copytree(os.path.join(ROOT, 'include'), tmp_path / 'include')
    shutil.copytree(os.path.join(ROOT, 'vision_b200', 'csrc'), tmp_path / 'vision_b200' / 'csrc')
    shutil.copy(os.path.join(ROOT, 'vision_b200', 'build.py'), tmp_path / 'vision_b200' / 'build.py')
    here, there = (_module(os.path.join(str(r), 'vision_b200', 'build.py')) for r in (ROOT, tmp_path))
    assert here._library_digest() == there._library_digest()
    assert [here._source_digest(s) for s in here.SOURCES] == [there._source_digest(s) for s in there.SOURCES]
    with open(tmp_path / 'vision_b200' / 'csrc' / 'vs_math.h', 'a') as f:
        f.write('\n')
    assert here._library_digest() != there._library_digest()
    assert here._source_digest('kernels.cu') != there._source_digest('kernels.cu')
