"""What makes a library that is linked to torch out of date, and under which name the extension module is found."""
import importlib.machinery
import os

import driss_torch_b200 as dt
from driss_torch_b200 import build


def test_rebuilt_for_another_torch_or_python(tmp_path):
    source, header, target, stamp = (tmp_path / n for n in ("a.cpp", "a.h", "a.so", "a.stamp"))
    for p in (source, header, target):
        p.touch()
    os.utime(target, (2e9, 2e9))
    made_for = build.made_for(["g++", "a.cpp"])
    assert build.out_of_date(target, [source, header], stamp, made_for)  # nobody has written for what it was made
    stamp.write_text(made_for)
    assert not build.out_of_date(target, [source, header], stamp, made_for)
    for other in (made_for.replace(build.sysconfig.get_config_var("SOABI"), "cpython-399"), made_for + " -g", made_for.replace("torch ", "torch 9.")):
        assert build.out_of_date(target, [source, header], stamp, other)
    os.utime(header, (2.1e9, 2.1e9))
    assert build.out_of_date(target, [source, header], stamp, made_for)


def test_extension_module_carries_the_python_abi():
    assert dt.direct.__file__.endswith("_direct" + importlib.machinery.EXTENSION_SUFFIXES[0])
    assert not (build.LIB / "_direct.so").exists()  # which any Python would load
