"""The closure's source holds no device function, and no overload of one, that nothing calls."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ark-cpp-mpi_gb300", "csrc")


def test_every_device_function_of_the_closure_is_used():
    with open(os.path.join(CSRC, "ark_closure.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    defined = re.findall(r"__device__ (?:__forceinline__ |__noinline__ )+[\w ]+? (\w+)\(", text)
    assert {"root2", "root3", "features_fp64", "features_of", "sroot6"} <= set(defined)
    for name in set(defined):
        # each definition (overloads too) needs a call beside it
        assert len(re.findall(rf"\b{name}\s*(?:<[^;<>]*>)?\(", text)) > defined.count(name), name
    assert len(defined) == len(set(defined)), [n for n in defined if defined.count(n) > 1]
