"""The combine grid releases its dependents behind its own wait, read off the kernel's source: a grid that may start from there
on then finds the attention grid's results complete, ahead of its own wait too."""
from test_kernel_ordering import body


def test_combine_releases_its_dependents_behind_its_wait():
    b = body("mxdsa_lib.cu", "mxdsa_combine_kernel")
    assert b.count("grid_dependency_wait()") == 1 and b.count("grid_launch_dependents()") == 1
    assert b.index("grid_dependency_wait()") < b.index("grid_launch_dependents()")
    assert "return" not in b[: b.index("grid_dependency_wait()")]      # blocks without work wait as well
