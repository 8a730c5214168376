"""Libraries that are loaded with their first use: no thread may see one whose functions do not yet know their argument types
(ctypes would pass 64-bit addresses as 32-bit integers).  No device needed."""
import pytest

from torchless_rs_b200.csrc import attention_f32, build, gemm_f32


@pytest.mark.parametrize("make", [gemm_f32.GemmF32, attention_f32.AttentionF32])
def test_a_library_is_seen_only_when_its_functions_know_their_types(make, monkeypatch):
    user, early, declared = make(), [], []

    class Function:
        def __setattr__(self, name, value):
            early.append(user.lib is not None)
            declared.append(name)

    class Library:
        def __getattr__(self, name):
            return Function()

    monkeypatch.setattr(build, "load_library", lambda name: Library())
    monkeypatch.setattr(gemm_f32, "register_error_word", lambda *a: None)
    user._load()
    assert "argtypes" in declared and not any(early)
    assert isinstance(user.lib, Library)


def test_error_words_are_read_while_another_library_is_loaded(monkeypatch):
    """A library that another thread loads registers its error word while this one reads those that are there."""
    from torchless_rs_b200.csrc import ops
    words = {}
    monkeypatch.setattr(ops, "_error_words", words)

    def take():
        ops.register_error_word("late", lambda: 0)
        return 0
    words["early"] = take
    ops.check_kernel_errors()
    assert set(words) == {"early", "late"}
    words["late"] = lambda: 3
    with pytest.raises(ops.KernelError, match="late: code 3"):
        ops.check_kernel_errors()
