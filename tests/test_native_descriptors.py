"""CPU: descriptors made by the native module (csrc/python/native.cpp). Nothing is launched."""
import pytest


def test_a_descriptor_takes_its_own_copy_of_a_lazily_cloned_tensor(aclnn):
    """A descriptor may be written through; a tensor that still shares its storage with the one it was cloned from must not be."""
    import torch

    for describe in (aclnn.from_torch, lambda t: aclnn.Tensor(t.shape, "float32", t)):
        source = torch.zeros(64)
        clone = torch._lazy_clone(source)
        assert torch._C._is_cow_tensor(clone)
        describe(clone)
        assert not torch._C._is_cow_tensor(clone) and clone.data_ptr() != source.data_ptr()
