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


def test_a_descriptor_is_an_ordinary_python_object(aclnn):
    """Attributes, weak references, subclasses that calls take, cycles that are collected: what a class written in Python has."""
    import gc
    import weakref

    import torch

    backing = torch.zeros(2, 3, dtype=torch.int8)
    t = aclnn.from_torch(backing)
    t.layer = "up"
    assert t.layer == "up" and t.__dict__ == {"layer": "up"} and weakref.ref(t)() is t

    class Named(aclnn.Tensor):
        def __init__(self, *args, **kwargs):
            self.name = "w"

    n = Named((2, 3), "int8", backing)
    assert isinstance(n, aclnn.Tensor) and n.name == "w" and n.shape == (2, 3) and n.handle
    with pytest.raises(aclnn.AclnnError):  # refused for its dtypes, not for its class
        aclnn.quant_matmul_v5(n, n, None, None, n)

    t.itself = n.other = t
    seen = weakref.ref(t)
    del t, n
    gc.collect()
    assert seen() is None


def test_strides_as_the_former_class_took_them(aclnn):
    assert aclnn.Tensor((2, 3), "int8", 0, (1,)).shape == (2, 3)  # what is missing is 0
    with pytest.raises(IndexError):
        aclnn.Tensor((2, 3), "int8", 0, (3, 1, 1))
