"""The drawn signs of a transform against the matrix they stand for."""
import pytest
import torch

from alto_b200 import hadamard as H


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("size", [16, 32, 64])
def test_signs_and_matrix_agree(size, dtype):
    state = {k: getattr(H.HadamardFactory, k) for k in ("block_size", "randomized", "dtype", "seed")}
    generator = H.HadamardFactory.generator.get_state()
    try:
        H.HadamardFactory.configure(block_size=size, randomized=True, dtype=dtype, seed=11)
        drawn = H.HadamardFactory.create_transform("cpu")
        after = H.HadamardFactory.generator.get_state()
        gen = torch.Generator().manual_seed(11)
        weight = H.random_hadamard_matrix(size, dtype, "cpu", gen)
        perm = torch.randperm(size, generator=gen)
        assert torch.equal(gen.get_state(), after) and torch.equal(perm, drawn.perm)
        plain = H.HadamardTransform(weight, perm)
        assert drawn.n == plain.n == size and drawn.is_fused == plain.is_fused == (size == 16)
        if drawn.is_fused:
            a, b = drawn.device_params(), plain.device_params()
            assert (a.n, a.perm, a.sign) == (b.n, b.perm, b.sign) and all(isinstance(v, int) for v in a.sign)
        assert torch.equal(drawn.weight, weight) and drawn.weight.dtype == dtype
        assert torch.equal(drawn.matrix(), plain.matrix())
        again = H.HadamardTransform(None, perm, torch.ones(size))
        for t in (drawn, again):                       # a matrix put in by hand counts, whatever was derived before
            t.device_matrix("cpu")
            t.weight = torch.ones(size, size)
            assert not t.is_fused and t.n == size and torch.equal(t.matrix(), torch.ones(size, size))
            assert torch.equal(t.device_matrix("cpu"), torch.ones(size, size))
            t.weight = weight
            assert t.is_fused == (size == 16) and torch.equal(t.device_matrix("cpu"), plain.device_matrix("cpu"))
            if size == 16:
                assert t.device_params().sign == plain.device_params().sign
            t.weight = torch.ones(2, 2)
            assert t.n == 2
    finally:
        for k, v in state.items():
            setattr(H.HadamardFactory, k, v)
        H.HadamardFactory.generator.set_state(generator)


def test_sizes_that_cannot_be_built_are_refused_when_drawn():
    state = H.HadamardFactory.block_size
    try:
        H.HadamardFactory.configure(block_size=6, randomized=True)
        with pytest.raises(ValueError):
            H.HadamardFactory.create_transform("cpu")
    finally:
        H.HadamardFactory.block_size = state


def test_a_factory_of_its_own_is_asked_for_both_parts(monkeypatch):
    generator = H.HadamardFactory.generator.get_state()

    class Sorted(H.HadamardFactory):
        block_size, randomized = 16, True

        @classmethod
        def _create_permutation(cls, weight):
            assert weight.shape == (16, 16)            # the matrix, whose rows it may look at
            return torch.argsort(weight[:, 0], stable=True)

    class Negated(H.HadamardFactory):
        block_size, randomized = 16, True

        @classmethod
        def _create_weight(cls, device):
            return -H.deterministic_hadamard_matrix(16)

    try:
        drawn = Sorted.create_transform("cpu")
        assert torch.equal(drawn.perm, torch.argsort(drawn.weight[:, 0], stable=True))
        assert torch.equal(Negated.create_transform("cpu").weight, -H.deterministic_hadamard_matrix(16))
        monkeypatch.setattr(H.HadamardFactory, "block_size", 16)
        monkeypatch.setattr(H.HadamardFactory, "_create_weight", lambda device: torch.ones(16, 16))
        assert torch.equal(H.HadamardFactory.create_transform("cpu").weight, torch.ones(16, 16))
    finally:
        H.HadamardFactory.generator.set_state(generator)


def test_a_transform_with_a_call_of_its_own_is_called():
    from alto_b200 import _lib as L
    from alto_b200 import _linear as E

    class Rows:                                        # what a bf16 matrix on a GPU answers
        dtype, shape, device, is_cuda = torch.bfloat16, (64, 128), torch.device("cpu"), True
        dim = lambda self: 2
        stride = lambda self, axis: (128, 1)[axis]
        data_ptr = lambda self: 0

    class Halved(H.HadamardTransform):
        def __call__(self, value, **options):
            return super().__call__(value, **options) / 2

    class Other:                                       # no matrix to ask for
        is_fused = False
        __call__ = lambda self, value, left_mul: value

    weight = H.deterministic_hadamard_matrix(32)
    ask = lambda transform: E.dense_in_quantizer(Rows(), transform, L.FMT_MXFP4, E.RTN)
    assert torch.equal(ask(H.HadamardTransform(weight, None)), weight)
    assert ask(Halved(weight, None)) is None and ask(Other()) is None
