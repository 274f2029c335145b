"""The allocation-free residual norm after calls that overlapped: two streams
of calls on worlds of other sizes (other grids) may spoil one another's
results, never those of the calls after them, direct or captured."""
import ctypes as C

import numpy as np
import pytest

from worldinagrain_b200 import abi

pytestmark = pytest.mark.gpu

SIZES = [(64, 64), (1024, 1024), (513, 777)]


class _State:
    """A world's field, blocks and cg as the norm reads them: every cell
    liquid, every block worked on, random residuals."""

    def __init__(self, width, height, seed):
        import torch
        from .test_zz_no_alloc import _entry
        self.fluid, self.f = _entry()
        self.d = abi.WorldDesc(width, height, 4, 0)
        c, b = width * height, ((width + 7) // 8) * ((height + 7) // 8)
        r = np.random.default_rng(seed).standard_normal(c).astype(np.float32)
        self.field = torch.ones(8 * c, dtype=torch.float32, device="cuda")
        self.blocks = torch.ones(5 * b + 9, dtype=torch.int32, device="cuda")
        cg = np.zeros((c, 4), dtype=np.float32)
        cg[:, 1] = r
        self.cg = torch.from_numpy(cg).cuda()
        self.want = float(np.sum(r.astype(np.float64) ** 2))
        self.out = torch.full((1,), -1.0, dtype=torch.float64, device="cuda")

    def call(self, stream):
        p = C.c_void_p
        rc = self.f(C.byref(self.d), p(self.field.data_ptr()), p(self.blocks.data_ptr()), p(self.cg.data_ptr()),
                    p(self.out.data_ptr()), p(stream.cuda_stream))
        assert rc == 0, self.fluid.lib().wig_fluid_last_error()

    def check(self):
        import torch
        torch.cuda.synchronize()
        got = float(self.out.item())
        # the two sums' orders differ: an FP64 sum of n terms of one sign
        # is within n 2^-53 of its value in any order
        assert abs(got - self.want) <= 1.0e-9 * self.want, (got, self.want)
        self.out.fill_(-1.0)


def test_calls_after_overlapping_ones_are_sound():
    import torch
    states = [_State(w, h, k) for k, (w, h) in enumerate(SIZES)]
    streams = [torch.cuda.Stream() for _ in states]
    torch.cuda.synchronize()
    for s, st in zip(streams, states):
        s.wait_stream(torch.cuda.current_stream())
        st.call(s)
        st.check()
    # each captured with its own stream's calls around it
    graphs = []
    for s, st in zip(streams, states):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            st.call(s)
        graphs.append(g)
    for _ in range(50):
        for s, st in zip(streams, states):
            for _ in range(5):
                st.call(s)
    torch.cuda.synchronize()
    for st in states:
        st.out.fill_(-1.0)
    for _ in range(3):
        for s, st, g in zip(streams, states, graphs):
            torch.cuda.synchronize()
            st.call(s)
            st.check()
            torch.cuda.synchronize()
            with torch.cuda.stream(s):
                g.replay()
            st.check()
    # overlapping replays too
    for _ in range(50):
        for s, g in zip(streams, graphs):
            with torch.cuda.stream(s):
                g.replay()
    torch.cuda.synchronize()
    for s, st, g in zip(streams, states, graphs):
        st.out.fill_(-1.0)
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            g.replay()
        st.check()
        st.call(s)
        st.check()
