"""GPU: the tensor-parallel exchange kernels of csrc/comm.cu (`--tensor-parallel-size N`, reference
benchmark-vllm/models.py:11) on ONE GPU.

* tp = 1: b2_comm_allreduce_rms_norm must equal b2_rms_norm with the fused residual add (residual bit for bit), and
  b2_comm_allgather_cols must be a copy.
tp = 2 is not emulated here: the ranks' kernels wait for one another.
The two-process CUDA-IPC path over NVLink is exercised by scripts/tp_check.py / bench.py --gpus N (needs >= 2 GPUs)."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


class Regions:
    """n comm regions on the current device + one b2_comm handle per emulated rank."""

    def __init__(self, n, max_rows, H, grows, gcols):
        from b200attn import _lib
        from b200attn.tp import _device_view
        self.lib, self.n, self.H, self.max_rows = _lib.load(), n, H, max_rows
        lib = self.lib
        nbytes = int(lib.b2_comm_region_bytes(n, max_rows, H, grows, gcols))
        self.ptrs = []
        for _ in range(n):
            p, h = C.c_void_p(), C.create_string_buffer(64)
            _lib.check(lib.b2_comm_alloc(nbytes, C.byref(p), h))
            self.ptrs.append(p.value)
        arr = (C.c_void_p * n)(*self.ptrs)
        self.comms = []
        for r in range(n):
            c = lib.b2_comm_create(r, n, arr, nbytes, max_rows, H, grows, gcols)
            assert c, lib.b2_last_error()
            self.comms.append(c)
        dev = torch.device("cuda", torch.cuda.current_device())
        self.inputs = [[_device_view(lib.b2_comm_input(c, s), max_rows * H * 2, dev).view(torch.bfloat16).view(max_rows, H)
                        for s in (0, 1)] for c in self.comms]
        self.gathered = [_device_view(lib.b2_comm_gathered(c), grows * gcols * 2, dev).view(torch.bfloat16).view(grows, gcols)
                         if grows else None for c in self.comms]

    def allreduce(self, r, slot, out, resid, w, T, eps, stream):
        from b200attn import _lib
        _lib.check(self.lib.b2_comm_allreduce_rms_norm(self.comms[r], slot, out.data_ptr(),
                                                       None if resid is None else resid.data_ptr(),
                                                       None if w is None else w.data_ptr(), T, self.H, self.H, eps,
                                                       stream.cuda_stream))

    def push(self, r, part, out, resid, w, eps, stream):
        from b200attn import _lib
        T = part.shape[0]
        _lib.check(self.lib.b2_comm_push_allreduce_rms_norm(self.comms[r], part.data_ptr(), part.stride(0), out.data_ptr(),
                                                            None if resid is None else resid.data_ptr(),
                                                            None if w is None else w.data_ptr(), T, self.H, self.H, eps,
                                                            stream.cuda_stream))

    def allgather(self, r, local, stream):
        from b200attn import _lib
        T, cols = local.shape
        _lib.check(self.lib.b2_comm_allgather_cols(self.comms[r], local.data_ptr(), local.stride(0), T, cols,
                                                   stream.cuda_stream))

    def close(self):
        torch.cuda.synchronize()
        for c in self.comms:
            self.lib.b2_comm_destroy(c)
        for p in self.ptrs:
            self.lib.b2_comm_free(p)


@pytest.mark.parametrize("H", [512, 4096, 8192])
def test_comm_tp1_equals_rms_norm(cuda, H):
    from b200attn import ops
    T = 37
    R = Regions(1, 64, H, 64, 1024)
    try:
        st = torch.cuda.current_stream()
        x = torch.randn(T, H, device="cuda").to(torch.bfloat16)
        w = torch.randn(H, device="cuda").to(torch.bfloat16)
        resid = torch.randn(T, H, device="cuda").to(torch.bfloat16)
        for slot in (0, 1, 0):
            R.inputs[0][slot][:T].copy_(x)
            r1, r2 = resid.clone(), resid.clone()
            out = torch.empty_like(x)
            R.allreduce(0, slot, out, r1, w, T, 1e-5, st)
            ref = ops.rms_norm(x, w, 1e-5, residual=r2)
            assert torch.equal(r1.view(torch.int16), r2.view(torch.int16))           # the residual stream: bit-exact
            # the norm: the two kernels sum the squares in a different thread order -> at most one bf16 ulp apart
            assert bool(((out.float() - ref.float()).abs() <= 2.0 ** -7 * ref.float().abs()).all())
            assert (out.view(torch.int16) != ref.view(torch.int16)).float().mean() < 0.01
            r3, out3 = resid.clone(), torch.empty_like(x)
            R.push(0, x, out3, r3, w, 1e-5, st)                                      # push variant: same arithmetic
            assert torch.equal(out3.view(torch.int16), out.view(torch.int16))
            assert torch.equal(r3.view(torch.int16), r2.view(torch.int16))
        # no weight: plain sum (+ residual); no residual: plain norm
        out = torch.empty_like(x)
        R.allreduce(0, 1, out, None, None, T, 1e-5, st)
        assert torch.equal(out.view(torch.int16), x.view(torch.int16))
        loc = torch.randn(T, 1024, device="cuda").to(torch.bfloat16)
        R.allgather(0, loc, st)
        assert torch.equal(R.gathered[0][:T].view(torch.int16), loc.view(torch.int16))
    finally:
        R.close()


def test_comm_two_emulated_ranks_on_one_gpu(cuda):
    pytest.skip("two ranks whose kernels wait for one another are not run as separate launches on one GPU: nothing guarantees that they "
                "run at the same time.  scripts/tp_check.py runs the exchange with a GPU a rank")
