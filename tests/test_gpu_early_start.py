"""What the kernels do before their dependency wait.  A writer that releases its dependents at once and writes late (late_writer.cu)
stands for an engine's own kernel: everything but the weights that B200_OPT_STABLE_WEIGHTS covers must come out as it wrote it.  And
with that option on, every path gives the bits that it gives with the option off."""
import ctypes as C
import os
import subprocess
import pytest
import torch

from util import pkg

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LATE_US = 300                                        # far longer than the host needs to enqueue the launches after the writer


def late_copy(dst, src):
    path = os.path.join(ROOT, 'tests', 'cpp', 'liblate_writer.so')
    if not os.path.exists(path):
        subprocess.check_call(['make', '-C', os.path.join(ROOT, 'glm-5.3-flash-cuda-server_b200'), 'gate'])
    f = C.CDLL(path).late_copy
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_uint, C.c_void_p]
    assert src.numel() * src.element_size() == dst.numel() * dst.element_size()
    assert f(dst.data_ptr(), src.data_ptr(), dst.numel() * dst.element_size(), LATE_US, torch.cuda.current_stream().cuda_stream) == 0


class stable_weights:
    def __enter__(self):
        pkg().set_option(pkg().OPT_STABLE_WEIGHTS, 1)

    def __exit__(self, *a):
        pkg().set_option(pkg().OPT_STABLE_WEIGHTS, 0)


@pytest.mark.parametrize('N,K,M', [(144, 4096, 1), (64, 2048, 4), (2048, 4096, 8)])
def test_a_bf16_matrix_is_no_stable_weight(N, K, M):
    """The option is a promise about NVFP4 weights.  A plain bf16 matrix written by the kernel before is read as it was written."""
    P = pkg()
    g = torch.Generator(device='cuda').manual_seed(N + M)
    old, new = [torch.randn((N, K), generator=g, device='cuda').to(torch.bfloat16) for _ in range(2)]
    x = torch.randn((M, K), generator=g, device='cuda')
    want = P.gemm(new, x)
    W, y = old.clone(), torch.empty_like(want)
    with stable_weights():
        for _ in range(5):
            W.copy_(old)
            P.gemm(W, x, y)
            late_copy(W, new)
            P.gemm(W, x, y)
            assert torch.equal(y, want)


# ---- every path: inputs that arrive late, and the option on against off ----------------------------

SMALL = dict(H=1024, I=512, E=16, topk=4)                    # one item per CTA and fewer
FULL = dict(H=4096, I=1536, E=16, topk=8)                    # several items per CTA from four tokens on


class Path:
    """One call of the library: run() -> outputs, and the buffers it reads that no promise covers, by name."""

    def __init__(self, name, seed=1):
        P = pkg()
        self.g = torch.Generator(device='cuda').manual_seed(seed)
        kind, *arg = name.split()
        M = int(arg[0]) if arg else 1
        self.late = {}
        getattr(self, kind)(P, M)

    def randn(self, *shape):
        return torch.randn(shape, generator=self.g, device='cuda')

    def weight(self, N, K):
        return pkg().quantize((self.randn(N, K) * 0.02).to(torch.bfloat16))

    def gemm(self, P, M):
        W, x, y, ws = self.weight(3000, 1024), self.randn(M, 1024), torch.empty((M, 3000), device='cuda'), P.split_workspace(M, 1024, 'cuda')
        self.late = {'x': x, 'gscale': W.gscale}
        self.run = lambda: [P.gemm(W, x, y, ws=ws if M > 1 else None)]

    def tall(self, P, M):                                    # several tiles per CTA
        W, x, y = self.weight(60000, 512), self.randn(M, 512), torch.empty((M, 60000), device='cuda')
        self.late = {'x': x, 'gscale': W.gscale}
        self.run = lambda: [P.gemm(W, x, y)]

    def short_k(self, P, M):                                 # the kernels for fewer than 256 columns
        W, x, y = self.weight(3000, 128), self.randn(M, 128), torch.empty((M, 3000), device='cuda')
        self.late = {'x': x, 'gscale': W.gscale}
        self.run = lambda: [P.gemm(W, x, y)]

    def siblings(self, P, M):
        Ws, x, ws = [self.weight(n, 2048) for n in (2048, 512, 64, 31)], self.randn(M, 2048), P.split_workspace(M, 2048, 'cuda')
        ys = [torch.empty((M, W.N), device='cuda') for W in Ws]
        self.late = {'x': x, 'gscale': Ws[1].gscale}
        self.run = lambda: P.gemv_multi(Ws, x, M, ys, ws=ws if M > 1 else None)

    def wide(self, P, M):
        W, x, y, ws = self.weight(3000, 1280), self.randn(M, 1280).to(torch.bfloat16), torch.empty((M, 3000), device='cuda'), P.gemm_bf16_workspace(M, 1280, 'cuda')
        self.late = {'x': x, 'gscale': W.gscale}
        self.run = lambda: [P.gemm_bf16(W, x, y, ws)]

    def exact(self, P, M):
        W, x, y = self.weight(3000, 1280), self.randn(M, 1280).to(torch.bfloat16), torch.empty((M, 3000), device='cuda')
        ws = torch.empty(P.lib().b200_nvfp4_gemm_bf16_exact_workspace_bytes(M, 1280), dtype=torch.uint8, device='cuda')
        self.late = {'x': x, 'gscale': W.gscale}
        self.run = lambda: [P.gemm_bf16_exact(W, x, y, ws)]

    def mlp(self, P, M):
        H, I = 1024, 2048
        gate, up, down, x = self.weight(I, H), self.weight(I, H), self.weight(H, I), self.randn(M, H)
        y, ws = torch.empty((M, H), device='cuda'), P.dense_mlp_workspace(M, H, I, 'cuda')
        self.late = {'x': x, 'gscale': down.gscale}
        self.run = lambda: [P.dense_mlp(x, gate, up, down, 10.0, y, ws)]

    def layer(self, P, M, H, I, E, topk):
        trip = [(self.weight(I, H), self.weight(I, H), self.weight(H, I)) for _ in range(E + 1)]
        L = P.MoeLayer((self.randn(E, H) * 0.02).to(torch.bfloat16), self.randn(E) * 0.1, trip[:E], trip[E], topk, H, I)
        assert P.moe_prepare(L)
        self.prepared = L
        return L

    def moe(self, P, M, **geometry):
        L = self.layer(P, M, **(geometry or FULL))
        x, y = self.randn(M, L.hidden), torch.empty((M, L.hidden), device='cuda')
        sel, wts = torch.empty((M, L.topk), dtype=torch.int32, device='cuda'), torch.empty((M, L.topk), device='cuda')
        self.late = {'x': x, 'router': L.router, 'bias': L.bias, 'gscale': L.shared[2].gscale}
        self.x = x
        self.step = lambda x: list(P.moe_forward(L, x, y, sel, wts))
        self.run = lambda: self.step(x)

    def moe_small(self, P, M):
        self.moe(P, M, **SMALL)

    def experts(self, P, M):
        L = self.layer(P, M, **SMALL)
        x, y, wts = self.randn(M, L.hidden), torch.empty((M, L.hidden), device='cuda'), self.randn(M, L.topk).abs()
        sel = torch.stack([torch.randperm(L.n_expert, generator=self.g, device='cuda')[:L.topk] for _ in range(M)]).to(torch.int32)
        self.late = {'x': x, 'sel': sel, 'wts': wts, 'gscale': L.shared[0].gscale}
        self.run = lambda: [P.moe_experts(L, x, sel, wts, y)]

    def quantise(self, P, M):
        w = self.randn(300, 1040).to(torch.bfloat16)
        out = P.quantize(w)
        self.late = {'x': w}
        self.run = lambda: (lambda t: [t.packed, t.scale, t.gscale])(P.quantize(w, out=out))

    def close(self):
        if hasattr(self, 'prepared'):
            pkg().moe_release(self.prepared)


PATHS = ['gemm 1', 'gemm 3', 'gemm 5', 'gemm 20', 'tall 1', 'tall 2', 'short_k 1', 'short_k 4', 'siblings 1', 'siblings 4', 'siblings 7', 'wide 40',
         'wide 700', 'exact 40', 'exact 300', 'mlp 1', 'mlp 5', 'mlp 20', 'moe 1', 'moe 4', 'moe 8', 'moe 12', 'moe 40', 'moe_small 1', 'moe_small 7',
         'experts 2', 'experts 11', 'experts 33', 'quantise']


@pytest.mark.parametrize('name', PATHS)
def test_what_a_late_writer_leaves_is_what_is_read(name):
    """Weights declared stable; activations, selections, gates, router, bias and global scales each written by a kernel that the
    call's launches overtake as far as they may."""
    P = pkg()
    path = Path(name)
    try:
        for key, buf in path.late.items():
            old = buf.clone()
            if key == 'gscale': new = old * 1.25
            elif key == 'sel': new = (buf.flip(1) + 1) % SMALL['E']
            else: new = (buf.float().flip(0).roll(1, -1) * 1.5).to(buf.dtype).contiguous()
            buf.copy_(new)
            want = [t.clone() for t in path.run()]
            with stable_weights():
                for _ in range(3):
                    buf.copy_(old)
                    path.run()
                    late_copy(buf, new)
                    got = path.run()
                    assert all(torch.equal(a, b) for a, b in zip(got, want)), key
            buf.copy_(old)
        assert P.device_status() == 0
    finally:
        path.close()


def replay(fn, times):
    """fn captured `times` over and replayed twice, with the options as they are now."""
    st, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        fn()
        st.synchronize()
        with torch.cuda.graph(g, stream=st):
            for _ in range(times): fn()
    for _ in range(2): g.replay()
    torch.cuda.synchronize()


@pytest.mark.parametrize('name', PATHS)
def test_stable_weights_change_no_bit(name):
    """One after the other without gaps, as plain launches and as a replayed graph."""
    P = pkg()
    path = Path(name)
    try:
        want = [t.clone() for t in path.run()]
        with stable_weights():
            for _ in range(30): got = path.run()
            assert all(torch.equal(a, b) for a, b in zip(got, want))
            for t in got: t.zero_()
            replay(path.run, 10)
            assert all(torch.equal(a, b) for a, b in zip(got, want))
        assert P.device_status() == 0
    finally:
        path.close()


@pytest.mark.parametrize('M', [1, 4, 8, 12, 40])
def test_layers_that_share_a_workspace(M):
    """Three layers with different experts and routers, each reading what the one before wrote, one scratch for all: a launch that
    read the scratch of its own layer too early would find the last one's records, digits or rows."""
    P = pkg()
    paths = [Path('moe %d' % M, seed=10 + k) for k in range(3)]
    try:
        ws = paths[0].prepared.workspace(M)
        for p in paths: p.prepared._ws[M] = ws
        x0 = paths[0].x

        def chain():
            outs = [paths[0].run()]
            for p in paths[1:]: outs.append(p.step(outs[-1][0]))
            return outs
        want = [[t.clone() for t in o] for o in chain()]
        assert not torch.equal(want[0][1], want[1][1])       # other selections
        with stable_weights():
            for _ in range(20): got = chain()
            assert all(torch.equal(a, b) for o, w in zip(got, want) for a, b in zip(o, w))
            for o in got:
                for t in o: t.zero_()
            replay(chain, 10)
            assert all(torch.equal(a, b) for o, w in zip(got, want) for a, b in zip(o, w))
            new = x0.clone()                                 # and once more behind a late writer of the first input
            for _ in range(3):
                x0.zero_()
                late_copy(x0, new)
                got = chain()
                assert all(torch.equal(a, b) for o, w in zip(got, want) for a, b in zip(o, w))
        assert P.device_status() == 0
    finally:
        for p in paths: p.close()
