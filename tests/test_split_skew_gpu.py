"""Keys of which half, 90% or 99% fall in one bucket, in random order, from 512 buckets
on: warps whose lanes of that bucket share one atomic, in whole and ragged tiles; the
stable split of the same keys by a stable sort."""
import pytest

pytestmark = pytest.mark.gpu

LONG = (1 << 22) + 8192  # beyond the one-launch form


@pytest.mark.parametrize("layout", ["ko", "soa", "aos"])
@pytest.mark.parametrize("buckets", [256, 512, 1024])
def test_one_heavy_bucket(cuda, edpp, buckets, layout):
    g = cuda.Generator(device="cuda")
    for n in (LONG, LONG + 1, LONG + 300, LONG + 511, LONG + 4097, 3000):
        for share in (0.3, 0.5, 0.9, 0.99):
            for heavy in (0, buckets // 3, buckets - 1):
                g.manual_seed(n + buckets + heavy)
                keys = cuda.randint(-2**31, 2**31 - 1, (n,), generator=g, device="cuda", dtype=cuda.int32)
                hot = cuda.rand(n, generator=g, device="cuda") < share
                keys = cuda.where(hot, keys & ~(buckets - 1) | heavy, keys)
                vals = cuda.arange(n, device="cuda", dtype=cuda.int32)
                b = keys & (buckets - 1)
                order = cuda.sort(b, stable=True)[1]
                counts = cuda.bincount(b, minlength=buckets)
                if layout == "aos":
                    o, _, s = edpp.split(cuda.stack([keys, vals], 1).contiguous(), buckets,
                                         layout="aos", bucket_start=True)
                    k, v = o[:, 0], o[:, 1]
                else:
                    k, v, s = edpp.split(keys, buckets, values=vals if layout == "soa" else None,
                                         layout=layout, bucket_start=True)
                assert cuda.equal(k, keys[order]), (n, share, heavy)
                assert v is None or cuda.equal(v, vals[order]), (n, share, heavy)
                assert cuda.equal(s, (cuda.cumsum(counts, 0) - counts).to(cuda.int32))
    assert edpp.sync_status() == edpp.EDPP_OK
