// Host side of the CUDA-core F stage: kernel shapes, twiddles, launches.
#include <cuda_runtime.h>
#include <cmath>
#include <cstdint>
#include <cstring>

#include "fxb_internal.h"
#include "fxb_kernels.h"

namespace fxb {

constexpr int kMaxTQ = 4;         // FFT iterations per CTA at most

// offset of the twiddles of radix-8 pass `pass` (stride 8^pass) in the table
static int tw_offset(int N, int pass)
{
	int o = 0, n8 = N / 8;
	for(int i = 0; i < pass; i++)
	{
		o += 7 * n8;
		n8 /= 8;
	}
	return o;
}

static int ilog2(int n)
{
	int l = 0;
	while((1 << l) < n)
		l++;
	return l;
}

int fstage_multi_class(int N, int nb)
{
	if(N < 32 || N > 8192)
		return -1;
	return 2 * (13 - ilog2(N)) + (nb == 2 ? 0 : 1);
}

int fstage_multi_tq(int N, int nb, int tq)
{
	FKind k;
	memset(&k, 0, sizeof(k));
	if(!fstage_plan(N, nb, 1, &k))
		return 1;
	const int cap = k.fpc == 1 ? kMaxTQ : kFsMultiFc / k.fpc;
	return tq < 1 ? 1 : (tq > cap ? cap : tq);
}

cudaError_t launch_fstage_multi(const FsMultiArgs &m, int nsm, cudaStream_t stream)
{
	return launch_fstage_multi_on(m, nsm, &stream, 1);
}

// plain VDIF, then raw reads; the long units first
cudaError_t launch_fstage_multi_on(const FsMultiArgs &m, int nsm, const cudaStream_t *streams, int nstream)
{
	int next = 0;
	for(int cls = 0; cls < kFsMultiClasses; cls++)
	{
		if(m.nunit[cls] <= 0)
			continue;
		cudaStream_t st = streams[(next++) % nstream];
		if((cls % kFsMultiPer) & 1)
			launch_fs_one_multi(m, cls, nsm, st);
		else
			launch_fs_pair_multi(m, cls, nsm, st);
	}
	return cudaGetLastError();
}

bool fstage_plan(int N, int nb, int out, FKind *k)
{
	if(N < 32 || N > 16384 || (N & (N - 1)))
		return false;
	k->N = N;
	k->nb = nb;
	if(nb == 2 && N > 8192)
		return false;                               // items of longer FFTs hold one band
	// two bands: one butterfly of both per thread; one band: two butterflies from
	// 4096 points, four at 16384
	k->kb = nb == 2 ? 1 : (N <= 2048 ? 1 : (N <= 8192 ? 2 : 4));
	const int tpf = N / (8 * k->kb);
	k->threads = tpf >= 256 ? tpf : 256;
	k->fpc = k->threads / tpf;
	const size_t side = (size_t)k->fpc * nb * (N + N / 8) * 8;
	k->pp = nb == 1 && 2 * side <= 80 * 1024 ? 1 : 0;
	k->smem = side * (k->pp ? 2 : 1);
	k->tq = kMaxTQ;
	k->out = out;
	k->items_fast = out == 1 ? 1 : 0;          // tensor-core spectra: a subband's stations side by side
	k->twn = tw_offset(N, ilog2(N) / 3);
	return k->smem <= 200 * 1024 && k->threads <= 1024;
}

// Twiddle table of FFT length N in the kernel's [pass][r - 1][p] layout
// (values computed in double): n = tw_offset(N, npass) entries.
void make_fstage_twiddles(int N, float2 *out32)
{
	int n8 = N / 8, s = 1, o = 0;
	while(n8 >= 1)
	{
		for(int r = 1; r < 8; r++)
			for(int p = 0; p < n8; p++)
			{
				const double ang = -2.0 * M_PI * (double)((int64_t)r * p * s % N) / (double)N;
				out32[o + (r - 1) * n8 + p] = make_float2((float)cos(ang), (float)sin(ang));
			}
		o += 7 * n8;
		n8 /= 8;
		s *= 8;
	}
}

void launch_fstage_kind(const FKind &k, FsArgs a, cudaStream_t stream)
{
	if(k.count <= 0 || a.T <= 0)
		return;
	a.first = k.first;
	a.pair0 = k.pair0;
	a.two = k.two;
	a.tq = k.tq;
	a.pp = k.pp;
	a.tw = k.tw;
	a.items_fast = k.items_fast;
	if(k.out == 1)
		k.nb == 2 ? launch_fs_pair_tc(k, a, stream) : launch_fs_one_tc(k, a, stream);
	else
		k.nb == 2 ? launch_fs_pair_f32(k, a, stream) : launch_fs_one_f32(k, a, stream);
}

}  // namespace fxb
