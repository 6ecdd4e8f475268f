// F stage of two-band work items, tensor-core-form spectra (see
// fxb_fstage_pair.cuh): the persistent launches, and complex sampling.
#include "fxb_fstage_pair.cuh"

namespace fxb {

// The units of one length (class 2 (13 - LOGN) of VAR 0: plain VDIF, 1: raw
// INTERLACEDVDIF reads), each in a kernel of its own: a kernel of several lengths has
// registers and an order of instructions that suit none.  2048 points among the
// shorter ones, 10 stations x 2 subbands x 2 bands of 8 bits: F stage 89 us, 81 alone;
// 16 threads read raw 311 and 289.
template <int VAR, int LOGN>
__global__ void __launch_bounds__(PShape<LOGN>::NT, PShape<LOGN>::MINB)
    k_fstage_pair_pw(const __grid_constant__ FsMultiArgs m)
{
	extern __shared__ __align__(16) ulonglong2 fsp[];
	constexpr int FPC = PShape<LOGN>::FPC, NFC = kMaxTQ * FPC < kFsMultiFc ? kMaxTQ * FPC : kFsMultiFc;
	__shared__ float lut8[260];
	__shared__ u64 lut4[16];
	__shared__ PairFeed<NFC> feed;
	fstage_pair_luts(lut8, lut4);
	pair_units(feed, m, kFsMultiPer * VAR + 2 * (13 - LOGN),
	           [&](const FsMultiUnit &w, const PairItem &I, const PairConst *fcs, const PairTwist *tws) {
		           const FsMultiKind &k = m.kinds[w.kind];
		           fstage_pair_unit<LOGN, true, VAR>(m.m[k.member], I, fcs, tws, w.t0, (w.nfc + FPC - 1) / FPC,
		                                             (const float2 *)k.tw, fsp, lut8, lut4);
	           });
}

template <int VAR, int LOGN>
static void launch_len(const FsMultiArgs &m, int nsm, cudaStream_t st)
{
	using SH = PShape<LOGN>;
	fs_launch_persistent(k_fstage_pair_pw<VAR, LOGN>, m, kFsMultiPer * VAR + 2 * (13 - LOGN), SH::MINB * nsm, SH::NT,
	                     (size_t)SH::FPC * SH::PADN * 16, st);
}

template <int VAR>
static void launch_cls(const FsMultiArgs &m, int c, int nsm, cudaStream_t st)
{
	switch(13 - c / 2)
	{
	case 5: launch_len<VAR, 5>(m, nsm, st); break;
	case 6: launch_len<VAR, 6>(m, nsm, st); break;
	case 7: launch_len<VAR, 7>(m, nsm, st); break;
	case 8: launch_len<VAR, 8>(m, nsm, st); break;
	case 9: launch_len<VAR, 9>(m, nsm, st); break;
	case 10: launch_len<VAR, 10>(m, nsm, st); break;
	case 11: launch_len<VAR, 11>(m, nsm, st); break;
	case 12: launch_len<VAR, 12>(m, nsm, st); break;
	default: launch_len<VAR, 13>(m, nsm, st); break;
	}
}

void launch_fs_pair_multi(const FsMultiArgs &m, int cls, int nsm, cudaStream_t st)
{
	if(cls >= kFsMultiPer)
		launch_cls<1>(m, cls - kFsMultiPer, nsm, st);
	else
		launch_cls<0>(m, cls, nsm, st);
}

// The constants of one FFT per thread (grid: FFTs, items): FP64 terms, frames of
// the window and, of raw reads, their place.  On their own so that the FFT
// kernels start from finished constants: formed inside them, a unit of four
// 2048-point FFTs spent about as long on this chain of loads and FP64
// operations as on one FFT.
__global__ void __launch_bounds__(128) k_pair_consts(const FsArgs a, int N, int mux, int cplx)
{
	const int t = blockIdx.x * blockDim.x + threadIdx.x;
	if(t >= a.T)
		return;
	const int item = a.pair0 + blockIdx.y;
	const PairItem &I = a.pitems[item];
	const FGroup &g = a.groups[I.group];
	const DevStation *Sp = a.st + I.station;
	const uint32_t fs = I.fs;
	const int nchan = cplx ? N : N / 2, S8 = N / 8, order = a.order;
	const uint8_t *vrow = a.valid + (int64_t)I.station * a.valid_stride;
	PairConst c;
	memset(&c, 0, sizeof(c));
	c.st = c.os[0] = c.os[1] = make_float2(1.0f, 0.0f);
	c.wp = a.sub[I.station].buf;
	const FftParam *pq = a.params + (int64_t)I.station * a.T + t;
	if(pq->status == kFftOk)
	{
		c.flags = kPActive | kPSame;
		const uint32_t g0 = (uint32_t)pq->nearest;
		c.fa = g0 / fs;
		c.so = g0 - c.fa * fs;
		c.stuck = pq->stuck;
		if(!mux)
			c.wp += (int64_t)c.fa * I.framebytes + I.header;
		const double invN = 1.0 / N;
		const int idl = pq->integerdelay;
		// LO offset: seconds since the job start of the FFT's first sample
		// (mode.cpp:686-694; the scan starts with the job) and the offset's
		// turns per sample
		const double walls = (double)a.sub[I.station].subsec + a.sub[I.station].subns / 1.0e9 +
		                     (double)t * N * Sp->sampletime / 1.0e6;
		const double low = g.corr ? looff_wall_turns(g.looff, walls) : 0.0;
		const double los = -g.looff * Sp->sampletime / 1.0e6;
		double postf[2] = {0.0, 0.0};
		for(int j = 0; j < (I.two ? 2 : 1); j++)
		{
			const double lo = j ? g.lofreq1 : g.lofreq;
			const double fraclo = a.fraclo ? (lo - (int)lo) * (double)idl : 0.0;
			float P0 = 0.0f, alpha = 0.0f, beta = 0.0f, gamma = 0.0f, eps = 0.0f;
			float2 st = make_float2(1.0f, 0.0f);
			if(order == 1)
			{
				P0 = frac_centered(lo * pq->b + fraclo + low);
				alpha = (float)(lo * pq->a * invN + los);
				st = cispi2(-(double)alpha * (double)S8);
			}
			else if(order == 2)
			{
				const double pa = pq->a, pb = pq->b;
				const double X1 = (double)Sp->asl * invN;
				P0 = frac_centered(lo * pq->c + fraclo + low);
				alpha = (float)(lo * (pb + pa * X1) * invN + los);
				beta = (float)(lo * 2.0 * pa * X1 * invN);
				gamma = (float)(lo * pb * Sp->asl * invN + los * Sp->asl);
				eps = (float)(lo * pa * X1 * X1);
			}
			else
			{
				double pr = (pq->averagedelay - idl) * lo;
				if(a.fraclo)
					pr += idl * (lo - (int)lo);
				pr -= walls * g.looff;
				postf[j] = -(double)(float)(pr - (int)pr);
			}
			if(j == 0)
			{
				c.P0 = P0;
				c.alpha = alpha;
				c.beta = beta;
				c.gamma = gamma;
				c.eps = eps;
				c.st = st;
				postf[1] = postf[0];
			}
			else
			{
				PairTwist w;
				w.P0 = P0;
				w.alpha = alpha;
				w.beta = beta;
				w.gamma = gamma;
				w.eps = eps;
				w.st = st;
				w.pad_ = 0;
				a.ptwist[(int64_t)(item - a.ptwist0) * a.T + t] = w;
				c.flags |= kPTwo;
			}
		}
		// per band: fse - clock offset (mode.cpp:1053-1059, 1099-1106); the
		// channel of an order-0 lower sideband falls with the bin
		const double sgn = I.lsb && (order == 0 || cplx) ? -1.0 : 1.0;
		for(int j = 0; j < 2; j++)
		{
			const double D = Sp->bw * (1.0 / nchan) * ((double)pq->fse - g.clk[j]);
			split_turns(D, c.dhi[j], c.dlo[j]);
			c.post[j] = (float)postf[j] + g.phase[j];
			if(j == 0 || g.clk[1] != g.clk[0])
				c.os[j] = cispi2(sgn * D * (double)S8);
			else
				c.os[1] = c.os[0];
		}
		if(g.clk[1] != g.clk[0] || c.post[1] != c.post[0])
			c.flags &= ~kPSame;
		// validity of the window's frames, one bit per frame relative to fa (k_fft_params)
		const uint32_t nwf = (c.so + (uint32_t)N - 1) / fs + 1;
		c.fmask = pq->fmask;
		if(pq->mflags & 1)
			c.flags |= kPNarrow;
		if(a.bandok)
		{
			// EDV4-blanked bands (INTERLACEDVDIF): the general decode path
			const uint32_t need = (1u << I.band0) | (1u << I.band1);
			for(uint32_t k = 0; k < nwf; k++)
			{
				const int64_t fk = (int64_t)c.fa + k;
				if(fk < a.valid_stride && vrow[fk] != 0 &&
				   (a.bandok[(int64_t)I.station * a.valid_stride + fk] & need) != need)
					c.flags |= kPBlank;
			}
		}
		const bool whole = nwf < 32 && c.fmask == (1u << nwf) - 1u && c.stuck >= N && !(c.flags & kPBlank);
		if(!mux && whole && fs >= (uint32_t)S8)
			c.flags |= I.adj ? kPFast : kPApart;
		if(mux && whole && nwf <= 2)
		{
			// valid frames of raw reads are complete slots: every thread is there
			c.flags |= kPFast;
			const int32_t *s0 = a.sub[I.station].mux_slot + (a.sub[I.station].mux_k0 + (int64_t)c.fa) * I.mnthr;
			const int32_t *s1 = nwf == 2 ? s0 + I.mnthr : s0;
			c.mi00 = s0[I.band0];
			c.mi01 = s0[I.band1];
			c.mi10 = s1[I.band0];
			c.mi11 = s1[I.band1];
		}
	}
	a.pconst[(int64_t)item * a.T + t] = c;
}

void launch_pair_consts(const FKind &k, const FsArgs &a0, cudaStream_t stream)
{
	FsArgs a = a0;
	a.pair0 = k.pair0;
	if(k.count > 0 && a.T > 0)
		k_pair_consts<<<dim3((a.T + 127) / 128, k.count), 128, 0, stream>>>(a, k.N, k.muxraw, k.cplx);
}

void launch_fs_pair_tc(const FKind &k, const FsArgs &a, cudaStream_t stream)
{
	if(k.cplx)
		launch_var<true, 2>(k, a, stream);
}

}  // namespace fxb
